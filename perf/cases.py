"""Performance cases of the Lindblad density-matrix dynamics: what a program that uses this package has it
do, through ``LindbladGPU``, from the smallest systems (launch latency) to operators far larger than L2.

The systems follow the synthetic generator's band structures (Si-like, GaAs-like, MoS2-like: k-points of
a parabolic band in an energy window, spin-split pairs, k-pairs inside an energy distance, operators
P = sum_m A_m (x) conj(A_m) of six phonon modes with Gaussian energy conservation plus an elastic
impurity term), made on the GPU from the seed alone. ``exact`` restates the same quantities in plain
torch (FP64 / complex128).
"""
import math

import numpy as np
import torch

from denmat_dynm_development_gb300.dmd import LindbladGPU

EV = 1.0 / 27.21138505
KELVIN = 1.3806488e-23 / 4.35974434e-18
FS = 41.341373336493
TESLA = 1.0 / 2.3505175675871e5
EWIN = 0.2 * EV
MEFF = 0.3
LATTICE = 10.68
ECBM = 0.05
DEGAUSS, NDEGAUSS = 10e-3 * EV, 5.0
MODES = [x * 1e-3 * EV for x in (8.0, 17.0, 26.0, 35.0, 44.0, 57.0)]
T300 = 300.0 * KELVIN

# kind: rk4 -- device-resident fixed-step RK4 between two measurements of S_z (the T1 run's loop);
#       func -- the right-hand side through the host-buffer callback (how an outside stepper drives it);
#       rkf45 -- one output interval of the adaptive stepper, DMD's own, on the linearized operators;
#       batch -- many initial states that share the operators (an ensemble of pumps);
#       adjoint -- the gradient of S_z(t) with respect to every operator element and the initial state;
#       ee -- the e-e operators rebuilt from the density matrix (Debye screening from rho).
# de: k-pairs closer than this (meV) in energy are kept; field: static B field (T), a coherent term.


def listed():
    c = []
    # A first test system, as in the example inputs: a few thousand pairs, all of it launches and latency.
    c.append(dict(name="rk4_f64_nk96", kind="rk4", prec="f64", nk=96, nb=2, de=60.0, field=0.5, steps=100))
    # The Si-like T1 run (nk = 500, 69k pairs, 50,000 steps of it for one lifetime): P sits in L2.
    c.append(dict(name="rk4_f64_nk500", kind="rk4", prec="f64", nk=500, nb=2, de=60.0, field=0.0, steps=50))
    # The GaAs-like production system, plain FP64 (the default arithmetic): P streams from HBM.
    c.append(dict(name="rk4_f64_nk10000", kind="rk4", prec="f64", nk=10000, nb=2, de=4.45, field=0.0, steps=4))
    # The callback that an outside ODE library calls, with a host copy in and out of every call.
    c.append(dict(name="func_f64_nk4001", kind="func", prec="f64", nk=4001, nb=2, de=4.45, field=0.1, steps=1))
    # DMD's own GaAs example: nk = 941, every pair stored, linearized, adaptive RKF45, one output interval.
    c.append(dict(name="rkf45_lin_f64_nk941", kind="rkf45", prec="f64", nk=941, nb=2, de=250.0, field=0.0, steps=1))
    # The double-float form of the same production run (a user's choice for speed at ~1e-14).
    c.append(dict(name="rk4_f64x_nk8000", kind="rk4", prec="f64x", nk=8000, nb=2, de=4.45, field=0.0, steps=8))
    # The reduced-storage form (P in complex64, rho as its deviation), for scans.
    c.append(dict(name="rk4_f32_nk6007", kind="rk4", prec="f32", nk=6007, nb=2, de=4.45, field=0.0, steps=8))
    # The MoS2-like four-band system, plain FP64.
    c.append(dict(name="rk4_f64_nb4_nk2000", kind="rk4", prec="f64", nk=2000, nb=4, de=2.0, field=0.1, steps=5))
    # An ensemble of 96 initial states on shared operators (tensor cores).
    c.append(dict(name="batch96_bf16x2_nk5000", kind="batch", prec="bf16x2", nk=5000, nb=2, de=4.45, field=0.0, steps=20,
                  states=96))
    # Gradients on the Si-like system, as in a fit of coupling scales to a lifetime.
    c.append(dict(name="adjoint_f64x_nk500", kind="adjoint", prec="f64x", nk=500, nb=2, de=60.0, field=0.0, steps=25))
    # e-e scattering updated with the state (eeMode = Pee_update).
    c.append(dict(name="ee_f64_nk400", kind="ee", prec="f64", nk=400, nb=2, de=20.0, field=0.0, steps=1))
    # Sparse operators (alg_sparseP), a fifth of the elements stored.
    c.append(dict(name="rk4_sparse_nb4_nk2000", kind="rk4", prec="f64", nk=2000, nb=4, de=2.0, field=0.0, steps=5,
                  fill=0.18))
    return c


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rk4", "rk4", "rk4", "func", "rkf45", "batch", "adjoint", "ee", "sparse"])
    nb = rng.choice([2, 2, 4])
    c = dict(kind=kind, prec="f64", nk=0, nb=nb, de=0.0, field=rng.choice([0.0, 0.0, 0.1, 1.0]), steps=1)
    if kind in ("rk4", "func"):
        c["prec"] = rng.choice(["f64", "f64", "f64x", "f32", "bf16x2"])
        if nb == 2:
            c["nk"] = log(60, 10000)
            # no more pairs than the largest listed case: about nk^2 / 2 * min(1, 3 de / 200)
            c["de"] = round(min(rng.uniform(3.0, 60.0), 200.0 / 3.0 * min(1.0, 2.0e6 / (0.5 * c["nk"] ** 2))), 3)
        else:
            c["nk"] = log(60, 2500)
            c["de"] = round(min(rng.uniform(0.6, 20.0), 200.0 / 3.0 * min(1.0, 4.0e4 / (0.5 * c["nk"] ** 2))), 3)
        c["steps"] = 1 if kind == "func" else max(2, min(60, 30000 // c["nk"]))
    elif kind == "rkf45":
        c.update(nb=2, nk=log(100, 941), de=round(rng.uniform(20.0, 250.0), 3), field=0.0)
    elif kind == "batch":
        c.update(prec="bf16x2", states=rng.choice([7, 16, 33, 96, 128]), steps=12)
        c["nk"] = log(200, 5000) if nb == 2 else log(200, 1500)
        c["de"] = round(rng.uniform(2.0, 4.45), 3) if nb == 2 else round(rng.uniform(0.6, 2.0), 3)
    elif kind == "adjoint":
        c.update(prec=rng.choice(["f64x", "f64x", "f64"]), steps=rng.randint(5, 25), field=0.0)
        c["nk"] = log(80, 500) if nb == 2 else log(80, 400)
        c["de"] = round(rng.uniform(10.0, 60.0), 3) if nb == 2 else round(rng.uniform(1.0, 4.0), 3)
    elif kind == "ee":
        c.update(prec=rng.choice(["f64", "f64x"]), nb=2, nk=log(60, 400), de=round(rng.uniform(5.0, 20.0), 3), field=0.0)
    else:
        c.update(kind="rk4", nb=4, nk=log(100, 2000), de=round(rng.uniform(0.6, 2.0), 3), steps=5, fill=round(rng.uniform(0.05, 0.35), 3))
    return c


# ---------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------
def _nk_full(nk):
    vol = LATTICE ** 3 / 4.0
    sphere = 4.0 / 3.0 * math.pi * (2.0 * MEFF * EWIN) ** 1.5
    return float(math.ceil((1.4 * nk * (2.0 * math.pi) ** 3 / vol / sphere) ** (1.0 / 3.0))) ** 3


def _pair_list(ebar, w):
    """every (k, k'), k <= k', with |ebar_k - ebar_k'| < w, k-major"""
    nk = ebar.size
    order = np.argsort(ebar, kind="stable")
    es = ebar[order]
    rank = np.empty(nk, np.int64)
    rank[order] = np.arange(nk)
    hi = np.searchsorted(es, es + w, side="left")
    n = hi - np.arange(nk)
    a = np.repeat(np.arange(nk), n)
    b = np.arange(a.size) - np.repeat(np.cumsum(n) - n, n) + a
    ka, kb = order[a], order[b]
    k1, k2 = np.minimum(ka, kb), np.maximum(ka, kb)
    o = np.argsort(k1 * nk + k2, kind="stable")
    return k1[o].astype(np.uint64), k2[o].astype(np.uint64)


def _npair(c):
    """k-pairs of the case (of a ball of mesh points: by its mean density)"""
    e = EWIN * ((np.arange(c["nk"]) + 0.5) / c["nk"]) ** (2.0 / 3.0)
    return int((np.searchsorted(e, e + c["de"] * 1e-3 * EV, side="left") - np.arange(c["nk"])).sum())


def _spin(rng, nk, nb):
    """S_x, S_y, S_z between the bands: spin matrices rotated by a small random mixing"""
    sig = 0.5 * np.array([[[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]], np.complex128)
    if nb > 2:
        sig = np.stack([np.kron(np.eye(nb // 2), s) for s in sig])
    a = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
    w, v = np.linalg.eigh(0.5 * (a + np.conj(np.swapaxes(a, 1, 2))) / math.sqrt(2.0 * nb))
    u = np.einsum("kij,kj,klj->kil", v, np.exp(0.1j * w), np.conj(v))
    s = np.einsum("kji,djl,klm->kdim", np.conj(u), sig, u)
    return 0.5 * (s + np.conj(np.swapaxes(s, 2, 3)))


def _operators(c, seed, e, k1, k2):
    """P1, P2 (complex128 [npair][nb^4], on the GPU, in chunks): yields (first pair, P1, P2)"""
    nb = e.shape[1]
    gen = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)
    eg = torch.as_tensor(e, device="cuda")
    step = (1 << 18) if nb == 2 else (1 << 14)
    amp = 20e-3 * EV * math.sqrt(1.0 / (DEGAUSS * math.sqrt(2.0 * math.pi)))

    def cgauss(shape):
        return torch.view_as_complex(torch.randn(*shape, 2, dtype=torch.float64, device="cuda", generator=gen)) * math.sqrt(0.5)

    def window(x):
        return torch.where(x.abs() < NDEGAUSS * DEGAUSS, torch.exp(-x * x / (4.0 * DEGAUSS ** 2)), torch.zeros_like(x))

    def outer(A, transpose):
        A = A.transpose(2, 3) if transpose else A
        n, m = A.shape[:2]
        X = A.reshape(n, m, nb * nb)
        M = torch.matmul(X.transpose(1, 2), X.conj())
        return M.reshape(n, nb, nb, nb, nb).permute(0, 1, 3, 2, 4).reshape(n, nb ** 4).contiguous()

    for p0 in range(0, k1.size, step):
        i1 = torch.as_tensor(k1[p0:p0 + step].astype(np.int64), device="cuda")
        i2 = torch.as_tensor(k2[p0:p0 + step].astype(np.int64), device="cuda")
        n = i1.numel()
        de = eg[i1][:, :, None] - eg[i2][:, None, :]
        A1, A2 = [], []
        for w in MODES:
            nq = 1.0 / math.expm1(w / T300)
            gp, gm = cgauss((n, nb, nb)) * window(de + w) * amp, cgauss((n, nb, nb)) * window(de - w) * amp
            A1 += [gp * math.sqrt(nq + 1.0), gm * math.sqrt(nq)]
            A2 += [gm * math.sqrt(nq + 1.0), gp * math.sqrt(nq)]
        imp = cgauss((n, nb, nb)) * window(de) * (0.1 * amp)  # elastic: the same amplitude both ways
        P1, P2 = outer(torch.stack(A1 + [imp], 1), False), outer(torch.stack(A2 + [imp], 1), True)
        if c.get("fill"):  # alg_sparseP: most elements of each operator are zero
            P1 = torch.where(torch.rand(P1.shape, device="cuda", generator=gen) < c["fill"], P1, torch.zeros_like(P1))
            P2 = torch.where(torch.rand(P2.shape, device="cuda", generator=gen) < c["fill"], P2, torch.zeros_like(P2))
        yield p0, P1, P2


def _system(c, seed):
    """bands, occupations, spin, pairs and states of the case (numpy); the operators come from _operators"""
    nk, nb = c["nk"], c["nb"]
    rng = np.random.default_rng([int(seed), nk, nb])
    s = dict(nk=nk, nb=nb)
    nkf = _nk_full(nk)
    if c["kind"] == "ee":  # a ball of mesh points: k1 + k3 - k2 is mostly on the set
        n = int(round(nkf ** (1.0 / 3.0)))
        R = 0.5 * LATTICE * np.array([[0.0, 1, 1], [1, 0, 1], [1, 1, 0]])
        B = 2.0 * math.pi * np.linalg.inv(R).T
        M = int(math.ceil(nk ** (1.0 / 3.0))) + 2
        g = np.stack(np.meshgrid(*[np.arange(-M, M + 1)] * 3, indexing="ij"), -1).reshape(-1, 3)
        e0 = (((g / n) @ B.T) ** 2).sum(1) / (2.0 * MEFF)
        sel = np.argsort(e0, kind="stable")[:nk]
        rng.shuffle(sel)
        e0, nkf = e0[sel], float(n) ** 3
        h = rng.standard_normal((4, 2 * nb, 2 * nb)) + 1j * rng.standard_normal((4, 2 * nb, 2 * nb))
        h = 0.5 * (h + np.conj(np.swapaxes(h, 1, 2))) / math.sqrt(4.0 * nb)
        w, v = np.linalg.eigh(h[0][None] + 4.0 * np.einsum("kd,dij->kij", g[sel] / n, h[1:]))
        U = np.einsum("kij,kj,klj->kil", v, np.exp(1j * w), np.conj(v))
        G = 2.0 * math.pi * np.linalg.inv(R)
        s.update(mesh=n, kidx=g[sel], kvec=g[sel] / n, U=np.ascontiguousarray(U[:, :, :nb]), GGT=G @ G.T,
                 cell=abs(np.linalg.det(R)))
    else:
        e0 = EWIN * ((rng.permutation(nk) + 0.5) / nk) ** (2.0 / 3.0)
    d = rng.uniform(0.0, 2e-3 * EV, (nk, max(1, nb // 2)))
    e = np.concatenate([np.stack([e0 + 0.05 * EV * i - 0.5 * d[:, i], e0 + 0.05 * EV * i + 0.5 * d[:, i]], 1)
                        for i in range(nb // 2)], 1) + ECBM
    f = 1.0 / (np.exp((e - (ECBM - 0.1 * EV)) / T300) + 1.0)
    sp = _spin(rng, nk, nb)
    fd, ed = f[:, :, None] - f[:, None, :], e[:, :, None] - e[:, None, :]
    near = np.abs(ed) < 1e-9
    ratio = np.where(near, -(f * (1.0 - f))[:, :, None] / T300, fd / np.where(near, 1.0, ed))

    def state(axis, tesla):
        """the response of first order to a field: f + (f_i - f_j) / (e_i - e_j) B S_ij"""
        return f[:, :, None] * np.eye(nb) + ratio * (tesla * TESLA) * sp[:, axis]

    k1, k2 = _pair_list(e0, c["de"] * 1e-3 * EV)
    s.update(e=e, f=f, nkf=nkf, prefac=2.0 * math.pi / nkf, sz=np.ascontiguousarray(sp[:, 2]), k1=k1, k2=k2)
    s["H"] = np.ascontiguousarray(c["field"] * TESLA * sp[:, 0]) if c["field"] else None
    if c["kind"] == "batch":  # polarised along x, y, z in turn, each with its own pump's random deviation
        x = 1e-4 * (rng.standard_normal((c["states"], nk, nb, nb)) + 1j * rng.standard_normal((c["states"], nk, nb, nb)))
        x *= f[None, :, :, None]
        s["rho"] = np.stack([state(q % 3, 0.1) for q in range(c["states"])]) + 0.5 * (x + np.conj(np.swapaxes(x, 2, 3)))
    else:
        s["rho"] = state(2, 0.1)
    s["rho"] = 0.5 * (s["rho"] + np.conj(np.swapaxes(s["rho"], -1, -2)))
    return s


def _linear(c, s, P1, P2, i1, i2):
    """operators of a linearized run: rates into k1 and k2 with the blocking of f folded in, and the
    losses on the diagonal pairs"""
    nb = s["nb"]
    f = torch.as_tensor(s["f"], device="cuda").mean(1)
    L1 = P1 * (1.0 - f[i1])[:, None]
    L2 = P2.conj() * (1.0 - f[i2])[:, None]
    loss = -torch.eye(nb * nb, dtype=torch.complex128, device="cuda").reshape(1, -1) * (2e-3 * s["nkf"] / (200.0 * FS))
    same = (i1 == i2)[:, None]
    return torch.where(same, L1 + loss, L1), torch.where(same, torch.zeros_like(L2), L2)


def _arrays(c, seed, s, host):
    """the operators of the whole case, as host arrays or on the GPU"""
    n4 = s["nb"] ** 4
    shape = (s["k1"].size, n4)
    if host:
        P1, P2 = np.empty(shape, np.complex128), np.empty(shape, np.complex128)
    else:
        P1 = torch.empty(shape, dtype=torch.complex128, device="cuda")
        P2 = torch.empty_like(P1)
    for p0, a, b in _operators(c, seed, s["e"], s["k1"], s["k2"]):
        n = a.shape[0]
        if c["kind"] == "rkf45":
            i1 = torch.as_tensor(s["k1"][p0:p0 + n].astype(np.int64), device="cuda")
            i2 = torch.as_tensor(s["k2"][p0:p0 + n].astype(np.int64), device="cuda")
            a, b = _linear(c, s, a, b, i1, i2)
        P1[p0:p0 + n] = a.cpu().numpy() if host else a
        P2[p0:p0 + n] = b.cpu().numpy() if host else b
    return P1, P2


def _ee_args(s):
    return dict(kvec=s["kvec"], kmesh=(s["mesh"],) * 3, U=s["U"], f=s["f"], GGT=s["GGT"], cell_size=s["cell"],
                nk_full=s["nkf"], temperature=T300, eps_background=12.9, meff=MEFF, formula="debye",
                nfree=float(s["f"].sum()) / (s["nkf"] * s["cell"]), update_screening=1, nv=0, degauss=DEGAUSS,
                ethr=DEGAUSS * NDEGAUSS, antisymmetry=0, scale=1.0, every_rhs=0)


def prepare(case, seed):
    c, s = case, _system(case, seed)
    P1, P2 = _arrays(c, seed, s, True)
    kind = c["kind"]
    g = LindbladGPU(nk=s["nk"], nb_dm=s["nb"], bstart=0, bend=s["nb"], e_dm=s["e"], k1st=s["k1"], k2nd=s["k2"], P1=P1, P2=P2,
                    prefac_eph=s["prefac"], Hcoh=s["H"], picture="interaction", expt=1, precision=c["prec"],
                    f_ref=s["f"], linear=kind == "rkf45", nrhs=c.get("states", 1), adjoint=kind == "adjoint",
                    ee=_ee_args(s) if kind == "ee" else None, sparse=bool(c.get("fill")))
    g.set_observable(0, s["sz"], s["f"], 1.0 / s["nkf"])
    y = np.ascontiguousarray(s["rho"]).view(np.float64).reshape(-1)
    return dict(c=c, g=g, y=y, t0=3.0 * FS, dydt=np.empty_like(y))


def run(state):
    c, g, y, t0 = state["c"], state["g"], state["y"], state["t0"]
    kind = c["kind"]
    if kind == "func":
        return g.func(t0, y, state["dydt"])
    if kind == "adjoint":
        n = c["steps"]
        sz, dP, dy = g.adjoint_rk4(t0, y, 1.0 * FS, n, [n // 2, n], [0.5, 1.0], want_dy0=True)
        return {"sz": sz, "dP": dP, "dy0": dy}
    g.set_state(t0, y)
    if kind == "ee":
        g.ee_update()
        P1, P2, n = g.ee_read()
        return {"P1": P1, "P2": P2, "n": n}
    if kind == "rkf45":
        h, evals = g.rkf45_apply(t0 + 100.0 * FS, 1.0 * FS, epsabs=1e-12)
        t, y = g.get_state()
        return {"y": y, "h": h, "evals": evals, "sz": g.measure(0)[0], "dydt": g.func(t, y)}
    g.rk4(1.0 * FS, c["steps"])
    if kind == "batch":
        return {"y": g.get_state()[1], "sz": g.measure_batch(0)[0]}
    sz = g.measure(0)[0]
    t, y = g.get_state()
    if c["prec"] in ("f32", "bf16x2"):
        return {"y": y, "sz": sz}
    return {"y": y, "sz": sz, "dydt": g.func(t, y)}  # the slope, for the instantaneous lifetime beside S_z


def _evals(c):
    return {"func": 1, "rk4": 4 * c["steps"] + (c["prec"] in ("f64", "f64x")), "batch": 4 * c["steps"], "rkf45": 13, "adjoint": 8 * c["steps"]}[c["kind"]]


def work(case):
    c, n, nb, nk, q = case, _npair(case), case["nb"], case["nk"], case.get("states", 1)
    if c["kind"] == "ee":
        # per pair and k3 on the set (about 0.6 of them) and inside the energy window: U_3^+ U_4, the
        # matrix elements and both contractions; P_ee written, P and the per-k arrays read
        flops = n * nk * 0.4 * (8 * (nb * nb * 2 * nb + 4 * nb ** 5 + 2 * nb ** 6) + 8 * nb ** 4)
        return {"bytes": n * 2 * nb ** 4 * 16 * 2.0 + nk * nb * nb * 16 * 6.0, "flops": float(flops)}
    # every right-hand side reads each stored operator element once (it depends on the state before it)
    # and reads and writes the states; an element enters both the k and the k' sum as complex x real
    width = {"f64": 16, "f64x": 16, "f32": 8, "bf16x2": 8}[c["prec"]]
    per_pair = 2 * nb ** 4 * width * c.get("fill", 1.0)
    state = 16.0 * nk * nb * nb * q
    if c["kind"] == "adjoint":  # forward, then per stage the operators again and the gradient read and written
        return {"bytes": 4.0 * c["steps"] * n * per_pair * 4, "flops": 4.0 * c["steps"] * n * 16 * nb ** 4 * 4}
    return {"bytes": _evals(c) * (n * per_pair + 3 * state),
            "flops": _evals(c) * float(n) * 16 * nb ** 4 * q * c.get("fill", 1.0)}


# ---------------------------------------------------------------------------------------------------------
# the same quantities in plain torch, FP64
# ---------------------------------------------------------------------------------------------------------
class _Exact:
    def __init__(self, c, seed):
        self.c, self.s = c, _system(c, seed)
        s = self.s
        cu = lambda a, t: None if a is None else torch.as_tensor(np.ascontiguousarray(a), dtype=t, device="cuda")  # noqa: E731
        self.nk, self.nb = s["nk"], s["nb"]
        self.P1, self.P2 = _arrays(c, seed, s, False)
        self.i1, self.i2 = cu(s["k1"].astype(np.int64), torch.int64), cu(s["k2"].astype(np.int64), torch.int64)
        self.both = (self.i1 < self.i2).to(torch.float64)
        self.e, self.f = cu(s["e"], torch.float64), cu(s["f"], torch.float64)
        self.H, self.sz = cu(s["H"], torch.complex128), cu(s["sz"], torch.complex128)
        self.one = torch.eye(self.nb, dtype=torch.complex128, device="cuda")
        self.de = self.e[:, :, None] - self.e[:, None, :]
        self.step = max(1, (1 << 26) // (self.nb ** 4 * 16))

    def phase(self, t):
        return torch.polar(torch.ones_like(self.de), self.de * t)

    def sums(self, r, w):
        """X, Y ([nk][nb^2][states]) of the coordinates r, w ([nk][nb^2][states])"""
        n2 = self.nb ** 2
        X, Y = torch.zeros_like(r), torch.zeros_like(r)
        for p in range(0, self.i1.numel(), self.step):
            a, b = self.i1[p:p + self.step], self.i2[p:p + self.step]
            m = self.both[p:p + self.step, None, None]
            P1, P2 = self.P1[p:p + self.step].reshape(-1, n2, n2), self.P2[p:p + self.step].reshape(-1, n2, n2)
            X = X.index_add(0, a, P1 @ r[b])
            if w is None:
                X = X.index_add(0, b, m * (P2 @ r[a]))
                continue
            X = X.index_add(0, b, m * (P2.conj() @ r[a]))
            Y = Y.index_add(0, a, P2.transpose(1, 2) @ w[b])
            Y = Y.index_add(0, b, m * (P1.conj().transpose(1, 2) @ w[a]))
        return X, Y

    def rhs(self, t, rho):
        """d rho / dt of [states][nk][nb][nb]"""
        nk, nb, q = self.nk, self.nb, rho.shape[0]
        D = self.phase(t)
        flat = lambda z: z.permute(1, 2, 3, 0).reshape(nk, nb * nb, q)  # noqa: E731
        full = lambda z: z.reshape(nk, nb, nb, q).permute(3, 0, 1, 2)  # noqa: E731
        if self.c["kind"] == "rkf45":
            X, _ = self.sums(flat(D.conj() * (rho - torch.diag_embed(self.f).to(rho.dtype))), None)
            z = D * full(X)
        else:
            X, Y = self.sums(flat(D.conj() * rho), flat(D.conj() * (self.one - rho)))
            z = (self.one - rho) @ (D * full(X)) - (D * full(Y)) @ rho
        out = 0.5 * self.s["prefac"] * (z + z.conj().transpose(2, 3))
        if self.H is not None:
            Ht = self.H * D
            out = out - 1j * (Ht @ rho - rho @ Ht)
        return out

    def rk4(self, t, h, y):
        k1 = self.rhs(t, y)
        k2 = self.rhs(t + 0.5 * h, y + 0.5 * h * k1)
        k3 = self.rhs(t + 0.5 * h, y + 0.5 * h * k2)
        k4 = self.rhs(t + h, y + h * k3)
        return y + h / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)

    def measure(self, t, y):
        d = y - torch.diag_embed(self.f).to(y.dtype)
        return torch.einsum("kib,qkbi->q", self.sz * self.phase(t), d).real / self.s["nkf"]

    def rkf45(self, t, t1, h, eps, y):
        """Fehlberg's pair with the standard step control (absolute tolerance), steps up to t1"""
        A = [1 / 4, 3 / 8, 12 / 13, 1.0, 1 / 2]
        B = [[1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
             [8341 / 4104, -32832 / 4104, 29440 / 4104, -845 / 4104],
             [-6080 / 20520, 41040 / 20520, -28352 / 20520, 9295 / 20520, -5643 / 20520]]
        C = [902880 / 7618050, 0.0, 3953664 / 7618050, 3855735 / 7618050, -1371249 / 7618050, 277020 / 7618050]
        E = [1 / 360, 0.0, -128 / 4275, -2197 / 75240, 1 / 50, 2 / 55]
        evals = 0
        while t < t1:
            K = [self.rhs(t, y)]
            evals += 1
            while True:
                last = h > t1 - t
                h = t1 - t if last else h
                del K[1:]
                for a, b in zip(A, B):
                    K.append(self.rhs(t + a * h, y + h * sum(u * k for u, k in zip(b, K))))
                    evals += 1
                r = float((h * torch.view_as_real(sum(u * k for u, k in zip(E, K)))).abs().max()) / eps
                if r > 1.1:
                    h *= max(0.2, 0.9 / r ** 0.2)
                    continue
                y = y + h * sum(u * k for u, k in zip(C, K))
                t = t1 if last else t + h
                if r < 0.5:
                    h *= min(5.0, max(1.0, 0.9 / max(r, 2.3e-308) ** (1 / 6)))
                break
        return y, h, evals


def _exact_ee(c, seed):
    """P_ee of every stored pair from rho (Lindblad form, Debye screening at rho's density)"""
    s = _system(c, seed)
    nk, nb, n = s["nk"], s["nb"], s["mesh"]
    dev = dict(device="cuda")
    e, U = torch.as_tensor(s["e"], **dev), torch.as_tensor(s["U"], **dev)
    rho = torch.as_tensor(s["rho"], **dev)
    D = torch.polar(torch.ones_like(e[:, :, None] - e[:, None, :]), (e[:, :, None] - e[:, None, :]) * (3.0 * FS))
    dm = rho * D.conj()
    dm1 = torch.eye(nb, dtype=torch.complex128, **dev) - dm
    dens = float(dm.diagonal(dim1=1, dim2=2).real.sum()) / (s["nkf"] * s["cell"])
    i1, i2 = (torch.as_tensor(s[k].astype(np.int64), **dev) for k in ("k1", "k2"))
    kidx = torch.as_tensor(s["kidx"].astype(np.int64), **dev)
    table = torch.full((n, n, n), -1, dtype=torch.int64, **dev)
    w = kidx % n
    table[w[:, 0], w[:, 1], w[:, 2]] = torch.arange(nk, **dev)
    q = torch.as_tensor(s["kvec"], **dev)
    q = q[i1] - q[i2]
    q = q - torch.floor(0.5 + q)
    q2 = torch.einsum("pd,de,pe->p", q, torch.as_tensor(s["GGT"], **dev), q)
    vq = 4 * math.pi / 12.9 / s["cell"] / (4 * math.pi * dens / 12.9 / T300 + q2)
    o12 = torch.einsum("pwa,pwb->pab", U[i1].conj(), U[i2]) * vq[:, None, None]
    P1 = torch.zeros((i1.numel(),) + (nb,) * 4, dtype=torch.complex128, **dev)
    P2 = torch.zeros_like(P1)
    for k3 in range(nk):
        m = (kidx[i1] + kidx[k3] - kidx[i2]) % n
        k4 = table[m[:, 0], m[:, 1], m[:, 2]]
        on = torch.nonzero((k4 >= 0) & (i1 != i2)).reshape(-1)
        if not on.numel():
            continue
        a, b, d = i1[on], i2[on], k4[on]
        de = e[a][:, :, None, None, None] - e[b][:, None, :, None, None] + e[k3][None, None, None, :, None] - e[d][:, None, None, None, :]
        delta = torch.where(de.abs() < DEGAUSS * NDEGAUSS, torch.exp(-0.25 * de * de / DEGAUSS ** 2), torch.zeros_like(de))
        o34 = torch.einsum("wa,pwb->pab", U[k3].conj(), U[d])
        A = delta * torch.einsum("pab,pcd->pabcd", o12[on], o34)
        Ar = torch.einsum("ij,pabjk,pkl->pabil", dm1[k3], A, dm[d])
        Ab = torch.einsum("ij,pabjk,pkl->pabil", dm[k3], A, dm1[d])
        P1.index_add_(0, on, torch.einsum("pacij,pbdij->pabcd", Ar, A.conj()))
        P2.index_add_(0, on, torch.einsum("pcaij,pdbij->pabcd", Ab, A.conj()))
    f = 1.0 / (DEGAUSS * math.sqrt(2 * math.pi)) / s["nkf"]
    return {"P1": (P1 * f).reshape(-1, nb ** 4), "P2": (P2 * f).reshape(-1, nb ** 4), "n": None}


def exact(case, seed):
    c = case
    if c["kind"] == "ee":
        return _exact_ee(c, seed)
    if c["kind"] == "batch" and c["nb"] == 4 and c["nk"] > 1000:
        return None  # over 20 s in FP64
    x = _Exact(c, seed)
    t, h = 3.0 * FS, 1.0 * FS
    y = torch.as_tensor(x.s["rho"], device="cuda").reshape(-1, x.nk, x.nb, x.nb)
    real = lambda z: torch.view_as_real(z).reshape(-1)  # noqa: E731
    if c["kind"] == "func":
        return real(x.rhs(t, y))
    if c["kind"] == "rkf45":
        y, h, evals = x.rkf45(t, t + 100.0 * FS, h, 1e-12, y)
        t += 100.0 * FS
        return {"y": real(y), "h": h, "evals": evals, "sz": float(x.measure(t, y)), "dydt": real(x.rhs(t, y))}
    if c["kind"] == "adjoint":
        y0 = y.clone().requires_grad_(True)
        x.P1.requires_grad_(True)
        x.P2.requires_grad_(True)
        seen, n, y = [], c["steps"], y0
        for i in range(n):
            y = x.rk4(t + i * h, h, y)
            if i + 1 in (n // 2, n):
                seen.append(x.measure(t + (i + 1) * h, y)[0])
        g1, g2, gy = torch.autograd.grad(0.5 * seen[0] + seen[1], [x.P1, x.P2, y0])
        return {"sz": torch.stack(seen).detach(), "dP": torch.stack([g1, g2]), "dy0": real(gy)}
    for i in range(c["steps"]):
        y = x.rk4(t + i * h, h, y)
    t += c["steps"] * h
    sz = x.measure(t, y)
    out = {"y": real(y), "sz": sz if c["kind"] == "batch" else float(sz)}
    if c["kind"] == "rk4" and c["prec"] in ("f64", "f64x"):
        out["dydt"] = real(x.rhs(t, y))
    return out
