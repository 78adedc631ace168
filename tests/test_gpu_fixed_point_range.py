"""Ranges of states and operators beside the exponents that the fixed-point contraction shares (csrc/dmd_pairs_fx.cuh): its sums
have to keep FP64's error at every k-point's own scale, not only beside the largest of all.

Bound. The scattering term is (prefac / 2) (C + C^+), C = (1 - rho) X - Y rho, X and Y sums over the pairs of n products. With
S the same sums of absolute values, a k-point's term is off by at most prefac nb (|1 - rho| S_X + |rho| S_Y) eps, largest
elements taken of each. FP64 sums (the oracle's side: a handle with DMD_FLAG_EE, on the FP64 pipe) have eps of some 2^-51 for n of a few
hundred; fixed-point ones are listed for FP64 from an error of 2^-49 (root mean square) on, four times that for the worst of some
thousand sums, and as much again for elements within 2^10 of their row block's: 2^-46 for both sides together.
"""
import numpy as np
import pytest

from test_gpu_fixed_point import built, handle, system  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -46


def scale(s, y, lines=slice(None)):
    """prefac nb (|1 - rho| S_X + |rho| S_Y) of every k-point (the window the whole density matrix), from these elements of X, Y"""
    nk, nb = s.nk, s.bend - s.bstart
    n2 = nb * nb
    k1, k2 = s.k1st.astype(np.int64), s.k2nd.astype(np.int64)
    P1, P2 = np.abs(np.asarray(s.P1)).reshape(-1, n2, n2), np.abs(np.asarray(s.P2)).reshape(-1, n2, n2)
    rho = np.ascontiguousarray(y).view(np.complex128).reshape(nk, n2)
    r, w = np.abs(rho), np.abs(np.eye(nb).reshape(-1) - rho)
    both = (k1 < k2)[:, None]
    X, Y = np.zeros((nk, n2)), np.zeros((nk, n2))
    np.add.at(X, k1, np.einsum("pab,pb->pa", P1, r[k2]))
    np.add.at(X, k2, both * np.einsum("pab,pb->pa", P2, r[k1]))
    np.add.at(Y, k1, np.einsum("pab,pa->pb", P2, w[k2]))
    np.add.at(Y, k2, both * np.einsum("pab,pa->pb", P1, w[k1]))
    return s.prefac_eph * nb * (w.max(1) * X[:, lines].max(1) + r.max(1) * Y[:, lines].max(1))


def handle_x(s):
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    return LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd,
                       P1=s.P1, P2=s.P2, prefac_eph=s.prefac_eph, picture=0, expt=1, precision="f64x")


def worst(s, y, t, make=handle):
    """the largest error of a k-point in units of its scale, against the FP64 pipe"""
    with make(s) as g, handle(s, pipe=True) as p:
        out, ref = g.func(t, y).reshape(s.nk, -1), p.func(t, y).reshape(s.nk, -1)
    u = scale(s, y)
    assert (out[u == 0] == 0).all()
    return float((np.abs(out - ref).max(1)[u > 0] / u[u > 0]).max())


def localised(rng, nk, nb, kind):
    """Hermitian rho_k of very different size from k-point to k-point"""
    if kind == "tail":      # a cold band: e^-E/kT over 2^-200
        w = np.exp2(-200.0 * np.arange(nk) / nk)
    elif kind == "random":  # neighbours in energy up to 2^60 apart
        w = np.exp2(-60.0 * rng.random(nk))
    elif kind == "spot":    # three k-points excited on a background of 1e-18
        w = np.full(nk, 1e-18)
        w[rng.integers(nk, size=3)] = 0.3
    else:                   # and on none
        w = np.zeros(nk)
        w[rng.integers(nk, size=3)] = 0.3
    x = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
    x = 0.05 * (x + np.conj(np.swapaxes(x, 1, 2))) + 0.5 * np.eye(nb)
    return w[:, None, None] * x


@pytest.mark.parametrize("hermitian", [True, False])
@pytest.mark.parametrize("kind", ["tail", "random", "spot", "alone"])
@pytest.mark.parametrize("nk,nb,density", [(33, 2, 1.0), (500, 2, 0.5), (9, 4, 1.0), (70, 4, 0.6)])
def test_states_of_wide_range(nk, nb, density, kind, hermitian, oracle, built):
    s = system(oracle, nk, nb, density, 17 + nk)
    rng = np.random.default_rng(nk)
    rank = np.argsort(np.argsort(s.e_dm.mean(1)))
    y = np.ascontiguousarray(localised(rng, nk, nb, kind)[rank]).view(np.float64).reshape(-1)
    if not hermitian:
        y = y * (1.0 + 0.3 * rng.standard_normal(y.size))
    assert worst(s, y, 13.0 * oracle.fs) < EPS


def test_many_weak_sums_in_a_run(oracle, built):
    """RK4 and RKF45 steps on a state whose sums are mostly listed: chained stages clear and count the lists of each"""
    s = system(oracle, 200, 2, 0.5, 9)
    rng = np.random.default_rng(3)
    rank = np.argsort(np.argsort(s.e_dm.mean(1)))
    y = np.ascontiguousarray(localised(rng, s.nk, 2, "tail")[rank]).view(np.float64).reshape(-1)
    out = []
    for pipe in (False, True):
        with handle(s, pipe=pipe) as g:
            g.set_state(0.0, y)
            g.rk4(0.2 * oracle.fs, 3)
            a = g.get_state()[1]
            g.rkf45_apply(g.get_state()[0] + 1.0 * oracle.fs, 0.2 * oracle.fs, epsabs=1e-9)
            out.append((a, g.get_state()[1], g.func(0.0, y)))
    for a, b in zip(*out):  # (each k-point's change over a step is far below its own largest neighbours' state)
        a, b = a.reshape(s.nk, -1), b.reshape(s.nk, -1)
        assert (np.abs(a - b).max(1) <= 1e-11 * np.abs(b).max(1)).all()


MEV = 1e-3 / 27.21138505
KELVIN = 1.3806488e-23 / 4.35974434e-18


def cold_band(oracle, nk, nb, T, de, seed):
    """a band of 200 meV at temperature T (kelvin) in equilibrium with its phonons: operators A (x) conj(A) of six modes,
    sqrt(n_q + 1) and sqrt(n_q) for emission and absorption, Gaussian energy conservation of 10 meV; pairs within `de` meV.
    Detailed balance pairs a large occupation with a small element and the reverse."""
    rng = np.random.default_rng(seed)
    s = system(oracle, nk, nb, 0.01, seed)
    e0 = 200.0 * MEV * ((rng.permutation(nk) + 0.5) / nk) ** (2.0 / 3.0)
    e = np.sort(e0[:, None] + rng.uniform(-1.0, 1.0, (nk, nb)) * MEV, axis=1)
    a, b = np.triu_indices(nk)
    keep = np.abs(e0[a] - e0[b]) < de * MEV
    k1, k2 = a[keep], b[keep]
    n = k1.size
    d = e[k1][:, :, None] - e[k2][:, None, :]
    A1, A2 = [], []
    for w in (8.0, 17.0, 26.0, 35.0, 44.0, 57.0):
        nq = 1.0 / np.expm1(w * MEV / (T * KELVIN))
        x = [(rng.standard_normal((n, nb, nb)) + 1j * rng.standard_normal((n, nb, nb))) *
             np.where(np.abs(d + u * w * MEV) < 50.0 * MEV, np.exp(-((d + u * w * MEV) / (20.0 * MEV)) ** 2), 0.0) for u in (1, -1)]
        A1 += [x[0] * np.sqrt(nq + 1.0), x[1] * np.sqrt(nq)]
        A2 += [x[1] * np.sqrt(nq + 1.0), x[0] * np.sqrt(nq)]

    def outer(A, transpose):
        A = np.stack(A, 1)
        A = np.swapaxes(A, 2, 3) if transpose else A
        X = A.reshape(n, -1, nb * nb)
        M = np.matmul(np.swapaxes(X, 1, 2), X.conj())
        return np.ascontiguousarray(M.reshape(n, nb, nb, nb, nb).transpose(0, 1, 3, 2, 4)).reshape(-1)

    f = 1.0 / (np.exp((e + 100.0 * MEV) / (T * KELVIN)) + 1.0)
    x = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
    dm = f[:, :, None] * np.eye(nb) + 1e-2 * (x + np.conj(np.swapaxes(x, 1, 2))) * np.sqrt(f[:, :, None] * f[:, None, :])
    return oracle.from_arrays(nk=nk, nb_dm=nb, bstart=0, bend=nb, e_dm=e, f_dm=f, k1st=k1.astype(np.uint64),
                              k2nd=k2.astype(np.uint64), P1=outer(A1, False), P2=outer(A2, True), prefac_eph=s.prefac_eph,
                              dm0=dm.reshape(nk, -1))


@pytest.mark.parametrize("T", [300.0, 77.0, 50.0, 30.0, 10.0])
@pytest.mark.parametrize("nk,nb,de", [(96, 2, 60.0), (300, 2, 60.0), (100, 2, 250.0), (60, 4, 40.0)])
def test_cold_bands(nk, nb, de, T, oracle, built):
    s = cold_band(oracle, nk, nb, T, de, nk + nb)
    y = oracle.y_of(s.dm0)
    assert worst(s, y, 13.0 * oracle.fs) < EPS
    rng = np.random.default_rng(5)
    assert worst(s, y * (1.0 + 1e-2 * rng.standard_normal(y.size)), 13.0 * oracle.fs) < EPS


@pytest.mark.parametrize("nb", [2, 4])
def test_spin_flip_elements_of_uneven_strength(nb, oracle, built):
    """k-points whose spin-flip elements (diagonal to off-diagonal) are 1e-6 of their neighbours' while the spin-conserving ones are
    alike: the off-diagonal elements of their terms, at the scale of those sums"""
    s = system(oracle, 96, nb, 0.6, 41)
    n2 = nb * nb
    off = np.array([a // nb != a % nb for a in range(n2)])
    odd = ((s.k1st | s.k2nd) & np.uint64(1)).astype(bool)
    mix = odd[:, None, None] & (off[:, None] != off[None, :])
    s.P1, s.P2 = (np.where(mix, 1e-6, 1.0) * np.asarray(P).reshape(-1, n2, n2) for P in (s.P1, s.P2))
    s.P1, s.P2 = s.P1.reshape(-1), s.P2.reshape(-1)
    y = oracle.y_of(s.dm0).copy()
    y.reshape(s.nk, n2, 2)[:, off] = 0.0
    t = 0.0
    with handle(s) as g, handle(s, pipe=True) as p:
        out, ref = (h.func(t, y).reshape(s.nk, n2, 2)[1::2, off] for h in (g, p))
    err = np.abs(out - ref).max((1, 2))
    u = scale(s, y, off)[1::2]
    assert u.max() < 1e-3 * scale(s, y)[1::2].max()
    assert (err < EPS * u).all()


@pytest.mark.parametrize("strength", [1e-2, 1e-4, 1e-25])
@pytest.mark.parametrize("nk,nb", [(70, 2), (400, 2), (40, 4)])
def test_a_weakly_coupled_k_point(nk, nb, strength, oracle, built):
    """its own terms at its own scale, in the f64 and the f64x form"""
    s = system(oracle, nk, nb, 0.6, 3)
    on = (s.k1st == 11) | (s.k2nd == 11)
    s.P1, s.P2 = (np.where(on, strength, 1.0)[:, None] * np.asarray(P).reshape(-1, nb ** 4) for P in (s.P1, s.P2))
    s.P1, s.P2 = s.P1.reshape(-1), s.P2.reshape(-1)
    y = oracle.y_of(s.dm0)
    assert worst(s, y, 5.0 * oracle.fs) < EPS
    assert worst(s, y, 5.0 * oracle.fs, handle_x) < EPS


def test_zero_pairs_and_strengths_in_every_row_block(oracle, built):
    """pairs of three strengths and none in every row block (three classes), one-sided and repeated pairs among them, and a
    state that is not finite: the split row blocks keep every pair's place"""
    s = system(oracle, 150, 2, 0.7, 77)
    rng = np.random.default_rng(1)
    w = np.array([1.0, 2.0 ** -25, 2.0 ** -50, 0.0])[rng.choice(4, s.k1st.size, p=[0.9, 0.04, 0.04, 0.02])][:, None]
    s.P1, s.P2 = ((w * np.asarray(P).reshape(-1, 16)).reshape(-1) for P in (s.P1, s.P2))
    y = oracle.y_of(s.dm0)
    assert worst(s, y, 5.0 * oracle.fs) < EPS
    v = y.copy()
    v[8 * 40] = np.nan
    with handle(s) as g, handle(s, pipe=True) as p:
        np.testing.assert_array_equal(np.isfinite(g.func(0.0, v)), np.isfinite(p.func(0.0, v)))


@pytest.mark.parametrize("fill", [0.44, 0.18, 0.05])
@pytest.mark.parametrize("nk,nb,density", [(40, 2, 1.0), (300, 2, 0.5), (120, 4, 0.3)])
def test_mostly_zero_operators(nk, nb, density, fill, oracle, built):
    """operators with most elements zero, in the dense form: columns without an element on the diagonal coordinates' lines, groups of one
    element. Off-diagonal coordinates 1e-3 of the diagonal ones, and a state that is not Hermitian."""
    s = system(oracle, nk, nb, density, 5 * nk + nb)
    rng = np.random.default_rng(2)
    s.P1, s.P2 = (np.where(rng.random(np.size(P)) < fill, np.asarray(P), 0.0) for P in (s.P1, s.P2))
    y = oracle.y_of(s.dm0)
    assert worst(s, y, 5.0 * oracle.fs) < EPS
    assert worst(s, y * (1.0 + 1e-2 * rng.standard_normal(y.size)), 5.0 * oracle.fs) < EPS
    rank = np.argsort(np.argsort(s.e_dm.mean(1)))
    for kind in ("spot", "tail", "random"):
        z = np.ascontiguousarray(localised(rng, nk, nb, kind)[rank]).view(np.float64).reshape(-1)
        assert worst(s, z, 5.0 * oracle.fs) < EPS
