"""The RK4 step whose finishes prepare the next stage (csrc/dmd_finish.cuh) against the same steps taken from the host
through dmd_func, which prepares every evaluation by itself: the operations and their order per element are the same, so
the states differ only by the order of the contraction's atomic sums. FP64 forms: 1e-13 of the state's change per
evaluation and the roundings of the state itself, 1e-14; FP32 forms: their products' 2^-24 of the change, 1e-5."""
import numpy as np
import pytest

from test_gpu_fixed_point import built, system  # noqa: F401

pytestmark = pytest.mark.gpu


def handle(s, prec, picture, expt, H):
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    return LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=0, bend=s.nb_dm, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1,
                       P2=s.P2, prefac_eph=s.prefac_eph, Hcoh=H, picture=picture, expt=expt, precision=prec, f_ref=s.f_dm)


def host_rk4(g, t, h, n, y):
    for _ in range(n):
        k1 = g.func(t, y)
        k2 = g.func(t + 0.5 * h, y + 0.5 * h * k1)
        k3 = g.func(t + 0.5 * h, y + 0.5 * h * k2)
        k4 = g.func(t + h, y + h * k3)
        y = y + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        t += h
    return y


@pytest.mark.parametrize("prec", ["f64", "f64x", "f32", "bf16x2"])
@pytest.mark.parametrize("nb,nk", [(2, 1), (2, 37), (4, 5), (4, 33)])
@pytest.mark.parametrize("picture,expt,with_H,herm", [(0, 1, False, True), (0, 1, True, False), (1, 0, True, True),
                                                      (1, 1, False, False), (0, 0, True, True)])
def test_fused_step(prec, nb, nk, picture, expt, with_H, herm, oracle, built):  # noqa: F811
    s = system(oracle, nk, nb, 0.8, 11 * nk + nb)
    rng = np.random.default_rng(3)
    H = None
    if with_H:
        x = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
        H = 1e-4 * (x + np.conj(np.swapaxes(x, 1, 2)))
    y = oracle.y_of(s.dm0)
    if not herm:
        y = y * (1.0 + 1e-2 * rng.standard_normal(y.size))
    t0, h, n = 7.0 * oracle.fs, 2.0 * oracle.fs, 5
    tol = 1e-5 if prec in ("f32", "bf16x2") else 1e-13
    with handle(s, prec, picture, expt, H) as g:
        ref = host_rk4(g, t0, h, n, y)
        change = np.abs(ref - y).max()
        for _ in range(2):  # a second run starts from its own state
            g.set_state(t0, y)
            g.rk4(h, 2)
            g.rk4(h, n - 2)
            out = g.get_state()[1]
            assert np.abs(out - ref).max() <= tol * 4 * n * change + 1e-14 * np.abs(ref).max()
        # the evaluation after it finds no flag or sum of the step that did not follow
        a, b = g.func(t0, y), g.func(t0, y)
        assert np.abs(a - b).max() <= tol * np.abs(b).max()


def test_group_follows_a_change_of_a_member(oracle, built):  # noqa: F811
    """a drift set after the group's first step is in its next one"""
    from denmat_dynm_development_gb300.dmd import Group
    s = system(oracle, 20, 2, 0.8, 5)
    y, h = oracle.y_of(s.dm0), 1.0 * oracle.fs
    with handle(s, "f64", 0, 1, None) as g, handle(s, "f64", 0, 1, None) as alone:
        eq = 1e-6 * np.eye(2)[None].repeat(s.nk, 0).astype(np.complex128)
        with Group([g]) as group:
            g.set_state(0.0, y)
            group.rk4(h, 1)
            g.set_ddmdt_eq(eq)
            group.rk4(h, 1)
        alone.set_state(0.0, y)
        alone.rk4(h, 1)
        alone.set_ddmdt_eq(eq)
        alone.rk4(h, 1)
        a, b = g.get_state()[1], alone.get_state()[1]
    assert np.abs(a - b).max() <= 1e-14 * np.abs(b).max()


def host_rkf45(f, t, t1, h, eps_abs, eps_rel, y):
    """Fehlberg's pair with the standard control on the new y (GSL's rkf45 driver), on the host"""
    A = [1 / 4, 3 / 8, 12 / 13, 1.0, 1 / 2]
    B = [[1 / 4], [3 / 32, 9 / 32], [1932 / 2197, -7200 / 2197, 7296 / 2197],
         [8341 / 4104, -32832 / 4104, 29440 / 4104, -845 / 4104],
         [-6080 / 20520, 41040 / 20520, -28352 / 20520, 9295 / 20520, -5643 / 20520]]
    C = [902880 / 7618050, 0.0, 3953664 / 7618050, 3855735 / 7618050, -1371249 / 7618050, 277020 / 7618050]
    E = [1 / 360, 0.0, -128 / 4275, -2197 / 75240, 1 / 50, 2 / 55]
    evals = rejected = 0
    while t < t1:
        K = [f(t, y)]
        evals += 1
        while True:
            last = h > t1 - t
            h = t1 - t if last else h
            del K[1:]
            for a, b in zip(A, B):
                K.append(f(t + a * h, y + h * sum(u * k for u, k in zip(b, K))))
                evals += 1
            yn = y + h * sum(u * k for u, k in zip(C, K))
            r = float((np.abs(h * sum(u * k for u, k in zip(E, K))) / (eps_rel * np.abs(yn) + eps_abs)).max())
            if r > 1.1:
                h *= max(0.2, 0.9 / r ** 0.2)
                rejected += 1
                continue
            y, t = yn, t1 if last else t + h
            if r < 0.5:
                h *= min(5.0, max(1.0, 0.9 / max(r, 2.3e-308) ** (1 / 6)))
            break
    return y, h, evals, rejected


@pytest.mark.parametrize("nb,nk", [(2, 37), (4, 9)])
@pytest.mark.parametrize("h0,eps_abs,eps_rel", [(50.0, 1e-12, 0.0), (0.5, 1e-11, 1e-9), (400.0, 1e-13, 0.0)])
def test_fused_rkf45(nb, nk, h0, eps_abs, eps_rel, oracle, built):  # noqa: F811
    """steps accepted, rejected and retried, and a second interval from where the first one ended; the same number of
    evaluations, the state within the roundings of its own updates (1e-12, evaluations as above)"""
    s = system(oracle, nk, nb, 0.8, 3 * nk + nb)
    s.prefac_eph = 2e-5  # a few hundred fs of relaxation: the control has something to do
    rng = np.random.default_rng(4)
    y = oracle.y_of(s.dm0) * (1.0 + (1e-3 * rng.standard_normal(2 * nk * nb * nb) if nb == 4 else 0.0))
    t, rejected = 2.0 * oracle.fs, 0
    with handle(s, "f64", 0, 1, None) as g:
        g.set_state(t, y)
        h = hg = h0 * oracle.fs
        for t1 in (t + 100.0 * oracle.fs, t + 150.0 * oracle.fs):
            y, h, evals, rej = host_rkf45(g.func, t, t1, h, eps_abs, eps_rel, y)
            rejected += rej
            g.set_state(t, g.get_state()[1])
            hg, n = g.rkf45_apply(t1, hg, epsabs=eps_abs, epsrel=eps_rel)
            assert n == evals
            assert abs(hg - h) <= 1e-4 * h  # (the ratio is a difference of slopes near the tolerance)
            tg, yg = g.get_state()
            assert tg == t1 and np.abs(yg - y).max() <= 1e-12 * np.abs(y).max()
            t, hg, y = t1, h, yg
            g.set_state(t, y)
    assert rejected > 0 or h0 < 1.0


@pytest.mark.parametrize("nk,nrhs,linear,expt,herm", [(1, 2, False, 1, True), (7, 5, False, 1, False), (37, 130, False, 0, True),
                                                      (64, 16, True, 1, True), (333, 33, False, 1, True)])
def test_fused_batch(nk, nrhs, linear, expt, herm, oracle, built):  # noqa: F811
    """k_stage_tc2: partly filled column groups, one and two blocks of states, runs that end inside a group, states that
    are not Hermitian; against the same steps from the host. Both round the slopes to FP32 in the same operations: the
    states differ by roundings of their own updates (4 n 2^-53) and by next inputs that round the other way (2^-24 of the
    change per evaluation)."""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = system(oracle, nk, 2, 0.8, 17 * nk + nrhs)
    rng = np.random.default_rng(6)
    y = np.concatenate([oracle.y_of(s.dm0)] * nrhs).reshape(nrhs, -1)
    x = 1e-3 * rng.standard_normal((nrhs, nk, 2, 2)) + 1e-3j * rng.standard_normal((nrhs, nk, 2, 2))
    if herm:
        x = 0.5 * (x + np.conj(np.swapaxes(x, 2, 3)))
    y = (y + (x * s.f_dm[None, :, :, None]).reshape(nrhs, -1).view(np.float64)).reshape(-1)
    t0, h, n = 7.0 * oracle.fs, 2.0 * oracle.fs, 4
    with LindbladGPU(nk=nk, nb_dm=2, bstart=0, bend=2, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1, P2=s.P2,
                     prefac_eph=s.prefac_eph, picture=0, expt=expt, precision="bf16x2", f_ref=s.f_dm, nrhs=nrhs,
                     linear=linear) as g:
        ref = host_rk4(g, t0, h, n, y)
        change = np.abs(ref - y).max()
        g.set_state(t0, y)
        g.rk4(h, 1)
        g.rk4(h, n - 1)
        out = g.get_state()[1]
        assert np.abs(out - ref).max() <= 4 * n * 2.0 ** -24 * change + 4 * n * 2.0 ** -53 * np.abs(ref).max()
        assert g.func(t0, y).tobytes() == g.func(t0, y).tobytes()
