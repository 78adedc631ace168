"""Ranges of states and operators beside the exponents that the fixed-point contraction shares (csrc/dmd_pairs_fx.cuh): its sums
have to keep FP64's error at every k-point's own scale, not only beside the largest of all.

Bound. The scattering term is (prefac / 2) (C + C^+), C = (1 - rho) X - Y rho, X and Y sums over the pairs of n products. With
S the same sums of absolute values, a k-point's term is off by at most prefac nb (|1 - rho| S_X + |rho| S_Y) eps, largest
elements taken of each. FP64 sums (the oracle's side: a handle with DMD_FLAG_EE, on the FP64 pipe) have eps of some 2^-51 for n of a few
hundred; fixed-point ones are listed for FP64 from an error of 2^-49 (root mean square) on, four times that for the worst of some
thousand sums, and as much again for pairs within 2^10 of each other's strength: 2^-46 for both sides together.
"""
import numpy as np
import pytest

from test_gpu_fixed_point import built, handle, system  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -46


def scale(s, y):
    """prefac nb (|1 - rho| S_X + |rho| S_Y) of every k-point (the window the whole density matrix)"""
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
    return s.prefac_eph * nb * (w.max(1) * X.max(1) + r.max(1) * Y.max(1))


def worst(s, y, t):
    """the largest error of a k-point in units of its scale, against the FP64 pipe"""
    with handle(s) as g, handle(s, pipe=True) as p:
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
