"""The fixed-point contraction of the FP64 form (csrc/dmd_pairs_fx.cuh) where it can go wrong: row blocks and
items with one pair and full ones, the last column block partly outside the k-points, one-sided, repeated and diagonal
pairs, operators and coordinates of very different size, states that are not Hermitian or not finite, and
operators without a fixed-point form. Against the oracle at the FP64 bound of the RHS (1e-12 normwise),
and for what the norm does not see, per k-point against the FP64-pipe contraction (a handle with DMD_FLAG_EE keeps it).

Bound per k-point: both forms round every product's operand and every partial sum at 2^-53 of the k-point's
sums or better, and n <= 2000 terms of random sign leave sqrt(n) 2^-53 < 1e-14 of sum |P| |r|; the finish cancels
up to three digits of it, so 1e-11 of the k-point's own largest dydt with a floor of 1e-14 of the largest of all.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built():
    import __graft_entry__ as G
    G.build()


def system(oracle, nk, nb, density, seed, spread=0.0):
    """random bands, occupations, states and operators; a share `density` of all (k, k') pairs, some one-sided, some
    twice; spread: P scaled by 2^-(0..spread) per pair"""
    rng = np.random.default_rng(seed)
    e = np.sort(rng.uniform(0.0, 0.01, (nk, nb)), axis=1) + rng.uniform(0.0, 0.02, (nk, 1))
    f = 1.0 / (np.exp(e / 2e-3) + 1.0)
    a, b = np.triu_indices(nk)
    keep = rng.random(a.size) < density
    keep[rng.integers(a.size)] = True
    k1, k2 = a[keep], b[keep]
    one = rng.random(k1.size) < 0.1  # k1 > k2: no reverse term
    k1, k2 = np.where(one, k2, k1), np.where(one, k1, k2)
    dup = rng.integers(0, k1.size, max(1, k1.size // 50))
    k1, k2 = np.concatenate([k1, k1[dup]]), np.concatenate([k2, k2[dup]])
    n, n4 = k1.size, nb ** 4
    P = rng.standard_normal((2, n, n4)) + 1j * rng.standard_normal((2, n, n4))
    P *= np.exp2(-spread * rng.random((1, n, 1)))
    P[:, rng.random(n) < 0.05] = 0.0
    x = rng.standard_normal((nk, nb, nb)) + 1j * rng.standard_normal((nk, nb, nb))
    dm = f[:, :, None] * np.eye(nb) + 1e-3 * (x + np.conj(np.swapaxes(x, 1, 2))) * f[:, :, None] * f[:, None, :]
    return oracle.from_arrays(nk=nk, nb_dm=nb, bstart=0, bend=nb, e_dm=e, f_dm=f, k1st=k1.astype(np.uint64),
                              k2nd=k2.astype(np.uint64), P1=P[0].reshape(-1), P2=P[1].reshape(-1), prefac_eph=1e-6,
                              dm0=dm.reshape(nk, -1))


def handle(s, pipe=False):
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    return LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd,
                       P1=s.P1, P2=s.P2, prefac_eph=s.prefac_eph, picture=0, expt=1, precision="f64", ee_flag=pipe)


def per_k(a, b, nk):
    a, b = a.reshape(nk, -1), b.reshape(nk, -1)
    big = np.abs(b).max(axis=1)
    return float((np.abs(a - b).max(axis=1) / np.maximum(big, 1e-3 * big.max())).max())


SHAPES = [(1, 2, 1.0), (2, 2, 1.0), (31, 2, 0.7), (33, 2, 1.0), (64, 2, 0.02), (200, 2, 0.5), (1500, 2, 0.6),
          (1, 4, 1.0), (9, 4, 1.0), (23, 4, 0.5), (150, 4, 0.4)]


@pytest.mark.parametrize("nk,nb,density", SHAPES)
def test_shapes_and_states(nk, nb, density, oracle, built):
    s = system(oracle, nk, nb, density, 100 * nb + nk)
    rng = np.random.default_rng(7)
    y = oracle.y_of(s.dm0)
    states = [y, y * (1.0 + 1e-2 * rng.standard_normal(y.size))]  # Hermitian, and not
    t = 13.0 * oracle.fs
    with handle(s) as g, handle(s, pipe=True) as p:
        for v in states:
            out, ref = g.func(t, v), oracle.rhs(s, t, v)
            assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
            assert per_k(out, p.func(t, v), nk) < 1e-11
        # non-finite entries reach the same elements as in FP64
        for bad in (np.nan, np.inf):
            v = y.copy()
            v[2 * nb * nb * (nk // 2)] = bad
            np.testing.assert_array_equal(np.isfinite(g.func(t, v)), np.isfinite(p.func(t, v)))


@pytest.mark.parametrize("scale", [1e-290, 1e-30, 1e30, 1e280])
@pytest.mark.parametrize("nb", [2, 4])
def test_scales(nb, scale, oracle, built):
    """operators near both ends of FP64's range, with a spread of 2^20 from pair to pair"""
    s = system(oracle, 40, nb, 0.8, 5 + nb, spread=20.0)
    s.P1 *= scale
    s.P2 *= scale
    s.prefac_eph = 1e-6 / scale if scale > 1e-280 else 1e280
    y = oracle.y_of(s.dm0)
    t = 5.0 * oracle.fs
    with handle(s) as g, handle(s, pipe=True) as p:
        out, ref = g.func(t, y), p.func(t, y)
        assert np.isfinite(ref).all() and np.abs(ref).max() > 0
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max()
        assert per_k(out, ref, s.nk) < 1e-11


@pytest.mark.parametrize("what", ["weak k-point", "nan", "inf"])
def test_operators_without_a_fixed_point_form(what, oracle, built):
    """a k-point coupled 1e-25 as strongly as its neighbours, or a non-finite element: the FP64 pipes, as before"""
    s = system(oracle, 70, 2, 0.8, 3)
    P1, P2 = s.P1.reshape(-1, 16).copy(), s.P2.reshape(-1, 16).copy()
    if what == "weak k-point":
        on = (s.k1st == 11) | (s.k2nd == 11)
        P1[on] *= 1e-25
        P2[on] *= 1e-25
    else:
        P1[5, 3] = np.nan if what == "nan" else np.inf
    s.P1, s.P2 = P1.reshape(-1), P2.reshape(-1)
    y = oracle.y_of(s.dm0)
    t = 5.0 * oracle.fs
    with handle(s) as g, handle(s, pipe=True) as p:
        out, ref = g.func(t, y).reshape(s.nk, -1), p.func(t, y).reshape(s.nk, -1)
        np.testing.assert_array_equal(np.isfinite(out), np.isfinite(ref))
        if what == "weak k-point":
            assert 0 < np.abs(ref[11]).max() < 1e-20 * np.abs(ref).max()
            assert np.abs(out[11] - ref[11]).max() < 1e-11 * np.abs(ref[11]).max()


@pytest.mark.parametrize("nk,nb,density,fill,spread", [(1, 4, 1.0, 1.0, 0.0), (13, 3, 1.0, 0.3, 40.0), (40, 4, 0.5, 0.3, 60.0),
                                                       (460, 4, 0.02, 0.25, 20.0), (1000, 4, 0.001, 0.5, 20.0),
                                                       (70, 2, 1.0, 1.0, 0.0), (2000, 1, 1.0, 1.0, None)])
def test_sparse_form(nk, nb, density, fill, spread, oracle, built):
    """k_pairs_sparse_fx: lists shorter than a chunk and long ones, 1 to 8 threads per list, elements of one list 2^-spread
    apart (a scale per list would lose them), sums that outgrow their exponent (None: 1.9 in every element); against the dense
    FP64-pipe form per k-point, and what a non-finite coordinate reaches"""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = system(oracle, nk, nb, density, 7 * nk + nb)
    rng = np.random.default_rng(nk)
    for name in ("P1", "P2"):
        P = np.array(getattr(s, name))
        P = np.where(P == 0.0, 1e-30, P) * np.exp2(-(spread or 0.0) * rng.random(P.size))
        P = np.full(P.size, 1.9 + 0.0j) if spread is None else np.where(rng.random(P.size) < fill, P, 0.0)
        setattr(s, name, P)
    kw = dict(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1, P2=s.P2,
              prefac_eph=s.prefac_eph, picture=0, expt=1, precision="f64")
    y = oracle.y_of(s.dm0)
    t = 13.0 * oracle.fs
    with LindbladGPU(sparse=True, **kw) as g, LindbladGPU(ee_flag=nb in (2, 4), **kw) as p:
        for v in (y, y * (1.0 + 1e-2 * rng.standard_normal(y.size))):
            assert per_k(g.func(t, v), p.func(t, v), nk) < 1e-11
        np.testing.assert_array_equal(g.func(t, 0.0 * y), p.func(t, 0.0 * y))  # (zeros of either sign)
        if fill == 1.0:  # (a zero that is not stored takes no NaN)
            for bad in (np.nan, np.inf):
                v = y.copy()
                v[2 * nb * nb * (nk // 2)] = bad
                np.testing.assert_array_equal(np.isfinite(g.func(t, v)), np.isfinite(p.func(t, v)))


def test_sparse_form_with_an_infinite_element(oracle, built):
    """operators without a fixed-point form stay on the FP64 pipe"""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = system(oracle, 20, 4, 1.0, 3)
    s.P1 = np.array(s.P1)
    s.P1[5] = np.inf
    kw = dict(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1, P2=s.P2,
              prefac_eph=s.prefac_eph, picture=0, expt=1, precision="f64")
    y = oracle.y_of(s.dm0)
    with LindbladGPU(sparse=True, **kw) as g:
        out = g.func(0.0, y)
    assert not np.isfinite(out).all() and np.isfinite(out).any()
