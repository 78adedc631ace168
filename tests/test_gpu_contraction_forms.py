"""Which contraction a handle takes when its operators have no fixed-point form, and with which work items: the time per
launch against the FP64-pipe contraction of the same operators (a handle with DMD_FLAG_EE keeps it)."""
import numpy as np
import pytest

from test_gpu_fixed_point import built, handle, system  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu


def uneven(oracle, nk, density, seed):
    """k-points of five strengths 2^-15 apart in turn: no exponent serves a row block's 32 columns"""
    s = system(oracle, nk, 2, density, seed)
    w = np.exp2(-15.0 * (np.arange(nk) % 5))
    w = (w[s.k1st.astype(np.int64)] * w[s.k2nd.astype(np.int64)])[:, None]
    s.P1 = (np.asarray(s.P1).reshape(-1, 16) * w).reshape(-1)
    s.P2 = (np.asarray(s.P2).reshape(-1, 16) * w).reshape(-1)
    return s


def contraction_us(oracle, s, **kw):
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    with LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1,
                     P2=s.P2, prefac_eph=s.prefac_eph, picture=0, expt=1, **kw) as g:
        g.set_state(0.0, oracle.y_of(s.dm0))
        g.rk4(oracle.fs, 5)
        g.set_profiling(True)
        g.rk4(oracle.fs, 20)
        ms, n = g.profile(1)
        return 1e3 * ms / n


def test_f64x_without_a_fixed_point_form_is_double_float(oracle, built):
    """the double-float contraction, not the FP64 pipe's: 225 against 700 us per launch on 2.5M pairs, 27 against 43 on 70k.
    A fifth less time than the f64 form's, and double-float sums: products to 2^-46, 330k pairs' normwise error below 1e-12"""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = uneven(oracle, 900, 0.8, 3)
    assert contraction_us(oracle, s, precision="f64x") < 0.8 * contraction_us(oracle, s, precision="f64")
    t, y, out = 3.0 * oracle.fs, oracle.y_of(s.dm0), []
    for prec in ("f64x", "f64"):
        with LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd,
                         P1=s.P1, P2=s.P2, prefac_eph=s.prefac_eph, picture=0, expt=1, precision=prec) as g:
            out.append(g.func(t, y))
    assert np.abs(out[0] - out[1]).max() < 1e-12 * np.abs(out[1]).max()


def test_f64x_operators_that_lose_and_regain_the_form(oracle, built):
    """dmd_add_operators chooses the form anew: an element becomes infinite, then the operators are other ones without it"""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = system(oracle, 60, 2, 0.8, 5)
    t, y = 3.0 * oracle.fs, oracle.y_of(s.dm0)
    P = [np.array(s.P1), np.array(s.P2)]
    w = np.exp2(-15.0 * (np.arange(60) % 5))
    w = (w[s.k1st.astype(np.int64)] * w[s.k2nd.astype(np.int64)])[:, None]
    U = [(p.reshape(-1, 16) * w).reshape(-1) for p in P]  # without the form
    with LindbladGPU(nk=s.nk, nb_dm=s.nb_dm, bstart=s.bstart, bend=s.bend, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd,
                     P1=P[0], P2=P[1], prefac_eph=s.prefac_eph, picture=0, expt=1, precision="f64x", adjoint=True) as g:
        for add, now in ((None, P), ([u - p for u, p in zip(U, P)], U), ([p - u for u, p in zip(U, P)], P)):
            if add is not None:
                g.add_operators(add[0], add[1], 1.0)
            s.P1, s.P2 = now
            ref = oracle.rhs(s, t, y)
            assert np.abs(g.func(t, y) - ref).max() < 1e-12 * np.abs(ref).max()
            g.set_state(t, y)
            g.rk4(1.0 * oracle.fs, 3)
            with handle(s) as fresh:  # FP64, from the operators as they are now
                fresh.set_state(t, y)
                fresh.rk4(1.0 * oracle.fs, 3)
                yr = fresh.get_state()[1]
            assert np.abs(g.get_state()[1] - yr).max() < 1e-12 * np.abs(yr).max()
