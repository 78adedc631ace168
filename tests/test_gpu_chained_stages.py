"""What a run of chained stages (csrc/dmd_finish.cuh) that ends in an error leaves behind: nothing."""
import numpy as np
import pytest

from test_gpu_fixed_point import built, handle, system  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu


def test_a_failed_rkf45_step_leaves_no_flag(oracle, built):
    """the step overflows, its last stage prepares coordinates that are not finite, and the step control gives up (a recoverable
    error): the next evaluation is the one that it was before, bit by bit. Two k-points: every sum has two terms, so that the
    order of the atomic sums does not show."""
    from denmat_dynm_development_gb300.dmd import DMDError
    s = system(oracle, 2, 2, 1.0, 4)
    s.k1st, s.k2nd = np.array([0, 0, 1], np.uint64), np.array([0, 1, 1], np.uint64)
    rng = np.random.default_rng(2)
    P = rng.standard_normal((2, 48)) + 1j * rng.standard_normal((2, 48))
    s.P1, s.P2 = P[0], P[1]
    y = oracle.y_of(s.dm0) * (1.0 + 0.1 * rng.standard_normal(16))
    with handle(s) as g:
        ref = g.func(0.0, y)
        for _ in range(5):
            np.testing.assert_array_equal(g.func(0.0, y), ref)
        g.set_state(0.0, 1e200 * np.ones(16))
        with pytest.raises(DMDError):
            g.rkf45_apply(1e3, 1.0, hmin=1e2, epsabs=1e-9)
        np.testing.assert_array_equal(g.func(0.0, y), ref)
