"""The batch's RK4 update (k_stage_tc2, csrc/dmd_batched_tc.cuh): y + h/6 (k1 + 2 k2 + 2 k3 + k4) of FP32 slopes, summed as exactly
as in FP64."""
import numpy as np
import pytest

from test_gpu_fixed_point import built, system  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [-2, 0, 2, 4, 6])
@pytest.mark.parametrize("nk,nrhs", [(7, 5), (40, 33)])
def test_update_is_as_exact_as_fp64(nk, nrhs, power, oracle, built):
    """One step, against the slopes of its own stages by dmd_func: with h a power of two the stages' inputs are exact sums rounded
    once, so the slopes are the same FP32 numbers. h is so long that the slopes grow from stage to stage and no two-float sum holds
    all of their bits. Bound: one rounding each of the product of h / 6, of the inner and of the outer sum, here and in the
    comparison: 2^-53 (2 |y| + 2 |result| + |h/6 sum|)."""
    from denmat_dynm_development_gb300.dmd import LindbladGPU
    s = system(oracle, nk, 2, 0.8, 5 * nk + nrhs)
    rng = np.random.default_rng(6)
    x = 1e-3 * (rng.standard_normal((nrhs, nk, 2, 2)) + 1j * rng.standard_normal((nrhs, nk, 2, 2)))
    x = 0.5 * (x + np.conj(np.swapaxes(x, 2, 3))) * s.f_dm[None, :, :, None] * s.f_dm[None, :, None, :]
    y = (oracle.y_of(s.dm0)[None] + x.reshape(nrhs, -1).view(np.float64)).reshape(-1)
    y = 0.5 * (y.reshape(-1, 2, 2, 2) + np.swapaxes(y.reshape(-1, 2, 2, 2), 1, 2) * np.array([1.0, -1.0])).reshape(-1)
    with LindbladGPU(nk=nk, nb_dm=2, bstart=0, bend=2, e_dm=s.e_dm, k1st=s.k1st, k2nd=s.k2nd, P1=s.P1, P2=s.P2,
                     prefac_eph=s.prefac_eph, picture=0, expt=0, precision="bf16x2", f_ref=s.f_dm, nrhs=nrhs) as g:
        k1 = g.func(0.0, y)
        h = 2.0 ** (power + np.ceil(np.log2(4.0 * np.abs(y).max() / np.abs(k1).max())))
        k2 = g.func(0.5 * h, y + 0.5 * h * k1)
        k3 = g.func(0.5 * h, y + 0.5 * h * k2)
        k4 = g.func(h, y + h * k3)
        g.set_state(0.0, y)
        g.rk4(h, 1)
        out = g.get_state()[1]
    for k in (k1, k2, k3, k4):
        np.testing.assert_array_equal(k, k.astype(np.float32))
    hi, lo = k1, np.zeros_like(k1)  # k1 + 2 k2 + 2 k3 + k4 by error-free sums
    for t in (2.0 * k2, 2.0 * k3, k4):
        z = hi + t
        b = z - hi
        hi, lo = z, lo + ((hi - (z - b)) + (t - b))
    ref = y + (h / 6.0 * hi + h / 6.0 * lo)
    assert (np.abs(out - ref) <= 2.0 ** -53 * (2.0 * np.abs(y) + 2.0 * np.abs(ref) + np.abs(h / 6.0 * hi))).all()
