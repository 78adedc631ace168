"""The nb = 2 gradient with the stages that fit (dmd_adjoint_rk4): where the memory does not hold 32 stages' vectors the gradient
passes take fewer, down to one."""
import os

import numpy as np
import pytest

from conftest import GOLDEN
from test_adjoint import _gpu, built, rel  # noqa: F401  (built: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stages", [20, 7, 1, 0])
def test_fewer_stages_where_memory_is_short(stages, oracle, built, monkeypatch):
    """11 steps, 44 stages. The outer products are added in the same order however many stages a pass takes, in double-floats; the
    backward chain's atomic sums differ in their last bits: 1e-11 of the gradient. No room for a single stage is an error."""
    from denmat_dynm_development_gb300.dmd import DMDError
    s = oracle.load(os.path.join(GOLDEN, "nb2_eimp_B"))
    y0, steps, w = oracle.y_of(s.dm0), np.array([5, 11]), np.array([0.5, 1.0])
    args = (s.t0, y0, 2.0 * oracle.fs, 11, steps, w)
    with _gpu(s, adjoint=True, precision="f64x") as g:
        _, dP, dy = g.adjoint_rk4(*args, bstart=s.nv_dm, want_dy0=True)
        monkeypatch.setenv("DMD_ADJ_ROOM", str(stages * 4 * s.nk * 4 * 16))
        if stages == 0:
            with pytest.raises(DMDError):
                g.adjoint_rk4(*args, bstart=s.nv_dm, want_dy0=True)
            return
        _, dP2, dy2 = g.adjoint_rk4(*args, bstart=s.nv_dm, want_dy0=True)
    assert rel(dP2, dP) < 1e-11 and rel(dy2, dy) < 1e-11
