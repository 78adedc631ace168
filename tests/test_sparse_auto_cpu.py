"""sparse="auto": the form that is the faster one for the operators' band count and fill."""
import pytest


@pytest.mark.parametrize("nb,fill,sparse", [(4, 0.44, False), (4, 0.31, True), (4, 0.09, True), (2, 0.44, False), (2, 0.31, False),
                                            (2, 0.27, True), (2, 0.09, True), (3, 0.35, True), (1, 0.45, False)])
def test_rule(nb, fill, sparse):
    from denmat_dynm_development_gb300.dmd import sparse_pays
    assert sparse_pays(nb, fill) is sparse
