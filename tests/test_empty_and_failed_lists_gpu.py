"""Interaction lists without pairs, and a plan whose lists could not be rebuilt."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m", [1, 900])
def test_targets_of_a_plan_without_points(cuda_lib, dtype, m):
    """Every target node has a row, of no sources: near and far sums are 0."""
    from electrodrive_gb300 import _lib

    plan = _lib.Plan(torch.empty(0, 3, dtype=dtype, device="cuda"), expansion_order=4)
    tg = plan.targets(torch.rand(m, 3, device="cuda").to(dtype))
    assert tg.n_p2p_pairs == 0 and tg.n_m2l_pairs == 0
    near = tg.stage(_lib.EDFMM_TARGETS_P2P)
    tg.stage(_lib.EDFMM_TARGETS_M2L)
    tg.stage(_lib.EDFMM_TARGETS_L2L)
    far = tg.stage(_lib.EDFMM_TARGETS_L2P)
    assert near.shape == (m,) and not bool(near.any()) and not bool(far.any())
