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


def test_a_plan_whose_lists_could_not_be_rebuilt_says_so(cuda_lib):
    """Lists of more than 2^31 pairs are refused; the plan then has none, every call that
    needs them is refused too, and a later rebuild makes it whole again."""
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(0)
    pts, q = torch.rand(60_000, 3, generator=g, device="cuda"), torch.rand(60_000, generator=g, device="cuda")
    one = torch.ones_like(q)
    plan = _lib.Plan(pts, leaf_size=1, mac_theta=0.8, expansion_order=2)
    want = plan.matvec(q, one)
    with pytest.raises(_lib.EdfmmError, match="2\\^31"):
        plan.rebuild_lists(1e-6)
    for call in (lambda: plan.matvec(q, one), plan.p2p, lambda: plan.stage("m2l", 0), plan.export_lists,
                 lambda: plan.convert(torch.float64)):
        with pytest.raises(_lib.EdfmmError, match="rebuil"):
            call()
    plan.rebuild_lists(0.8)
    assert torch.equal(plan.matvec(q, one), want)
