"""M2L as a stage of its own, overlapped with its predecessor: instance flags and
interaction lists that the kernel just before it has written are the ones it uses."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_flags_written_just_before_the_stage(cuda_lib, dtype):
    """Rows of inactive instances keep their locals; the flags change in the stream
    between two stages, without a synchronisation."""
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(0)
    n = 1200
    pts = torch.rand(2 * n, 3, generator=g, device="cuda").to(dtype)
    q = torch.rand(2 * n, generator=g, device="cuda").to(dtype)
    plan = _lib.Plan(pts, leaf_size=16, expansion_order=4, instance_offsets=[0, n, 2 * n])
    both = [q, -2.0 * q]
    want = []
    for c in both:
        plan.set_charges(c)
        plan.stage("p2m"), plan.stage("m2m"), plan.stage("m2l", 0)
        want.append(plan.expansions()[1].clone())
    roots = (plan.export_tree()["node_levels"] == 0).nonzero().flatten()
    nodes = int(roots[1])  # first node of the second instance
    flags = torch.ones(2, device="cuda", dtype=torch.float64)
    new = torch.tensor([[1.0, 0.0], [0.0, 1.0]], device="cuda", dtype=torch.float64)
    plan.set_instance_mask(flags)
    for k in range(40):
        flags.fill_(1.0)
        plan.set_charges(both[0])
        plan.stage("p2m"), plan.stage("m2m"), plan.stage("m2l", 0)
        plan.set_charges(both[1])
        plan.stage("p2m"), plan.stage("m2m")
        flags.copy_(new[k % 2])
        plan.stage("m2l", 0)
        got = plan.expansions()[1]
        a, b = (1, 0) if k % 2 == 0 else (0, 1)  # which charges each instance's locals belong to
        assert torch.equal(got[:nodes], want[a][:nodes]) and torch.equal(got[nodes:], want[b][nodes:])


def test_lists_rebuilt_just_before_the_stage(cuda_lib):
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(1)
    pts, q = torch.rand(3000, 3, generator=g, device="cuda"), torch.rand(3000, generator=g, device="cuda")
    plan = _lib.Plan(pts, leaf_size=16, mac_theta=0.5, expansion_order=4)
    plan.set_charges(q)
    want = {}
    for theta in (0.4, 0.6):
        ref = _lib.Plan(pts, leaf_size=16, mac_theta=theta, expansion_order=4)
        ref.set_charges(q)
        ref.stage("p2m"), ref.stage("m2m"), ref.stage("m2l", 0)
        want[theta] = ref.expansions()[1]
    plan.stage("p2m"), plan.stage("m2m")
    for k in range(10):
        theta = (0.4, 0.6)[k % 2]
        plan.rebuild_lists(theta)
        plan.stage("m2l", 0)
        assert torch.equal(plan.expansions()[1], want[theta])
