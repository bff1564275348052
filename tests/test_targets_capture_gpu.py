"""The first evaluation of a set of targets may lie inside a stream capture: it allocates nothing."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, 2, 4])  # both fields, near only, far only
@pytest.mark.parametrize("m", [1, 700])
def test_first_evaluation_inside_a_capture(cuda_lib, m, flags):
    from electrodrive_gb300._lib import Plan

    g = torch.Generator(device="cuda").manual_seed(m)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=torch.float64)
    c, t, s, a = rand(5000, 3), rand(m, 3) * 1.4, rand(5000), rand(5000)
    plan = Plan(c, expansion_order=6)
    ref = plan.targets(t).potential(s, a, flags=flags)  # loads the kernels
    tg = plan.targets(t)
    out = torch.zeros(m, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tg.potential(s, a, out=out, flags=flags)
    graph.replay()
    assert torch.equal(out, ref)
