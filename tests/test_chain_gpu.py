"""Far-field kernels that start before their predecessors end: repeated matvecs
with changing charges, on the default and on another stream, back to back and
captured, must equal the first one of the same charges bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,leaf", [(1, 64), (70, 64), (700, 16), (2500, 64), (30_000, 8)])
def test_back_to_back_matvecs(cuda_lib, dtype, n, leaf):
    from electrodrive_gb300._lib import Plan

    rng = np.random.default_rng(n)
    pts = torch.as_tensor(rng.random((n, 3)), dtype=dtype, device="cuda")
    plan = Plan(pts, leaf_size=leaf, expansion_order=8)
    one = torch.ones(n, dtype=dtype, device="cuda")
    qs = [torch.as_tensor(rng.normal(size=n), dtype=dtype, device="cuda") for _ in range(4)]
    want = []
    for q in qs:
        want.append(plan.matvec(q, one).clone())
        torch.cuda.synchronize()
    got = [torch.empty_like(q) for q in qs for _ in range(25)]
    for r in range(25):
        for i, q in enumerate(qs):
            plan.matvec(q, one, out=got[4 * r + i])
    torch.cuda.synchronize()
    assert all(torch.equal(g, want[i % 4]) for i, g in enumerate(got))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        out = [plan.matvec(q, one) for q in qs]
        graph = torch.cuda.CUDAGraph()
        res = torch.empty_like(one)
        with torch.cuda.graph(graph, stream=side):
            plan.matvec(qs[0], one, out=res)
        graph.replay()
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(out, want)) and torch.equal(res, want[0])
