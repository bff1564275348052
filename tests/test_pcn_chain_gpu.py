"""Training steps of the warm-start network with overlapped launches (outside a
capture) against the same kernels replayed from a graph (ordinary launches):
the same bits, so no kernel reads what its predecessor has not finished."""
import numpy as np
import pytest
import torch

from oracle import pcn_ref as R


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 300, 4097])
def test_overlapped_steps_match_a_graph(cuda_lib, n):
    from electrodrive_gb300.core.warm_start import PointCloudNet

    rng = np.random.default_rng(n)
    T = lambda x: torch.as_tensor(x, device="cuda")
    f = T(rng.normal(size=(n, R.INPUTS)).astype(np.float32))
    s, a = T(rng.uniform(0.5, 2.0, n)), T(rng.uniform(0.5, 1.5, n) / n)
    sigma = s * T(1 + 0.3 * rng.normal(size=n))
    theta = R.init(3)

    def gradients(net):
        y = net.forward(f)
        _, dy = net.loss(y, s, sigma, a)
        net.backward(dy)

    one, two = PointCloudNet(theta), PointCloudNet(theta)
    gradients(two)  # allocates the workspace
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        gradients(two)
    for _ in range(20):
        gradients(one)
        one.adam(1e-3)
    for _ in range(20):
        graph.replay()
        two.adam(1e-3)
    assert torch.equal(one.grads, two.grads)
    assert torch.equal(one.params, two.params)
