"""M2L reads the multipoles by columns of 32 nodes (FP32 and two-float; the FP64
kernel reads rows): trees whose node count is at, below and above a group."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points_with_nodes(target):
    """The first points of a random cloud whose tree has at least `target` nodes."""
    from electrodrive_gb300 import _lib

    pts = np.random.default_rng(3).random((4000, 3)).astype(np.float32)
    for n in range(target, 4000):
        p = torch.as_tensor(pts[:n]).cuda()
        if _lib.Plan(p, leaf_size=8, max_depth=32, mac_theta=0.5, expansion_order=2).info.n_nodes >= target:
            return p
    raise AssertionError("no such tree")


@pytest.mark.parametrize("mode", ["float32", "two_float"])
@pytest.mark.parametrize("nodes", [31, 32, 33, 65, 400])
def test_m2l_columns_at_group_edges(cuda_lib, mode, nodes):
    """Potentials of positive charges against the FP64 kernel.  FP32 (its own
    tree): both results are within the truncation bound of order 8 at theta
    0.5, 2 (1/3)^9 * 4/3, so within twice that of one another.  Two-float (the
    same tree): 2^-44 an operation over the about 64 of a coefficient's chain,
    times 16 for the growth of the coefficients."""
    from electrodrive_gb300 import _lib

    p = _points_with_nodes(nodes)
    q = torch.as_tensor(np.random.default_rng(nodes).random(p.shape[0]) + 0.5).cuda()
    one = torch.ones_like(q)

    def potential(points, two_float=False):
        plan = _lib.Plan(points, leaf_size=8, max_depth=32, mac_theta=0.5, expansion_order=8)
        if two_float:
            plan.set_arithmetic("two_float")
        assert plan.info.n_m2l_pairs > 0
        return plan.matvec(q.to(points.dtype), one.to(points.dtype)).double()

    want = potential(p.double())
    if mode == "float32":
        got, tol = potential(p), 2 * 2 * 3.0 ** -9 * 4 / 3
    else:
        got, tol = potential(p.double(), True), 64 * 16 * 2.0 ** -44
    assert float(((got - want).abs() / want).max()) <= tol
