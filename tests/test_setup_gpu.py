"""Tree and interaction lists at the edges of the set-up's branches: nodes of
1024 points (a level of blocks per node or of chunks), lists that outgrow their
first room, rows sorted as bitmaps, in a warp, and (above 65,536 nodes) in a
block, and launch orders of more than one chunk of 1024."""
import numpy as np
import pytest
import torch

from test_tree_lists_gpu import _compare_tree, _plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,leaf,depth,theta,dtype", [
    ("cube", 1023, 64, 32, 0.5, np.float32),
    ("cube", 1024, 1024, 32, 0.5, np.float64),
    ("cube", 1025, 1024, 32, 0.5, np.float64),
    ("cube", 8 * 1024, 1, 32, 0.5, np.float32),    # every level down to single points
    ("cube", 9_000, 64, 3, 0.5, np.float64),       # leaves above leaf_size at max_depth
    ("cube", 30_011, 3, 32, 0.3, np.float32),      # lists and fronts that grow, rows above 512
    ("sphere", 80_021, 1, 32, 0.4, np.float32),    # above 65,536 nodes: no bitmaps, long rows in blocks
])
def test_tree_and_lists_match_oracle_at_branch_edges(cuda_lib, oracle, kind, n, leaf, depth, theta, dtype):
    rng = np.random.default_rng(n + leaf)
    pts = rng.random((n, 3)) if kind == "cube" else rng.normal(size=(n, 3))
    if kind == "sphere":
        pts /= np.linalg.norm(pts, axis=1, keepdims=True)
    pts = pts.astype(dtype)
    t = oracle.build_tree(pts, leaf, depth)
    lists = oracle.build_lists(t, theta)
    plan = _plan(pts, leaf, depth, theta, p=2)
    _compare_tree(plan.export_tree(), t)
    p2p, m2l = plan.export_lists()
    assert np.array_equal(p2p.cpu().numpy(), lists.p2p_pairs)
    assert np.array_equal(m2l.cpu().numpy(), lists.m2l_pairs)
    # the launch orders are permutations: every point's row is summed once
    ones = torch.ones(n, dtype=torch.as_tensor(pts).dtype, device="cuda")
    a = plan.matvec(ones, ones)
    b = _plan(pts, leaf, depth, theta, p=2).matvec(ones, ones)
    assert torch.equal(a, b) and bool((a > 0).all())
