"""Near field (P2P) where its packing can go wrong: leaves of 1 to over 64
points (every number of targets per lane), rows shorter and longer than a
32-entry batch and a source chunk, few leaves (four warps per leaf) and many,
pairs too close for the exact coordinate split, geometries far from the origin
and at extreme scales; in FP32, FP64 and two-float arithmetic, against the
oracle's P2P on the same tree.  And the far field with levels on both sides of
the warp-per-node limit.

Tolerances (charges positive): an FP64 term's error is below 2^-51 and a sum of
k terms adds at most k 2^-53, so (k + 16) 2^-51 per target with k the longest
row; two-float terms are good to 2^-42; FP32 2^-21 for a term plus chains of at
most 64 + k / 64 additions of 2^-24."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    p = rng.random((n, 3))
    if kind == "surface":
        p = p - 0.5
        p /= np.linalg.norm(p, axis=1, keepdims=True)
    elif kind == "offset":
        p = p + np.array([4000.0, 0.0, -17.0])
    elif kind == "close":
        p[1::2] = p[: n - n % 2 : 2] + 1e-9 * rng.random((n // 2, 3))
        p[5] = p[3]
    elif kind == "tiny":
        p = p * 1e-12
    elif kind == "extreme":
        p = p * 1e120
    return p


@pytest.mark.parametrize("kind,n,leaf", [("cube", 1, 64), ("cube", 2, 64), ("cube", 33, 1), ("cube", 500, 3),
                                         ("cube", 700, 64), ("cube", 1200, 200), ("surface", 3000, 64),
                                         ("surface", 20000, 32), ("cube", 9000, 64), ("close", 900, 64),
                                         ("offset", 2000, 64), ("tiny", 800, 64), ("extreme", 800, 64)])
@pytest.mark.parametrize("mode", ["float32", "native", "two_float"])
def test_p2p_packing(cuda_lib, oracle, kind, n, leaf, mode):
    from electrodrive_gb300 import _lib

    if mode != "native" and kind in ("close", "tiny", "extreme"):
        pytest.skip("below or beyond FP32's range")
    npdt = np.float32 if mode == "float32" else np.float64
    rng = np.random.default_rng(n + leaf)
    pts = _points(kind, n, rng).astype(npdt)
    q = rng.uniform(0.5, 1.5, n).astype(npdt)
    t = oracle.build_tree(pts, leaf, 32)
    lists = oracle.build_lists(t, 0.5)
    ref = oracle.p2p(t.points_tree, q[t.index_map], t.node_ranges, lists.p2p_pairs, float(np.finfo(npdt).eps))
    plan = _lib.Plan(torch.as_tensor(pts).cuda(), leaf_size=leaf, mac_theta=0.5, expansion_order=6)
    if mode == "two_float":
        plan.set_arithmetic("two_float")
    plan.set_charges(torch.as_tensor(q).cuda())
    phi = plan.p2p().cpu().numpy().astype(np.float64)
    k = n
    tol = {"float32": 2.0 ** -21 + (64 + k / 64) * 2.0 ** -24, "native": (k + 16) * 2.0 ** -51,
           "two_float": 2.0 ** -42}[mode]
    assert np.all(np.abs(phi - ref) <= tol * np.abs(ref) + 1e-300)


def test_native_after_two_float_has_the_current_charges(cuda_lib):
    """Leaving two-float mode rebuilds the split points with the charges that are set."""
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(1)
    pts = torch.rand(4000, 3, generator=g, device="cuda", dtype=torch.float64)
    q = torch.rand(4000, generator=g, device="cuda", dtype=torch.float64)
    a, b = _lib.Plan(pts, expansion_order=6), _lib.Plan(pts, expansion_order=6)
    a.set_charges(2.0 * q)
    a.set_arithmetic("two_float")
    a.set_charges(q)
    a.set_arithmetic("native")
    b.set_charges(q)
    assert torch.equal(a.p2p(), b.p2p())


@pytest.mark.parametrize("p", [6, 8])
def test_levels_on_both_sides_of_the_warp_limit(cuda_lib, p):
    """300,000 points: levels of 8 to over 6,144 nodes, FP32 against FP64 at the same order."""
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(p)
    pts = torch.rand(300000, 3, generator=g, device="cuda")
    q = torch.rand(300000, generator=g, device="cuda")
    one = torch.ones_like(q)
    v = _lib.Plan(pts, expansion_order=p).matvec(q, one)
    ref = _lib.Plan(pts.double(), expansion_order=p).matvec(q.double(), one.double())
    assert float(torch.linalg.norm(v - ref) / torch.linalg.norm(ref)) < 2e-6
