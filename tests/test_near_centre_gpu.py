"""FP64 near field of geometries away from the origin: the split coordinates
have a centre on the axes where the points' extent is small against their
distance.  Against the oracle's P2P on the same tree; an FP64 term's error is
below 2^-51 and a sum of n terms adds at most n 2^-53, so (n + 16) 2^-51; two-float
terms are good to 2^-42."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

OFFSETS = [(0.0, 0.0, 0.0), (16.0, 0.0, 0.0), (16.0, 15.9, -17.0), (-1e4, 0.3, 0.0), (1e6, -3e5, 2e4), (1e8, 0.0, -1e8),
           (1e6, 1e6, 1e6)]


def _points(kind, n, off, rng):
    p = rng.random((n, 3))
    if kind == "plane":
        p[:, 0] = 0.5  # no extent on an axis
    elif kind == "pair":
        p[1::2] = p[: n - n % 2 : 2] + 2.0 ** -26 * rng.random((n // 2, 3))
    return p + np.asarray(off)


@pytest.mark.parametrize("off", OFFSETS)
@pytest.mark.parametrize("kind,n", [("cube", 1), ("cube", 2), ("cube", 700), ("plane", 600), ("pair", 400)])
@pytest.mark.parametrize("mode", ["native", "two_float"])
def test_near_sums_away_from_the_origin(cuda_lib, oracle, off, kind, n, mode):
    from electrodrive_gb300 import _lib

    rng = np.random.default_rng(n)
    pts, q = _points(kind, n, off, rng), rng.uniform(0.5, 1.5, n)
    t = oracle.build_tree(pts, 64, 32)
    lists = oracle.build_lists(t, 0.5)
    ref = oracle.p2p(t.points_tree, q[t.index_map], t.node_ranges, lists.p2p_pairs, float(np.finfo(np.float64).eps))
    plan = _lib.Plan(torch.as_tensor(pts).cuda(), mac_theta=0.5, expansion_order=6)
    plan.set_arithmetic(mode)
    plan.set_charges(torch.as_tensor(q).cuda())
    phi = plan.p2p().cpu().numpy()
    tol = (n + 16) * 2.0 ** -51 if mode == "native" else 2.0 ** -42
    assert np.all(np.abs(phi - ref) <= tol * np.abs(ref))


@pytest.mark.parametrize("mode", ["native", "two_float"])
def test_each_instance_of_a_batch_has_its_own_centre(cuda_lib, mode):
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(2)
    sizes = [1, 700, 33, 1500]
    pts = [torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) + torch.tensor(off, device="cuda")
           for n, off in zip(sizes, ([1e6, 0.0, 0.0], [0.0, 0.0, 0.0], [-50.0, 0.0, 1e4], [1e7, -1e7, 0.0]))]
    q = [torch.rand(n, generator=g, device="cuda", dtype=torch.float64) for n in sizes]
    both = _lib.Plan(torch.cat(pts), expansion_order=6, instance_offsets=np.cumsum([0] + sizes).tolist())
    both.set_arithmetic(mode)
    got = both.matvec(torch.cat(q), torch.ones(sum(sizes), device="cuda", dtype=torch.float64)).split(sizes)
    for p, c, v in zip(pts, q, got):
        one = _lib.Plan(p, expansion_order=6)
        one.set_arithmetic(mode)
        assert torch.equal(v, one.matvec(c, torch.ones_like(c)))


@pytest.mark.parametrize("mode", ["native", "two_float"])
def test_near_field_is_as_fast_away_from_the_origin(cuda_lib, mode):
    """Pairs closer than 2^-19 of the largest |coordinate| once went through the split and
    then through IEEE FP64: 6 (native) and 10 (two-float) times the time."""
    from electrodrive_gb300 import _lib

    g = torch.Generator(device="cuda").manual_seed(3)
    p = torch.randn(20011, 3, generator=g, device="cuda", dtype=torch.float64)
    p /= p.norm(dim=1, keepdim=True)
    us = []
    for x in (0.0, 1e6):
        plan = _lib.Plan(p + torch.tensor([x, 0.0, 0.0], device="cuda", dtype=torch.float64), expansion_order=6)
        plan.set_arithmetic(mode)
        plan.set_charges(torch.ones(20011, device="cuda", dtype=torch.float64))
        times = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            plan.p2p()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        us.append(sorted(times)[len(times) // 2])
    assert us[1] <= 3.0 * us[0]
