"""Point charges: the potential is one FP64 sum rounded once however many
charges there are, positions have three coordinates, and the field stays a
torch expression of positions and points that ask for gradients."""
import numpy as np
import pytest
import torch

from electrodrive_gb300.utils.config import K_E

pytestmark = pytest.mark.gpu


def _cancelling(rng, k):
    """k charges whose first half is cancelled by the second, a little further out."""
    u = rng.normal(size=(k // 2, 3))
    r = 3.0 * u / np.linalg.norm(u, axis=1, keepdims=True)
    q = rng.uniform(0.5, 1.5, k // 2)
    return list(zip(np.concatenate([q, -q]).tolist(), np.concatenate([r, 1.001 * r]).tolist()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,k", [(1, 32), (300, 34), (129, 64), (1000, 200)])
def test_potential_of_many_charges_is_rounded_once(cuda_lib, dtype, n, k):
    """One rounding of the sum in the points' type, and (k + 16) FP64 roundings of the
    terms; the add form rounds twice more (the sum, and the sum with V)."""
    from electrodrive_gb300.core.bem_near import add_point_charges, point_charge_potential

    rng = np.random.default_rng(n + k)
    pts = torch.as_tensor(rng.normal(size=(n, 3)), dtype=dtype, device="cuda")
    ch = _cancelling(rng, k)
    q, r = (torch.as_tensor([c[i] for c in ch], dtype=torch.float64, device="cuda") for i in (0, 1))
    t = K_E * q / (pts.double()[:, None] - r[None]).norm(dim=2)
    ref, size = t.sum(1), (k + 16) * 2.0 ** -52 * t.abs().sum(1)
    u = torch.finfo(dtype).eps / 2
    v = point_charge_potential(pts, ch)
    assert bool(((v.double() - ref).abs() <= u * ref.abs() + size).all())
    w = torch.full((n,), 3.0, dtype=dtype, device="cuda")
    add_point_charges(pts, ch, V=w)
    assert bool(((w.double() - 3.0 - ref).abs() <= u * (2 * ref.abs() + 3.0) + size + 3.0 * 2.0 ** -52).all())


@pytest.mark.parametrize("charges", [[(1.0, (0.0, 2.0))], [(1.0, (0.0, 2.0, 0.0, 1.0))], [(1.0, ())],
                                     [(1.0, (0.0, 0.0, 2.0)), (1.0, (0.0, 2.0))]])
def test_positions_without_three_coordinates_are_refused(cuda_lib, charges):
    from electrodrive_gb300.core.bem import BEMSolution
    from electrodrive_gb300.core.bem_near import add_point_charges, point_charge_potential

    pts = torch.rand(5, 3, device="cuda", dtype=torch.float64)
    with pytest.raises(ValueError):
        point_charge_potential(pts, charges)
    with pytest.raises(ValueError):
        add_point_charges(pts, charges, V=torch.zeros(5, device="cuda", dtype=torch.float64))
    one = torch.ones(1, device="cuda", dtype=torch.float64)
    sol = BEMSolution(centroids=torch.zeros(1, 3, device="cuda", dtype=torch.float64), areas=one, sigma=one,
                      charges=charges)
    with pytest.raises(ValueError):
        sol.eval_V_E_batched(pts)


def _field(points, charges):
    """K_E sum q (x - r) / |x - r|^3 in torch."""
    d = points[:, None] - torch.stack([torch.as_tensor(r, dtype=points.dtype, device=points.device)
                                       for _, r in charges])[None]
    q = torch.tensor([float(c) for c, _ in charges], dtype=points.dtype, device=points.device)
    return (K_E * q[:, None] * d / d.norm(dim=2, keepdim=True) ** 3).sum(1)


def _case():
    rng = np.random.default_rng(3)
    pts = torch.as_tensor(rng.normal(size=(7, 3)), device="cuda")
    pos = [torch.as_tensor(2.0 + rng.random(3), device="cuda") for _ in range(2)]
    return pts, [(0.5, pos[0]), (-1.5, pos[1])]


def _close(a, b):
    return float((a - b).norm()) <= 1e-13 * float(b.norm())


def test_field_has_derivatives_to_points_and_positions(cuda_lib):
    from electrodrive_gb300.core.bem_near import point_charge_field

    pts, ch = _case()
    assert _close(point_charge_field(pts, ch), _field(pts, ch))
    for leaf in (pts, ch[0][1]):
        leaf.requires_grad_(True)
        e = point_charge_field(pts, ch)
        assert e.requires_grad
        got, = torch.autograd.grad(e.square().sum(), leaf)
        assert _close(got, torch.autograd.grad(_field(pts, ch).square().sum(), leaf)[0])
        leaf.requires_grad_(False)


def test_field_under_vmap_and_forward_mode(cuda_lib):
    from electrodrive_gb300.core.bem_near import point_charge_field

    pts, ch = _case()
    batch = torch.stack([pts, 2.0 * pts])
    got = torch.func.vmap(lambda p: point_charge_field(p, ch))(batch)
    assert _close(got[0], _field(pts, ch)) and _close(got[1], _field(2.0 * pts, ch))
    t = torch.ones_like(pts)
    got = torch.func.jvp(lambda p: point_charge_field(p, ch), (pts,), (t,))[1]
    assert _close(got, torch.func.jvp(lambda p: _field(p, ch), (pts,), (t,))[1])


def test_evaluation_keeps_the_charges_part_of_the_fields_gradient(cuda_lib):
    """eval_V_E_batched: the induced part has no graph, the point charges' part has one."""
    from electrodrive_gb300.core.bem import BEMSolution

    pts, ch = _case()
    one = torch.ones(1, device="cuda", dtype=torch.float64)
    sol = BEMSolution(centroids=torch.zeros(1, 3, device="cuda", dtype=torch.float64), areas=one, sigma=one, charges=ch)
    plain = sol.eval_V_E_batched(pts)
    for leaf in (pts, ch[1][1]):
        leaf.requires_grad_(True)
        v, e = sol.eval_V_E_batched(pts)
        got, = torch.autograd.grad(e.sum(), leaf)
        assert _close(got, torch.autograd.grad(_field(pts, ch).sum(), leaf)[0])
        leaf.requires_grad_(False)
        assert _close(v.detach(), plain[0]) and _close(e.detach(), plain[1])
    assert not plain[1].requires_grad
