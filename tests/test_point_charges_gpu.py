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
