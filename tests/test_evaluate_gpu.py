"""Potential and field in one pass: the sums of the two separate passes (another
split of the panels, so to rounding), tiles of 32 and 64 targets and their edges."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("m,n", [(1, 1), (31, 129), (33, 5), (64, 1000), (2433, 300), (10_000, 257)])
def test_potential_and_field_in_one_pass(cuda_lib, dtype, m, n):
    """Relative to the sum of the terms' sizes: each pass rounds a term about 16
    times and adds n of them."""
    from electrodrive_gb300.core.bem_near import (field_at_targets, potential_at_targets,
                                                  potential_field_at_targets)

    rng = np.random.default_rng(m + n)
    T = lambda x: torch.as_tensor(x, dtype=dtype, device="cuda")
    t, c = T(rng.normal(size=(m, 3))), T(rng.normal(size=(n, 3)))
    s, a = T(rng.normal(size=n)), T(rng.random(n) + 0.5)
    t[0] = c[0]  # a coincident pair: the clamped distance
    v, e = potential_field_at_targets(t, c, s, a, k_e=2.0)
    tol = 2 * (n + 16) * torch.finfo(dtype).eps
    size_v = potential_at_targets(t, c, s.abs(), a, k_e=2.0)
    assert bool(((v - potential_at_targets(t, c, s, a, k_e=2.0)).abs() <= tol * size_v).all())
    d = torch.cdist(t.double(), c.double()).clamp_min(1e-12)
    size_e = (2.0 * (s * a).abs().double() / d ** 2).sum(1, keepdim=True)
    w = field_at_targets(t, c, s, a, k_e=2.0)
    assert bool(((e.double() - w.double()).abs() <= tol * size_e)[1:].all())
    assert bool(torch.isfinite(e).all()) and torch.equal(torch.isfinite(w), torch.isfinite(e))
