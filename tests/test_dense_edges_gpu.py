"""The dense kernels where a tile is padded and where a charge is not finite.

FP32 tolerance: a term rounds about 16 times and a target adds n of them, so
(n + 32) 2^-23 of the sum of the terms' sizes."""
import numpy as np
import pytest
import torch

from electrodrive_gb300.utils.config import K_E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 65])
@pytest.mark.parametrize("n", [1, 2, 129, 256, 257, 1025])
def test_fp32_field_at_the_origin(cuda_lib, m, n):
    """Targets at and next to the coordinate origin, odd and even numbers of panels, with
    the physical constant (K_E / r^3 overflows FP32 below r = 3e-10)."""
    from electrodrive_gb300.core.bem_near import field_at_targets, potential_field_at_targets

    rng = np.random.default_rng(n)
    T = lambda x: torch.as_tensor(x, dtype=torch.float32, device="cuda")
    p = rng.normal(size=(n, 3)) + 0.3
    c = T(p / np.linalg.norm(p, axis=1, keepdims=True))
    s, a = T(1e-11 * rng.uniform(0.5, 1.5, n)), T(rng.uniform(0.5, 1.5, n))
    t = torch.zeros(m, 3, device="cuda")
    t[1:] = T(10.0 ** rng.uniform(-14, -6, (m - 1, 1)) * rng.normal(size=(m - 1, 3)))
    d = t.double()[:, None] - c.double()[None]
    term = (K_E * (s.double() * a.double()) / d.norm(dim=2) ** 3)[..., None] * d
    tol = (n + 32) * 2.0 ** -23 * term.norm(dim=2).sum(1, keepdim=True)
    for e in (field_at_targets(t, c, s, a), potential_field_at_targets(t, c, s, a)[1]):
        assert bool(((e.double() - term.sum(1)).abs() <= tol).all())


@pytest.mark.parametrize("kernel", ["float32", "float64", "table"])
@pytest.mark.parametrize("n,i", [(1, 0), (2, 1), (129, 128), (300, 5), (2049, 700)])
def test_a_charge_that_is_not_finite_stays_out_of_its_own_row(cuda_lib, kernel, n, i):
    """The sum over j != i without a self term: row i is that of the other panels, and
    every other row is not finite, which the operator returns as 0."""
    from electrodrive_gb300 import _lib
    from electrodrive_gb300.core.operators import DenseOperator

    rng = np.random.default_rng(n)
    dt = torch.float32 if kernel == "float32" else torch.float64
    T = lambda x: torch.as_tensor(x, dtype=dt, device="cuda")
    c, s, a = T(rng.random((n, 3))), T(rng.uniform(0.5, 1.5, n)), T(rng.uniform(0.5, 1.5, n))
    s[i] = float("inf")
    if kernel == "table":
        op = DenseOperator(c, a, None, k_e=1.0)
        assert op.tabulate()
        v = op(s)
    else:
        v = _lib.dense_matvec(c, s, a, None, k_e=1.0)
    keep = torch.arange(n, device="cuda") != i
    term = (s * a).double()[keep] / (c.double()[keep] - c.double()[i]).norm(dim=1)
    assert abs(float(v[i]) - float(term.sum())) <= (n + 32) * torch.finfo(dt).eps * float(term.sum())
    assert not bool(v[keep].any())
