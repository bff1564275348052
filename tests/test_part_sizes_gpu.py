"""Kernels whose blocks take a part of the rows chosen by the size: the Krylov
steps, the warm-start network and the point charges, at the edges of the parts."""
import numpy as np
import pytest
import torch

from oracle import pcn_ref as R
from test_warm_start import _blocks, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,restart", [
    (63, 8, 8), (65, 8, 10), (5120, 70, 80), (19_457, 12, 12), (38_784, 12, 12), (38_785, 12, 12), (310_273, 12, 30)])
def test_krylov_steps_at_part_edges(cuda_lib, n, steps, restart):
    """Diagonal operator with entries 1..1000: the basis is orthonormal and the
    rotations' residual is the true one, to the n-term bound of each inner
    product (n u, u = 2^-53) times the steps."""
    from electrodrive_gb300.core.bem_solver import _Krylov

    rng = np.random.default_rng(n)
    d = torch.as_tensor(np.logspace(0, 3, n), device="cuda")
    b = torch.as_tensor(rng.normal(size=n), device="cuda")
    kr = _Krylov(n, restart, torch.float64, torch.device("cuda"))
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    kr.start(b, torch.zeros_like(b), None)
    for j in range(steps):
        kr.arnoldi(j, d * kr.V[j], None)
    kr.update(steps, x)
    tol = steps * n * 2.0 ** -53
    V = kr.V[:steps + 1]
    assert float((V @ V.T - torch.eye(steps + 1, dtype=torch.float64, device="cuda")).abs().max()) <= tol
    beta = float(torch.linalg.vector_norm(b))
    res = float(torch.linalg.vector_norm(b - d * x))
    assert abs(res - float(kr.scal[4 + steps - 1])) <= 1000 * tol * beta  # |A| = 1000
    assert res < beta


@pytest.mark.parametrize("n", [5, 63, 65, 129, 1025, 20_011])
def test_network_at_part_edges(cuda_lib, n):
    """Against the oracle, which rounds to BF16 at the same places: within 1e-2
    (potential) and 3e-2 (gradients) and the whole effect of that rounding,
    which shows how far the quantity is conditioned."""
    from electrodrive_gb300.core.warm_start import PointCloudNet

    c, nr, a, b, s, sigma = _problem(n, 5)
    theta = R.init(7)
    theta[R.NPARAMS - 129:R.NPARAMS - 1] = np.random.default_rng(8).normal(0, 0.05, 128).astype(np.float32)
    net = PointCloudNet(theta)
    T = lambda v: torch.as_tensor(v, device="cuda")
    f = net.features(T(c), T(nr), T(a), T(b))
    fr = R.features(c, nr, a, b)
    assert np.abs(f.cpu().numpy() - fr).max() < 1e-5
    y = net.forward(f)
    yg = y.cpu().numpy()
    yr, cache = R.forward(theta, fr)
    yu, cache_u = R.forward(theta, fr, emulate_bf16=False)
    assert np.linalg.norm(yg - yr) <= 1e-2 * np.linalg.norm(yr) + np.linalg.norm(yr - yu)
    l, dy = net.loss(y, T(s), T(sigma), T(a))
    lr_, dyr = R.loss(yg.astype(np.float64), s, sigma, a)
    assert abs(float(l) - lr_) <= 1e-9 * lr_
    assert np.abs(dy.cpu().numpy() - dyr).max() <= 1e-6 * np.abs(dyr).max()
    g = net.backward(dy).cpu().numpy()
    gr = R.backward(theta, cache, dyr)
    gu = R.backward(theta, cache_u, dyr, emulate_bf16=False)
    for name, (lo, hi) in _blocks().items():
        err = np.linalg.norm(g[lo:hi] - gr[lo:hi])
        assert err <= 3e-2 * np.linalg.norm(gr[lo:hi]) + np.linalg.norm(gr[lo:hi] - gu[lo:hi]), name


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n,k", [(1, 1), (257, 32), (1000, 33), (5, 70)])
def test_point_charges_past_one_parameter_block(cuda_lib, dtype, n, k):
    """Potential and field against torch in FP64, to (k + 8) roundings of the
    sum of the terms' sizes."""
    from electrodrive_gb300.core.bem_near import add_point_charges

    rng = np.random.default_rng(n + k)
    pts = torch.as_tensor(rng.normal(size=(n, 3)), dtype=dtype, device="cuda")
    q, r = rng.normal(size=k), 3.0 + rng.random((k, 3))
    V = torch.ones(n, dtype=dtype, device="cuda")
    E = torch.ones(n, 3, dtype=dtype, device="cuda")
    add_point_charges(pts, list(zip(q, r)), V=V, E=E, k_e=2.0)
    d = pts.double()[:, None, :] - torch.as_tensor(r, device="cuda")[None]
    dist = d.norm(dim=-1)
    tv = 2.0 * torch.as_tensor(q, device="cuda") / dist
    te = (tv / dist ** 2)[..., None] * d
    # the difference of a point and a charge carries one rounding of the point's size
    eps = torch.finfo(dtype).eps * (k + 8) * (1.0 + float((6.0 / dist).max()))
    assert bool(((V.double() - 1 - tv.sum(1)).abs() <= eps * (1 + tv.abs().sum(1))).all())
    assert bool(((E.double() - 1 - te.sum(1)).abs() <= 3 * eps * (1 + te.abs().sum(1))).all())
