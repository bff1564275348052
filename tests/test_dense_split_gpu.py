"""The dense kernels at the edges of their tiles and of the exact coordinate
split: remainders of the 64- and 128-target tiles and of the source tiles,
one to eight blocks per cluster, geometries far from the origin, at extreme
scales, with coincident and nearly coincident points and with non-finite
coordinates.

Tolerance: a term's error is below 2^-51 relative (the oracle's 2^-51 too) and
a sum of n positive terms adds at most n 2^-53, so (n + 16) 2^-51 per panel in
FP64; FP32 the same with 2^-22 and tile-wise sums (at most 256 + n / 256 terms
in a chain)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _geometry(kind, n, rng):
    c = rng.random((n, 3))
    if kind == "offset":
        c = c + np.array([1000.0, -300.0, 0.0])
    elif kind == "tiny":
        c = c * 1e-9  # r^2 below 1e-17; nothing reaches the 1e-24 clamp
    elif kind == "huge":
        c = c * 1e90
    elif kind == "extreme":
        c = c * 1e140  # beyond the split's range of scales
    elif kind == "close":  # pairs down to 1e-9 apart, and coincident ones
        c[1::2] = c[:n - n % 2:2] + rng.choice([0.0, 1e-9, 1e-7, 1e-5], (n // 2, 1)) * rng.random((n // 2, 3))
    return c


@pytest.mark.parametrize("kind", ["cube", "offset", "tiny", "huge", "extreme", "close"])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 127, 130, 515, 2049])
@pytest.mark.parametrize("dt", [torch.float64, torch.float32])
def test_dense_tile_edges(cuda_lib, oracle, kind, n, dt):
    from electrodrive_gb300 import _lib

    if dt == torch.float32 and kind in ("huge", "extreme"):
        pytest.skip("beyond FP32")
    rng = np.random.default_rng(n)
    npdt = np.float64 if dt == torch.float64 else np.float32
    c = _geometry(kind, n, rng).astype(npdt)
    s, a = rng.uniform(0.5, 1.5, n).astype(npdt), rng.uniform(0.5, 1.5, n).astype(npdt)
    ref = oracle.dense_matvec(c, s, a, None, ke=1.0)
    T = lambda x: torch.as_tensor(x, device="cuda")
    v = _lib.dense_matvec(T(c), T(s), T(a), None, k_e=1.0).cpu().numpy().astype(np.float64)
    tol = (n + 16) * 2.0 ** -51 if dt == torch.float64 else (256 + n / 256 + 16) * 2.0 ** -22
    assert np.all(np.abs(v - ref) <= tol * np.abs(ref))


@pytest.mark.parametrize("m,n", [(1, 1), (63, 130), (64, 2049), (129, 5120), (3000, 65), (80000, 3)])
def test_targets_tile_edges(cuda_lib, m, n):
    from electrodrive_gb300.core.bem_near import field_at_targets, potential_at_targets

    g = torch.Generator(device="cuda").manual_seed(m + n)
    c, t = (torch.rand(k, 3, generator=g, device="cuda", dtype=torch.float64) for k in (n, m))
    t = t + torch.tensor([1.5, 0.0, 0.0], device="cuda", dtype=torch.float64)
    s, a = (0.5 + torch.rand(n, generator=g, device="cuda", dtype=torch.float64) for _ in range(2))
    d = t[:, None, :] - c[None, :, :]
    r2 = (d * d).sum(2)
    V = (s * a / r2.sqrt()).sum(1)
    E = ((s * a / (r2 * r2.sqrt()))[:, :, None] * d).sum(1)
    Vg = potential_at_targets(t, c, s, a, k_e=1.0)
    Eg = field_at_targets(t, c, s, a, k_e=1.0)
    assert bool(((Vg - V).abs() <= (n + 16) * 2.0 ** -51 * V).all())
    scale = (s * a / r2).sum(1, keepdim=True)  # sum of the terms' magnitudes
    assert bool(((Eg - E).abs() <= (n + 32) * 2.0 ** -51 * scale).all())


def test_dense_nonfinite_coordinates(cuda_lib):
    """A source at infinity adds nothing to the others; its own row and a NaN
    coordinate follow the formula r^2 = max(r^2, 1e-24) as device arithmetic
    evaluates it, and no row is left non-finite."""
    from electrodrive_gb300 import _lib

    n = 300
    g = torch.Generator(device="cuda").manual_seed(0)
    c = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64)
    c[17, 1] = float("inf")
    s = a = torch.ones(n, device="cuda", dtype=torch.float64)
    v = _lib.dense_matvec(c, s, a, None, k_e=1.0)
    keep = torch.arange(n, device="cuda") != 17
    r = torch.cdist(c[keep], c[keep], compute_mode="donot_use_mm_for_euclid_dist")
    r.fill_diagonal_(float("inf"))
    ref = (1.0 / r).sum(1)
    assert bool(torch.isfinite(v).all())
    assert bool(((v[keep] - ref).abs() <= (n + 16) * 2.0 ** -51 * ref).all())
