"""The warm-start network's merged launches at small and ragged row counts:
the casts of weights and features (fewer and more feature values than weights),
the context of the column sums, and the head's three results (sum of dy, column
sums, masked rows), against the oracle.

The layers are identities, so a row's activations are its features plus the
context.  u = 2^-24: a chain of k FP32 adds is off by at most k u times the sum
of absolute values; a stored activation may round to the neighbouring BF16
value (2^-8 of it, 2^-7 after two layers).
"""
import numpy as np
import pytest
import torch

from oracle import pcn_ref as R

U = 2.0 ** -24


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 15, 17, 255, 257, 1023, 1025, 4099])
def test_small_row_counts(cuda_lib, n):
    from electrodrive_gb300.core.warm_start import PointCloudNet

    rng = np.random.default_rng(n)
    P = R.unpack(np.zeros(R.NPARAMS, np.float32))
    P["W1"] = np.eye(R.WIDTH, R.INPUTS)
    P["b1"] = rng.integers(-32, 64, R.WIDTH) / 64.0
    P["W2"] = np.eye(R.WIDTH)
    P["W3"] = np.eye(R.WIDTH)
    P["V2"] = rng.normal(0, 0.05, (R.WIDTH, R.WIDTH))
    P["b2"] = rng.normal(0, 0.5, R.WIDTH)
    P["w4"] = rng.normal(0, 0.2, R.WIDTH)
    P["b4"] = np.array([0.25])
    theta = R.pack(P).astype(np.float32)
    f = rng.normal(size=(n, R.INPUTS)).astype(np.float32)
    dy = rng.normal(size=n).astype(np.float32)

    net = PointCloudNet(theta)
    y = net.forward(torch.as_tensor(f, device="cuda")).cpu().numpy().astype(np.float64)
    g = R.unpack(net.backward(torch.as_tensor(dy, device="cuda")).cpu().numpy().astype(np.float64))
    yr, cache = R.forward(theta, f)
    dy64 = dy.astype(np.float64)
    gr = R.unpack(R.backward(theta, cache, dy64))
    Q = {k: np.asarray(v, np.float64) for k, v in R.unpack(theta).items()}
    h3, w4 = cache["h3"], Q["w4"]

    c2 = np.abs(Q["V2"]) @ np.abs(cache["g"]) + np.abs(Q["b2"])
    step = h3 * 2.0 ** -7 + c2 * (n + R.WIDTH) * 2 * U  # of a stored h3
    assert np.all(np.abs(y - yr) <= step @ np.abs(w4) + (h3 @ np.abs(w4) + 0.25) * R.WIDTH * U)
    assert abs(g["b4"][0] - gr["b4"][0]) <= (n / 256 + 14) * U * np.abs(dy64).sum()
    assert np.all(np.abs(g["w4"] - gr["w4"]) <= np.abs(dy64) @ (step + h3 * n * U))
    # rows of dz3 are equal but where the ReLU may turn over
    turned = (h3 <= step) * np.abs(dy64)[:, None] * np.abs(w4)
    rows = np.abs(dy64).sum() * np.abs(w4)
    assert np.all(np.abs(g["b3"] - gr["b3"]) <= (turned.sum(axis=0) + n * U * rows) * (1 + 2.0 ** -8))
