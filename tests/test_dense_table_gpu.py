"""The tabulated FP64 operator against the one from the coordinates (another
order of the sum): tiles of 64 rows, clusters of eight blocks, close pairs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,extent", [(1, 1.0), (2, 1.0), (63, 1e-6), (64, 1.0), (65, 1e8), (511, 1.0), (513, 1.0), (3001, 1.0)])
def test_table_matches_the_operator(cuda_lib, n, extent):
    """n additions and about four roundings a term: (n + 4) 2^-52 of the sum of
    the terms' sizes on either side."""
    from electrodrive_gb300.core.operators import DenseOperator

    rng = np.random.default_rng(n)
    c = rng.normal(size=(n, 3)) * extent
    if n > 60:
        c[5] = c[4]                                   # coincident: the clamped distance
        c[9] = c[8] + np.array([1e-9, 0, 0]) * extent  # closer than the split resolves
    a = rng.random(n) + 0.5
    s = torch.as_tensor(rng.normal(size=n), device="cuda")
    op = DenseOperator(torch.as_tensor(c), torch.as_tensor(a), torch.as_tensor(rng.random(n)), k_e=2.0)
    want, size = op(s).clone(), op(s.abs()).clone()
    assert op.tabulate() and op.tabulate()
    got = op(s)
    assert bool(((got - want).abs() <= 2 * (n + 4) * 2.0 ** -52 * size).all())


def test_table_is_declined(cuda_lib):
    from electrodrive_gb300.core.operators import DenseOperator

    c, a = torch.rand(300, 3), torch.rand(300)
    assert not DenseOperator(c, a, dtype=torch.float32).tabulate()
    assert not DenseOperator(c, a).tabulate(max_bytes=300 * 300 * 8)  # rows are padded to 64
