"""When the dense operator takes its table of 1 / r, and what was captured before."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operator(n=400):
    from electrodrive_gb300.core.operators import DenseOperator

    rng = np.random.default_rng(n)
    c, a = torch.as_tensor(rng.random((n, 3))), torch.as_tensor(rng.uniform(0.5, 1.5, n) / n)
    return DenseOperator(c, a, torch.full((n,), 50.0 * n), k_e=1.0), torch.as_tensor(rng.normal(size=n), device="cuda")


def test_graphs_captured_before_the_table_are_not_replayed(cuda_lib):
    """The coordinates are destroyed once the table holds all that the operator needs: a
    replay of an older capture would read them."""
    from electrodrive_gb300.core.bem_solver import gmres_restart

    op, b = _operator()
    solve = lambda: gmres_restart(op, b, restart=4, tol=1e-12, maxiter=200, use_graph=True)
    for _ in range(3):
        x, info = solve()
        assert info["code"] == 0 and info["iters"] > 8
    assert op.tabulate()
    op.c.zero_()
    for _ in range(3):
        y, info = solve()
        assert info["code"] == 0
        assert float((y - x).norm()) <= 1e-10 * float(x.norm())
