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


def test_memory_the_allocator_holds_free_counts_as_free(cuda_lib, monkeypatch):
    op, _ = _operator()
    held = torch.empty(2 << 30, dtype=torch.uint8, device="cuda")
    del held  # reserved by the caching allocator, not by the program
    assert torch.cuda.memory_reserved() - torch.cuda.memory_allocated() >= 2 << 30
    total = torch.cuda.mem_get_info()[1]
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (16 << 20, total))
    assert op.tabulate()
    torch.cuda.empty_cache()


def test_a_device_short_of_memory_declines_the_table(cuda_lib, monkeypatch):
    op, s = _operator()
    torch.cuda.empty_cache()
    total = torch.cuda.mem_get_info()[1]
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda *a: (16 << 20, total))
    assert not op.tabulate() and op.table is None
    assert bool(torch.isfinite(op(s)).all())


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


@pytest.mark.parametrize("operator,fp64,dense_table", [("dense", True, True), ("dense", False, False), ("fmm", True, False)])
def test_a_solve_says_whether_it_used_the_table(cuda_lib, operator, fp64, dense_table):
    from electrodrive_gb300.core.bem import bem_solve
    from electrodrive_gb300.core.bem_mesh import icosphere
    from electrodrive_gb300.utils.config import BEMConfig

    spec = dict(conductors=[dict(type="sphere", radius=1.0, center=[0.0, 0.0, 0.0], potential=0.0)],
                charges=[dict(type="point", q=1.0, pos=[0.0, 0.0, 2.0])])
    res = bem_solve(spec, BEMConfig(fp64=fp64, gmres_tol=1e-6), mesh=icosphere(2), operator=operator)
    assert res["mesh_stats"]["dense_table"] is dense_table
