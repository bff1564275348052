"""M2M and L2L with a block per node, every order and type (their terms are
dealt to the threads by tables of the order), and FP32 levels on either side of
the rule between a block and a thread per node."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("p", range(1, 9))
def test_m2m_gives_the_multipoles_of_the_root(cuda_lib, p, dtype):
    """Shifted multipoles of a deep tree against P2M at the root of a tree that
    is one leaf (the same box).  A level adds at most 81 terms of size 2^n q / n!
    an output, so four levels stay within 4 * 81 * 2^n u sum(q) / n!."""
    from electrodrive_gb300 import _lib

    rng = np.random.default_rng(p)
    pts = torch.as_tensor(rng.random((3000, 3)), dtype=dtype, device="cuda")
    q = torch.as_tensor(rng.random(3000), dtype=dtype, device="cuda")

    def root(leaf):
        plan = _lib.Plan(pts, leaf_size=leaf, max_depth=32, mac_theta=0.5, expansion_order=p)
        plan.set_charges(q)
        plan.stage("p2m")
        plan.stage("m2m")
        return plan.expansions()[0][0].to(torch.complex128).cpu()

    got, want = root(16), root(4096)
    u, c = torch.finfo(dtype).eps / 2, 0
    for n in range(p + 1):
        tol = 4 * 81 * 2.0 ** n * u * float(q.sum()) / math.factorial(n)
        assert float((got[c:c + n + 1] - want[c:c + n + 1]).abs().max()) <= tol, n
        c += n + 1


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,leaf,p", [(2500, 8, 2), (2500, 8, 5), (60_000, 6, 5), (120_000, 16, 3)])
def test_matvec_matches_oracle_at_the_level_rule(cuda_lib, oracle, n, leaf, p, dtype):
    """Against the oracle's FMM of the same order (FP64): rounding only, so 2^-24
    (2^-53) times the 10^4 operations of a result's longest sums, relative to the
    largest potential (charges of one sign)."""
    from electrodrive_gb300 import _lib

    rng = np.random.default_rng(n + p)
    pts = rng.random((n, 3)).astype(dtype)
    q = (rng.random(n) + 0.5).astype(dtype)
    t = oracle.build_tree(pts, leaf, 32)
    want = oracle.fmm_matvec(t, oracle.build_lists(t, 0.5), pts, q, np.ones_like(q), None, p=p, ke=1.0)
    plan = _lib.Plan(torch.as_tensor(pts).cuda(), leaf_size=leaf, max_depth=32, mac_theta=0.5, expansion_order=p)
    Q = torch.as_tensor(q).cuda()
    got = plan.matvec(Q, torch.ones_like(Q)).cpu().numpy()
    u = np.finfo(dtype).eps / 2
    assert np.abs(got - want).max() <= 1e4 * u * np.abs(want).max()
