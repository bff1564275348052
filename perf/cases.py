"""Performance cases: what users of electrodrive_gb300 run, through its public entry points.

Each case is a dict of plain values; ``prepare`` makes what a program holds
before the call (inputs from the seed, plans and operators), ``run`` is one
pass through the public API, ``work`` the bytes and operations the pass
cannot do without and ``exact`` the same outputs in 64 bits from plain torch.

Kinds and the sizes they stand for (``draw`` spreads over the same ranges):

``fmm``       ``bem_matvec_gpu(backend="external", matvec_impl=LaplaceFmm3D.matvec)``:
              the operator application, 500 to 1,048,576 points in the unit cube (FP32)
              or on a sphere (FP64), expansion orders 6 to 8, leaf size 64
``operator``  the operators of the solves on a torus mesh (near-pair correction
              included): the FP32 inner operator and the FP64 stopping-test operator in
              two-float arithmetic, 5,000 to 200,000 panels
``dense``     ``bem_matvec_gpu`` below the FMM threshold of 20,000 panels
``evaluate``  ``BEMSolution.eval_V_E_batched``: potential and field of a solution at
              50 to 20,000 points
``apply``     ``create_bem_fmm_backend(...).apply``: tree, lists and one matvec per call
``batch``     the FP32 operator of many sphere dimers solved together
``solve``     ``bem_solve`` of a grounded sphere with a point charge, dense FP64 GMRES
``train``     one training step of the warm-start network (forward, loss, backward, Adam)

The mixed-precision solves have no case of their own: their FP64 result is
shaped by the rounding of FP32 inner iterations to about their 1e-6 residual,
so it cannot be compared; nearly all of their time is the operators above.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from electrodrive_gb300.core.batch import BatchSystem, dimer_case_device
from electrodrive_gb300.core.bem import BEMSolution, bem_solve, build_operator
from electrodrive_gb300.core.bem_kernel import bem_matvec_gpu
from electrodrive_gb300.core.bem_mesh import generate_mesh, icosphere
from electrodrive_gb300.core.bem_near import NearCorrection
from electrodrive_gb300.core.mesh_device import torus_mesh_device
from electrodrive_gb300.core.warm_start import PointCloudNet
from electrodrive_gb300.fmm3d import FmmConfig, create_bem_fmm_backend, make_laplace_fmm_backend
from electrodrive_gb300.utils.config import BEMConfig

K_E = 1.0 / (4.0 * math.pi * 8.854187817e-12)
DTYPES = {"float32": torch.float32, "float64": torch.float64}
ALL_PAIRS_MAX = 250_000  # above this the all-pairs sum in 64 bits takes over 20 s


def listed():
    return [
        # a small geometry: latency of the call and of its launches
        {"name": "fmm_cube_f32_2k", "kind": "fmm", "points": "cube", "n": 2003, "dtype": "float32", "order": 8},
        # the matvec benchmark's own size
        {"name": "fmm_cube_f32_1m", "kind": "fmm", "points": "cube", "n": 1048576, "dtype": "float32", "order": 8},
        # a double-precision operator on a surface, just above the dense threshold
        {"name": "fmm_sphere_f64_20k", "kind": "fmm", "points": "sphere", "n": 20011, "dtype": "float64", "order": 8},
        # the inner operator of the 200,000-panel torus solve (one application per inner iteration)
        {"name": "operator_torus_f32_200k", "kind": "operator", "nu": 500, "nv": 200, "dtype": "float32", "order": 6},
        # the stopping-test operator of a 50,000-panel torus solve
        {"name": "operator_torus_f64_50k", "kind": "operator", "nu": 250, "nv": 100, "dtype": "float64", "order": 8},
        # the default single-precision operator just below the FMM threshold
        {"name": "dense_f32_20k", "kind": "dense", "n": 19997, "dtype": "float32"},
        # the double-precision operator of the 5,120-panel sphere
        {"name": "dense_f64_5k", "kind": "dense", "n": 5120, "dtype": "float64"},
        # potential and field of a 5,120-panel solution at 1,000 exterior points
        {"name": "evaluate_f64_5k_1k", "kind": "evaluate", "n": 5120, "m": 1000, "dtype": "float64"},
        # the legacy bridge: every call builds tree and lists
        {"name": "apply_cube_f32_100k", "kind": "apply", "n": 100003},
        # many uneven geometries in one operator application
        {"name": "batch_dimers_f32_24", "kind": "batch", "instances": 24, "order": 6},
        # a whole solve: 5,120 panels, GMRES(50) to 1e-8 in FP64
        {"name": "solve_sphere_f64_5k", "kind": "solve", "n": 5120},
        # one step of the warm-start network's training on a 30,000-panel geometry
        {"name": "train_30k", "kind": "train", "nu": 200, "nv": 75},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fmm", "fmm", "fmm", "operator", "operator", "dense", "dense", "evaluate", "apply", "batch",
                       "solve", "train"])
    if kind == "fmm":
        if rng.random() < 0.6:
            return {"kind": kind, "points": "cube", "n": _log_int(rng, 500, 1048576), "dtype": "float32",
                    "order": rng.choice([6, 7, 8, 8])}
        return {"kind": kind, "points": "sphere", "n": _log_int(rng, 500, 60000), "dtype": "float64",
                "order": rng.choice([6, 8])}
    if kind == "operator":
        f32 = rng.random() < 0.6
        panels = _log_int(rng, 5000, 200000 if f32 else 50000)
        nv = max(16, int(math.sqrt(panels / 2 * rng.uniform(0.25, 0.6))))
        return {"kind": kind, "nu": panels // (2 * nv), "nv": nv, "dtype": "float32" if f32 else "float64",
                "order": rng.choice([6, 7, 8]) if f32 else 8}
    if kind == "dense":
        f32 = rng.random() < 0.5
        return {"kind": kind, "n": _log_int(rng, 300, 20000 if f32 else 6000),
                "dtype": "float32" if f32 else "float64"}
    if kind == "evaluate":
        return {"kind": kind, "n": _log_int(rng, 300, 6000), "m": _log_int(rng, 50, 20000),
                "dtype": rng.choice(["float32", "float64"])}
    if kind == "apply":
        return {"kind": kind, "n": _log_int(rng, 1000, 200000)}
    if kind == "batch":
        return {"kind": kind, "instances": rng.randint(2, 24), "order": rng.choice([6, 7, 8])}
    if kind == "solve":
        return {"kind": kind, "n": _log_int(rng, 500, 5000)}
    return {"kind": kind, "nu": _log_int(rng, 40, 250), "nv": rng.randint(25, 100)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)


def _sphere_points(gen, n):
    p = torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)
    return p / torch.linalg.norm(p, dim=1, keepdim=True)


def _points(case, seed):
    """Points, panel areas, charge densities in [-1, 1] and disk self terms, FP64."""
    g, n = _gen(seed), case["n"]
    if case.get("points", "cube") == "cube":
        c, a = _rand(g, n, 3), torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)
    else:
        c, a = _sphere_points(g, n), (4.0 * math.pi / n) * (0.5 + _rand(g, n))
    return c, a, 2.0 * _rand(g, n) - 1.0, _disk(a)


def _disk(areas):
    """The reference's default self terms: V_i += self_i sigma_i A_i, the equal-area disk."""
    return 2.0 * math.pi * K_E * torch.sqrt(areas / math.pi) / areas


def _torus(case, seed):
    g = _gen(seed)
    r = float(0.3 + 0.1 * _rand(g, 1))
    m = torus_mesh_device(1.0, r, case["nu"], case["nv"])
    return m, 0.5 + _rand(g, m.n_panels), _disk(m.areas)


def _charges(seed):
    rng = np.random.default_rng(seed)
    u = rng.normal(size=3)
    return [(float(rng.uniform(0.5, 1.5)), tuple(float(x) for x in u / np.linalg.norm(u) * rng.uniform(1.6, 2.4)))]


def _sphere_solution(case, seed):
    """Panels of a unit sphere with a smooth density, and points outside it."""
    g, n = _gen(seed), case["n"]
    c, a = _sphere_points(g, n), (4.0 * math.pi / n) * (0.5 + _rand(g, n))
    s = 1e-11 * (1.0 + 0.8 * c[:, 2] + 0.1 * _rand(g, n))
    t = _sphere_points(g, case["m"]) * (1.2 + 1.8 * _rand(g, case["m"], 1))
    dt = DTYPES[case["dtype"]]
    return [x.to(dt) for x in (c, a, s, t)]


def _batch(case, seed):
    """The batch benchmark's dimers (their own 2,000 to 40,000 panels), densities from the seed."""
    cases = [dimer_case_device(10 + k) for k in range(case["instances"])]
    n = sum(m.n_panels for m, _ in cases)
    return cases, 0.5 + _rand(_gen(seed), n).to(torch.float32)


def _solve_input(case, seed):
    spec = dict(conductors=[dict(type="sphere", radius=1.0, center=[0.0, 0.0, 0.0], potential=0.0)],
                charges=[dict(type="point", q=q, pos=list(p)) for q, p in _charges(seed)])
    if case["n"] == 5120:
        return icosphere(4), spec
    return generate_mesh(spec, math.sqrt(8.0 * math.pi / case["n"])), spec


def _train_input(case, seed):
    m, rough, _ = _torus(case, seed)
    pos = torch.tensor(_charges(seed)[0][1], device="cuda", dtype=torch.float64)
    b = 1.0 / torch.linalg.norm(m.centroids - pos, dim=1)
    sigma = b * (1.0 + 0.3 * m.centroids[:, 2] + 0.05 * rough)
    return dict(centroids=m.centroids.contiguous(), normals=m.normals.contiguous(), areas=m.areas.contiguous(), b=b,
                scale=b.clone(), sigma=sigma)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fmm":
        dt = DTYPES[case["dtype"]]
        c, a, s, si = (x.to(dt) for x in _points(case, seed))
        c, a = c.cpu(), a.cpu()  # the backend takes its geometry from the host
        fmm = make_laplace_fmm_backend(c, a, max_leaf_size=64, theta=0.5, expansion_order=case["order"])
        return dict(kind=kind, fmm=fmm, c=c, a=a, s=s, si=si)
    if kind == "operator":
        dt = DTYPES[case["dtype"]]
        m, s, si = _torus(case, seed)
        near = NearCorrection(m.centroids, m.areas, m.panel_vertices, distance_factor=1.5, order=2, depth=3, dtype=dt)
        op = build_operator(m.centroids, m.areas, si.to(dt), dtype=dt, kind="fmm", near=near,
                            expansion_order=case["order"])
        if dt == torch.float64:
            op.base.plan.set_arithmetic("two_float")
        return dict(kind=kind, op=op, s=s.to(dt))
    if kind == "dense":
        dt = DTYPES[case["dtype"]]
        c, a, s, si = (x.to(dt).contiguous() for x in _points(dict(case, points="sphere"), seed))
        return dict(kind=kind, c=c, a=a, s=s, si=si)
    if kind == "evaluate":
        c, a, s, t = _sphere_solution(case, seed)
        return dict(kind=kind, sol=BEMSolution(centroids=c, areas=a, sigma=s, charges=_charges(seed)), t=t)
    if kind == "apply":
        c, a, s, _ = (x.to(torch.float32) for x in _points(case, seed))
        return dict(kind=kind, backend=create_bem_fmm_backend(FmmConfig(precision="single")), c=c.cpu(), a=a.cpu(),
                    s=s)
    if kind == "batch":
        cases, s = _batch(case, seed)
        return dict(kind=kind, system=BatchSystem(cases, inner_expansion_order=case["order"]), s=s)
    if kind == "solve":
        mesh, spec = _solve_input(case, seed)
        return dict(kind=kind, mesh=mesh, spec=spec, cfg=BEMConfig(fp64=True, gmres_restart=50, gmres_tol=1e-8))
    x = _train_input(case, seed)
    net = PointCloudNet(seed=int(seed))
    return dict(kind=kind, net=net, x=x, f=net.features(x["centroids"], x["normals"], x["areas"], x["b"]))


def run(state):
    kind = state["kind"]
    if kind == "fmm":
        return bem_matvec_gpu(state["s"], state["c"], state["a"], self_integrals=state["si"], backend="external",
                              matvec_impl=state["fmm"].matvec)
    if kind == "operator":
        return state["op"](state["s"])
    if kind == "dense":
        return bem_matvec_gpu(state["s"], state["c"], state["a"], self_integrals=state["si"])
    if kind == "evaluate":
        return state["sol"].eval_V_E_batched(state["t"])
    if kind == "apply":
        return state["backend"].apply(state["c"], state["s"], state["a"])
    if kind == "batch":
        return state["system"].op32(state["s"])
    if kind == "solve":
        return bem_solve(state["spec"], state["cfg"], mesh=state["mesh"], operator="dense")["surface_charge_density"]
    net, x = state["net"], state["x"]
    y = net.forward(state["f"])
    loss, dy = net.loss(y, x["scale"], x["sigma"], x["areas"])
    net.backward(dy)
    net.adam(1e-3)
    return dict(y=y, loss=loss, grads=net.grads, params=net.params)


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _fmm_work(n, size, order, cube, shared=1):
    """One FMM application: points, areas, charges and self terms read, potentials
    written.  Operations as this geometry needs them at leaf 64 and theta 0.5: about
    4,500 (volume) or 1,400 (surface) near interactions per point of 20 flops and 29 or
    12 multipole translations per point of 4,116 flops at order 8 (cubic in the order);
    never more than all pairs of one instance."""
    per = (4500 * 20 + 29 * 4116 * (order / 8) ** 3) if cube else (1400 * 20 + 12 * 4116 * (order / 8) ** 3)
    return {"bytes": 7 * size * n, "flops": min(per * n, 20.0 * n * n / shared)}


def work(case):
    kind = case["kind"]
    size = 8 if case.get("dtype") == "float64" else 4
    if kind == "fmm":
        return _fmm_work(case["n"], size, case["order"], case["points"] == "cube")
    if kind == "operator":
        n = 2 * case["nu"] * case["nv"]
        w = _fmm_work(n, size, case["order"], False)
        return {"bytes": w["bytes"] + 8 * n * (size + 4), "flops": w["flops"] + 16 * n}  # about 8 near pairs per panel
    if kind == "dense":
        return {"bytes": 7 * size * case["n"], "flops": 20.0 * case["n"] ** 2}
    if kind == "evaluate":
        return {"bytes": size * (5 * case["n"] + 7 * case["m"]), "flops": 45.0 * case["n"] * case["m"]}
    if kind == "apply":
        return _fmm_work(case["n"], 4, 8, True)
    if kind == "batch":
        return _fmm_work(21000 * case["instances"], 4, case["order"], False, case["instances"])  # about 21,000 each
    if kind == "solve":
        return {"bytes": 8 * 14 * case["n"], "flops": 51 * 20.0 * case["n"] ** 2}
    n = 2 * case["nu"] * case["nv"]
    return {"bytes": n * (16 * 4 + 3 * 8 + 4), "flops": 6.0 * n * (16 * 128 + 2 * 128 * 128 + 128)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _rows(n, m):
    return range(0, m, max(1, 400_000_000 // max(n, 1)))


def _all_pairs(c, q, clamp):
    """sum over j != i of q_j / max(|c_i - c_j|, clamp) in FP64."""
    out, step = torch.empty_like(q), max(1, 400_000_000 // max(len(q), 1))
    for i in _rows(len(q), len(q)):
        r = torch.zeros(min(step, len(q) - i), len(q), dtype=torch.float64, device=q.device)
        for k in range(3):
            r += (c[i:i + step, k, None] - c[None, :, k]) ** 2
        r = 1.0 / r.sqrt_().clamp_(min=clamp)
        at = torch.arange(len(r), device=q.device)
        r[at, at + i] = 0.0
        out[i:i + step] = r @ q
    return out


def _near_term(m, sigma):
    """The near-pair correction: for 0 < |C_i - C_j| <= 1.5 (R_i + R_j), R = sqrt(A / pi),
    sigma_j (K_E sum of the 3-point rule on 64 equal sub-triangles - K_E A_j / |C_i - C_j|)."""
    c, a, pv = m.centroids, m.areas, m.panel_vertices
    n, R = len(a), torch.sqrt(a / math.pi)
    step = max(1, 200_000_000 // n)
    out = torch.zeros_like(a)
    cells = [(i, j, up) for i in range(8) for j in range(8 - i) for up in ((1, -1) if i + j < 7 else (1,))]
    rule = [((i + (u if up > 0 else 1 - u)) / 8, (j + (v if up > 0 else 1 - v)) / 8) for i, j, up in cells
            for u, v in ((1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3))]
    for i in range(0, n, step):
        d = sum((c[i:i + step, k, None] - c[None, :, k]) ** 2 for k in range(3)).sqrt()
        ti, sj = ((d > 0) & (d <= 1.5 * (R[i:i + step, None] + R[None, :]))).nonzero(as_tuple=True)
        ti = ti + i
        near = torch.zeros(len(ti), dtype=torch.float64, device=a.device)
        v0, e1, e2 = pv[sj, 0], pv[sj, 1] - pv[sj, 0], pv[sj, 2] - pv[sj, 0]
        for u, v in rule:
            near += 1.0 / torch.linalg.norm(v0 + u * e1 + v * e2 - c[ti], dim=1)
        w = K_E * a[sj] * (near / len(rule) - 1.0 / torch.linalg.norm(c[ti] - c[sj], dim=1))
        out.index_add_(0, ti, w * sigma[sj])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fmm", "dense", "apply"):
        if case["n"] > ALL_PAIRS_MAX:
            return None
        dt = DTYPES[case.get("dtype", "float32")]
        pts = dict(case, points="sphere") if kind == "dense" else case
        c, a, s, si = (x.to(dt).double() for x in _points(pts, seed))
        eps = 1e-12 if kind == "dense" else torch.finfo(dt).eps
        v = K_E * _all_pairs(c, s * a, eps)
        return v if kind == "apply" else v + si * s * a
    if kind == "operator":
        if 2 * case["nu"] * case["nv"] > ALL_PAIRS_MAX:
            return None
        m, s, si = _torus(case, seed)
        s = s.to(DTYPES[case["dtype"]]).double()
        v = K_E * _all_pairs(m.centroids, s * m.areas, torch.finfo(DTYPES[case["dtype"]]).eps)
        return v + si * s * m.areas + _near_term(m, s)
    if kind == "evaluate":
        c, a, s, t = (x.double() for x in _sphere_solution(case, seed))
        V, E = torch.zeros_like(t[:, 0]), torch.zeros_like(t)
        step = max(1, 20_000_000 // len(a))
        for i in range(0, len(t), step):
            d = t[i:i + step, None, :] - c[None, :, :]
            r = torch.linalg.norm(d, dim=2)
            V[i:i + step] = K_E * (1.0 / r) @ (s * a)
            E[i:i + step] = K_E * torch.einsum("ij,ijk->ik", s * a / r ** 3, d)
        for q, p in _charges(seed):
            d = t - torch.tensor(p, device=t.device, dtype=torch.float64)
            r = torch.linalg.norm(d, dim=1, keepdim=True)
            V, E = V + K_E * q / r[:, 0], E + K_E * q * d / r ** 3
        return V, E
    if kind == "batch":
        cases, s = _batch(case, seed)
        out, at = [], 0
        system = BatchSystem(cases, inner_expansion_order=case["order"])  # its self terms are inputs here
        for m, _ in cases:
            q = s[at:at + m.n_panels].double() * m.areas
            out.append(K_E * _all_pairs(m.centroids, q, torch.finfo(torch.float32).eps)
                       + system.self_corr[at:at + m.n_panels] * q)
            at += m.n_panels
        return torch.cat(out)
    if kind == "solve":
        mesh, spec = _solve_input(case, seed)
        c, a = (torch.as_tensor(x, dtype=torch.float64, device="cuda") for x in (mesh.centroids, mesh.areas))
        r = torch.cdist(c, c, compute_mode="donot_use_mm_for_euclid_dist")
        A = K_E * a[None, :] / r.clamp(min=1e-12)
        A.fill_diagonal_(0.0)
        A += torch.diag(2.0 * math.pi * K_E * torch.sqrt(a / math.pi))
        b = torch.zeros_like(a)
        for q, p in _charges(seed):
            b -= K_E * q / torch.linalg.norm(c - torch.tensor(p, device="cuda", dtype=torch.float64), dim=1)
        return torch.linalg.solve(A, b).cpu().numpy()
    x = _train_input(case, seed)
    c, a, b = x["centroids"], x["areas"], x["b"]
    d = c - c.mean(0)
    R2 = (d * d).sum(1).mean()
    f = torch.zeros(len(a), 16, dtype=torch.float64, device=a.device)
    f[:, :3], f[:, 3:6] = d / R2.sqrt(), x["normals"]
    f[:, 6], f[:, 7] = torch.log(a / R2), b / (b * b).mean().sqrt()
    p0 = PointCloudNet(seed=int(seed)).params.double()
    p = p0.clone().requires_grad_()
    W1, b1, W2, V2, b2, W3, b3, w4, b4 = torch.split(p, [2048, 128, 16384, 16384, 128, 16384, 128, 128, 1])
    h = torch.relu(f @ W1.view(128, 16).T + b1)
    h = torch.relu(h @ W2.view(128, 128).T + V2.view(128, 128) @ h.mean(0) + b2)
    y = torch.relu(h @ W3.view(128, 128).T + b3) @ w4 + b4
    e = x["scale"] * (1.0 + y) - x["sigma"]
    loss = (a * e * e).sum() / (a * x["sigma"] ** 2).sum()
    g, = torch.autograd.grad(loss, p)
    return dict(y=y.detach(), loss=loss.detach().reshape(1), grads=g, params=p0 - 1e-3 * g / (g.abs() + 1e-8))
