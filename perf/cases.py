"""The work a program has this library do, as timed cases.

A case is a plain dict; `kind` says which calls it makes:

  jacobian    Newton Jacobian and residual of one iterate
  newton      the same, then the residual alone at a trial point (a line-search step)
  system      K(nu), M(sigma), a source vector and a coil vector on one mesh, from device arrays
  assembler   the same four through the Assembler facade, from {tag: value} maps, MATLAB storage
  batch       K + j omega M of many meshes of uneven size in one call
  hbfem       harmonic-balance residual and DC block
  transient   backward-Euler steps of the E-core problem from rest: Newton, line search, CG;
              then the element flux densities of each step
  predict     reluctivity inference of the MLP over all elements
  gradient    forward and backward pass of the MLP on one minibatch
  mex         one call of the MATLAB gateway's entry point: host arrays in, sparse matrix out
  setup       a new mesh: edges, dofs, CSR pattern, assembly plan and its first Jacobian

Meshes are jittered Kuhn boxes (six tetrahedra per hexahedron, node jitter of a tenth of the
spacing) with an iron block on a 200-point B-H curve and an aluminium slab in air. Edge values
are scaled so that |B| is of the order of one tesla, where the curve bends.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

AIR, IRON, ALUMINIUM = 1, 2, 3
NU0 = 1.0 / (4e-7 * math.pi)
SIGMA_AL = 3.526e7
_PERMS = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))
_EDGES = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))
_MLP_SHAPES = ((64, 4), (64,), (64, 64), (64,), (64, 64), (64,), (64,), (1,))


# ---- the cases -------------------------------------------------------------------------------


def listed():
    return [
        # a tutorial-sized problem in a Newton loop: latency and launches
        {"name": "jacobian_8", "kind": "jacobian", "nx": 8, "ny": 8, "nz": 8},
        # an ordinary nonlinear solve: one iteration with its line-search evaluation
        {"name": "newton_60", "kind": "newton", "nx": 60, "ny": 60, "nz": 60},
        # the largest single mesh of the benchmark, 8 million tetrahedra
        {"name": "jacobian_110", "kind": "jacobian", "nx": 110, "ny": 110, "nz": 110},
        # a magnetostatic or frequency problem's matrices and right-hand sides, sides of no round number
        {"name": "system_53", "kind": "system", "nx": 53, "ny": 47, "nz": 41},
        # the same for a script that works with the Assembler class and material maps
        {"name": "assembler_17", "kind": "assembler", "nx": 17, "ny": 16, "nz": 15},
        # a frequency sweep over independent meshes
        {"name": "batch_16", "kind": "batch", "count": 16, "n_min": 8, "n_max": 48},
        # harmonic balance with the first three odd harmonics, 32 time samples
        {"name": "hbfem_40", "kind": "hbfem", "nx": 40, "ny": 40, "nz": 40, "harmonics": 3, "samples": 32},
        # the E-core transient at the size of the transient benchmark
        {"name": "transient_40", "kind": "transient", "nx": 40, "ny": 40, "nz": 20, "steps": 1},
        # reluctivity of every element of the largest mesh
        {"name": "predict_8m", "kind": "predict", "rows": 7986000},
        # one minibatch of the predictor's training
        {"name": "gradient_32k", "kind": "gradient", "rows": 32768},
        # MATLAB's Newton loop: the gateway's mesh cache is warm, the matrix goes back to the host
        {"name": "mex_30", "kind": "mex", "nx": 30, "ny": 30, "nz": 30},
        # a program's start, or one more mesh of a design study
        {"name": "setup_40", "kind": "setup", "nx": 40, "ny": 40, "nz": 40},
    ]


# per kind: smallest and largest number of hexahedra per side (geometric mean of the three)
_SIDES = {"jacobian": (4, 80), "newton": (6, 64), "system": (6, 56), "assembler": (4, 24), "hbfem": (6, 40),
          "mex": (6, 30), "setup": (6, 44), "transient": (8, 24)}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(sorted(_SIDES) + ["batch", "predict", "gradient"])
    if kind == "batch":
        n_min = rng.randint(4, 12)
        return {"kind": kind, "count": rng.randint(2, 20), "n_min": n_min, "n_max": rng.randint(n_min + 4, 44)}
    if kind == "predict":
        return {"kind": kind, "rows": _log(rng, 1000, 7900000)}
    if kind == "gradient":
        return {"kind": kind, "rows": _log(rng, 100, 32768)}
    lo, hi = _SIDES[kind]
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if kind == "transient":  # the core needs some elements across its legs in x and y
        n = max(10, int(round(n)))
        return {"kind": kind, "nx": n, "ny": n + rng.randint(-2, 2), "nz": max(6, n // 2 + rng.randint(-1, 1)),
                "steps": rng.randint(1, 2)}
    fx, fy = rng.uniform(0.75, 1.3), rng.uniform(0.75, 1.3)
    case = {"kind": kind, "nx": max(2, int(round(n * fx))), "ny": max(2, int(round(n * fy))),
            "nz": max(2, int(round(n / (fx * fy))))}
    if kind == "hbfem":
        case["harmonics"] = rng.randint(1, 4)
        case["samples"] = rng.choice((16, 24, 32))
    return case


# ---- inputs ------------------------------------------------------------------------------------


def _rng(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * (seed + 1) + salt)


def _f64(shape, g):
    return torch.randn(shape, generator=g, dtype=torch.float64, device="cuda")


def _box(case, seed, salt=0):
    """P [Nn, 3], T [Ne, 4] (int64), tags [Ne] and the largest spacing h of a jittered Kuhn box
    whose longest side is 1."""
    n = (case["nx"], case["ny"], case["nz"])
    g = _rng(seed, salt)
    h = 1.0 / max(n)
    ax = [torch.arange(k + 1, dtype=torch.float64, device="cuda") for k in n]
    kk, jj, ii = torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij")  # x fastest
    idx = torch.stack([ii.reshape(-1), jj.reshape(-1), kk.reshape(-1)], 1)
    top = torch.tensor(n, dtype=torch.float64, device="cuda")
    d = torch.rand(idx.shape, generator=g, dtype=torch.float64, device="cuda") * 0.2 - 0.1
    d = torch.where((idx == 0) | (idx == top), torch.zeros_like(d), d)
    P = (idx + d) * h
    ah = [torch.arange(k, device="cuda") for k in n]
    hk, hj, hi = torch.meshgrid(ah[2], ah[1], ah[0], indexing="ij")
    sx, sy = n[0] + 1, (n[0] + 1) * (n[1] + 1)
    base = (hi + sx * hj + sy * hk).reshape(-1)
    step = (1, sx, sy)
    T = torch.empty((base.numel(), 6, 4), dtype=torch.int64, device="cuda")
    for t, perm in enumerate(_PERMS):
        v = base
        T[:, t, 0] = v
        for a in range(3):
            v = v + step[perm[a]]
            T[:, t, a + 1] = v
    T = T.reshape(-1, 4)
    c = (P[T].sum(1) * 0.25) / (top * h)
    u = torch.rand(7, generator=g, dtype=torch.float64, device="cuda")
    lo, ext = 0.2 + 0.2 * u[:3], 0.3 + 0.15 * u[3:6]
    tags = torch.full((T.shape[0],), AIR, dtype=torch.int32, device="cuda")
    z0 = 0.03 + 0.07 * u[6]
    tags[(c[:, 2] >= z0) & (c[:, 2] <= z0 + 0.1)] = ALUMINIUM
    tags[((c >= lo) & (c <= lo + ext)).all(1)] = IRON
    return P, T, tags, h


def _num_edges(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mx, my, mz = nx + 1, ny + 1, nz + 1
    axes = nx * my * mz + mx * ny * mz + mx * my * nz
    faces = nx * ny * mz + nx * my * nz + mx * ny * nz
    return axes + faces + nx * ny * nz


def _num_nodes(case):
    return (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)


def _num_elems(case):
    return 6 * case["nx"] * case["ny"] * case["nz"]


def _field(case, h, g, cols=None):
    """Edge values of a field of about one tesla: noise of the size of a face's flux."""
    shape = (_num_edges(case),) if cols is None else (_num_edges(case), cols)
    return 0.2 * h * h * _f64(shape, g)


def _materials():
    from magpackage_b200 import synth

    return synth.standard_materials()


def _coefficients(tags, g):
    """Per-element reluctivity, conductivity and current density as a linear problem has them."""
    nu = torch.where(tags == IRON, NU0 / 1000.0, NU0).double()
    sigma = torch.where(tags == ALUMINIUM, SIGMA_AL, 0.0).double()
    js = 1e6 * _f64((tags.numel(), 3), g) * (tags != ALUMINIUM).double()[:, None]
    return nu, sigma, js


_MAP_NU = {AIR: NU0, IRON: NU0 / 1000.0, ALUMINIUM: NU0}
_MAP_SIGMA = {AIR: 1.0, IRON: 1e3, ALUMINIUM: SIGMA_AL}  # a little conductivity regularises the air
_COIL = {"id": IRON, "direction": (0.6, 0.0, 0.8), "turns": 100.0, "area": 1e-3}


def _mlp_inputs(case, seed):
    g = _rng(seed, 5)
    fan = (4, None, 64, None, 64, None, 64, None)
    parts = []
    for shape, f in zip(_MLP_SHAPES, fan):
        w = torch.randn(shape, generator=g, device="cuda")
        parts.append((w * math.sqrt((1.0 if shape == (64,) else 2.0) / f) if f else 0.1 * w).reshape(-1))
    params = torch.cat(parts)
    feats = torch.randn((case["rows"], 4), generator=g, device="cuda")
    target = torch.randn(case["rows"], generator=g, device="cuda")
    return params, feats, target


def _harmonics(case):
    return [2 * i + 1 for i in range(case["harmonics"])]


def _sweep(case):
    """(side, angular frequency) of each mesh of a batch."""
    n = case["count"]
    t = [i / max(n - 1, 1) for i in range(n)]
    return [(int(round(case["n_min"] + (case["n_max"] - case["n_min"]) * x)), 2.0 * math.pi * 10.0 * 1000.0 ** x)
            for x in t]


def _plan(P, T, tags):
    from magpackage_b200.plan import AssemblyPlan, generate_edges

    edges, t2e, sign = generate_edges(T.int())
    return AssemblyPlan(P, T.int(), t2e, int(edges.shape[0]), tags, sign)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("predict", "gradient"):
        from magpackage_b200.mlp import MLP

        params, st["feats"], st["target"] = _mlp_inputs(case, seed)
        st["mlp"] = MLP(params.cpu().numpy())
        if kind == "predict":
            st["rows"] = torch.arange(case["rows"], dtype=torch.int32, device="cuda")
            st["nu"] = torch.empty(case["rows"], dtype=torch.float64, device="cuda")
        return st
    if kind == "transient":
        from magpackage_b200.transient import TransientConfig, TransientProblem

        st["problem"] = prob = TransientProblem(TransientConfig(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed))
        st["x0"] = torch.zeros(prob.num_dofs, dtype=torch.float64, device="cuda")
        b0 = torch.zeros(prob.iron.numel(), dtype=torch.float32, device="cuda")
        st["b"], st["steps"] = (b0, b0), case["steps"]
        return st
    if kind == "batch":
        from magpackage_b200.plan import ComplexBatch

        plans, nus, sigmas, omegas = [], [], [], []
        for i, (n, omega) in enumerate(_sweep(case)):
            P, T, tags, _ = _box({"nx": n, "ny": n, "nz": n}, seed, 100 + i)
            nu, sigma, _ = _coefficients(tags, _rng(seed, 50 + i))
            plans.append(_plan(P, T, tags))
            nus.append(nu)
            sigmas.append(sigma)
            omegas.append(omega)
        st["batch"] = ComplexBatch(plans, nus, sigmas, omegas)
        return st

    P, T, tags, h = _box(case, seed)
    g = _rng(seed, 1)
    if kind in ("assembler", "setup"):
        from magpackage_b200.assembler import Assembler, DofHandler, Mesh, Winding

        host = (P.cpu().numpy(), T.int().cpu().numpy(), tags.cpu().numpy())
        if kind == "setup":
            st["host"], st["sol"], st["materials"] = host, _field(case, h, g), _materials()
            return st
        mesh = Mesh(*host)
        dh = DofHandler(mesh)
        dh.distribute_dofs()
        st["assembler"] = asm = Assembler(mesh, dh)
        asm.plan.row_ptr
        st["js"] = {IRON: (0.0, 2e6, 0.0)}
        st["winding"] = Winding.create("coil", _COIL["id"], _COIL["turns"], 1.0, _COIL["area"], _COIL["direction"])
        return st
    if kind == "mex":
        from magpackage_b200.material import pack_material_data
        from magpackage_b200.plan import generate_edges
        from magpackage_b200.quadrature import reference_data

        _, t2e, sign = generate_edges(T.int())
        f = lambda a: np.ascontiguousarray(a.cpu().numpy(), dtype=np.float64)  # noqa: E731
        st["mesh"] = [f(P), f(T + 1), f(t2e + 1), f(sign), f(tags)]
        st["sol"] = f(_field(case, h, g))
        qw, _, curl = reference_data(2)
        st["ref"] = [np.ascontiguousarray(a, dtype=np.float64) for a in (qw, curl)]
        st["mat"] = [np.ascontiguousarray(a, dtype=np.float64) for a in pack_material_data(_materials()).as_tuple()]
        return st

    st["plan"] = plan = _plan(P, T, tags)
    if kind == "system":
        st["nu"], st["sigma"], st["js"] = _coefficients(tags, g)
        return st
    from magpackage_b200.material import pack_material_data

    plan.set_materials(pack_material_data(_materials()))
    if kind == "hbfem":
        from magpackage_b200.hbfem import AFT

        st["aft"] = AFT(_harmonics(case), n_time_steps=case["samples"])
        st["sol"] = tuple(_field(case, h, g, case["harmonics"]).T.contiguous() for _ in range(2))
        return st
    st["sol"] = _field(case, h, g)
    if kind == "newton":
        st["trial"] = st["sol"] + 0.1 * _field(case, h, g)
    return st


# ---- one pass ----------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "jacobian":
        return state["plan"].jacobian(state["sol"])
    if kind == "newton":
        vals, res = state["plan"].jacobian(state["sol"])
        _, trial = state["plan"].jacobian(state["trial"], calc_j=False)
        return vals, res, trial
    if kind == "system":
        p = state["plan"]
        return (p.stiffness(state["nu"]), p.mass(state["sigma"]), p.source(state["js"]),
                p.winding(_COIL["id"], _COIL["direction"], _COIL["turns"] / _COIL["area"]))
    if kind == "assembler":
        a = state["assembler"]
        K, M = a.assemble_stiffness(_MAP_NU), a.assemble_mass_weighted(_MAP_SIGMA)
        return (a.assemble_source(state["js"]), a.assemble_winding(state["winding"]),
                K.row_ptr, K.col_idx, K.values, M.row_ptr, M.col_idx, M.values)
    if kind == "batch":
        return state["batch"].assemble()
    if kind == "hbfem":
        from magpackage_b200.hbfem import assemble_hbfem

        return assemble_hbfem(state["plan"], state["sol"], state["aft"])
    if kind == "transient":
        from magpackage_b200.transient import run as steps

        n = state["steps"]
        rec = steps(state["problem"], 1, n, state["x0"], state["b"], keep_x=tuple(range(1, n + 1)))
        return [t for _, x in rec.x for t in (x,) + state["problem"].plan.element_b(x)]
    if kind == "predict":
        state["mlp"].predict_nu(state["feats"], state["rows"], state["nu"], 0.5, 5.0, 1.0, 1e6)
        return state["nu"]
    if kind == "gradient":
        return state["mlp"].gradient(state["feats"], state["target"], 2.0 / state["feats"].shape[0])
    if kind == "mex":
        return _run_mex(state)
    from magpackage_b200.assembler import Assembler, DofHandler, Mesh

    mesh = Mesh(*state["host"])
    dh = DofHandler(mesh)
    dofs = dh.distribute_dofs()
    K, res = Assembler(mesh, dh, matlab_storage=False).assemble_jacobian(state["sol"], state["materials"])
    return K.values, res, K.row_ptr, K.col_idx, mesh.Edges, mesh.T2E_Sign, dofs


def _run_mex(state):
    """mag_mex_jacobian_sparse and the copy of its result, as the gateway calls them."""
    from magpackage_b200 import _lib

    L, p = _lib.lib(), _lib.dptr
    P, T, D, S, G = state["mesh"]
    sol, (qw, curl), pk = state["sol"], state["ref"], state["mat"]
    res, h = np.empty(sol.size), C.c_void_p()
    _lib.check(L.mag_mex_jacobian_sparse(
        p(P), P.shape[0], p(T), T.shape[0], p(D), p(S), p(G), p(sol), sol.size, p(qw), qw.size, p(curl), p(pk[0]),
        p(pk[1]), p(pk[2]), pk[0].size, p(pk[3]), pk[3].size, p(pk[4]), pk[4].size, p(pk[5]), p(pk[6]), p(pk[7]), 1,
        C.byref(h), p(res)))
    n, nz = C.c_int64(), C.c_int64()
    _lib.check(L.mag_sparse_info(h, C.byref(n), C.byref(nz)))
    jc, ir = np.empty(n.value + 1, dtype=np.uint64), np.empty(max(nz.value, 1), dtype=np.uint64)
    pr = np.empty(max(nz.value, 1))
    u64 = C.POINTER(C.c_uint64)
    _lib.check(L.mag_sparse_copy(h, jc.ctypes.data_as(u64), ir.ctypes.data_as(u64), p(pr)))
    _lib.check(L.mag_sparse_destroy(h))
    return jc.view(np.int64), ir.view(np.int64), pr, res


# ---- what a pass cannot do without ---------------------------------------------------------------
# Element flops: geometry 45, curls 54, B and the material 80, six residual entries 40, 36 matrix
# entries of 7 operations each; mass: inverse 50, four points of 6 basis vectors (90) and 21 products (126).


def _nnz(case):
    """Structural nonzeros of the Nedelec matrix: an edge couples with itself, and with each other edge
    that shares a triangle (two ordered pairs for each of 3 pairs) or lies opposite in a tetrahedron."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ne = _num_elems(case)
    tri = (4 * ne + 4 * (nx * ny + ny * nz + nx * nz)) // 2
    return _num_edges(case) + 6 * tri + 6 * ne


def work(case):
    kind = case["kind"]
    if kind in ("predict", "gradient"):
        n = case["rows"]
        fl = 2.0 * (4 * 64 + 2 * 64 * 64 + 64)
        if kind == "predict":
            return {"bytes": 28.0 * n, "flops": fl * n}
        return {"bytes": 24.0 * n + 4 * 8769, "flops": 3.0 * fl * n}
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        for n, _ in _sweep(case):
            c = {"nx": n, "ny": n, "nz": n}
            ne = _num_elems(c)
            tot["bytes"] += 57.0 * ne + 24.0 * _num_nodes(c) + 16.0 * _nnz(c)
            tot["flops"] += ne * (350.0 + 0.1 * 900.0)
        return tot
    ne, nn, E, nnz = _num_elems(case), _num_nodes(case), _num_edges(case), _nnz(case)
    mesh = 41.0 * ne + 24.0 * nn  # nodes, dofs and tag of each element, coordinates
    if kind == "jacobian":
        return {"bytes": mesh + 16.0 * E + 8.0 * nnz, "flops": 470.0 * ne}
    if kind == "newton":
        return {"bytes": 2 * mesh + 32.0 * E + 8.0 * nnz, "flops": 690.0 * ne}
    if kind in ("system", "assembler"):
        return {"bytes": 4 * mesh + 40.0 * ne + 16.0 * E + 16.0 * nnz, "flops": ne * (350.0 + 900.0 + 150.0)}
    if kind == "hbfem":
        K, N = case["harmonics"], case["samples"]
        per = N * (6 * 4 * K + 36 + 40 + 66) + 4 * N * 6 * 4 * K + 300
        return {"bytes": mesh + 32.0 * K * E + 8.0 * nnz, "flops": float(per) * ne}
    if kind == "transient":  # per step about 4 Newton iterations; CG iterations grow with the side
        it = 4.0 * case["steps"] * 20.0 * case["nx"]
        return {"bytes": 4 * case["steps"] * (mesh + 8.0 * nnz) + it * (12.0 * nnz + 80.0 * E),
                "flops": it * (2.0 * nnz + 20.0 * E)}
    if kind == "mex":  # the arrays MATLAB holds are doubles; the matrix comes back as jc, ir, pr
        return {"bytes": 8.0 * (3 * nn + 17 * ne) + 24.0 * E + 16.0 * nnz, "flops": 470.0 * ne}
    # host mesh in; edges, element dofs and signs, pattern and values out
    return {"bytes": 24.0 * nn + 20.0 * ne + 30.0 * ne + 32.0 * E + 12.0 * nnz, "flops": 470.0 * ne}


# ---- the same outputs in 64 bits, with plain torch ---------------------------------------------


def _exact_mesh(P, T, pattern=True):
    nn = P.shape[0]
    i = torch.tensor([a for a, _ in _EDGES], device="cuda")
    j = torch.tensor([b for _, b in _EDGES], device="cuda")
    a, b = T[:, i], T[:, j]
    keys, dofs = torch.unique(torch.minimum(a, b) * nn + torch.maximum(a, b), return_inverse=True)
    m = {"E": keys.numel(), "dofs": dofs, "sign": torch.where(a < b, 1.0, -1.0).double()}
    X = P[T]
    J = (X[:, 1:] - X[:, :1]).transpose(1, 2)  # columns v_k - v_0
    det = (J[:, :, 0] * torch.linalg.cross(J[:, :, 1], J[:, :, 2])).sum(1)
    # gradients of the barycentric coordinates: rows of J^-1
    r = torch.stack([torch.linalg.cross(J[:, :, 1], J[:, :, 2]), torch.linalg.cross(J[:, :, 2], J[:, :, 0]),
                     torch.linalg.cross(J[:, :, 0], J[:, :, 1])], 1) / det[:, None, None]
    grad = torch.cat([-r.sum(1, keepdim=True), r], 1)
    m["ga"], m["gb"] = grad[:, i], grad[:, j]
    m["i"], m["j"], m["adet"] = i, j, det.abs()
    m["curl"] = 2.0 * torch.linalg.cross(m["ga"], m["gb"]) * m["sign"][:, :, None]
    if pattern:
        E = m["E"]
        pairs, m["slot"] = torch.unique((dofs[:, :, None] * E + dofs[:, None, :]).reshape(-1), return_inverse=True)
        m["nnz"] = pairs.numel()
        m["pairs"] = pairs
    return m


def _scatter_matrix(m, block):
    return torch.zeros(m["nnz"], dtype=block.dtype, device="cuda").index_add_(0, m["slot"], block.reshape(-1))


def _scatter_vector(m, v):
    return torch.zeros(m["E"], dtype=v.dtype, device="cuda").index_add_(0, m["dofs"].reshape(-1), v.reshape(-1))


def _exact_nu(tags, s):
    """nu and d nu / d s at s = |B|^2 [Ne, ...] from the packed B-H table of the iron."""
    mat = _materials()[IRON]
    brk = torch.as_tensor(mat.breaks, dtype=torch.float64, device="cuda")
    coef = torch.as_tensor(mat.coefs, dtype=torch.float64, device="cuda")
    x = s.clamp(max=float(mat.max_bsq))
    k = (torch.searchsorted(brk, x, right=True) - 1).clamp(0, coef.shape[0] - 1)
    t, c = x - brk[k], coef[k]
    v = ((c[..., 0] * t + c[..., 1]) * t + c[..., 2]) * t + c[..., 3]
    dv = (3.0 * c[..., 0] * t + 2.0 * c[..., 1]) * t + c[..., 2]
    v = v + torch.where(s > mat.max_bsq, dv * (s - mat.max_bsq), 0.0)
    out = (v > mat.nu0) | (v < 1e-7)
    v, dv = torch.where(out, mat.nu0, v), torch.where(out, 0.0, dv)
    iron = (tags == IRON).reshape((-1,) + (1,) * (s.dim() - 1))
    return torch.where(iron, v, NU0), torch.where(iron, dv, 0.0)


def _exact_newton(m, tags, sol, matrix=True):
    C_, w = m["curl"], m["adet"] / 6.0
    B = (sol[m["dofs"]][:, :, None] * C_).sum(1)
    nu, dnu = _exact_nu(tags, (B * B).sum(1))
    b = (C_ * B[:, None]).sum(2)
    res = _scatter_vector(m, (nu * w)[:, None] * b)
    if not matrix:
        return None, res
    K = (nu * w)[:, None, None] * (C_ @ C_.transpose(1, 2))
    K += (2.0 * dnu * w)[:, None, None] * b[:, :, None] * b[:, None, :]
    return _scatter_matrix(m, K), res


def _exact_stiffness(m, nu):
    return _scatter_matrix(m, (nu * m["adet"] / 6.0)[:, None, None] * (m["curl"] @ m["curl"].transpose(1, 2)))


def _moments():
    """sum_q w_q and the sums of w_q L_a, w_q L_a L_b over the 4-point rule on the unit tetrahedron."""
    a, b = 0.58541020, 0.13819660
    q = torch.full((4, 3), b, dtype=torch.float64, device="cuda")
    for k in range(3):
        q[k, k] = a
    lam = torch.cat([1.0 - q.sum(1, keepdim=True), q], 1)
    return lam.sum(0) / 24.0, lam.T @ lam / 24.0


def _exact_mass(m, sigma):
    _, I = _moments()
    i, j, ga, gb = m["i"], m["j"], m["ga"], m["gb"]
    ii, ij, jj = I[i][:, i], I[i][:, j], I[j][:, j]
    M = ii * (gb @ gb.transpose(1, 2)) - ij * (gb @ ga.transpose(1, 2))
    M = M - ij.T * (ga @ gb.transpose(1, 2)) + jj * (ga @ ga.transpose(1, 2))
    s = m["sign"]
    return _scatter_matrix(m, (sigma * m["adet"])[:, None, None] * M * (s[:, :, None] * s[:, None, :]))


def _exact_load(m, js):
    f, _ = _moments()
    W = f[m["i"]][None, :, None] * m["gb"] - f[m["j"]][None, :, None] * m["ga"]
    return _scatter_vector(m, m["adet"][:, None] * m["sign"] * (W * js[:, None]).sum(2))


def _coil_density(tags):
    d = torch.tensor(_COIL["direction"], dtype=torch.float64, device="cuda") * (_COIL["turns"] / _COIL["area"])
    return (tags == _COIL["id"]).double()[:, None] * d


def _exact_hbfem(m, tags, sol, case):
    N = case["samples"]
    N = max(N, 2 * max(_harmonics(case)) + 1)
    h = torch.tensor(_harmonics(case), dtype=torch.float64, device="cuda")
    theta = torch.arange(N, dtype=torch.float64, device="cuda") * (2.0 * math.pi / N)
    arg = h[:, None] * theta[None, :]
    sr, si = sol
    R = torch.zeros((case["harmonics"], m["E"]), dtype=torch.complex128, device="cuda")
    dc = torch.zeros(m["adet"].numel(), dtype=torch.float64, device="cuda")
    P = (2.0 / N) * torch.polar(torch.ones_like(arg), -arg)
    for t in range(N):
        x = torch.cos(arg[:, t]) @ sr - torch.sin(arg[:, t]) @ si
        B = (x[m["dofs"]][:, :, None] * m["curl"]).sum(1)
        nu, _ = _exact_nu(tags, (B * B).sum(1))
        dc += nu / N
        r = _scatter_vector(m, (nu * m["adet"] / 6.0)[:, None] * (m["curl"] * B[:, None]).sum(2))
        R += P[:, t, None] * r[None, :]
    return R, _exact_stiffness(m, dc)


def _exact_mlp(params, feats, target=None, chunk=1 << 20):
    p, w = params.double(), []
    for shape in _MLP_SHAPES:
        n = math.prod(shape)
        w.append(p[:n].reshape(shape))
        p = p[n:]
    ys = []
    for f in feats.split(chunk):
        z = f.double()
        for k in (0, 2, 4):
            z = torch.nn.functional.silu(z @ w[k].T + w[k + 1])
        ys.append(z @ w[6] + w[7])
    y = torch.cat(ys)
    if target is None:
        return y, None
    leaves = [t.clone().requires_grad_() for t in w]
    z = feats.double()
    for k in (0, 2, 4):
        z = torch.nn.functional.silu(z @ leaves[k].T + leaves[k + 1])
    out = z @ leaves[6] + leaves[7]
    dy = (out.detach() - target.double()) * (2.0 / feats.shape[0])
    grads = torch.autograd.grad((out * dy).sum(), leaves)
    return y, torch.cat([g.reshape(-1) for g in grads])


def exact(case, seed):
    kind = case["kind"]
    if kind == "transient":  # a nonlinear solve to a tolerance, on a mesh too large for a dense one
        return None
    if kind == "predict":
        params, feats, _ = _mlp_inputs(case, seed)
        y, _ = _exact_mlp(params, feats)
        return torch.exp(0.5 * y + 5.0).clamp(1.0, 1e6)
    if kind == "gradient":
        return _exact_mlp(*_mlp_inputs(case, seed))
    if kind == "batch":
        out = []
        for i, (n, omega) in enumerate(_sweep(case)):
            P, T, tags, _ = _box({"nx": n, "ny": n, "nz": n}, seed, 100 + i)
            nu, sigma, _ = _coefficients(tags, _rng(seed, 50 + i))
            m = _exact_mesh(P, T)
            out.append(torch.complex(_exact_stiffness(m, nu), omega * _exact_mass(m, sigma)))
        return out
    P, T, tags, h = _box(case, seed)
    g = _rng(seed, 1)
    m = _exact_mesh(P, T, pattern=kind not in ("assembler", "mex"))
    if kind == "system":
        nu, sigma, js = _coefficients(tags, g)
        return (_exact_stiffness(m, nu), _exact_mass(m, sigma), _exact_load(m, js),
                _exact_load(m, _coil_density(tags)))
    if kind == "assembler":  # the stored entries depend on which sums are exactly zero
        js = torch.zeros((tags.numel(), 3), dtype=torch.float64, device="cuda")
        js[tags == IRON] = torch.tensor((0.0, 2e6, 0.0), dtype=torch.float64, device="cuda")
        return (_exact_load(m, js), _exact_load(m, _coil_density(tags))) + (None,) * 6
    if kind == "hbfem":
        sol = tuple(_field(case, h, g, case["harmonics"]).T.contiguous() for _ in range(2))
        return _exact_hbfem(m, tags, sol, case)
    sol = _field(case, h, g)
    if kind == "mex":
        return None, None, None, _exact_newton(m, tags, sol, matrix=False)[1]
    vals, res = _exact_newton(m, tags, sol)
    if kind == "jacobian":
        return vals, res
    if kind == "setup":
        return (vals, res) + (None,) * 5
    trial = sol + 0.1 * _field(case, h, g)
    return vals, res, _exact_newton(m, tags, trial, matrix=False)[1]
