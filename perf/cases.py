"""The workloads that a program built on this framework runs, for measurement.

A case names one of the solve path's public entry points and the mesh, element
and precision it runs on:

  apply        FEMatrix.apply / apply_f32: y = A x on an assembled finest-level
               matrix (BlockFEMatrix::apply), the product every Krylov method
               and residual evaluation runs
  assemble     assembly of one level (element loop, CSR values, right-hand side)
               into the caller's device arrays
  cycle        Solver.apply_preconditioner: one multigrid V cycle in FP64
               (damped Jacobi on convection-diffusion, nodal Vanka on Stokes)
  linearise    the Navier-Stokes Picard step's reassembly around a velocity on
               every level, followed by the product with the new matrix
  request      reset, assemble and solve one convection-diffusion or Stokes
               problem whose mesh is resident: what the serving loop does per
               request
  batch        assemble several problems of one mesh and solve them together
  steps        two implicit time steps from the initial condition

Meshes are uniform with cells = root * 2^refine per side, as the framework's
own requests use them (one root cell, or 3, 5, 7 for the sizes in between).
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import mymoonmd_gb300 as m
from mymoonmd_gb300 import workloads
from mymoonmd_gb300._lib import check, lib


# ------------------------------------------------------------------ cases ---
def listed():
    return [
        # the smallest call: the preconditioner of a small 2D problem's Krylov loop
        dict(name="cycle_2d_q1_32", kind="cycle", dim=2, elem=1, root=1, refine=5, levels=4, eps=0.1),
        # the outer product of the 3D Q2 convection-diffusion request
        dict(name="apply_3d_q2_32", kind="apply", dim=3, elem=2, root=1, refine=5, dtype="fp64", eps=1e-2),
        # the mixed form's FP32 product on a mesh between the powers of two
        dict(name="apply_f32_3d_q2_24", kind="apply", dim=3, elem=2, root=3, refine=3, dtype="fp32", eps=1e-2),
        # assembly of a mid-size 3D level by a caller that owns its memory
        dict(name="assemble_3d_q2_16", kind="assemble", dim=3, elem=2, root=1, refine=4, eps=1e-2),
        # the plain FP64 form's preconditioner: Jacobi V(2,2)
        dict(name="cycle_3d_q2_16", kind="cycle", dim=3, elem=2, root=1, refine=4, levels=3, eps=1e-2),
        # the Stokes preconditioner in FP64: nodal Vanka V(1,1)
        dict(name="cycle_stokes_12", kind="cycle", flow="stokes", root=3, nu=1.0),
        # the Picard loop's reassembly of a mid-size Navier-Stokes problem
        dict(name="linearise_12", kind="linearise", root=3, nu=0.1),
        # the 2D Q1 128^2 workload in its plain FP64 form, to 1e-10
        dict(name="request_2d_q1_128_fp64", kind="request", dim=2, elem=1, root=1, refine=7, levels=4, eps=0.1,
             precision="fp64", reduction=1e-10, restart=20),
        # the 3D Q2 32^3 workload, mixed form, to 1e-8: the benchmark's request
        dict(name="request_3d_q2_32_mixed", kind="request", dim=3, elem=2, root=1, refine=5, levels=4, eps=1e-2,
             precision="mixed", reduction=1e-8, restart=30),
        # the Stokes P2/P1 24^3 workload, mixed form, to 1e-8
        dict(name="request_stokes_24_mixed", kind="request", flow="stokes", root=6, nu=1.0, precision="mixed",
             reduction=1e-8, restart=30),
        # eight requests of the stream on one 2D mesh, solved in lockstep
        dict(name="batch_2d_q2_64", kind="batch", dim=2, elem=2, root=1, refine=6, levels=5, eps=0.1,
             precision="mixed", reduction=1e-8, restart=30, n=8),
        # time-dependent convection-diffusion, two Crank-Nicolson steps
        dict(name="steps_3d_q2_12", kind="steps", dim=3, elem=2, root=3, refine=2, levels=3, eps=1e-2,
             precision="mixed", reduction=1e-8, restart=30, scheme="crank_nicolson", tau=0.01),
    ]


# finest cells per side: (dimension, element) -> range of the requests
_RANGE = {(2, 1): (16, 256), (2, 2): (16, 256), (3, 1): (8, 32), (3, 2): (6, 32)}
# a product above a launch's own few microseconds
_RANGE_APPLY = {(2, 1): (192, 640), (2, 2): (96, 320), (3, 1): (24, 48), (3, 2): (10, 32)}
# a level whose element matrices fit the allocation-free assembly's array
_RANGE_NOALLOC = {(2, 1): (16, 256), (2, 2): (16, 200), (3, 1): (6, 32), (3, 2): (4, 16)}


def _draw_mesh(rng, dim, elem, ranges, min_refine):
    """root cells and refinements with root * 2^refine log-uniform over the range
    (2D Q2 multigrid on 5 or 7 root cells is left out: its coarse direct solve
    is inaccurate there)"""
    lo, hi = ranges[dim, elem]
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    roots = (1, 3) if (dim, elem) == (2, 2) and min_refine else (1, 3, 5, 7)
    fits = [(r, k) for r in roots for k in range(min_refine, 9) if lo <= (r << k) <= hi]
    near = min(abs(math.log((r << k) / want)) for r, k in fits)
    return rng.choice([f for f in fits if abs(math.log((f[0] << f[1]) / want)) <= near + 0.15])


def _levels(dim, root, refine):
    """multigrid levels down to about 4 (2D) or 3-5 (3D) cells per side"""
    levels = 1
    while levels <= refine and (root << refine) >> levels >= (4 if dim == 2 else 3):
        levels += 1
    return max(2, levels)


def draw(rng):
    kind = rng.choice(["apply", "apply", "assemble", "cycle", "cycle_stokes", "linearise", "request", "request",
                       "request_stokes", "batch", "steps"])
    if kind in ("cycle_stokes", "linearise", "request_stokes"):
        # 4, 8, ... 24 cubes per side, log-uniform; viscosity over two decades
        root = int(round(math.exp(rng.uniform(math.log(1.0), math.log(6.0 if kind == "request_stokes" else 5.0)))))
        nu = round(10.0 ** rng.uniform(-1.0, 1.0 if kind != "linearise" else 0.0), 4)
        if kind == "linearise":
            return dict(kind=kind, root=root, nu=nu)
        if kind == "cycle_stokes":
            return dict(kind="cycle", flow="stokes", root=root, nu=nu)
        return dict(kind="request", flow="stokes", root=root, nu=nu, precision=rng.choice(["mixed", "mixed", "fp64"]),
                    reduction=1e-8, restart=30)
    dim, elem = rng.choice([2, 3]), rng.choice([1, 2])
    # below about 1e-2 the damped-Jacobi multigrid of many meshes stops at the
    # iteration cap, in every precision
    c = dict(kind=kind, dim=dim, elem=elem, eps=round(10.0 ** rng.uniform(-1.7, 0.0), 5))
    if kind == "apply":
        c["root"], c["refine"] = _draw_mesh(rng, dim, elem, _RANGE_APPLY, 0)
        c["dtype"] = rng.choice(["fp64", "fp32"])
        return c
    if kind == "assemble":
        c["root"], c["refine"] = _draw_mesh(rng, dim, elem, _RANGE_NOALLOC, 0)
        return c
    small = kind in ("batch", "steps")
    ranges = {k: (lo, hi // 2 if small else hi) for k, (lo, hi) in _RANGE.items()}
    c["root"], c["refine"] = _draw_mesh(rng, dim, elem, ranges, 1)
    c["levels"] = _levels(dim, c["root"], c["refine"])
    if kind == "cycle":
        return c
    c.update(precision=rng.choice(["mixed", "mixed", "fp64"]), reduction=1e-8, restart=30)
    if kind == "batch":
        c.update(precision="mixed", n=rng.randint(2, 8))
    if kind == "steps":
        c.update(scheme=rng.choice(["crank_nicolson", "backward_euler"]), tau=rng.choice([0.005, 0.01, 0.02]))
    return c


# -------------------------------------------------------------- preparation --
@functools.lru_cache(maxsize=1)
def _context():
    return m.Context(0)


@functools.lru_cache(maxsize=4)
def _disc(geometry, root, refine, levels, kind, elem):
    """the mesh hierarchy with its spaces: a program makes it once per mesh"""
    return m.Discretization(geometry, root, refine, levels, kind, elem, ctx=_context())


class _Dev:
    """a device array of the framework, for torch.as_tensor (the tensor keeps
    this object, and with it the array's owner)"""

    def __init__(self, owner, ptr, n, typestr="<f8"):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=(int(n),), typestr=typestr, version=3)


def _tensor(v):
    return torch.as_tensor(_Dev(v, v.ptr.value, v.n, "<f8" if v.dtype == np.float64 else "<f4"), device="cuda")


def _solution(p):
    sol, rhs = ctypes.c_void_p(), ctypes.c_void_p()
    check(lib.pm_problem_solution_dev(p.handle, ctypes.byref(sol), ctypes.byref(rhs)), p.ctx.handle)
    return torch.as_tensor(_Dev(p, sol.value, p.size()[0]), device="cuda")


def _database(case):
    db = m.ParameterDatabase.solve_path_database()
    db["solver_type"] = "iterative"
    db["iterative_solver_type"] = "fgmres"
    db["preconditioner"] = "multigrid"
    db["residual_tolerance"] = 0.0
    db["residual_reduction"] = case.get("reduction", 1e-8)
    db["max_n_iterations"] = 500
    db["gmres_restart"] = case.get("restart", 30)
    db["gpu_precision"] = case.get("precision", "fp64")
    if "dim" in case:
        db["multigrid_n_levels"] = case.get("levels", 2)
        db["multigrid_smoother"] = "jacobi"
        db["multigrid_smoother_coarse"] = "direct_solve"
        db["jacobi_damp"] = 0.8
        db["multigrid_n_pre_smooth"] = 2
        db["multigrid_n_post_smooth"] = 2
    else:
        db["multigrid_n_levels"] = 3
        db["multigrid_smoother"] = "nodal_vanka"
        db["multigrid_smoother_coarse"] = "nodal_vanka_jacobi"
        db["multigrid_vanka_damp_factor"] = 0.8
        db["multigrid_n_pre_smooth"] = 1
        db["multigrid_n_post_smooth"] = 1
    return db


def _coefficients(case, seed, k=0):
    """diffusion and convection of the seed's problem: eps up to a fifth above the
    case's, each component of b up to a third below (1, 0.5, 0.25)"""
    r = np.random.RandomState((seed * 17 + k) % (1 << 31))
    eps = case["eps"] * (1.0 + 0.2 * r.uniform())
    b = np.array([1.0, 0.5, 0.25][: case["dim"]]) * (1.0 - r.uniform(0.0, 1.0 / 3.0, case["dim"]))
    return float(eps), tuple(float(v) for v in b)


def _vector(seed, n):
    return np.random.RandomState(seed % (1 << 31)).standard_normal(n)


def _cd_disc(case, levels):
    geometry = m.GEO_SQUARE_QUAD if case["dim"] == 2 else m.GEO_CUBE_HEXA
    return _disc(geometry, case["root"], case["refine"], levels, m.KIND_CD, case["elem"])


def _cd_problem(case, seed, levels, k=0):
    db = _database(case)
    if case["kind"] in ("apply", "assemble"):
        db["preconditioner"] = "no_preconditioner"
    eps, b = _coefficients(case, seed, k)
    return m.ConvectionDiffusion(_context(), _cd_disc(case, levels), m.cd_coeffs(eps, b, 0.0, True), db,
                                 quad_points=3)


def _flow_disc(case):
    # 4 * root cubes per side, each 6 tetrahedra, three levels
    rq = workloads.stokes_request(4 * case["root"])
    return _disc(rq["geometry"], rq["root_n"], rq["n_refine"], rq["n_levels"], rq["kind"], rq["elem"])


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    state = dict(kind=kind, ctx=ctx)
    if kind == "apply":
        p = _cd_problem(case, seed, 1)
        p.assemble()
        A = p.matrix(-1)
        dtype = np.float64 if case["dtype"] == "fp64" else np.float32
        if dtype == np.float32:
            A.make_fp32()
        else:
            A.make_sliced64()
        n = A.n_rows
        state.update(problem=p, A=A, x=m.DeviceVector.from_numpy(ctx, _vector(seed, n).astype(dtype)),
                     y=m.DeviceVector(ctx, n, dtype), fp32=dtype == np.float32)
        state["out"] = [_tensor(state["y"])]
    elif kind == "assemble":
        p = _cd_problem(case, seed, 1)
        vals = m.DeviceVector(ctx, p.matrix(-1).nnz)
        rhs = m.DeviceVector(ctx, p.size()[0])
        state.update(problem=p, vals=vals, rhs=rhs, out=[_tensor(vals), _tensor(rhs)])
    elif kind == "cycle":
        flow = case.get("flow") == "stokes"
        if flow:
            p = m.StokesProblem(ctx, _flow_disc(case), case["nu"], _database(case))
        else:
            p = _cd_problem(case, seed, case["levels"])
        p.assemble()
        solver = p.solver()
        solver.update_matrix(p.matrix(-1))
        n = p.size()[0]
        z = _vector(seed, n)
        if flow:  # a residual: exact zeros in the Dirichlet rows
            nv, na, _ = p.blocks()
            for b in range(3):
                z[b * nv + na:(b + 1) * nv] = 0.0
        else:
            z[p.size()[1]:] = 0.0
        state.update(problem=p, solver=solver, z=m.DeviceVector.from_numpy(ctx, z), r=m.DeviceVector(ctx, n))
        state["out"] = [_tensor(state["r"])]
    elif kind == "linearise":
        db = _database(case)
        db.add("example", -3)
        db.add("problem_type", 5)
        p = m.StokesProblem(ctx, _flow_disc(case), case["nu"], db)
        p.assemble_linear_terms()
        n = p.size()[0]
        p.set_solution(_vector(seed, n))  # the velocity of the last iterate
        A = p.matrix(-1)
        state.update(problem=p, A=A, x=m.DeviceVector.from_numpy(ctx, _vector(seed + 1, n)),
                     y=m.DeviceVector(ctx, n))
        state["out"] = [_tensor(state["y"])]
    elif kind == "request":
        if case.get("flow") == "stokes":
            # viscosity within 10 per cent of the case's
            nu = case["nu"] * (1.0 + 0.1 * np.random.RandomState(seed % (1 << 31)).uniform(-1.0, 1.0))
            p = m.StokesProblem(ctx, _flow_disc(case), float(nu), _database(case))
        else:
            p = _cd_problem(case, seed, case["levels"])
        state.update(problem=p, out=[_solution(p)])
    elif kind == "batch":
        ps = [_cd_problem(case, seed, case["levels"], k) for k in range(case["n"])]
        state.update(problems=ps, out=[_solution(p) for p in ps])
    else:
        db = _database(case)
        db.merge(m.ParameterDatabase.default_time_database())
        db["time_discretization"] = case["scheme"]
        db["time_step_length"] = case["tau"]
        eps, b = _coefficients(case, seed)
        p = m.TimeConvectionDiffusion(ctx, _cd_disc(case, case["levels"]), m.cd_coeffs(eps, b, 0.0, True), db,
                                      quad_points=3)
        state.update(problem=p, out=[_solution(p)])
    ctx.synchronize()
    return state


def run(state):
    kind = state["kind"]
    if kind == "apply":
        if state["fp32"]:
            state["A"].apply_f32(state["x"], state["y"])
        else:
            state["A"].apply(state["x"], state["y"])
    elif kind == "assemble":
        state["problem"].assemble_level_noalloc(0, state["vals"], state["rhs"])
    elif kind == "cycle":
        state["solver"].apply_preconditioner(state["z"], state["r"])
    elif kind == "linearise":
        state["problem"].assemble_nonlinear_term()
        state["A"].apply(state["x"], state["y"])
    elif kind == "request":
        p = state["problem"]
        p.reset_solution()
        p.assemble()
        p.solve()
    elif kind == "batch":
        for p in state["problems"]:
            p.reset_solution()
            p.assemble()
        m.solve_batched(state["problems"], slots=8)
    else:
        p = state["problem"]
        p.assemble_initial_time()
        for _ in range(2):
            p.next_time_step()
            p.assemble()
            p.solve()
    return state["out"]


# ------------------------------------------------------------------- work ---
def _cd_size(dim, elem, cells):
    """unknowns and stored entries of the Qk matrix on cells^dim cells: an
    inner vertex couples to 2k + 1 nodes per direction, an inner midpoint to 3"""
    n = (elem * cells + 1) ** dim
    active = (elem * cells - 1) ** dim
    per_dir = 3 * (cells - 1) if elem == 1 else 5 * (cells - 1) + 3 * cells
    return n, per_dir ** dim + n - active


def _flow_size(cubes):
    """unknowns and (about) stored entries of the combined P2/P1 matrix; the
    24^3 mesh holds 14.18 million entries for its 368,572 unknowns"""
    n = 3 * (2 * cubes + 1) ** 3 + (cubes + 1) ** 3
    return n, 14.18e6 * (cubes / 24.0) ** 3


def _all_levels(case):
    if "dim" in case:
        cells = case["root"] << case["refine"]
        return [_cd_size(case["dim"], case["elem"], cells >> l) for l in range(case.get("levels", 1))]
    return [_flow_size(4 * case["root"] >> l) for l in range(3)]


def work(case):
    """bytes of the matrices, vectors and mesh that a pass reads or writes, each
    once (a solve's iterations read the matrices again; their number depends on
    the data), and the multiply-adds of the sums over those entries, twice"""
    kind = case["kind"]
    levels = _all_levels(case)
    n, nnz = levels[0]
    if kind == "apply":
        eb = 8 if case["dtype"] == "fp64" else 4
        return dict(bytes=nnz * (eb + 4) + 4 * (n + 1) + 2 * n * eb, flops=2 * nnz)
    total_n, total_nnz = sum(v[0] for v in levels), sum(v[1] for v in levels)
    if kind == "cycle":
        sweeps = 5 if "dim" in case else 3
        return dict(bytes=12 * total_nnz + 4 * total_n + 16 * n, flops=2 * sweeps * total_nnz)
    if "dim" in case:
        cells = [((case["root"] << case["refine"]) >> l) ** case["dim"] for l in range(len(levels))]
        nloc = (case["elem"] + 1) ** case["dim"]
        # one coefficient-weighted sum of 6 (2D) or 10 (3D) reference matrices per cell
        flops = sum(cells) * nloc ** 2 * 2 * (6 if case["dim"] == 2 else 10)
        nbytes = 8 * total_nnz + 8 * total_n + sum(cells) * 8 * case["dim"] * 2 ** case["dim"]
    else:
        cells = [6 * (4 * case["root"] >> l) ** 3 for l in range(3)]
        flops = sum(cells) * (100 * 36 + 120 * 3) * 2
        nbytes = 8 * total_nnz + 8 * total_n + sum(cells) * 96
    times = dict(batch=case.get("n", 1), steps=2).get(kind, 1)
    if kind not in ("assemble", "linearise"):  # the solve: the new matrices read, the solution written
        nbytes += 12 * total_nnz + 8 * n
        flops += 2 * total_nnz
    return dict(bytes=times * nbytes, flops=times * flops)


# ------------------------------------------------- plain 64-bit reference ---
# The same discrete problems in numpy / torch: the cells in the order of the
# regular refinement (child i of a cell starts at its vertex i), the unknowns
# in the order in which the cells first touch them, inner ones before the
# Dirichlet ones, the element integrals on the tensor Gauss rule with three
# points per direction.
_HEX_CHILD = [[0, 8, 12, 11, 15, 16, 26, 24], [1, 9, 12, 8, 13, 19, 26, 16], [2, 10, 12, 9, 17, 22, 26, 19],
              [3, 11, 12, 10, 20, 24, 26, 22], [4, 23, 25, 14, 15, 24, 26, 16], [5, 14, 25, 18, 13, 16, 26, 19],
              [6, 18, 25, 21, 17, 19, 26, 22], [7, 21, 25, 23, 20, 22, 26, 24]]
_HEX_MEAN = [[0, 1], [1, 2], [2, 3], [0, 3], [0, 1, 2, 3], [1, 5], [4, 5], [0, 4], [0, 1, 4, 5], [2, 6], [5, 6],
             [1, 2, 5, 6], [3, 7], [6, 7], [2, 3, 6, 7], [4, 7], [0, 3, 4, 7], [4, 5, 6, 7], list(range(8))]
_QUAD_CHILD = [[0, 4, 8, 7], [1, 5, 8, 4], [2, 6, 8, 5], [3, 7, 8, 6]]
_QUAD_MEAN = [[0, 1], [1, 2], [2, 3], [0, 3], [0, 1, 2, 3]]


def _ref_cells(dim, root, refine):
    """integer vertex coordinates (cells x vertices x dim) per refinement, and the scale"""
    unit = 2 << refine
    corner = [[0, 0], [1, 0], [1, 1], [0, 1]]
    if dim == 3:
        corner = [c + [k] for k in (0, 1) for c in corner]
    grid = np.stack(np.meshgrid(*[np.arange(root)] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
    out = [(grid[:, None, :] + np.array(corner)[None]) * unit]
    child, mean = (_QUAD_CHILD, _QUAD_MEAN) if dim == 2 else (_HEX_CHILD, _HEX_MEAN)
    for _ in range(refine):
        v = out[-1]
        pts = np.concatenate([v] + [v[:, s].mean(1, keepdims=True).astype(np.int64) for s in mean], 1)
        out.append(pts[:, np.array(child)].reshape(-1, v.shape[1], dim))
    return out, unit * root


def _ref_space(v, scale, dim, k):
    """dofmap (cells x local), the node of every unknown, number of inner unknowns"""
    axes = [v[:, 1] - v[:, 0], v[:, 3] - v[:, 0]] + ([v[:, 4] - v[:, 0]] if dim == 3 else [])
    steps = np.stack(np.meshgrid(*[np.arange(k + 1)] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
    nodes = v[:, None, 0] + sum(a[:, None, :] * steps[None, :, d, None] // k for d, a in enumerate(axes))
    key = np.zeros(nodes.shape[:2], dtype=np.int64)
    for d in range(dim):
        key = key * (scale + 1) + nodes[..., d]
    _, first, inv = np.unique(key.ravel(), return_index=True, return_inverse=True)
    xyz = nodes.reshape(-1, dim)[first]
    outer = ((xyz == 0) | (xyz == scale)).any(1)
    order = np.lexsort((first, outer))
    number = np.empty_like(order)
    number[order] = np.arange(order.size)
    return number[inv].reshape(key.shape), xyz[order], int((~outer).sum())


def _ref_basis(k, x):
    if k == 1:
        return np.stack([(1 - x) / 2, (1 + x) / 2], -1), np.stack([0 * x - 0.5, 0 * x + 0.5], -1)
    return (np.stack([x * (x - 1) / 2, 1 - x * x, x * (x + 1) / 2], -1), np.stack([x - 0.5, -2 * x, x + 0.5], -1))


def _ref_tensor(parts):
    """tensor products in the local order (first direction fastest)"""
    out = parts[0]
    for p in parts[1:]:
        out = p[..., :, None] * out[..., None, :]
        out = out.reshape(out.shape[:-2] + (-1,))
    return out


class _Level:
    """one level: unknowns, sorted pattern and (with coefficients) the matrix"""

    def __init__(self, v, scale, dim, k, device):
        self.v, self.scale, self.dim, self.k, self.device = v, scale, dim, k, device
        self.dofs, self.nodes, self.n_active = _ref_space(v, scale, dim, k)
        self.n = len(self.nodes)

    def assemble(self, eps, b, mass=False):
        dim, k, dev = self.dim, self.k, self.device
        g = np.array([-math.sqrt(0.6), 0.0, math.sqrt(0.6)])
        w1 = np.array([5.0, 8.0, 5.0]) / 9.0
        pts = np.stack(np.meshgrid(*[g] * dim, indexing="ij")[::-1], -1).reshape(-1, dim)
        w = _ref_tensor([w1] * dim)
        vals = [_ref_basis(k, pts[:, d]) for d in range(dim)]
        phi = torch.tensor(_ref_tensor([f for f, _ in vals]), device=dev)
        dphi = torch.tensor(np.stack([_ref_tensor([vals[d][1 if d == a else 0] for d in range(dim)])
                                      for a in range(dim)]), device=dev)
        w = torch.tensor(w, device=dev)
        x = torch.tensor(self.v / self.scale, device=dev)
        edges = [1, 3, 4][:dim]
        J = torch.stack([(x[:, e] - x[:, 0]) / 2 for e in edges], -1)  # columns: directions
        x0 = x[:, 0] + J.sum(-1)
        det, G = torch.linalg.det(J).abs(), torch.linalg.inv(J).transpose(1, 2)
        if mass:
            M = torch.einsum("q,qi,qj->ij", w, phi, phi)
            K = det[:, None, None] * M
        else:
            S = torch.einsum("q,aqi,bqj->abij", w, dphi, dphi)
            C = torch.einsum("q,qi,aqj->aij", w, phi, dphi)
            Gab = eps * torch.einsum("cda,cdb->cab", G, G)
            bG = torch.einsum("d,cda->ca", torch.tensor(b, dtype=torch.float64, device=dev), G)
            K = det[:, None, None] * (torch.einsum("cab,abij->cij", Gab, S) + torch.einsum("ca,aij->cij", bG, C))
        xq = x0[:, None] + torch.einsum("cda,qa->cqd", J, torch.tensor(pts, device=dev))
        s, c = torch.sin(math.pi * xq), torch.cos(math.pi * xq)
        u = s.prod(-1)
        f = eps * dim * math.pi ** 2 * u
        for d in range(dim):
            f = f + b[d] * math.pi * c[..., d] * torch.cat([s[..., :d], s[..., d + 1:]], -1).prod(-1)
        F = torch.einsum("c,q,cq,qi->ci", det, w, f, phi)
        dofs = torch.tensor(self.dofs, device=dev)
        na, n = self.n_active, self.n
        rhs = torch.zeros(n, dtype=torch.float64, device=dev).index_add(0, dofs.ravel(), F.ravel())
        rhs[na:] = 0.0
        nb = dofs.shape[1]
        key = (dofs[:, :, None] * n + dofs[:, None, :]).expand(-1, nb, nb).ravel()
        keep = key < na * n
        diag = torch.arange(na, n, device=dev)
        key, val = torch.cat([key[keep], diag * n + diag]), torch.cat([K.ravel()[keep], torch.ones_like(diag).double()])
        key, inv = torch.unique(key, return_inverse=True)
        self.vals = torch.zeros(key.numel(), dtype=torch.float64, device=dev).index_add(0, inv, val)
        self.rows, self.cols = key // n, key % n
        return rhs

    def apply(self, x, vals=None):
        vals = self.vals if vals is None else vals
        return torch.zeros_like(x).index_add(0, self.rows, vals * x[self.cols])

    def solve(self, rhs):
        """dense solve on the inner unknowns (zero Dirichlet values)"""
        na = self.n_active
        D = torch.zeros(na, na, dtype=torch.float64, device=rhs.device)
        keep = (self.rows < na) & (self.cols < na)
        D[self.rows[keep], self.cols[keep]] = self.vals[keep]
        out = torch.zeros_like(rhs)
        out[:na] = torch.linalg.solve(D, rhs[:na])
        return out

    def prolongation(self, fine):
        """(rows, columns, values) from this level to `fine` (inner rows only)"""
        nchild = 2 ** self.dim
        parent = np.arange(len(fine.v)) // nchild
        pv = self.v[parent]
        _, first = np.unique(fine.dofs.ravel(), return_index=True)
        cell = first // fine.dofs.shape[1]
        pv = pv[cell]
        J = np.stack([pv[:, e] - pv[:, 0] for e in [1, 3, 4][: self.dim]], -1).astype(float)
        xi = 2 * np.linalg.solve(J, (fine.nodes - pv[:, 0])[..., None].astype(float))[..., 0] - 1
        val = _ref_tensor([_ref_basis(self.k, xi[:, d])[0] for d in range(self.dim)])
        rows = np.repeat(np.arange(fine.n), val.shape[1])
        cols = self.dofs[parent[cell]].ravel()
        keep = (val.ravel() != 0) & (rows < fine.n_active)
        dev = self.device
        return [torch.tensor(a[keep], device=dev) for a in (rows, cols, val.ravel())]


def _ref_levels(case, count):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    cells, scale = _ref_cells(case["dim"], case["root"], case["refine"])
    return [_Level(v, scale, case["dim"], case["elem"], device) for v in cells[len(cells) - count:]]


def _ref_cycle(levels, z):
    """V(2,2) with damped Jacobi 0.8 and the direct solve on the coarsest level"""
    def smooth(lv, b, x):
        d = torch.zeros_like(b)
        on = lv.rows == lv.cols
        d[lv.rows[on]] = lv.vals[on]
        for _ in range(2):
            x = x + 0.8 * (b - lv.apply(x)) / d
        return x

    def cycle(l, b):
        lv = levels[l]
        if l == 0:
            return lv.solve(b)
        x = smooth(lv, b, torch.zeros_like(b))
        rows, cols, val = levels[l - 1].prolongation(lv)
        r = b - lv.apply(x)
        rc = torch.zeros(levels[l - 1].n, dtype=b.dtype, device=b.device).index_add(0, cols, val * r[rows])
        rc[levels[l - 1].n_active:] = 0.0
        e = cycle(l - 1, rc)
        x = x.index_add(0, rows, val * e[cols])
        return smooth(lv, b, x)

    return cycle(len(levels) - 1, z)


def exact(case, seed):
    """the outputs of run() in 64 bits; None for the Stokes and Navier-Stokes
    cases and for systems too large for a dense solve in a few seconds"""
    kind = case["kind"]
    if "dim" not in case:
        return None
    inner = (case["elem"] * (case["root"] << case["refine"]) - 1) ** case["dim"]
    if kind in ("request", "batch", "steps") and inner * (case.get("n", 1) ** (1 / 3)) > 17000:
        return None
    eps, b = _coefficients(case, seed)
    if kind == "cycle":
        levels = _ref_levels(case, case["levels"])
        for lv in levels:
            lv.assemble(eps, b)
        z = _vector(seed, levels[-1].n)
        z[levels[-1].n_active:] = 0.0
        return [_ref_cycle(levels, torch.tensor(z, device=levels[-1].device))]
    lv = _ref_levels(case, 1)[0]
    if kind == "batch":
        return [lv.solve(lv.assemble(*_coefficients(case, seed, k))) for k in range(case["n"])]
    rhs = lv.assemble(eps, b)
    if kind == "assemble":
        return [lv.vals, rhs]
    if kind == "apply":
        x = torch.tensor(_vector(seed, lv.n), device=lv.device)
        if case["dtype"] == "fp32":
            x = x.float().double()
        return [lv.apply(x)]
    if kind == "request":
        return [lv.solve(rhs)]
    # (M + theta tau A) u1 = M u0 - (1 - theta) tau A u0 + tau f, u0 = 0
    A = lv.vals
    lv.assemble(eps, b, mass=True)
    M, tau = lv.vals, case["tau"]
    theta = 0.5 if case["scheme"] == "crank_nicolson" else 1.0
    lv.vals = M + theta * tau * A
    u = torch.zeros_like(rhs)
    for _ in range(2):
        u = lv.solve(lv.apply(u, M) - (1 - theta) * tau * lv.apply(u, A) + tau * rhs)
    return [u]
