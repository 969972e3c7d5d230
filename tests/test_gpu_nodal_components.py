"""Nodal Vanka on a matrix whose velocity blocks differ between the components, as a
program gets it that writes its own values into the assembled pattern (an anisotropic
viscosity): the default sweep over packed patches against the sweep over the CSR rows
(nodal_sliced 0), and back to equal blocks.

Tolerance: one cycle within rounding, 1e-12 in FP64 and 1e-5 in FP32, as the packed
sweep is held to on equal blocks."""
import numpy as np
import pytest

import mymoonmd_gb300 as m
from test_gpu_stokes import rel, stokes_db

pytestmark = pytest.mark.gpu
CHANGES = ["one_entry", "component_1", "component_2", "none"]


def write(prob, levels, change):
    """values of every level with the velocity block of one component changed"""
    for l in range(levels):
        A = prob.matrix(l)
        rp, ci = A.structure()
        v = A.values()
        nv = prob.disc.level_info(l, 0)["n_dofs"]
        rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
        if change == "one_entry":
            inner = np.flatnonzero((rows // nv == 1) & (ci // nv == 1) & (np.diff(rp)[rows] > 1) & (rows == ci))
            v[inner[len(inner) // 2]] *= 1.25
        elif change != "none":
            d = int(change[-1])
            v[(rows // nv == d) & (ci // nv == d) & (np.diff(rp)[rows] > 1)] *= 1.5
        A.set_values(v)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("coarse", ["nodal_vanka_jacobi", "nodal_vanka"])
def test_cycle_with_different_velocity_blocks(ctx, coarse, precision):
    db = stokes_db(2, "nodal_vanka", 0.8, coarse=coarse, precision=precision)
    db["multigrid_coarse_max_n_iterations"] = 4
    db["multigrid_coarse_residual"] = 0.0
    out = {}
    try:
        for sliced in (8, 0):
            ctx.set_option("nodal_sliced", sliced)
            disc = m.Discretization(m.GEO_CUBE_TETRA, 2, 1, 2, m.KIND_STOKES, 12)
            prob = m.StokesProblem(ctx, disc, 1.0, db)
            n = prob.size()[0]
            z, r = m.DeviceVector.from_numpy(ctx, np.random.default_rng(5).standard_normal(n)), m.DeviceVector(ctx, n)
            for change in CHANGES:
                prob.assemble()
                write(prob, 2, change)
                prob.solver().update_matrix(prob.matrix(-1))
                prob.solver().apply_preconditioner(z, r)
                out[sliced, change] = r.numpy()
            prob.close()
            disc.close()
    finally:
        ctx.set_option("nodal_sliced", 8)
    tol = 1e-12 if precision == "fp64" else 1e-5
    for change in CHANGES:
        assert rel(out[8, change], out[0, change]) <= tol, change
    for change in CHANGES[:3]:
        assert rel(out[0, change], out[0, "none"]) > tol, change  # the change is seen at all


def test_solve_across_a_change_of_the_blocks(ctx):
    """the captured steps of a solve follow the change: FGMRES on equal, different and
    equal blocks again, against the CSR-row sweep"""
    db = stokes_db(2, "nodal_vanka", 0.8, coarse="nodal_vanka_jacobi", max_it=100, reduction=1e-8, precision="fp64")
    db["multigrid_coarse_max_n_iterations"] = 10
    db["multigrid_coarse_residual"] = 0.1
    out = {}
    try:
        for sliced in (8, 0):
            ctx.set_option("nodal_sliced", sliced)
            disc = m.Discretization(m.GEO_CUBE_TETRA, 2, 1, 2, m.KIND_STOKES, 12)
            prob = m.StokesProblem(ctx, disc, 1.0, db)
            out[sliced] = []
            for change in ("none", "none", "component_1", "component_1", "none"):
                prob.reset_solution()
                prob.assemble()
                write(prob, 2, change)
                prob.solve()
                out[sliced].append((prob.last_info()[0], prob.solution()))
            prob.close()
            disc.close()
    finally:
        ctx.set_option("nodal_sliced", 8)
    for (it8, x8), (it0, x0) in zip(out[8], out[0]):
        assert it8 == it0
        assert rel(x8, x0) <= 1e-7
