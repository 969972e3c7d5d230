"""The nodal Vanka sweep with one kernel per colour over packed patches
(nodal_sliced 8, the default) against the sweep over the CSR rows (nodal_sliced 0):
patches of 14 to 75 nodes, one patch per colour up to a hundred, as the fine
levels' smoother and, additive and in colours, in the coarse level's loop with its
stopping test never, at once and in between.

Tolerance: one cycle within rounding, 1e-12 in FP64 and 1e-5 in FP32, as the sweep
over sliced rows is held to."""
import numpy as np
import pytest

import mymoonmd_gb300 as m
from test_gpu_stokes import rel, stokes_db

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("coarse,stop", [("nodal_vanka_jacobi", 0.0), ("nodal_vanka", 0.0), ("nodal_vanka", 1e30),
                                         ("nodal_vanka", 0.1)])
@pytest.mark.parametrize("root,refine", [(1, 1), (2, 1), (1, 2), (3, 2)])
def test_cycle_of_packed_patches(ctx, root, refine, coarse, stop, precision):
    db = stokes_db(refine + 1, "nodal_vanka", 0.8, coarse=coarse, precision=precision)
    db["multigrid_coarse_max_n_iterations"] = 4
    db["multigrid_coarse_residual"] = stop
    out = {}
    try:
        for sliced in (8, 0):
            ctx.set_option("nodal_sliced", sliced)
            disc = m.Discretization(m.GEO_CUBE_TETRA, root, refine, refine + 1, m.KIND_STOKES, 12)
            prob = m.StokesProblem(ctx, disc, 1.0, db)
            prob.assemble()
            prob.solver().update_matrix(prob.matrix(-1))
            z = np.random.default_rng(5).standard_normal(prob.size()[0])
            zd, rd = m.DeviceVector.from_numpy(ctx, z), m.DeviceVector(ctx, z.size)
            for _ in range(2):  # the second pass finds the first one's buffers
                prob.solver().apply_preconditioner(zd, rd)
            out[sliced] = rd.numpy()
            prob.close()
            disc.close()
    finally:
        ctx.set_option("nodal_sliced", 8)
    assert rel(out[8], out[0]) <= (1e-12 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("coarse", ["nodal_vanka_jacobi", "nodal_vanka"])
@pytest.mark.parametrize("root,refine", [(3, 1), (5, 1), (7, 1), (4, 2)])
def test_fp64_colours_around_one_block_per_sm(ctx, root, refine, coarse):
    """colours of up to 8, 27, 64 and 64 patches: on clusters of three blocks up to a
    third of the SMs, on one block per patch above it, both in one sweep"""
    test_cycle_of_packed_patches(ctx, root, refine, coarse, 0.0, "fp64")
