"""Shapes 442 (FP64) and 482 (FP32) of the sliced sweeps pick the steps in flight by the
matrix: every choice gives the bits of the fixed shapes with the same lanes, in
products and in cycles, on long rows (3D Q2) and short ones (3D Q1), small and large.
Values that are no shape stay refused."""
import numpy as np
import pytest

import mymoonmd_gb300 as m
from test_gpu_early_launch import cd_db

pytestmark = pytest.mark.gpu
OPTION = {"fp64": "fp64_sliced_spmv", "mixed": "fp32_sliced_spmv"}
CHOSEN = {"fp64": 442, "mixed": 482}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("elem,root,refine,levels", [(2, 1, 2, 2), (2, 1, 4, 3), (2, 7, 2, 3), (1, 1, 4, 3),
                                                     (1, 1, 5, 4), (1, 3, 4, 4)])
def test_bits_of_the_fixed_shapes(ctx, elem, root, refine, levels, precision):
    disc = m.Discretization(m.GEO_CUBE_HEXA, root, refine, levels, m.KIND_CD, elem, ctx=ctx)
    prob = m.ConvectionDiffusion(ctx, disc, m.cd_coeffs(0.1, (1.0, 0.5, 0.25), 0.0, True), cd_db(precision, levels),
                                 quad_points=3)
    prob.assemble()
    s, A, n = prob.solver(), prob.matrix(-1), prob.size()[0]
    s.update_matrix(A)
    A.make_sliced64()
    A.make_fp32()
    dtype = np.float64 if precision == "fp64" else np.float32
    v = np.random.default_rng(3).standard_normal(n)
    z, r = m.DeviceVector.from_numpy(ctx, v), m.DeviceVector(ctx, n)
    x, y = m.DeviceVector.from_numpy(ctx, v.astype(dtype)), m.DeviceVector(ctx, n, dtype)
    out = {}
    try:
        for shape in (441, 481, CHOSEN[precision]):
            ctx.set_option(OPTION[precision], shape)
            s.apply_preconditioner(z, r)
            (A.apply if precision == "fp64" else A.apply_f32)(x, y)
            out[shape] = (r.numpy(), y.numpy())
    finally:
        ctx.set_option(OPTION[precision], CHOSEN[precision])
    prob.close()
    disc.close()
    for shape in (441, 481):
        for a, b in zip(out[shape], out[CHOSEN[precision]]):
            assert np.isfinite(a).all() and np.array_equal(a, b)


@pytest.mark.parametrize("option,values", [("fp64_sliced_spmv", (443, 482, 842)), ("fp32_sliced_spmv", (442, 483, 882))])
def test_other_values_are_refused(ctx, option, values):
    for v in values:
        with pytest.raises(m.PmError):
            ctx.set_option(option, v)
