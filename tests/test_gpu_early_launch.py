"""Launches with programmatic stream serialization (option pdl 1) against plain ones
(pdl 0): the same kernels in the same order, so the same bits, cycle after cycle, on
hierarchies whose small levels have several launches in flight; and the coarse inverse,
whose panels are launched that way."""
import numpy as np
import pytest

import mymoonmd_gb300 as m
from test_gpu_coarse_inverse import csr, system
from test_gpu_stokes import stokes_db

pytestmark = pytest.mark.gpu


def cd_db(precision, levels):
    db = m.ParameterDatabase.solve_path_database()
    db["solver_type"] = "iterative"
    db["iterative_solver_type"] = "fgmres"
    db["preconditioner"] = "multigrid"
    db["gpu_precision"] = precision
    db["multigrid_n_levels"] = levels
    db["multigrid_smoother"] = "jacobi"
    db["multigrid_smoother_coarse"] = "direct_solve"
    db["jacobi_damp"] = 0.8
    db["multigrid_n_pre_smooth"] = 2
    db["multigrid_n_post_smooth"] = 3
    return db


def cycles(ctx, prob, count=30):
    s = prob.solver()
    s.update_matrix(prob.matrix(-1))
    n = prob.size()[0]
    out = []
    for k in range(count):
        z, r = m.DeviceVector.from_numpy(ctx, np.random.default_rng(k).standard_normal(n)), m.DeviceVector(ctx, n)
        s.apply_preconditioner(z, r)
        s.apply_preconditioner(r, z)
        out.append(z.numpy())
    return np.array(out)


def both(ctx, run):
    try:
        ctx.set_option("pdl", 0)
        plain = run()
    finally:
        ctx.set_option("pdl", 1)
    return plain, run()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("geometry,elem,refine,levels", [
    (m.GEO_SQUARE_QUAD, 1, 4, 3), (m.GEO_SQUARE_QUAD, 1, 6, 5), (m.GEO_SQUARE_QUAD, 2, 5, 4),
    (m.GEO_CUBE_HEXA, 1, 3, 2), (m.GEO_CUBE_HEXA, 1, 4, 4), (m.GEO_CUBE_HEXA, 2, 3, 3), (m.GEO_CUBE_HEXA, 2, 4, 3)])
def test_cycles_have_the_bits_of_plain_launches(ctx, geometry, elem, refine, levels, precision):
    b = (1.0, 0.5, 0.25)[:2 if geometry == m.GEO_SQUARE_QUAD else 3]
    disc = m.Discretization(geometry, 1, refine, levels, m.KIND_CD, elem, ctx=ctx)
    prob = m.ConvectionDiffusion(ctx, disc, m.cd_coeffs(0.1, b, 0.0, True), cd_db(precision, levels), quad_points=3)
    prob.assemble()
    plain, early = both(ctx, lambda: cycles(ctx, prob))
    prob.close()
    disc.close()
    assert np.isfinite(plain).all() and np.array_equal(plain, early)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_stokes_cycles_have_the_bits_of_plain_launches(ctx, precision):
    db = stokes_db(3, "nodal_vanka", 0.8, coarse="nodal_vanka_jacobi", precision=precision)
    disc = m.Discretization(m.GEO_CUBE_TETRA, 2, 2, 3, m.KIND_STOKES, 12)
    prob = m.StokesProblem(ctx, disc, 1.0, db)
    prob.assemble()
    plain, early = both(ctx, lambda: cycles(ctx, prob, 10))
    prob.close()
    disc.close()
    assert np.isfinite(plain).all() and np.array_equal(plain, early)


@pytest.mark.parametrize("n", [9, 81, 225, 343, 1025])
def test_direct_solves_have_the_bits_of_plain_launches(ctx, n):
    a, b = system(n)
    A = csr(ctx, a)

    def run():
        out = []
        for _ in range(5):
            s = m.Solver(ctx, {"solver_type": "direct"})
            s.update_matrix(A)
            x = np.zeros(n)
            s.solve(b, x)
            s.close()
            out.append(x)
        return np.array(out)

    plain, early = both(ctx, run)
    A.close()
    assert (plain == plain[0]).all() and np.array_equal(plain, early)


@pytest.mark.parametrize("fp32", [False, True])
def test_product_right_after_new_values(ctx, fp32):
    """the first product after the sliced values were filled, launch after launch"""
    disc = m.Discretization(m.GEO_CUBE_HEXA, 1, 4, 1, m.KIND_CD, 2, ctx=ctx)
    db = cd_db("fp64", 1)
    db["preconditioner"] = "no_preconditioner"
    prob = m.ConvectionDiffusion(ctx, disc, m.cd_coeffs(0.1, (1.0, 0.5, 0.25), 0.0, True), db, quad_points=3)
    prob.assemble()
    A = prob.matrix(-1)
    A.make_sliced64()
    v, n = A.values(), A.n_rows
    dtype = np.float32 if fp32 else np.float64
    x = m.DeviceVector.from_numpy(ctx, np.random.default_rng(1).standard_normal(n).astype(dtype))
    y = m.DeviceVector(ctx, n, dtype)

    def product(scale):
        A.set_values(scale * v)  # a power of two: the products scale exactly
        if fp32:
            A.make_fp32()
            A.apply_f32(x, y)
        else:
            A.apply(x, y)
        return y.numpy()

    one = product(1.0)
    for k in range(1, 40):
        assert np.array_equal(product(2.0 ** (k % 7)), one * dtype(2.0 ** (k % 7)))
    prob.close()
    disc.close()
