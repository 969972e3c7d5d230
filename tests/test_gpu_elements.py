"""Element kernels of the convection-diffusion assembly: the factored kernels
(direction by direction on axis-aligned quadrilaterals and hexahedra, reference
tensors elsewhere) against the per-quadrature-point loop, on the generated mesh,
on sheared cells and on a mesh where only some cells are sheared, for cell counts
around the kernels' cells per block (8 to 64).

Tolerance: an entry sums at most 8 cells x 64 points x 4 products; each form
rounds within 512 x 1.1e-16 of the sum of magnitudes (6e-14), so two forms agree
within 2e-13 of the largest entry (the sums of magnitudes stay below twice it
for the coefficients used)."""
import numpy as np
import pytest

import mymoonmd_gb300 as m

pytestmark = pytest.mark.gpu

TOL = 2e-13


def assembled(ctx, disc, cf, quad, loop, verts):
    db = m.ParameterDatabase.solve_path_database()
    db["solver_type"] = "iterative"
    db["iterative_solver_type"] = "jacobi"
    db["preconditioner"] = "no_preconditioner"
    db["max_n_iterations"] = 1
    ctx.set_option("assembly_quadrature_loop", loop)
    try:
        p = m.ConvectionDiffusion(ctx, disc, cf, db, quad_points=quad)
        p.run_host(cf, verts, np.zeros(p.size()[0]))
        out = p.matrix(-1).values(), p.rhs()
        p.close()
        return out
    finally:
        ctx.set_option("assembly_quadrature_loop", 0)


@pytest.mark.parametrize("dim,root,refine", [(2, 1, 1), (2, 3, 1), (2, 5, 2), (3, 1, 1), (3, 3, 0), (3, 5, 0)])
@pytest.mark.parametrize("elem,quad", [(1, 2), (1, 3), (2, 3), (2, 4)])
def test_factored_elements_equal_the_quadrature_loop(ctx, dim, root, refine, elem, quad):
    disc = m.Discretization(m.GEO_SQUARE_QUAD if dim == 2 else m.GEO_CUBE_HEXA, root, refine, 1, m.KIND_CD, elem)
    try:
        shear = np.array([[1.0, 0.3, 0.1], [0.0, 1.1, -0.2], [0.05, 0.0, 0.9]])[:dim, :dim]
        flat = disc.cell_vertices(0)
        some = flat.copy()
        some[len(some) // 2:] = some[len(some) // 2:] @ shear.T
        for verts in (None, flat @ shear.T, some):
            arg = None if verts is None else [np.ascontiguousarray(verts)]
            for cf in (m.cd_coeffs(0.3, (1.0, -0.5, 0.25), 0.7, True), m.cd_coeffs(0.0, (0.0, 0.0, 0.0), 1.0, False, 2.0),
                       m.cd_coeffs(0.2, (0.4, 0.1, -0.3), 0.0, poly=[1.0, 2.0, -1.0, 0.5, 0.3, 0.2, 0.1, 0.4, 0.6, 0.7])):
                A, f = assembled(ctx, disc, cf, quad, 0, arg)
                A1, f1 = assembled(ctx, disc, cf, quad, 1, arg)
                assert np.abs(A - A1).max() <= TOL * np.abs(A1).max()
                assert np.abs(f - f1).max() <= TOL * np.abs(f1).max()
    finally:
        disc.close()
