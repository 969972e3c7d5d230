"""The dense inverse behind the direct coarse solve, by panels of 8 (FP64) and
16 (FP32) columns on one to four rows per thread, at the edges of its panels, warps
and size classes; matrices with condition number 10 whose
rows are shuffled, so that every panel swaps rows.

Tolerance: the rounding errors of n elimination steps add up like sqrt(n) u
times the condition number; 20 sqrt(n) 10 u of the solution's norm."""
import numpy as np
import pytest

import mymoonmd_gb300 as m

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 31, 32, 33, 64, 81, 96, 127, 128, 129, 160, 169, 225, 257, 320]
U = {"fp64": 2.0 ** -53, "mixed": 2.0 ** -24}


def system(n):
    r = np.random.default_rng(n)
    q, _ = np.linalg.qr(r.standard_normal((n, n)))
    w, _ = np.linalg.qr(r.standard_normal((n, n)))
    a = (q * np.geomspace(1.0, 10.0, n)) @ w
    return a[r.permutation(n)], r.standard_normal(n)


def csr(ctx, a):
    n = len(a)
    return m.FEMatrix.from_csr(ctx, np.arange(n + 1) * n, np.tile(np.arange(n), n), a.ravel())


def close(x, ref, n, precision):
    return np.linalg.norm(x - ref) <= 20 * np.sqrt(n) * 10 * U[precision] * np.linalg.norm(ref)


@pytest.mark.parametrize("n", SIZES + [343, 640, 641, 1023, 1024, 1025, 2048, 2049])
def test_direct_solve(ctx, n):
    a, b = system(n)
    A = csr(ctx, a)
    s = m.Solver(ctx, {"solver_type": "direct"})
    s.update_matrix(A)
    x = np.zeros(n)
    s.solve(b, x)
    s.close()
    A.close()
    assert close(x, np.linalg.solve(a, b), n, "fp64")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", SIZES + [343, 639, 640, 641])
def test_coarse_solve_of_a_cycle(ctx, n, precision):
    """two levels joined by the identity, no smoothing: the cycle is the coarse
    solve, in FP32 for the mixed form"""
    a, b = system(n)
    A, C = csr(ctx, a), csr(ctx, a)
    s = m.Solver(ctx, {"solver_type": "iterative", "iterative_solver_type": "fgmres", "preconditioner": "multigrid",
                       "multigrid_n_levels": 2, "multigrid_smoother": "jacobi",
                       "multigrid_smoother_coarse": "direct_solve", "multigrid_n_pre_smooth": 0,
                       "multigrid_n_post_smooth": 0, "gpu_precision": precision})
    eye = (np.arange(n + 1), np.arange(n), np.ones(n))
    s.set_multigrid_level(0, 2, C, eye)
    s.set_multigrid_level(1, 2, A)
    s.update_matrix(A)
    z, r = m.DeviceVector.from_numpy(ctx, b), m.DeviceVector(ctx, n)
    s.apply_preconditioner(z, r)
    x = r.numpy()
    s.close()
    A.close()
    C.close()
    assert close(x, np.linalg.solve(a, b), n, precision)


def test_singular_matrix_is_refused(ctx):
    a, b = system(40)
    a[:, 17] = a[:, 3]
    a[:, 3] = 0.0
    A = csr(ctx, a)
    s = m.Solver(ctx, {"solver_type": "direct"})
    s.update_matrix(A)
    with pytest.raises(m.PmError):
        s.solve(b, np.zeros(40))
    s.close()
    A.close()
