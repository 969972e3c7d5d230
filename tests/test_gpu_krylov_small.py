"""FGMRES at the edges of its reductions (two entries per thread and block) and of
its small dense kernels (one warp, two entries of y per lane): the residual that
the rotations report against the residual of the solution that the back
substitution gives, with a well conditioned matrix.

Tolerance: the Arnoldi relation, the basis and the back substitution each hold to
about k u times the condition number (at most 20) of |b|; 100 k u 20 |b|."""
import numpy as np
import pytest

import mymoonmd_gb300 as m

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def system(ctx, n):
    """upper bidiagonal with a spread diagonal: k steps reduce the residual slowly"""
    r = np.random.default_rng(n)
    d = np.linspace(1.0, 10.0, n)
    off = 0.5 * np.ones(n - 1)
    a = np.zeros(2 * n - 1)
    a[0::2], a[1::2] = d, off
    cols = np.zeros(2 * n - 1, dtype=np.int64)
    cols[0::2], cols[1::2] = np.arange(n), np.arange(1, n)
    rp = np.minimum(np.arange(n + 1) * 2, 2 * n - 1)
    b = r.standard_normal(n)

    def apply(x):
        y = d * x
        y[:-1] += off * x[1:]
        return y

    return m.FEMatrix.from_csr(ctx, rp, cols, a), b, apply


def solve(ctx, n, k, restart):
    A, b, apply = system(ctx, n)
    s = m.Solver(ctx, {"solver_type": "iterative", "iterative_solver_type": "fgmres", "preconditioner": "no_preconditioner",
                       "residual_tolerance": 0.0, "residual_reduction": 0.0, "max_n_iterations": k,
                       "gmres_restart": restart, "divergence_factor": 1e9})
    s.update_matrix(A)
    x = np.zeros(n)
    try:
        s.solve(b, x)
    finally:
        info = s.last_info()
        s.close()
        A.close()
    return info, np.linalg.norm(b - apply(x)), np.linalg.norm(b)


@pytest.mark.parametrize("k", [1, 2, 16, 17, 31, 32, 33, 34, 47, 59, 60])
def test_reported_residual_is_that_of_the_solution(ctx, k):
    info, res, nb = solve(ctx, 3000, k, 60)
    assert info[0] == k
    assert abs(info[1] - res) <= 100 * k * U * 20 * nb


@pytest.mark.parametrize("n", [2, 511, 512, 513, 1023, 1025, 304 * 512 - 1, 304 * 512, 304 * 512 + 1, 200001])
def test_sizes_of_the_reductions(ctx, n):
    k = min(8, n - 1)
    info, res, nb = solve(ctx, n, k, 30)
    assert abs(info[1] - res) <= 100 * k * U * 20 * nb


@pytest.mark.parametrize("lens", [(1, 7, 8, 9), (31, 32, 33), (40, 64, 65), (125,)])
def test_jacobi_finds_the_diagonal_of_any_row(ctx, lens):
    """rows of several lengths, the diagonal entry anywhere in the row; a quotient and a product round twice"""
    n = 200
    r = np.random.default_rng(sum(lens))
    rp, cols, vals, d = [0], [], [], r.uniform(1.0, 2.0, n)
    for i in range(n):
        k = lens[i % len(lens)]
        c = sorted([j for j in r.permutation(n) if j != i][:k - 1] + [i])
        cols += c
        vals += [d[i] if j == i else 0.0 for j in c]
        rp.append(len(cols))
    A = m.FEMatrix.from_csr(ctx, rp, cols, vals)
    s = m.Solver(ctx, {"solver_type": "iterative", "iterative_solver_type": "fgmres", "preconditioner": "jacobi",
                       "jacobi_damp": 1.0})
    s.update_matrix(A)
    b = r.standard_normal(n)
    z, y = m.DeviceVector.from_numpy(ctx, b), m.DeviceVector(ctx, n)
    s.apply_preconditioner(z, y)
    out = y.numpy()
    s.close()
    A.close()
    assert np.all(np.abs(out - b / d) <= 4 * U * np.abs(b / d))
