"""The dense inverse at the upper end of its panels (four rows per thread, 4,096 rows)
and, one row further, column by column: sparse matrices with singular values within
[0.5, 10.5] whose rows are shuffled, so that every step swaps rows.

Tolerance: the rounding errors of n elimination steps add up like sqrt(n) u times the
condition number; 20 sqrt(n) 21 u of the solution's norm."""
import numpy as np
import pytest

import mymoonmd_gb300 as m

pytestmark = pytest.mark.gpu


def solve(ctx, n):
    """the error of the direct solve and its tolerance; the solver stays open"""
    r = np.random.default_rng(n)
    d = np.linspace(1.0, 10.0, n) * r.choice([-1.0, 1.0], n)
    x = r.standard_normal(n)
    b = d * x
    b[:-1] += 0.5 * x[1:]  # upper bidiagonal
    order = r.permutation(n)
    rp, ci, v = [0], [], []
    for i in order:
        ci += [i, i + 1] if i + 1 < n else [i]
        v += [d[i], 0.5] if i + 1 < n else [d[i]]
        rp.append(len(ci))
    A = m.FEMatrix.from_csr(ctx, np.array(rp), np.array(ci), np.array(v))
    s = m.Solver(ctx, {"solver_type": "direct"})
    s.update_matrix(A)
    out = np.zeros(n)
    s.solve(b[order], out)
    return s, A, np.linalg.norm(out - x), 20 * np.sqrt(n) * 21 * 2.0 ** -53 * np.linalg.norm(x)


@pytest.mark.parametrize("n", [3071, 3072, 3073, 4095, 4096, 4097])
def test_direct_solve(ctx, n):
    s, A, err, tol = solve(ctx, n)
    s.close()
    A.close()
    assert err <= tol


def test_memory_held_by_a_direct_solver(ctx):
    """the inverse and one matrix beside it, not more"""
    torch = pytest.importorskip("torch")
    s, A, _, _ = solve(ctx, 3073)  # every kernel is loaded
    s.close()
    A.close()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info(0)[0]
    s, A, _, _ = solve(ctx, 4096)
    held = before - torch.cuda.mem_get_info(0)[0]
    s.close()
    A.close()
    assert held <= 2.25 * 8 * 4096 ** 2
