"""SpMV on ragged random rows at the edges of the launch rules: short rows (two
lanes), sliced FP64 rows with eight or four steps in flight (the line is at 128
slices of eight rows per SM), slices whose last group of steps is partial, sizes
that leave blocks partly empty; FP32 with sixteen steps in flight.

Tolerance per row: the k products of a row are summed in some order, (k + 2) u of
sum_j |a_ij x_j|; FP32 also rounds a and x."""
import numpy as np
import pytest

import mymoonmd_gb300 as m

pytestmark = pytest.mark.gpu
LINE = 128 * 152 * 8


def matrix(ctx, n, longest):
    """rows of 0 to `longest` consecutive entries near the diagonal"""
    r = np.random.default_rng(n + longest)
    length = np.minimum(r.integers(0, longest + 1, n), n)
    first = np.clip(np.arange(n) - length // 2, 0, n - length)
    rp = np.concatenate([[0], np.cumsum(length)])
    cols = np.repeat(first - rp[:-1], length) + np.arange(rp[-1])
    vals, x = r.standard_normal(rp[-1]), r.standard_normal(n)
    rows = np.repeat(np.arange(n), length)
    y = np.bincount(rows, vals * x[cols], minlength=n)
    scale = np.bincount(rows, np.abs(vals * x[cols]), minlength=n)
    return m.FEMatrix.from_csr(ctx, rp, cols, vals), x, y, scale, length


SIZES = [1, 3, 31, 129, 1024, 4913, LINE - 8, LINE, LINE + 1, LINE + 9]


@pytest.mark.parametrize("longest", [9, 30, 70])
@pytest.mark.parametrize("n", SIZES)
def test_spmv_of_ragged_rows(ctx, n, longest):
    A, x, ref, scale, length = matrix(ctx, n, longest)
    A.make_fp32()
    A.make_sliced64()
    xd, yd = m.DeviceVector.from_numpy(ctx, x), m.DeviceVector(ctx, n)
    A.apply(xd, yd)
    out = yd.numpy()
    x32, y32 = m.DeviceVector.from_numpy(ctx, x.astype(np.float32)), m.DeviceVector(ctx, n, np.float32)
    A.apply_f32(x32, y32)
    out32 = y32.numpy()
    A.close()
    assert np.all(np.abs(out - ref) <= 2 * (length + 2) * 2.0 ** -53 * scale)
    assert np.all(np.abs(out32 - ref) <= (length + 4) * 2.0 ** -24 * scale)
