"""pm_matrix_get_structure and pm_matrix_get_values write nnz entries and no more,
whatever nnz is modulo four (the device's column array is padded)."""
import ctypes

import numpy as np
import pytest

import mymoonmd_gb300 as m
from mymoonmd_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8, 33])
def test_exactly_the_entries_are_written(ctx, n):
    cols = np.arange(n, dtype=np.int32)
    A = m.FEMatrix.from_csr(ctx, np.arange(n + 1), cols, np.arange(n) + 1.0)
    rp = np.full(n + 1 + 8, -7, dtype=np.int32)
    ci = np.full(n + 8, -7, dtype=np.int32)
    v = np.full(n + 8, -7.0)
    ptr = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    check(lib.pm_matrix_get_structure(A.handle, ptr(rp), ptr(ci)), ctx.handle)
    check(lib.pm_matrix_get_values(A.handle, ptr(v)), ctx.handle)
    A.close()
    assert np.array_equal(rp[:n + 1], np.arange(n + 1)) and (rp[n + 1:] == -7).all()
    assert np.array_equal(ci[:n], cols) and (ci[n:] == -7).all()
    assert np.array_equal(v[:n], np.arange(n) + 1.0) and (v[n:] == -7.0).all()
