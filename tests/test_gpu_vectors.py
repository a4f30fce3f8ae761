"""Dat arithmetic, dot products and the CG solve at the sizes where their
kernels change path: pieces of 16 bytes and what is left of them, pointers off
a 16-byte boundary, groups of 32 rows, rows longer than a warp's chunk, and
matrices whose rows take a group of lanes."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def b200(backend):
    from pyop2_b200 import b200
    return b200


OPS = [np.add, np.subtract, np.multiply, np.divide]


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 1023, 1024, 4096, 4099])
@pytest.mark.parametrize("dtype,code", [(np.float64, 0), (np.float32, 1), (np.int32, 2)])
@pytest.mark.parametrize("shift", [0, 1])
def test_binop(b200, n, dtype, code, shift):
    from pyop2_b200._lib import call
    rng = np.random.default_rng(n)
    x = rng.integers(1, 50, n + 1).astype(dtype)
    y = rng.integers(1, 50, n + 1).astype(dtype)
    item = np.dtype(dtype).itemsize
    dx, dy = b200._upload(x), b200._upload(y)
    for op in range(3 if code == 2 else 4):
        for scalar in (False, True):
            out = b200._upload(np.zeros(n + 1, dtype))
            call("op2b_vec_binop", out.ptr + shift * item, dx.ptr + shift * item,
                 0 if scalar else dy.ptr + shift * item, 3.0, n, op, code, 0)
            got = np.zeros(n + 1, dtype)
            out.to_host(got)
            want = np.zeros(n + 1, dtype)
            want[shift:shift + n] = OPS[op](x[shift:shift + n], dtype(3) if scalar else y[shift:shift + n])
            np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("n", [0, 1, 2, 255, 256, 257, 2049, 300001, 1500003])
@pytest.mark.parametrize("shift", [0, 1])
def test_dot(b200, n, shift):
    """Whole numbers: exact in any order, so equal; and twice the same bits."""
    from pyop2_b200._lib import call
    rng = np.random.default_rng(n)
    x, y = (rng.integers(-9, 10, n + 2).astype(np.float64) for _ in range(2))
    dx, dy = b200._upload(x), b200._upload(y)
    for a, b, da, db in ((x, y, dx, dy), (x, x, dx, dx)):
        r = C.c_double(-1.0)
        call("op2b_vec_dot", da.ptr + 8 * shift, db.ptr + 8 * shift, n, C.byref(r), 0)
        assert r.value == float(a[shift:shift + n] @ b[shift:shift + n])


def _spd(n, per_row, long_rows, rng):
    """Symmetric, diagonally dominant (condition number below 4), as CSR."""
    a = np.zeros((n, n))
    for i in range(n):
        k = min(n, 700 if i in long_rows else rng.integers(1, 2 * per_row + 1))
        j = rng.choice(n, k, replace=False)
        a[i, j] = a[j, i] = rng.uniform(-1, 1, k)
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, 2.0 * np.maximum(np.abs(a).sum(1), 1.0))
    nz = a != 0
    rowptr = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
    return a, rowptr, np.nonzero(nz)[1].astype(np.int32), a[nz]


@pytest.mark.parametrize("n,per_row,long_rows", [(1, 1, ()), (31, 3, ()), (33, 4, ()), (513, 5, ()),
                                                 (1200, 6, (0, 40, 1199)), (900, 20, ()), (700, 60, ()),
                                                 (300, 140, ())])
@pytest.mark.parametrize("jacobi", [0, 1])
def test_cg_matches_dense_solve(b200, n, per_row, long_rows, jacobi):
    """The preconditioned residual ends below 1e-12 of the first, and the
    condition number is below 4 (8 with the rows' scaling): 1e-10 on x."""
    from pyop2_b200._lib import call
    rng = np.random.default_rng(n + per_row)
    a, rowptr, colidx, vals = _spd(n, per_row, long_rows, rng)
    want = rng.standard_normal(n)
    b = a @ want
    dr, dc, dv, db = (b200._upload(v) for v in (rowptr, colidx, vals, b))
    dx = b200.DeviceBuffer(8 * n)
    its, reason = C.c_int32(), C.c_int32()
    hist = np.zeros(301)
    call("op2b_cg_solve", dr.ptr, dc.ptr, dv.ptr, n, len(vals), dx.ptr, db.ptr, jacobi, 1e-12, 0.0, 1e5, 300,
         C.byref(its), C.byref(reason), hist.ctypes.data_as(C.POINTER(C.c_double)), 0)
    x = np.zeros(n)
    dx.to_host(x)
    assert reason.value == 1
    assert np.linalg.norm(x - want) <= 1e-10 * np.linalg.norm(want)
    z0 = b / np.diag(a) if jacobi else b
    assert abs(hist[0] - np.linalg.norm(z0)) <= 1e-12 * hist[0]
    assert (hist[:its.value] > 1e-12 * hist[0]).all() and hist[its.value] <= 1e-12 * hist[0]


def test_cg_limits(b200):
    """No iterations allowed, a solution at the start, a right-hand side that
    is not finite, and a history longer than its first copy."""
    from pyop2_b200._lib import call
    n = 300
    a = 2.0 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
    nz = a != 0
    rowptr = np.concatenate([[0], np.cumsum(nz.sum(1))]).astype(np.int32)
    dr, dc, dv = (b200._upload(v) for v in (rowptr, np.nonzero(nz)[1].astype(np.int32), a[nz]))
    dx = b200.DeviceBuffer(8 * n)

    def solve(b, max_it, rtol=1e-14):
        its, reason, hist = C.c_int32(), C.c_int32(), np.zeros(max_it + 1)
        db = b200._upload(np.asarray(b, dtype=np.float64))
        call("op2b_cg_solve", dr.ptr, dc.ptr, dv.ptr, n, int(rowptr[-1]), dx.ptr, db.ptr, 1, rtol, 0.0, 1e9,
             max_it, C.byref(its), C.byref(reason), hist.ctypes.data_as(C.POINTER(C.c_double)), 0)
        return its.value, reason.value, hist
    assert solve(np.ones(n), 0)[:2] == (0, 4)
    assert solve(np.zeros(n), 10)[:2] == (0, 1)
    assert solve(np.full(n, np.nan), 10)[:2] == (0, 3)
    assert solve(np.ones(n), 7)[:2] == (7, 4)
    rng = np.random.default_rng(0)
    its, reason, hist = solve(rng.standard_normal(n), 290, 0.0)
    assert its == 290 and reason == 4 and (hist > 0).all()
