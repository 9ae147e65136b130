"""The mixed solve's inner solve where a column of the FP32 correction leaves the
range of its type: the column stays as it was, whole, the others are what they
are without it, and the solve says when nothing is left to go on with."""
import ctypes

import numpy as np
import pytest

from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu


def inner_solve(gpu_lib, A, b, x0, max_iter):
    ops = gpu_lib.CudaOps()
    try:
        h = ops.mat(A)
        k = b.shape[1]
        hb, hx = ops.multivec(h, k, b), ops.multivec(h, k, x0)
        it, out = ctypes.c_int(), ctypes.c_ulonglong()
        st = ops.lib.GCGE_MixedInnerSolve(
            h, None, ctypes.c_double(0.0), hb, hx, ctypes.c_int(k), ctypes.c_int(max_iter),
            ctypes.c_double(0.0), ctypes.c_double(1e-4), ctypes.byref(it), ctypes.byref(out))
        assert st == gpu_lib.GCGE_OK
        return ops.download(hx, 0, k), it.value, out.value
    finally:
        ops.close()


@pytest.mark.parametrize("max_iter", [1, 30])
@pytest.mark.parametrize("n,k", [(1000, 3), (4160, 13), (120000, 12), (120001, 20), (90000, 40)])
def test_column_out_of_range_stays_whole(gpu_lib, n, k, max_iter):
    """S is diagonal, +-1 in its first 64 rows and within [1, 2] below, and one
    column's residual has a p^T S p of 1e-36: the first step is 2.6e38 times that
    residual, so its entries of 10 overflow and its entries of 1 do not.  n and k
    on either side of the small operators' kernel."""
    rng = np.random.default_rng(n + k)
    s = rng.uniform(1.0, 2.0, n).astype(np.float32).astype(np.float64)
    s[:64] = np.where(np.arange(64) % 2 == 0, 1.0, -1.0)
    s[n - 1] = 1.0
    A = P.diag_matrix(s)
    bad = k // 2
    x0 = np.round(rng.uniform(-8, 8, (n, k)))
    x0[n - 1, bad] = 0.0
    r = rng.standard_normal((n, k)).astype(np.float32).astype(np.float64)
    r[:64] = 0.0
    r[:, bad] = 0.0
    r[:64, bad] = 1.0
    r[4:6, bad] = 10.0
    r[n - 1, bad] = 1e-18
    b = r + s[:, None] * x0
    x, it, out = inner_solve(gpu_lib, A, b, x0, max_iter)
    assert out == 1 << bad
    np.testing.assert_array_equal(x[:, bad], x0[:, bad])
    b2 = b.copy()
    b2[:, bad] = s * x0[:, bad]  # no correction at all in that column
    x2, _, out2 = inner_solve(gpu_lib, A, b2, x0, max_iter)
    assert out2 == 0 and np.all(np.isfinite(x2))
    keep = np.arange(k) != bad
    np.testing.assert_array_equal(x[:, keep], x2[:, keep])
    assert np.any(x2[:, keep] != x0[:, keep])


@pytest.mark.parametrize("scale", [1e6, 1e12, 1e18, 1e30])
def test_operators_far_from_unit_scale(gpu_lib, scale):
    """From 1e12 on p^T S p leaves FP32's range in every column of the first W, and
    the mixed solve reports it; FP64 solves them all."""
    A = P.laplace2d(30, 29)
    A = P.CSRMatrix(A.n, A.indptr, A.indices, A.data * scale)
    X0 = P.initial_block(A.n, 12, seed=1)
    args = (A, None, 8, 4, 12, 20)
    if scale > 1e9:
        with pytest.raises(gpu_lib.GCGEError) as e:
            gpu_lib.solve(*args, X0=X0, precision=gpu_lib.PREC_MIXED)
        assert e.value.status == 5
    else:
        r = gpu_lib.solve(*args, X0=X0, precision=gpu_lib.PREC_MIXED)
        assert r.status == gpu_lib.GCGE_OK and r.nconv >= 8
    r = gpu_lib.solve(*args, X0=X0, precision=gpu_lib.PREC_FP64)
    assert r.status == gpu_lib.GCGE_OK and r.nconv >= 8
