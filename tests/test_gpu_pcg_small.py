"""The block CG of small operators (register-resident units, one cluster or one
block per SM, with and without the fused p update) at the sizes where its
dispatch and its partition change: fewer slices than blocks, one and two units
per warp, odd numbers of 16-byte column groups, rows of uneven length, and the
first sizes that go back to the three-phase kernel; against the CPU restatement
of BlockPCG (src/ops_lin_sol.c:140-437).

Tolerances: the operators have a condition number below 100, so 30 steps in a
precision u leave a relative difference below 30 x 100 u; FP64 3.3e-13 and FP32
1.8e-4, taken ten times over for the sums' length."""
import ctypes

import numpy as np
import pytest

from gcge_gb300 import problems as P
from oracle.gcg_oracle import GCGOracle, GCGParams

pytestmark = pytest.mark.gpu


def shifted(A, shift):
    """A + shift I."""
    rows = np.repeat(np.arange(A.n), np.diff(A.indptr))
    data = A.data + np.where(rows == A.indices, shift, 0.0)
    return P.CSRMatrix(A.n, A.indptr, A.indices, data)


def oracle(A, b, x0, rate):
    p = GCGParams(nev_init=1, nev_max=1, block_size=1, cg_max_iter=30, cg_rate=rate,
                  cg_tol=1e-14, cg_tol_type="abs")
    o = GCGOracle(A.to_scipy(), None, p)
    x = np.array(x0, order="F", copy=True)
    return x, o.block_pcg(np.asfortranarray(b), x)


def columns(n, k, seed):
    """Right-hand sides that leave at different steps: noise, constants, peaks."""
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((n, k))
    b[:, 1::3] = 1.0
    b[:, 2::3] = 0.0
    b[rng.integers(0, n, k), np.arange(k)] += 5.0
    return b


CASES = [(5, 4, 1), (11, 13, 3), (33, 31, 2), (64, 65, 4), (64, 65, 13), (64, 65, 40),
         (128, 128, 4), (120, 130, 20), (128, 128, 40), (200, 160, 12), (230, 220, 5),
         (230, 220, 20), (300, 290, 12)]


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nx,ny,k", CASES)
def test_small_operator_matches_oracle(gpu_lib, nx, ny, k, fp32):
    A = shifted(P.laplace2d(nx, ny), 0.1)
    b = columns(A.n, k, nx + k)
    x0 = 0.1 * np.random.default_rng(1).standard_normal(b.shape)
    if fp32:
        b, x0 = (v.astype(np.float32).astype(np.float64) for v in (b, x0))
    ref, it_ref = oracle(A, b, x0, 1e-4)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=30, rate=1e-4, tol=1e-14, fp32=fp32)
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    assert err < (1.8e-3 if fp32 else 3.3e-12), err
    assert abs(it - it_ref) <= (1 if fp32 else 0)


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("n,k", [(700, 6), (5000, 9), (20000, 4)])
def test_uneven_rows_match_oracle(gpu_lib, n, k, fp32):
    A = P.rgg_laplacian(n, 9.0, 3, shift=1.0)
    b = columns(n, k, n)
    if fp32:
        b = b.astype(np.float32).astype(np.float64)
    x0 = np.zeros_like(b)
    ref, it_ref = oracle(A, b, x0, 1e-4)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=30, rate=1e-4, tol=1e-14, fp32=fp32)
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    assert err < (1.8e-3 if fp32 else 3.3e-12), err
    assert abs(it - it_ref) <= (1 if fp32 else 0)


@pytest.mark.parametrize("k", [4, 20])
def test_no_iteration_and_wide_operator(gpu_lib, k):
    """max_iter 0 returns x0; a 27-point operator in FP64 takes the unfused form."""
    A = P.mass3d(14)
    A = P.CSRMatrix(A.n, A.indptr, A.indices, A.data * 15.0 ** 3)
    b = columns(A.n, k, 5)
    x0 = np.random.default_rng(2).standard_normal(b.shape)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=0, rate=1e-4, tol=1e-14)
    assert it == 0
    np.testing.assert_array_equal(x, x0)
    ref, it_ref = oracle(A, b, x0, 1e-4)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=30, rate=1e-4, tol=1e-14)
    assert it == it_ref
    assert np.linalg.norm(x - ref) / np.linalg.norm(ref) < 3.3e-12


def test_relative_tolerance_through_the_linear_solver_hook(gpu_lib):
    """"rel" norms of b, column ranges with offsets, 27 rows of an odd grid."""
    A = shifted(P.laplace2d(61, 47), 0.1)
    k = 6
    b, x0 = columns(A.n, k, 9), np.zeros((A.n, k))
    ops = gpu_lib.CudaOps()
    try:
        h = ops.mat(A)
        bv, xv = ops.multivec(h, k, b), ops.multivec(h, k, x0)
        ops.lib.MultiLinearSolverSetup_BlockPCG(
            ctypes.c_int(30), ctypes.c_double(1e-30), ctypes.c_double(1e-6), b"rel", None, None,
            None, None, None, ops.ptr)
        vp, ip = ctypes.c_void_p, ctypes.POINTER(ctypes.c_int)
        fn = ctypes.cast(ops.ptr.contents.MultiLinearSolver,
                         ctypes.CFUNCTYPE(None, vp, vp, vp, ip, ip, vp))
        two = ctypes.c_int * 2
        fn(h, bv, xv, two(0, 0), two(k, k), ctypes.cast(ops.ptr, vp))
        ops.check("MultiLinearSolver")
        x = ops.download(xv, 0, k)
    finally:
        ops.close()
    p = GCGParams(nev_init=1, nev_max=1, block_size=1, cg_max_iter=30, cg_rate=1e-30,
                  cg_tol=1e-6, cg_tol_type="rel")
    ref = x0.copy(order="F")
    GCGOracle(A.to_scipy(), None, p).block_pcg(np.asfortranarray(b), ref)
    assert np.linalg.norm(x - ref) / np.linalg.norm(ref) < 3.3e-12


@pytest.mark.parametrize("nx,ny,k", [(100, 74, 8), (100, 74, 12), (100, 75, 7), (64, 65, 20)])
def test_cluster_and_grid_forms_in_fp32(gpu_lib, nx, ny, k):
    """Either side of the cluster form's rule: one and two units a warp."""
    A = shifted(P.laplace2d(nx, ny), 0.1)
    b = columns(A.n, k, nx + k).astype(np.float32).astype(np.float64)
    x0 = np.zeros_like(b)
    ref, it_ref = oracle(A, b, x0, 1e-4)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=30, rate=1e-4, tol=1e-14, fp32=True)
    assert np.linalg.norm(x - ref) / np.linalg.norm(ref) < 1.8e-3
    assert abs(it - it_ref) <= 1
