"""The block CG in the form that each test names (the library reports it): the
three-phase kernel at the widths whose gathers differ, with whole 16-byte column
groups leaving early (its gather then changes), a start away from zero and "rel"
norms; the small operators' forms on a worker's share of the SMs; a barrier wait
that runs out in the three-phase kernel; against the CPU restatement of BlockPCG
(src/ops_lin_sol.c:140-437).

Tolerances: the operators have a condition number below 100, so 30 steps in a
precision u leave a relative difference below 30 x 100 u; FP64 3.3e-13 and FP32
1.8e-4, taken ten times over for the sums' length."""
import ctypes

import numpy as np
import pytest

from gcge_gb300 import problems as P
from oracle.gcg_oracle import GCGOracle, GCGParams

pytestmark = pytest.mark.gpu

CLUSTER, UNITS, PHASES = 1, 2, 3


def shifted(A, shift):
    """A + shift I."""
    rows = np.repeat(np.arange(A.n), np.diff(A.indptr))
    return P.CSRMatrix(A.n, A.indptr, A.indices, A.data + np.where(rows == A.indices, shift, 0.0))


def oracle(A, b, x0, rate, tol=1e-14, tol_type="abs"):
    p = GCGParams(nev_init=1, nev_max=1, block_size=1, cg_max_iter=30, cg_rate=rate,
                  cg_tol=tol, cg_tol_type=tol_type)
    x = np.array(x0, order="F", copy=True)
    return x, GCGOracle(A.to_scipy(), None, p).block_pcg(np.asfortranarray(b), x)


def mode(nx, ny, i, j):
    """Eigenvector of the 5-point Laplacian: its column leaves after one step."""
    x = np.sin(np.arange(1, nx + 1) * i * np.pi / (nx + 1))
    y = np.sin(np.arange(1, ny + 1) * j * np.pi / (ny + 1))
    return np.outer(y, x).ravel()


def columns(nx, ny, k, L, seed):
    """Noise; from two groups of L columns on, the first group has nothing to do
    and the second leaves after one step."""
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((nx * ny, k))
    if k > 2 * L:
        b[:, :L] = 0.0
        for c in range(L, 2 * L):
            b[:, c] = mode(nx, ny, c, 2 * c + 1)
    return b


def check(gpu_lib, A, b, x0, fp32, form):
    if fp32:
        b, x0 = (v.astype(np.float32).astype(np.float64) for v in (b, x0))
    ref, it_ref = oracle(A, b, x0, 1e-4)
    x, it = gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=30, rate=1e-4, tol=1e-14, fp32=fp32)
    assert gpu_lib.load().GCGE_TestBlockPCGForm() == form
    err = np.linalg.norm(x - ref) / np.linalg.norm(ref)
    assert err < (1.8e-3 if fp32 else 3.3e-12), err
    assert abs(it - it_ref) <= (1 if fp32 else 0)


@pytest.mark.parametrize("fp32,nx,ny,k", [
    (True, 420, 400, 8), (True, 330, 320, 12), (True, 230, 220, 24), (True, 230, 220, 28),
    (True, 230, 220, 31), (True, 230, 220, 36), (True, 230, 220, 40), (True, 290, 281, 20),
    (False, 230, 220, 24), (False, 230, 220, 27), (False, 230, 220, 32), (False, 230, 220, 36),
    (False, 230, 220, 40)])
@pytest.mark.parametrize("start", ["zero", "noise"])
def test_three_phase_kernel(gpu_lib, fp32, nx, ny, k, start):
    A = shifted(P.laplace2d(nx, ny), 0.1)
    b = columns(nx, ny, k, 4 if fp32 else 2, nx + k)
    x0 = np.zeros_like(b)
    if start == "noise":
        x0 = 0.1 * np.random.default_rng(1).standard_normal(b.shape)
    check(gpu_lib, A, b, x0, fp32, PHASES)


def test_three_phase_kernel_with_relative_norms(gpu_lib):
    A = shifted(P.laplace2d(300, 290), 0.1)
    k = 12
    b, x0 = columns(300, 290, k, 2, 9), np.zeros((A.n, k))
    b *= 10.0 ** np.linspace(-6, 6, k)
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
        assert ops.lib.GCGE_TestBlockPCGForm() == PHASES
        x = ops.download(xv, 0, k)
    finally:
        ops.close()
    ref, _ = oracle(A, b, x0, 1e-30, 1e-6, "rel")
    live = np.linalg.norm(ref, axis=0) > 0
    np.testing.assert_array_equal(x[:, ~live], 0.0)
    err = np.linalg.norm(x - ref, axis=0)[live] / np.linalg.norm(ref, axis=0)[live]
    assert err.max() < 3.3e-12, err


@pytest.mark.parametrize("fp32,nx,ny,k,form", [
    (True, 64, 65, 4, CLUSTER), (True, 64, 65, 20, UNITS), (True, 90, 88, 20, PHASES),
    (False, 40, 39, 2, CLUSTER), (False, 64, 65, 13, UNITS), (False, 120, 130, 20, PHASES)])
@pytest.mark.parametrize("workers", [8])
def test_share_of_the_sms(gpu_lib, fp32, nx, ny, k, form, workers):
    """As a server's workers run: an eighth of the SMs (19 blocks) each."""
    A = shifted(P.laplace2d(nx, ny), 0.1)
    b = columns(nx, ny, k, 4 if fp32 else 2, nx + k)
    x0 = 0.1 * np.random.default_rng(1).standard_normal(b.shape)
    lib = gpu_lib.load()
    before = lib.GCGE_TestBlockPCGShare(workers)
    try:
        check(gpu_lib, A, b, x0, fp32, form)
    finally:
        assert lib.GCGE_TestBlockPCGShare(before) == workers


@pytest.mark.parametrize("nx,ny,k,form", [(300, 290, 12, PHASES), (200, 200, 8, UNITS)])
def test_barrier_timeout_in_each_grid_form(gpu_lib, nx, ny, k, form):
    """One block leaves before its first grid barrier: the others' bounded waits
    (100 ms) run out, the call returns GCGE_ERR_CUDA, and the next one succeeds."""
    A = P.laplace2d(nx, ny)
    ops = gpu_lib.CudaOps()
    try:
        h = ops.mat(A)
        hb = ops.multivec(h, k, np.random.default_rng(3).standard_normal((A.n, k)))
        hx = ops.multivec(h, k)
        st = ops.lib.GCGE_TestBlockPCGBarrierTimeout(h, hb, hx, ctypes.c_int(k),
                                                     ctypes.c_double(100.0))
        assert st == gpu_lib.GCGE_ERR_CUDA and ops.lib.GCGE_TestBlockPCGForm() == form
        it = ctypes.c_int()
        st = ops.lib.GCGE_BlockPCG(h, None, ctypes.c_double(0.0), hb, hx, ctypes.c_int(k),
                                   ctypes.c_int(30), ctypes.c_double(1e-2),
                                   ctypes.c_double(1e-14), ctypes.c_int(0), ctypes.byref(it))
        assert st == gpu_lib.GCGE_OK and it.value > 0
        assert ops.lib.GCGE_TestBlockPCGForm() == form
    finally:
        ops.close()
