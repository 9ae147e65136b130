"""The FP64 products over every tile shape their dispatch chooses: Q^T P
(DenseMatQtAP with matA = NULL, app/app_lapack.c:64-183), alpha X C + Y
diag(beta) (MultiVecLinearComb, app/app_lapack.c:463-534) and A X
(app/app_ccs.c:50-139), at sizes on both sides of tile, chunk and cluster
edges, against extended-precision host arithmetic.

Bound, entry by entry: a sum of K products in any order differs from the exact
one by at most K u / (1 - K u) times the sum of their magnitudes (u = 2^-53);
the split sums and the scaling by alpha and beta add a few roundings."""
import numpy as np
import pytest

from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu

EXT = np.longdouble
U = 2.0 ** -53


def _within(got, exact, scale, terms):
    err = np.abs(got.astype(EXT) - exact).astype(np.float64)
    bound = (terms + 8) * U * scale
    bad = err > bound
    assert not bad.any(), (np.argwhere(bad)[:4], err[bad][:4], bound[bad][:4])


@pytest.mark.parametrize("n,m,w", [
    (1, 1, 1), (15, 16, 4), (31, 17, 5), (33, 3, 64), (180, 180, 180), (200, 140, 20),
    (257, 400, 3), (400, 400, 400), (1024, 4, 4), (1500, 33, 37), (2000, 60, 36),
    (4160, 40, 6), (4161, 64, 41), (16384, 60, 4), (20011, 20, 40), (30000, 65, 33),
    (50001, 180, 20), (6000, 100, 13)])
def test_gram_fp64_shapes(gpu_lib, n, m, w):
    rng = np.random.default_rng(n + 31 * m + w)
    Q, R = rng.standard_normal((n, m)), rng.standard_normal((n, w))
    exact = Q.astype(EXT).T @ R.astype(EXT)
    _within(gpu_lib.dense_gram(Q, R), exact, np.abs(Q).T @ np.abs(R), n)


@pytest.mark.parametrize("n,k,m", [
    (1, 1, 1), (16, 32, 4), (17, 33, 5), (180, 180, 180), (200, 160, 21), (400, 400, 400),
    (257, 31, 3), (4160, 40, 6), (4161, 64, 41), (16384, 60, 4), (20011, 20, 40),
    (78000, 9, 20), (100003, 33, 33), (3000, 500, 13)])
@pytest.mark.parametrize("beta", [False, True])
def test_lincomb_fp64_shapes(gpu_lib, n, k, m, beta):
    rng = np.random.default_rng(n + 31 * k + m)
    X, C, Y = (rng.standard_normal(s) for s in ((n, k), (k, m), (n, m)))
    b = rng.standard_normal(m) if beta else None
    alpha = -0.75 if beta else 1.0
    exact = EXT(alpha) * (X.astype(EXT) @ C.astype(EXT))
    scale = abs(alpha) * (np.abs(X) @ np.abs(C))
    if beta:
        exact = exact + Y.astype(EXT) * b.astype(EXT)
        scale = scale + np.abs(Y) * np.abs(b)
    _within(gpu_lib.dense_lincomb(X, C, Y, beta=b, alpha=alpha), exact, scale, k)


def test_spmm_every_width(gpu_lib):
    A, _ = P.vardiff3d(11)
    S = A.to_scipy()
    rng = np.random.default_rng(7)
    X = rng.standard_normal((A.n, 43))
    ops = gpu_lib.CudaOps()
    try:
        h = ops.mat(A)
        x, y = ops.multivec(h, 43, X), ops.multivec(h, 43)
        exact, scale = (S.toarray().astype(EXT) @ X.astype(EXT)), abs(S) @ np.abs(X)
        for k in range(1, 44):
            ops.axpby(0.0, None, 0.0, y, (0, 0), (43, 43))
            ops.mat_dot(h, x, y, (0, 0), (k, k))
            got = ops.download(y, 0, 43)
            _within(got[:, :k], exact[:, :k], scale[:, :k], 7)
            assert not got[:, k:].any()
    finally:
        ops.close()
