"""The tensor-core digit products (ozaki_tc.cu) at the sizes where their tiles
change: row tiles split evenly, row groups shared by two and four warps, right
operands of one, two and several column tiles, contractions that end inside a
stage, a 16-k step, a 128-k chunk and a 432-k window, and operands whose
exponents sit at both ends of the range.

Bound, entry by entry: a product of two truncated operands is off by less than
2 x 2^-55 x 2 of the largest |x||y| of its row and column (the exponents are
rounded up to a power of two on both sides, hence 2^-51), K of them are added
exactly and the sum is rounded once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXT = np.longdouble
U = 2.0 ** -53


def _check(got, exact, K, xmax, ymax):
    bound = K * 2.0 ** -51 * np.outer(xmax, ymax) + 4 * U * np.abs(exact.astype(np.float64))
    err = np.abs(got.astype(EXT) - exact).astype(np.float64)
    assert np.all(err <= bound), float(np.max(err / bound))


@pytest.mark.parametrize("n,m,w", [
    (40, 8, 3), (128, 17, 16), (129, 33, 17), (1000, 64, 33), (3000, 65, 20), (4097, 128, 48),
    (5000, 129, 20), (6001, 180, 20), (2500, 257, 49), (9000, 360, 40), (20000, 72, 13),
    (70000, 96, 1)])
def test_gram_tiles(gpu_lib, n, m, w):
    rng = np.random.default_rng(n + m + w)
    Q, R = rng.standard_normal((n, m)), rng.standard_normal((n, w))
    got = gpu_lib.dense_gram(Q, R, emulated=True)
    _check(got, Q.astype(EXT).T @ R.astype(EXT), n, np.abs(Q).max(0), np.abs(R).max(0))


@pytest.mark.parametrize("n,k,m", [
    (40, 16, 3), (128, 17, 16), (129, 32, 17), (200, 33, 48), (1000, 100, 20), (1025, 112, 33),
    (1500, 113, 7), (2050, 144, 49), (3000, 180, 100), (2500, 432, 20), (2500, 433, 20),
    (20000, 60, 8), (135, 400, 320)])
def test_lincomb_tiles(gpu_lib, n, k, m):
    rng = np.random.default_rng(n + k + m)
    X, C, Y = (rng.standard_normal(s) for s in ((n, k), (k, m), (n, m)))
    got = gpu_lib.dense_lincomb(X, C, Y, beta=np.ones(m), alpha=-1.0, emulated=True)
    exact = Y.astype(EXT) - X.astype(EXT) @ C.astype(EXT)
    bound = np.abs(Y).max()
    xmax, cmax = np.abs(X).max(1), np.abs(C).max(0)
    err = np.abs(got.astype(EXT) - exact).astype(np.float64)
    tol = k * 2.0 ** -51 * np.outer(xmax, cmax) + 8 * U * (np.abs(exact.astype(np.float64)) + bound)
    assert np.all(err <= tol), float(np.max(err / tol))


@pytest.mark.parametrize("scale", [2.0 ** -1000, 2.0 ** -940, 1.0, 2.0 ** 500])
def test_gram_exponent_range(gpu_lib, scale):
    """Columns down to where subnormals begin, against the same product scaled
    exactly into the normal range."""
    rng = np.random.default_rng(4)
    Q, R = rng.standard_normal((700, 20)), rng.standard_normal((700, 5))
    Q[::7, 3] = 0.0
    got = gpu_lib.dense_gram(Q * scale, R, emulated=True)
    exact = Q.astype(EXT).T @ R.astype(EXT)
    # (subnormal inputs lose no bits at these scales: 2^-1000 x a normal number)
    _check(got.astype(EXT) / EXT(scale), exact, 700, np.abs(Q).max(0), np.abs(R).max(0))
