"""The digit products where their work is divided: k ranges of whole 32-k stages (one
stage, an odd number, a range that ends inside a drain chunk, fewer rows than a
stage), several row and column tiles, and right operands of 49 to 64 columns.

Bound, entry by entry: a product of two truncated operands is off by less than
2 x 2^-55 x 2 of the largest |x||y| of its row and column (the exponents are
rounded up to a power of two on both sides, hence 2^-51), K of them are added
exactly and the sum is rounded once (per work item of a Gram product, whose
partial sums are then added in FP64: 152 of them at most, 152 x 2^-53 of the sum of
their magnitudes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EXT = np.longdouble
U = 2.0 ** -53


def check(got, exact, K, xmax, ymax, mag):
    bound = K * 2.0 ** -51 * np.outer(xmax, ymax) + 156 * U * mag
    err = np.abs(got.astype(EXT) - exact).astype(np.float64)
    assert np.all(err <= bound), float(np.max(err / bound))


@pytest.mark.parametrize("n,m,w", [
    (2, 3, 2), (30, 12, 5), (32, 40, 40), (4864, 20, 20), (4866, 20, 20), (14592, 20, 20),
    (24322, 33, 16), (2000, 200, 60), (4160, 130, 30), (9000, 130, 20), (1216, 260, 60),
    (10002, 40, 49), (3000, 64, 64), (700, 200, 200)])
def test_gram_ranges(gpu_lib, n, m, w):
    rng = np.random.default_rng(n + m + w)
    Q, R = rng.standard_normal((n, m)), rng.standard_normal((n, w))
    got = gpu_lib.dense_gram(Q, R, emulated=True)
    check(got, Q.astype(EXT).T @ R.astype(EXT), n, np.abs(Q).max(0), np.abs(R).max(0),
          np.abs(Q).T @ np.abs(R))


@pytest.mark.parametrize("n,k,m", [
    (130, 8, 49), (1000, 40, 50), (3000, 60, 64), (2050, 144, 60), (5000, 433, 57), (20002, 33, 63)])
def test_lincomb_of_two_even_column_tiles(gpu_lib, n, k, m):
    rng = np.random.default_rng(n + k + m)
    X, C, Y = (rng.standard_normal(s) for s in ((n, k), (k, m), (n, m)))
    beta = rng.standard_normal(m)
    got = gpu_lib.dense_lincomb(X, C, Y, beta=beta, alpha=-1.0, emulated=True)
    exact = Y.astype(EXT) * beta.astype(EXT) - X.astype(EXT) @ C.astype(EXT)
    check(got, exact, k, np.abs(X).max(1), np.abs(C).max(0),
          np.abs(X) @ np.abs(C) + np.abs(Y * beta))
