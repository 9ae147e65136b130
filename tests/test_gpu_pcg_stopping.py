"""Stopping rule of the block CG (src/ops_lin_sol.c:383-394) at bounds that a test
on squares could get wrong: negative ones never stop a column, one that is not a
number stops it at its first test, zero ones stop it at a zero residual."""
import numpy as np
import pytest

from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu

# n k: the small operators' kernel as a cluster and as a grid, the three-phase kernel
SIZES = [(20, 19, 3), (128, 128, 5), (300, 290, 12)]


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nx,ny,k", SIZES)
def test_negative_and_nan_bounds(gpu_lib, nx, ny, k, fp32):
    A = P.laplace2d(nx, ny)
    rng = np.random.default_rng(nx)
    b = rng.standard_normal((A.n, k))
    x0 = np.zeros_like(b)

    def solve(rate, tol):
        return gpu_lib.block_pcg(A, None, 0.0, b, x0, max_iter=9, rate=rate, tol=tol, fp32=fp32)
    x, it = solve(0.0, 0.0)
    assert it == 9
    for rate, tol in [(-1.0, -1.0), (-10.0, -1e300), (-1e-3, 0.0), (-np.inf, -np.inf)]:
        y, it = solve(rate, tol)
        assert it == 9, (rate, tol)
        np.testing.assert_array_equal(x, y)
    _, it = solve(np.nan, 1e-30)
    assert it == 1
    _, it = solve(np.inf, 0.0)
    assert it == 1
    _, it = solve(0.0, np.nan)  # no column starts
    assert it == 0
    _, it = solve(0.999999, -1.0)
    assert 1 <= it <= 9
