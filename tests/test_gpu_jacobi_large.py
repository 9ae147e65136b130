"""The dense eigensolver's cluster Jacobi over its range, up to the largest projected
dimension that its shared memory takes (466 rows at least)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("s", [111, 129, 207, 260, 341, 400, 463, 465, 466])
def test_dense_eig_cluster_range(gpu_lib, s):
    rng = np.random.default_rng(s)
    d = np.cumsum(0.5 + rng.random(s)) * np.where(rng.random(s) < 0.3, -1.0, 1.0)
    M = rng.standard_normal((s, s)) * 0.2
    M = 0.5 * (M + M.T) + np.diag(d)
    ev, Z = gpu_lib.dense_eig(M)
    ref = np.linalg.eigvalsh(M)
    scale = np.abs(ref).max()
    # backward error of a refined FP64 decomposition: products of length s, each
    # rounding to s eps relative to |M|
    tol = 16 * s * EPS
    assert np.all(np.diff(ev) >= 0)
    assert np.abs(ev - ref).max() <= tol * scale
    assert np.abs(M @ Z - Z * ev).max() <= tol * scale
    assert np.abs(Z.T @ Z - np.eye(s)).max() <= tol
