"""The dense eigensolver at the edges of its Jacobi kernels: one pair, an odd size
next to an even one, one to three 2x2 blocks a thread, and the step from one CTA to
the cluster."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("s", [1, 2, 3, 4, 31, 33, 63, 64, 65, 66, 90, 91, 103, 104, 105, 128])
def test_dense_eig_jacobi_edges(gpu_lib, s):
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
