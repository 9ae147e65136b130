"""Eigenvalues of higher multiplicity than the block size: the convergence test
locks a cluster whole (src/ops_eig_sol_gcg.c:266-273) and looks at one block at
a time, so such a cluster is locked only by a check that covers it.

Tolerances: a pair whose relative residual is below 7.4e-10 has an eigenvalue
accurate to about its square over the gap, far below the 1e-10 of the other
parity tests."""
import numpy as np
import pytest

from gcge_gb300 import problems as P

pytestmark = pytest.mark.gpu


def cube_solve(gpu_lib, seed, mixed):
    """A request of the serving workload: the cube's eigenvalues have up to six
    members, the block four columns, the tolerance is 7.4e-10."""
    A = P.laplace3d(44)
    bs, ni, nm = P.gcge_block_rule(22)
    assert bs == 4
    return gpu_lib.solve(A, None, 22, bs, ni, nm, X0=P.initial_block(A.n, ni, seed=seed),
                         tol=(1e300, 7.427257145118223e-10),
                         precision=gpu_lib.PREC_MIXED if mixed else gpu_lib.PREC_FP64)


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("seed", [1, 2, 3, 4, 5, 6, 7, 8])
def test_cluster_wider_than_the_block(gpu_lib, seed, mixed):
    r = cube_solve(gpu_lib, seed, mixed)
    assert r.status == gpu_lib.GCGE_OK and r.nconv >= 22
    k = 2 - 2 * np.cos(np.arange(1, 45) * np.pi / 45)
    lam = np.sort((k[:, None, None] + k[None, :, None] + k[None, None, :]).ravel())[:22] * 45.0 ** 2
    assert np.max(np.abs(r.eval[:22] - lam) / lam) < 1e-10
    V = r.evec[:, :22]
    res = np.linalg.norm(P.laplace3d(44).to_scipy() @ V - V * r.eval[:22], axis=0)
    assert np.all(res <= 7.5e-10 * r.eval[:22])


@pytest.mark.parametrize("seed", [1, 2, 3, 4, 5, 6, 7, 8])
def test_stall_far_from_the_tolerance_goes_over_to_fp64(gpu_lib, seed):
    """From some starting blocks the mixed solve stalls at a few hundred times
    its tolerance; FP64 takes about 95 iterations, so twice as many are a stall
    that was not noticed."""
    r = cube_solve(gpu_lib, seed, True)
    assert r.status == gpu_lib.GCGE_OK and r.niter < 190
