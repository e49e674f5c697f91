"""Node kernels of the HSS Cholesky factor at the edges of their sizes: leaves of 20 to 128
rows (odd ones, 32 and 33, more than shared memory holds three matrices of), nodes that
keep nothing, and right-hand sides below, at and above a CTA's eight warps."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp
from oracle import hsschol_ref as ref

pytestmark = pytest.mark.gpu


def _check(A, ni, nrhs, seed):
    n = A.shape[0]
    f = hp.HssChol(torch.tensor(np.asfortranarray(A).ravel(order="F"), device="cuda"), ni, 1e-12, 128)
    B = np.random.default_rng(seed).standard_normal((n, nrhs))
    Bt = torch.tensor(np.asfortranarray(B).ravel(order="F"), device="cuda")
    f.solve(Bt)
    X = Bt.cpu().numpy().reshape(n, nrhs, order="F")
    f.free()
    # backward error: a node drops at most tol ||A||, and there are fewer than 100 nodes
    assert np.linalg.norm(A @ X - B) <= 1e-10 * np.linalg.norm(A, 2) * np.linalg.norm(X)


@pytest.mark.parametrize("n,ni,nrhs", [(400, 20, 1), (500, 31, 7), (512, 32, 8), (530, 33, 9),
                                       (900, 64, 16), (1000, 100, 3), (1024, 128, 17)])
def test_kernel_matrix(n, ni, nrhs):
    _check(ref.kernel_matrix(n, 0.2, 1e-2, seed=n), ni, nrhs, ni)


@pytest.mark.parametrize("ni", [32, 63])
def test_nothing_kept(ni):
    n = 8 * ni
    rng = np.random.default_rng(ni)
    A = np.zeros((n, n))
    for k in range(0, n, ni):  # block diagonal: every node's rank is 0
        G = rng.standard_normal((ni, ni))
        A[k:k + ni, k:k + ni] = G @ G.T + np.eye(ni)
    _check(A, ni, 2, ni)
