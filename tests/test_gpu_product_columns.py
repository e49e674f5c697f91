"""Every product kernel writing a merge's new vectors straight into the columns of the
slots that its roots took: split products staged and inside the CTA, FP64 tiles, the
element kernel, alone and mixed, in a tridiagonal and a bidiagonal solve."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu

KERNELS = [dict(precision=1, split_min_m=1, split_min_log2=1), dict(precision=1, gemm_path=1),
           dict(precision=0, small_nk=1), dict(precision=0), dict(precision=1)]


# the acceptance of the full solves: residual and orthogonality 1e-12 (Frobenius over n)
@pytest.mark.parametrize("cfg", KERNELS)
def test_tridiagonal(cfg):
    n = 777
    d = np.full(n, 2.0) + 1e-3 * np.random.default_rng(0).standard_normal(n)  # extended vectors
    e = np.ones(n)
    w, ee = torch.tensor(d, device="cuda"), torch.tensor(e, device="cuda")
    z = torch.full((n * n,), float("nan"), dtype=torch.float64, device="cuda")
    old = hp.set_config(**cfg)
    try:
        hp.mdstedc_dev(w, ee, z)
    finally:
        hp.restore_config(old)
    T = torch.tensor(np.diag(d) + np.diag(e[:-1], 1) + np.diag(e[:-1], -1), device="cuda")
    Q = z.view(n, n).T
    assert float(torch.linalg.norm(T @ Q - Q * w)) / (n * 4.0) <= 1e-12
    assert float(torch.linalg.norm(Q.T @ Q - torch.eye(n, dtype=Q.dtype, device="cuda"))) / n <= 1e-12


@pytest.mark.parametrize("cfg", KERNELS)
def test_bidiagonal(cfg):
    n = 531
    rng = np.random.default_rng(1)
    B = np.diag(2.0 + 1e-3 * rng.standard_normal(n)) + np.diag(np.ones(n - 1), 1)
    w, ee = (torch.tensor(x, device="cuda") for x in (np.diag(B).copy(), np.append(np.diag(B, 1), 0.0)))
    u = torch.full((n * n,), float("nan"), dtype=torch.float64, device="cuda")
    v = u.clone()
    old = hp.set_config(**cfg)
    try:
        hp.mdbdsdc_dev(w, ee, u, v)
    finally:
        hp.restore_config(old)
    s, U, VT = w.cpu().numpy(), u.view(n, n).T.cpu().numpy(), v.view(n, n).T.cpu().numpy()
    assert np.linalg.norm(U * s @ VT - B) / (n * 3.0) <= 1e-12
    assert np.linalg.norm(U.T @ U - np.eye(n)) / n <= 1e-12
    assert np.linalg.norm(VT @ VT.T - np.eye(n)) / n <= 1e-12
