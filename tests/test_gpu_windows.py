"""Merges restricted to the rows on which their columns hold data: localized and
extended columns side by side, rotated columns of different supports."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu


def _tridiagonal(kind, n, rng):
    d, e = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n - 1)
    if kind == "glued":  # equal blocks, weakly coupled: rotations at every level
        blk = 37
        d = np.resize(rng.uniform(-1, 1, blk), n)
        e = np.resize(np.append(rng.uniform(0.5, 1, blk - 1), 1e-9), n)[:n - 1]
    elif kind == "mixed":  # a flat stretch (extended columns) inside disorder
        d[n // 3:n // 2], e[n // 3:n // 2] = 0.1, 1.0
    elif kind == "stepped":  # a stretch whose columns never reach the cut at n / 2
        e[n // 2 - 40:n // 2 - 30] *= 1e-8
    return d, e


# the acceptance of the full solves: eigenvalues within 1e-13 ||T||, residual and
# orthogonality 1e-12 (Frobenius norms over n)
@pytest.mark.parametrize("kind", ["random", "glued", "mixed", "stepped"])
@pytest.mark.parametrize("n,cfg", [(999, dict(smlsiz=8)), (2600, dict(smlsiz=12, precision=1)),
                                   (2600, dict(smlsiz=25, bsmlz=150, hss_leaf=64, tol=1e-14)),
                                   (9001, dict(smlsiz=12, precision=1, predictor=2))])
def test_tridiagonal_windows(kind, n, cfg):
    d, e = _tridiagonal(kind, n, np.random.default_rng(n))
    dd = torch.tensor(d, device="cuda")
    ee = torch.tensor(np.append(e, 0.0), device="cuda")
    w, z = dd.clone(), torch.full((n * n,), float("nan"), dtype=torch.float64, device="cuda")
    old = hp.set_config(**cfg)
    try:
        hp.mdstedc_dev(w, ee, z)
    finally:
        hp.restore_config(old)
    Q = z.view(n, n).T
    tn = float(np.abs(d).max() + 2 * np.abs(e).max())
    R = dd[:, None] * Q - Q * w[None, :]
    R[:-1] += ee[:n - 1, None] * Q[1:]
    R[1:] += ee[:n - 1, None] * Q[:-1]
    assert float(torch.linalg.norm(R)) / (n * tn) <= 1e-12
    g = torch.randn(n, 8, dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(1))
    assert float(torch.linalg.norm(Q.T @ (Q @ g) - g)) / (8 ** 0.5 * n) <= 1e-12
    if n <= 2600:
        T = torch.diag(dd) + torch.diag(ee[:n - 1], 1) + torch.diag(ee[:n - 1], -1)
        assert float((w - torch.linalg.eigvalsh(T)).abs().max()) <= 1e-13 * tn


@pytest.mark.parametrize("kind", ["random", "glued", "mixed"])
@pytest.mark.parametrize("lower", [False, True])
@pytest.mark.parametrize("n,cfg", [(700, dict()), (2500, dict(smlsiz=8, precision=1, predictor=2)),
                                   (1500, dict(bsmlz=60, hss_leaf=64, tol=1e-14))])
def test_bidiagonal_windows(kind, lower, n, cfg):
    d, e = _tridiagonal(kind, n, np.random.default_rng(n + 1))
    d = np.abs(d) + 0.05
    old = hp.set_config(**cfg)
    try:
        s, U, VT = hp.svd_bidiagonal(d, e, lower=lower)
    finally:
        hp.restore_config(old)
    B = np.diag(d) + np.diag(e, -1 if lower else 1)
    bn = float(np.abs(d).max() + np.abs(e).max())
    assert np.abs(s - np.linalg.svd(B, compute_uv=False)).max() <= 1e-13 * bn
    assert np.linalg.norm(B @ VT.T - U * s) / (n * bn) <= 1e-12
    assert np.linalg.norm(U.T @ U - np.eye(n)) / n <= 1e-12
    assert np.linalg.norm(VT @ VT.T - np.eye(n)) / n <= 1e-12
