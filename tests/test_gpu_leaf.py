"""Leaf kernels of the tridiagonal and bidiagonal divide and conquer: every lane
count per leaf (it follows the number of leaves) at the edges of the row counts."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu

# a leaf of m rows takes about 1.7 sweeps per eigenvalue of m / 2 rotations, below
# 900 rotations at m = 32, each of which may turn a column by 4 eps
ORTH = 900 * 4 * 2.0 ** -53


@pytest.mark.parametrize("count", [1, 700, 2500, 5000, 12000, 40000])
@pytest.mark.parametrize("lo,hi", [(1, 8), (2, 12), (9, 13), (15, 16), (17, 17), (25, 32)])
def test_tridiagonal_leaves(count, lo, hi):
    # every problem is one leaf
    rng = np.random.default_rng(count + hi)
    sizes = rng.integers(lo, hi + 1, count).astype(np.int32)
    sizes[-1] = hi
    o, oz = hp.batch_offsets(sizes)
    d0 = torch.tensor(rng.uniform(-1, 1, int(o[-1])), device="cuda")
    e0 = torch.tensor(rng.uniform(-1, 1, int(o[-1])), device="cuda")
    d, z = d0.clone(), torch.empty(int(oz[-1]), dtype=torch.float64, device="cuda")
    old = hp.set_config(smlsiz=32)
    try:
        hp.mdstedc_batch_dev(sizes, d, e0.clone(), z)
    finally:
        hp.restore_config(old)
    for m in range(lo, hi + 1):
        ps = np.flatnonzero(sizes == m)
        if not len(ps):
            continue
        r = torch.tensor(o[ps], device="cuda")[:, None] + torch.arange(m, device="cuda")
        D, E, w = d0[r], e0[r][:, :m - 1], d[r]
        Q = z[torch.tensor(oz[ps], device="cuda")[:, None] + torch.arange(m * m, device="cuda")]
        Q = Q.view(-1, m, m).transpose(1, 2)
        T = torch.diag_embed(D)
        if m > 1:
            T = T + torch.diag_embed(E, 1) + torch.diag_embed(E, -1)
        ref = torch.linalg.eigvalsh(T)
        tn = 3.0  # |d| + 2 |e|
        assert float((w - ref).abs().max()) <= 1e-13 * tn
        assert float((T @ Q - Q * w[:, None, :]).abs().max()) <= 2 * ORTH * tn
        eye = torch.eye(m, dtype=torch.float64, device="cuda")
        assert float((Q.transpose(1, 2) @ Q - eye).abs().max()) <= ORTH


@pytest.mark.parametrize("kind", ["equal", "zero_diagonal", "graded", "tiny"])
def test_tridiagonal_leaf_special(kind):
    m = 24
    d, e = np.full(m, 2.0), np.zeros(m - 1)
    if kind == "zero_diagonal":
        d[:], e[:] = 0.0, 1.0
    elif kind == "graded":
        d = 10.0 ** -np.arange(0.0, m)
        e = 0.1 * np.sqrt(d[1:] * d[:-1])
    elif kind == "tiny":  # off-diagonals whose squares underflow
        d, e = np.zeros(m), np.full(m - 1, 1e-180)
    w, Q = hp.eigh_tridiagonal(d, e)
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    tn = np.abs(T).sum(1).max()
    assert np.abs(w - np.linalg.eigvalsh(T)).max() <= 1e-13 * tn
    assert np.abs(T @ Q - Q * w).max() <= 2 * ORTH * tn
    assert np.abs(Q.T @ Q - np.eye(m)).max() <= ORTH


# leaves: 1, 2 of 16 (17 columns), 32 of 31 / 32, 64 of 15, 512 of 4, 4096 of 4,
# 8192 of 2 rows
@pytest.mark.parametrize("n,smlsiz", [(32, 32), (33, 25), (1023, 32), (1001, 25), (2047, 8),
                                      (16383, 4), (20000, 4)])
def test_bidiagonal_leaves(n, smlsiz):
    rng = np.random.default_rng(n)
    d = torch.tensor(1.0 - rng.uniform(0.0, 1.0, n), device="cuda")
    e = torch.tensor(1.0 - rng.uniform(0.0, 1.0, n), device="cuda")
    s = d.clone()
    u, vt = (torch.empty(n * n, dtype=torch.float64, device="cuda") for _ in range(2))
    old = hp.set_config(precision=1, predictor=2, smlsiz=smlsiz)
    try:
        hp.mdbdsdc_dev(s, e, u, vt)
    finally:
        hp.restore_config(old)
    U, VT = u.view(n, n).T, vt.view(n, n).T
    g = torch.randn(n, 8, dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(1))
    # probes: ||X g|| estimates ||X||_F; the acceptance of the full solves, 1e-12 n
    vg = VT.T @ g
    bv = d[:, None] * vg
    bv[:-1] += e[:n - 1, None] * vg[1:]
    assert float(torch.linalg.norm(bv - U @ (s[:, None] * g))) / (8 ** 0.5 * n) <= 1e-12 * 2.0
    for X in (U, VT.T):
        y = X.T @ (X @ g) - g
        assert float(torch.linalg.norm(y)) / (8 ** 0.5 * n) <= 1e-12
    if n <= 2047:
        B = torch.diag(d) + torch.diag(e[:n - 1], 1)
        ref = np.linalg.svd(B.cpu().numpy(), compute_uv=False)
        assert np.abs(s.cpu().numpy() - ref).max() <= 1e-13 * 2.0
