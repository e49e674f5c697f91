"""NaN inputs end in INFO > 0, not in finite numbers that look like results."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kd", [(5, 2), (20, 4), (40, 32)])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("where", ["diagonal", "off"])
def test_band_leaf(n, kd, sign, where):
    """One leaf, no merges: a NaN on or off its diagonal."""
    rng = np.random.default_rng(n)
    ab = np.asfortranarray(rng.uniform(-1.0, 1.0, (kd + 1, n)))
    ab[kd if where == "diagonal" else kd - 1, n // 2] = np.copysign(np.nan, sign)
    old = hp.set_config(smlsiz=25)
    try:
        with pytest.raises(hp.HssError, match=r"INFO=[1-9]"):
            hp.eigh_banded(ab)
        ab[np.isnan(ab)] = 0.5
        w, q = hp.eigh_banded(ab)
    finally:
        hp.restore_config(old)
    assert np.isfinite(w).all() and np.linalg.norm(q.T @ q - np.eye(n)) <= 1e-12 * n


BAD = [np.nan, -np.nan, np.inf, -np.inf]


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _new(n):
    return torch.empty(n, dtype=torch.float64, device="cuda")


def _refused(run, w):
    """The call fails and leaves no numbers in w."""
    with pytest.raises(hp.HssError, match=r"INFO=1: "):
        run()
    assert bool(torch.isnan(w).all())


@pytest.mark.parametrize("bad", [np.inf, -np.inf])
@pytest.mark.parametrize("at", [0, 64, 198])
def test_tridiagonal_merges(bad, at):
    """(A NaN, or an infinite diagonal entry, is split off as the reference splits it.)"""
    n = 200
    rng = np.random.default_rng(1)
    d0, e0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    e1 = e0.copy()
    e1[at] = bad
    d = _dev(d0)
    _refused(lambda: hp.mdstedc_dev(d, _dev(e1), _new(n * n)), d)
    sizes = np.array([50, n, 30], dtype=np.int32)
    d = _dev(np.concatenate([d0[:50], d0, d0[:30]]))
    e = _dev(np.concatenate([e0[:50], e1, e0[:30]]))
    _refused(lambda: hp.mdstedc_batch_dev(sizes, d, e, _new(int((sizes.astype(int) ** 2).sum()))), d)
    w, q = hp.eigh_tridiagonal(d0, e0[:n - 1])
    t = np.diag(d0) + np.diag(e0[:n - 1], 1) + np.diag(e0[:n - 1], -1)
    assert np.abs(w - np.linalg.eigvalsh(t)).max() <= 1e-13


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("where", [("d", 0), ("d", 100), ("e", 50), ("e", 198)])
def test_bidiagonal_merges(bad, where):
    n = 200
    rng = np.random.default_rng(2)
    x = {"d": rng.uniform(0.1, 1, n), "e": rng.uniform(0.1, 1, n)}
    x[where[0]][where[1]] = bad
    d = _dev(x["d"])
    _refused(lambda: hp.mdbdsdc_dev(d, _dev(x["e"]), _new(n * n), _new(n * n)), d)
    with pytest.raises(hp.HssError):
        hp.svd_bidiagonal(x["d"], x["e"][:n - 1], lower=True)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("n,kd", [(200, 4), (150, 16)])
def test_band_merges(n, kd, bad):
    """In a leaf's inside, on its diagonal, in the coupling of two leaves.  (An infinity
    inside a leaf is not looked for: its rotations are all skipped.)"""
    rng = np.random.default_rng(3)
    ab = rng.uniform(-1, 1, (n, kd + 1))  # ab[j, kd + i - j] = A(i, j)
    for j, o in ((3, 0), (3, 1), (n // 2, kd), (n // 2, 1)):
        if np.isinf(bad) and j == 3:
            continue
        x = ab.copy()
        x[j, kd - o] = bad
        w = _new(n)
        _refused(lambda: hp.mdsbevd_dev(kd, _dev(x), w, _new(n * n)), w)


@pytest.mark.parametrize("bad", BAD)
@pytest.mark.parametrize("n,sb", [(20, 3), (300, 1), (300, 5), (200, 16)])
def test_banded_svd(n, sb, bad):
    """Anywhere: leaf, appended rows, extra columns (and in a single leaf)."""
    rng = np.random.default_rng(4)
    ab = rng.uniform(0, 1, (n, sb + 1))
    s = _new(n)
    for j in {sb, n // 2 - 1, n // 2, n // 2 + sb // 2, n // 2 + sb, n // 4, n - 1}:
        for o in {0, sb}:
            x = ab.copy()
            x[j, sb - o] = bad
            _refused(lambda: hp.mdbdsvd_dev(sb, _dev(x), s, _new(n * n), _new(n * n)), s)
    # entries outside the matrix are not read
    ab[0, :sb] = bad
    hp.mdbdsvd_dev(sb, _dev(ab), s, _new(n * n), _new(n * n))
    a = np.zeros((n, n))
    for o in range(sb + 1):
        a += np.diag(ab[o:, sb - o], o)
    ref = np.linalg.svd(a, compute_uv=False)
    assert np.abs(s.cpu().numpy() - ref).max() <= 1e-13 * ref[0]
