"""What the kernels promise to the last bits: the helpers that replace sqrt and divides
against numpy's (correctly rounded) ones, the Jacobi angle against extended precision, and
the leaf solvers against their iterations as plain loops (tests/device_check.cu)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest
import torch

import hsspack_gb300 as hp
from hsspack_gb300 import build as hb

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("check") / "device_check.so")
    subprocess.run([hb._nvcc()] + hb.ARCH + hb.FLAGS +
                   ["-shared", os.path.join(HERE, "device_check.cu"), "-o", so], check=True)
    x = ctypes.CDLL(so)
    x.check_work_bytes.restype = ctypes.c_longlong
    return x


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ops(lib, op, a, b=None, c=None, z=None):
    t = [_dev(v if v is not None else a) for v in (a, b, c)]
    out = [torch.zeros_like(t[0]), torch.zeros_like(t[0]), _dev(z if z is not None else a)]
    torch.cuda.synchronize()
    assert lib.check_ops(op, len(a), *[_p(v) for v in t + out]) == 0
    return [v.cpu().numpy() for v in out]


def _operands(n, seed, lo, hi):
    """Random mantissas and signs, exponents of lo .. hi; a share just below a power of two
    and one with few bits."""
    rng = np.random.default_rng(seed)
    m = rng.uniform(1.0, 2.0, n)
    m[: n // 8] = 2.0 - 2.0 ** -52 * rng.integers(1, 5, n // 8)
    m[n // 8: n // 4] = 1.0 + 2.0 ** -rng.integers(1, 53, n // 4 - n // 8)
    return np.ldexp(m * rng.choice([-1.0, 1.0], n), rng.integers(lo, hi, n))


N = 1 << 20


def test_roots(lib):
    x = np.abs(_operands(N, 1, -960, 960))
    r = np.sqrt(x)
    got = _ops(lib, 0, x)
    assert np.array_equal(got[0], r)
    assert np.array_equal(got[1], 1.0 / r)


@pytest.mark.parametrize("lo,hi", [(-479, 479), (-3, 3), (-1000, 1000)])
def test_quotients(lib, lo, hi):
    a, b = _operands(N, 2, lo, hi), _operands(N, 3, lo, hi)[::-1].copy()
    with np.errstate(all="ignore"):
        ref = a / b
    assert np.array_equal(_ops(lib, 1, a, b)[0], ref)
    if hi < 1000:
        assert np.array_equal(_ops(lib, 2, b)[0], 1.0 / b)


def test_quotients_next_to_a_midpoint(lib):
    """a / b at a distance of 2^-54 ulps from the middle of two doubles, the closest there
    is: b q = a 2^54 -+ 1 with an odd q.  There the result may be either neighbour."""
    rng = np.random.default_rng(4)
    a, b = [], []
    while len(a) < 4096:
        x = int(rng.integers(1 << 52, 1 << 53)) | 1
        s = 1 if len(a) % 2 else -1
        q = -s * pow(x, -1, 1 << 54) % (1 << 54)
        y, rest = divmod(x * q + s, 1 << 54)
        assert rest == 0
        if q >> 53 and 0 < y < 1 << 53:
            a.append(float(y))
            b.append(float(x))
    a, b = np.array(a), np.array(b)
    ref = a / b
    assert (np.abs(_ops(lib, 1, a, b)[0] - ref) <= np.spacing(ref)).all()


def test_reflector(lib):
    alpha = _operands(N, 5, -200, 200)
    sg = np.abs(_operands(N, 6, -400, 400))[::-1].copy()
    beta, tau, scale = _ops(lib, 3, alpha, sg)
    x = np.longdouble(alpha) * alpha + sg  # one rounding more than the kernel's fma
    ok = np.abs(beta) - np.sqrt(x).astype(np.float64)
    assert (np.abs(ok) <= np.spacing(np.abs(beta))).all() and (beta * alpha < 0).all()
    L = np.longdouble
    exact = 1 + np.abs(L(alpha)) / np.sqrt(L(alpha) * alpha + sg)
    # 1 / |beta| within an ulp times a factor of at most 1, and one rounding
    assert (np.abs(L(tau) - exact) <= 1.5 * 2.0 ** -52).all()
    assert np.array_equal(scale, 1.0 / (alpha - beta))


@pytest.mark.parametrize("spread", [2, 40, 300])
def test_jacobi_tangent(lib, spread):
    """Root of smaller modulus of c t^2 + x t - c, x = b - a.  The last step rounds once
    and its residual's error is at most half an ulp of t more: two ulps, four where the
    operands' range calls for the plain formula."""
    rng = np.random.default_rng(spread)
    n = 1 << 18
    a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-spread, spread, n))
    b = a * np.ldexp(rng.uniform(0.5, 1, n), rng.integers(-60, 60, n))
    b[: n // 4] = a[: n // 4] * (1.0 + np.ldexp(rng.uniform(-1, 1, n // 4), -rng.integers(0, 53, n // 4)))
    b[b == a] *= 1.5
    c = np.sqrt(a) * np.sqrt(b) * np.ldexp(rng.uniform(-1, 1, n), -rng.integers(0, 40, n))
    t, go, _ = _ops(lib, 4, a, b, c, np.full(n, 1e-30))
    L = np.longdouble
    x = L(b - a)
    ref = 2 * L(c) / (x + np.copysign(np.sqrt(x * x + 4 * L(c) * L(c)), x))
    go = go != 0
    assert go.sum() > n // 2
    err = np.abs((t - ref) / L(1) / np.spacing(np.abs(ref.astype(np.float64))))[go]
    assert err.max() <= (2.0 if spread <= 300 else 4.0), float(err.max())


def test_jacobi_threshold(lib):
    """Every pair with c^2 > jtol^2 a b in FP64 is rotated, none with less than 0.9999 of it."""
    rng = np.random.default_rng(9)
    n = 1 << 18
    a = np.ldexp(rng.uniform(1, 2, n), rng.integers(-200, 200, n))
    b = a * np.ldexp(rng.uniform(0.5, 1, n), rng.integers(-20, 20, n))
    j2 = (2.0 ** -52 * rng.integers(16, 129, n)) ** 2
    c = np.sqrt(j2 * a * b) * (1.0 + np.ldexp(rng.uniform(-1, 1, n), -rng.integers(1, 53, n)))
    c *= rng.choice([-1.0, 1.0], n)
    go = _ops(lib, 4, a, b, c, j2)[1] != 0
    assert go[c * c > j2 * a * b].all() and not go[c * c < 0.9999 * j2 * a * b].any()


def _plain(lib, svd, sizes, d, e):
    off = np.concatenate([[0], np.cumsum(sizes)[:-1]]).astype(np.int32)
    zoff = np.concatenate([[0], np.cumsum(sizes.astype(np.int64) ** 2)])
    work = torch.empty(lib.check_work_bytes() * len(sizes), dtype=torch.uint8, device="cuda")
    new = lambda n: torch.empty(int(n), dtype=torch.float64, device="cuda")
    w, u, v = new(sizes.sum()), new(zoff[-1]), new(zoff[-1])
    ms, of, zo = _dev(sizes), _dev(off), _dev(zoff[:-1].copy())
    torch.cuda.synchronize()
    assert lib.check_leaves(svd, len(sizes), _p(ms), _p(of), _p(zo), _p(d), _p(e), _p(work), _p(w),
                            _p(u), _p(v)) == 0
    return w, u, v


@pytest.mark.parametrize("count,most", [(1, 32), (40, 32), (1500, 16), (3000, 32), (6000, 24),
                                        (20000, 32), (30000, 16), (60000, 12), (60000, 8)])
def test_tridiagonal_leaves(lib, count, most):
    """Single-leaf problems, with every number of lanes per leaf, bit for bit."""
    rng = np.random.default_rng(count + most)
    sizes = rng.integers(2, most + 1, count).astype(np.int32)
    sizes[0] = most
    n = int(sizes.sum())
    d0, e = _dev(rng.uniform(-1, 1, n)), _dev(rng.uniform(-1, 1, n))
    w, z, _ = _plain(lib, 0, sizes, d0, e)
    d, zb = d0.clone(), torch.empty_like(z)
    old = hp.set_config(smlsiz=32)
    try:
        hp.mdstedc_batch_dev(sizes, d, e, zb)
    finally:
        hp.restore_config(old)
    assert torch.equal(d, w) and torch.equal(zb, z)


@pytest.mark.parametrize("n", list(range(2, 33)))
def test_bidiagonal_leaf(lib, n):
    rng = np.random.default_rng(n)
    old = hp.set_config(smlsiz=32)
    try:
        for _ in range(4):
            d0, e0 = rng.uniform(0.05, 1, n), rng.uniform(0.05, 1, n)
            d0[rng.integers(n)] = 1.0  # the norm, so nothing is scaled
            d, e = _dev(d0), _dev(e0)
            w, u, v = _plain(lib, 1, np.array([n], dtype=np.int32), d, e)
            uo, vo = torch.empty_like(u), torch.empty_like(v)
            hp.mdbdsdc_dev(d, e, uo, vo)
            assert torch.equal(d, w.flip(0))
            assert torch.equal(uo.view(n, n), u.view(n, n).flip(0))
            assert torch.equal(vo.view(n, n), v.view(n, n).flip(0).T)
    finally:
        hp.restore_config(old)


def _digit_rows(x):
    """Seven rounded base-256 digits (ties up) of the rows of x scaled to below 2^60 by the
    exponent of the row's largest entry, and those exponents."""
    e = np.frexp(np.abs(x).max(axis=1))[1]
    q = [[int(v) for v in np.ldexp(r, 60 - int(ei))] for r, ei in zip(x, e)]
    d = []
    for row in q:
        digs = []
        for v in row:
            ds = []
            for s in range(7):
                sh = 53 - 8 * s
                t = (v + (1 << (sh - 1))) >> sh
                ds.append(t)
                v -= t << sh
            digs.append(ds)
        d.append(digs)
    return d, e


@pytest.mark.parametrize("k", [8, 127, 128, 129, 300])
@pytest.mark.parametrize("path", [0, 1])
def test_split_product_bits(k, path):
    """The split products' own arithmetic in Python integers: digit products of groups 0 to 6,
    exact sums, one rounding (path 1: one per window of 128, added up).  Entries of at least
    2^-7 of their row's largest, so the scaled integers are exact."""
    rng = np.random.default_rng(k)
    m, n = 140, 40
    A, B = (rng.uniform(0.01, 1.0, s) * rng.choice([-1.0, 1.0], s) for s in ((m, k), (k, n)))
    A *= np.ldexp(1.0, rng.integers(-30, 30, (m, 1)))
    A[:, 0] = np.abs(A).max(axis=1)
    B[0] = 1.0
    dA, dB = (_dev(x.ravel(order="F")) for x in (A, B))
    dC = torch.empty(m * n, dtype=torch.float64, device="cuda")
    old = hp.set_config(gemm_path=path, split_min_log2=15)
    try:
        hp.gemm_dev(dA, dB, dC, m, n, k, m, k, m, precision=1)
    finally:
        hp.restore_config(old)
    C = dC.cpu().numpy().reshape(m, n, order="F")
    rows, cols = [0, 31, 32, 127, 128, 139], [0, 15, 16, 31, 32, 39]
    da, ea = _digit_rows(A[rows])
    db, eb = _digit_rows(B[:, cols].T)
    for i, r in enumerate(rows):
        for j, c in enumerate(cols):
            parts = []
            for w0 in range(0, k, 128) if path else [0]:
                v = 0
                for t in range(w0, min(k, w0 + 128) if path else k):
                    for s in range(7):
                        for p in range(7 - s):
                            v += (da[i][t][s] * db[j][t][p]) << (8 * (6 - s - p))
                parts.append(v)
            # weight of group 6: 2^(e + f - 30 - 32)
            ref = 0.0
            for v in parts:
                ref += np.ldexp(float(v), int(ea[i] + eb[j]) - 62)
            assert C[r, c] == ref, (r, c, C[r, c], ref)
