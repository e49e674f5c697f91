"""What the kernels promise to the last bits: the leaf solvers against their iterations as
plain loops (tests/device_check.cu)."""
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
