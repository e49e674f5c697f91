"""Products through the entry points that run no eigensolve, on device memory that
held something else before: the products' error word has to be cleared by each."""
import ctypes

import numpy as np
import pytest
import torch

import hsspack_gb300 as hp
from helpers import interlace_grid

pytestmark = pytest.mark.gpu


@pytest.fixture
def used_memory():
    """The library's buffers given back, and the small blocks it will get next filled."""
    hp.finalize()
    torch.zeros(1, device="cuda")
    cu = ctypes.CDLL("libcuda.so.1")
    ptrs = []
    for _ in range(16384):
        p = ctypes.c_uint64()
        assert cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(4)) == 0
        assert cu.cuMemsetD32_v2(p, ctypes.c_uint(1), ctypes.c_size_t(1)) == 0
        ptrs.append(p)
    torch.cuda.synchronize()
    keep = ptrs[::64]  # the slabs stay with the process
    for i, p in enumerate(ptrs):
        if i % 64:
            assert cu.cuMemFree_v2(p) == 0
    yield
    for p in keep:
        assert cu.cuMemFree_v2(p) == 0


@pytest.mark.parametrize("entry", ["dhssmm", "cauchyhssmm", "dhssevc", "svdhssupdat"])
def test_products_on_used_memory(entry, used_memory):
    n = 600
    rng = np.random.default_rng(0)
    F, D = interlace_grid(n)
    u, v = rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 1.0, n)
    C = u[:, None] * v[None, :] / (D[:, None] - F[None, :])
    B = rng.standard_normal((n, n))

    def dev(a):
        return torch.tensor(np.ascontiguousarray(a), device="cuda")

    old = hp.set_config(precision=1)
    try:
        if entry == "dhssmm":
            b = dev(B.T)
            hp.dhssmm_dev(dev(C.T), b, 64, 1e-11)
            out, ref = b.cpu().numpy().T, C @ B
        elif entry == "cauchyhssmm":
            b = dev(B.T)
            hp.cauchyhssmm_dev(dev(D), dev(F), dev(u), dev(v), b, 64, 1e-14)
            out, ref = b.cpu().numpy().T, C @ B
        elif entry == "svdhssupdat":
            # right singular vectors of [diag(f); z^T], the rows of the result
            f, z = np.sort(rng.uniform(0.1, 1.0, n)), rng.uniform(0.5, 1.0, n)
            vt = dev(np.eye(n).ravel())
            k = hp.svdhssupdat_dev(torch.zeros(n, dtype=torch.float64, device="cuda"), dev(f), dev(z),
                                   vt, 1e-14, 64)
            assert k == n
            V = vt.cpu().numpy().reshape(n, n, order="F")
            A = np.vstack([np.diag(f), z])
            G = V @ (A.T @ A) @ V.T
            out, ref = G, np.diag(np.diag(G))
        else:
            # C(i, j) = u_i v_j / (F_i - lam_j), lam_j = D_j between F_j and F_{j+1}
            dr = np.append(D[:-1] - F[1:], 0.0)
            q = dev(B.T)
            hp.dhssevc_dev(dev(F), dev(u), dev(v), dev(D - F), dev(dr), q, n, n, ni=64, tol=1e-14)
            out = q.cpu().numpy().T
            ref = B @ (u[:, None] * v[None, :] / (F[:, None] - D[None, :]))
    finally:
        hp.restore_config(old)
    # the tests of these entries allow 1e-11 for the compression
    assert np.linalg.norm(out - ref) / np.linalg.norm(ref) <= 1e-11
