"""Split-BF16 products at the edges of their digits and exactness windows: operands
whose digit planes are all at the ends of their range, K around the window of 128
and the stages of 16, against the exact rational product."""
from fractions import Fraction

import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu


def _edge_values(rng, shape):
    # bytes 0x7f, 0x80, 0xff, 0x00 below the leading bits: digits 127, +-128, 0 and
    # the carries between them
    byte = rng.choice(np.array([0x00, 0x7f, 0x80, 0xff], dtype=np.int64), size=shape + (6,))
    m = np.full(shape, 0x1f, dtype=np.int64)  # 5 leading ones, then 48 bits
    for k in range(6):
        m = (m << 8) | byte[..., k]
    return np.ldexp(m.astype(np.float64), -53) * rng.choice([-1.0, 1.0], size=shape)


@pytest.mark.parametrize("kind", ["edges", "same_sign", "full"])
@pytest.mark.parametrize("k", [1, 16, 17, 112, 127, 128, 129, 144, 256, 300])
def test_split_digits_exact(kind, k):
    rng = np.random.default_rng(k)
    m, n = 130, 33  # a second row panel of 2 rows, a second column tile of 1
    A, B = _edge_values(rng, (m, k)), _edge_values(rng, (k, n))
    if kind == "same_sign":
        A, B = np.abs(A), np.abs(B)
    elif kind == "full":  # the largest group sums: every digit at an end
        A[:] = np.ldexp(float(0x1f7f7f7f7f7f7f), -53)
        B[:] = -A[0, 0]
    dA, dB = (torch.tensor(x.ravel(order="F"), device="cuda") for x in (A, B))
    dC = torch.empty(m * n, dtype=torch.float64, device="cuda")
    hp.gemm_dev(dA, dB, dC, m, n, k, m, k, m, precision=1)
    C = dC.cpu().numpy().reshape(m, n, order="F")
    rows, cols = [0, 1, 31, 32, 64, 127, 128, 129], [0, 1, 15, 16, 31, 32]
    for i in rows:
        for j in cols:
            a, b = [Fraction(x) for x in A[i]], [Fraction(x) for x in B[:, j]]
            exact = sum(x * y for x, y in zip(a, b))
            scale = sum(abs(x * y) for x, y in zip(a, b))
            # 56-bit operands, dropped products below 2^-56 each side, one rounding
            assert abs(Fraction(C[i, j]) - exact) <= scale * Fraction(1, 2 ** 50), (i, j)
