"""The pivot decisions of the HSS compression do not depend on the scale of u and v: with
both multiplied by a power of two every FP64 operation scales exactly, so the product is
the same to the last bit but for the factor."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu


def _poles(n, weak, strong):
    """Interlacing poles one apart, but 1e-4 apart around index `weak` and 1e-8 around
    `strong`, two ends of one leaf.  Its row and column searches stop at the entries of 1e4
    at the weak end; the next pivot, in the smooth part, is below the tolerance, and only
    the search over all that is left finds the entries of 1e8 at the strong end."""
    step = np.ones(2 * n)
    step[2 * (weak - 1):2 * (weak + 1)] = 1e-4
    step[2 * (strong - 1):2 * (strong + 1)] = 1e-8
    x = np.concatenate([[0.0], np.cumsum(step)])
    return x[0:2 * n:2], x[1:2 * n + 1:2]


@pytest.mark.parametrize("exponent", [-60, -100, 40])
@pytest.mark.parametrize("n,seed", [(512, 0), (512, 1), (256, 2)])
def test_product_scales_exactly(n, seed, exponent):
    ni, tol, sc = 64, 1e-4, 2.0 ** exponent
    F, D = _poles(n, 64, 128)
    rng = np.random.default_rng(seed)
    u, v = rng.uniform(0.5, 1.0, n), rng.uniform(0.5, 1.0, n)
    B = rng.standard_normal((n, 32))
    C = u[:, None] * v[None, :] / (D[:, None] - F[None, :])

    def product(s):
        dev = [torch.tensor(np.ascontiguousarray(a), device="cuda") for a in (D, F, u * s, v * s, B.T)]
        hp.cauchyhssmm_dev(*dev, ni, tol)
        y = dev[4].cpu().numpy().T / s / s
        # what is dropped of a block is below tol times its largest entry, per entry
        err = np.linalg.norm(y - C @ B) / (np.linalg.norm(C) * np.linalg.norm(B, 2))
        return y, err, hp.get_stats()["max_rank"]

    old = hp.set_config(precision=0)
    try:
        y1, e1, r1 = product(1.0)
        y2, e2, r2 = product(sc)
    finally:
        hp.restore_config(old)
    assert e1 <= 1e-3 and e2 <= 1e-3, (e1, e2)
    assert r1 == r2
    assert np.array_equal(y1, y2)
