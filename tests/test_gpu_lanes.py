"""Lane groups and searches that follow a level's sizes: eigenvector blocks with 4 to
32 lanes per column, products found by warps that straddle several of them."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu


# few merges of many roots (32 lanes per column), one large problem, and many small
# ones (4 lanes), whose bottom merges have one to a few roots
@pytest.mark.parametrize("count,n,smlsiz,kind", [(1, 70, 16, "random"), (1, 3000, 32, "chain"),
                                                 (1, 6000, 8, "random"), (300, 97, 4, "random"),
                                                 (2000, 33, 2, "random"), (900, 130, 8, "chain")])
@pytest.mark.parametrize("precision", [0, 1])
def test_vector_blocks(count, n, smlsiz, kind, precision):
    rng = np.random.default_rng(n)
    d = rng.uniform(-1, 1, (count, n))
    e = rng.uniform(-1, 1, (count, n))
    if kind == "chain":
        d, e = 2.0 + 1e-3 * d, 1.0 + 1e-3 * e
    d0, e0 = (torch.tensor(x, device="cuda") for x in (d, e))
    w, z = d0.reshape(-1).clone(), torch.empty(count * n * n, dtype=torch.float64, device="cuda")
    old = hp.set_config(smlsiz=smlsiz, precision=precision, bsmlz=10 ** 6)
    try:
        hp.mdstedc_batch_dev(np.full(count, n, dtype=np.int32), w, e0.reshape(-1).clone(), z)
    finally:
        hp.restore_config(old)
    w, Q = w.view(count, n), z.view(count, n, n).transpose(1, 2)
    T = torch.diag_embed(d0) + torch.diag_embed(e0[:, :-1], 1) + torch.diag_embed(e0[:, :-1], -1)
    tn = float(d0.abs().max() + 2 * e0.abs().max())
    # the acceptance of the full solves, per problem
    R = T @ Q - Q * w[:, None, :]
    assert float(torch.linalg.norm(R, dim=(1, 2)).max()) / (n * tn) <= 1e-12
    G = Q.transpose(1, 2) @ Q - torch.eye(n, dtype=torch.float64, device="cuda")
    assert float(torch.linalg.norm(G, dim=(1, 2)).max()) / n <= 1e-12
    few = slice(0, 8)
    assert float((w[few] - torch.linalg.eigvalsh(T[few])).abs().max()) <= 1e-13 * tn
