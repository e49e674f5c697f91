"""The batch's final ordering at the edges of its 16-byte stores: odd and even columns, a
base that is and is not 16-byte aligned, one-row problems; nothing outside is written."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp
from helpers import rand_tridiag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
def test_batch_outputs(shift):
    sizes = [1, 2, 3, 31, 64, 65, 66, 1, 257, 130]
    probs = [rand_tridiag(n, n) for n in sizes]
    s, D, E = hp.pack_batch(probs)
    oz = np.concatenate([[0], np.cumsum(np.array(sizes, dtype=np.int64) ** 2)])
    buf = torch.full((int(oz[-1]) + 2 + shift,), float("nan"), dtype=torch.float64, device="cuda")
    z = buf[1 + shift:-1]
    d, e = torch.tensor(D, device="cuda"), torch.tensor(E, device="cuda")
    hp.mdstedc_batch_dev(s, d, e, z)
    assert bool(torch.isnan(buf[:1 + shift]).all()) and bool(torch.isnan(buf[-1]))
    w, at = d.cpu().numpy(), 0
    for p, (n, (dd, ee)) in enumerate(zip(sizes, probs)):
        Q = z[int(oz[p]):int(oz[p + 1])].view(n, n).T.cpu().numpy()
        T = np.diag(dd) + np.diag(ee, 1) + np.diag(ee, -1)
        W = w[at:at + n]
        at += n
        # the acceptance of the full solves
        tn = np.abs(T).sum(axis=1).max()
        assert np.linalg.norm(T @ Q - Q * W) / (n * tn) <= 1e-12
        assert np.linalg.norm(Q.T @ Q - np.eye(n)) / n <= 1e-12
