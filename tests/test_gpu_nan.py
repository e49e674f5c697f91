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
