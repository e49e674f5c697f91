"""An HSS merge that cannot be built ends in INFO at every entry that runs merges, not in an
uncaught C++ exception.  A leaf size of 1 makes a tree of 1500 leaves on one level, which the
construction refuses on the host."""
import numpy as np
import pytest
import torch

import hsspack_gb300 as hp

pytestmark = pytest.mark.gpu

N = 1500


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _new(n):
    return torch.empty(n, dtype=torch.float64, device="cuda")


def _calls():
    d, e = 2.0 + 1e-3 * np.sin(np.arange(N)), np.ones(N)
    ab = 1.0 + 1e-3 * np.random.default_rng(0).uniform(-1, 1, (N, 3))  # little deflates
    sizes = np.array([N, 40], dtype=np.int32)
    return {
        "mdstedc_dev": lambda: hp.mdstedc_dev(_dev(d), _dev(e), _new(N * N)),
        "mdstedc_v_dev": lambda: hp.mdstedc_v_dev(_dev(d), _dev(e), _dev(np.eye(N))),
        "mdstedc_batch_dev": lambda: hp.mdstedc_batch_dev(
            sizes, _dev(np.concatenate([d, d[:40]])), _dev(np.concatenate([e, e[:40]])),
            _new(N * N + 1600)),
        "mdstedc": lambda: hp.eigh_tridiagonal(d, e[:N - 1]),
        "mdsbevd_dev": lambda: hp.mdsbevd_dev(2, _dev(ab), _new(N), _new(N * N)),
        "mdsbedc": lambda: hp.eigh_banded(np.asfortranarray(ab.T)),
        "mdbdsdc_dev": lambda: hp.mdbdsdc_dev(_dev(np.ones(N)), _dev(e), _new(N * N), _new(N * N)),
        "mdbdsdc": lambda: hp.svd_bidiagonal(np.ones(N), e[:N - 1]),
        "mdbdsvd_dev": lambda: hp.mdbdsvd_dev(2, _dev(ab), _new(N), _new(N * N), _new(N * N)),
    }


@pytest.mark.parametrize("name", ["mdstedc_dev", "mdstedc_v_dev", "mdstedc_batch_dev", "mdstedc",
                                  "mdsbevd_dev", "mdsbedc", "mdbdsdc_dev", "mdbdsdc", "mdbdsvd_dev"])
def test_refused_merge(name):
    old = hp.set_config(bsmlz=1030, hss_leaf=1)
    try:
        with pytest.raises(hp.HssError, match="too wide"):
            _calls()[name]()
    finally:
        hp.restore_config(old)
    w, q = hp.eigh_tridiagonal(np.arange(30.0), np.ones(29))
    assert np.linalg.norm(q.T @ q - np.eye(30)) <= 1e-13
