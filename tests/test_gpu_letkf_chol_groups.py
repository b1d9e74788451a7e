"""FP64 Cholesky local analyses of up to 32 members with an analysis per warp and
per four warps: point counts on both sides of the rule (two points per SM),
local lists at the edges of the gathered rows and of the filtered block, against
the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
CHOL, UPD, RTPS = _lib.MG_SQRT_CHOLESKY, _lib.MG_UPDATE_COMPAT, _lib.MG_RTPS


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("k", [2, 8, 9, 15, 16, 17, 31, 32])
@pytest.mark.parametrize("flags,n_var", [(_lib.MG_COMPAT, 1), (CHOL, 5), (CHOL | UPD, 2), (CHOL | RTPS, 3)])
def test_both_group_sizes(dev, flags, n_var, k, few):
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    ncol = 2 * sms if few else 2 * sms + 1
    g = np.random.default_rng(10 * k + flags)
    p, n = 150, ncol * n_var
    X = g.standard_normal((k, n)) + 3.0
    HX = g.standard_normal((p, k)) + 1.0
    yo, rvar = g.standard_normal(p) + 1.0, g.uniform(0.2, 2.0, p)
    counts = g.integers(0, 20, ncol)
    counts[:12] = [0, 1, 15, 16, 17, 31, 32, 33, 127, 128, 129, 150]
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([np.sort(g.choice(p, c, replace=False)) for c in counts]).astype(np.int32)
    dist = g.uniform(0.0, 9.9, len(idx))
    rho = 0.9 if flags & RTPS else 1.07
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    Xd = T(X)
    _, st = K.letkf_batched(Xd, col_base=T(np.arange(ncol, dtype=np.int64)), nlev=1, n_var=n_var, lev_stride=ncol,
                            var_stride=ncol, HX=T(HX), yo=T(yo), rvar=T(rvar), loc_off=T(off), loc_idx=T(idx),
                            loc_dist=T(dist), hsupport=10.0, rho=rho, flags=flags)
    w = np.array([ob.gaspari_cohn(b / 5.0) for b in dist])
    if flags & _lib.MG_R_IDENTITY:
        w[:] = 1.0
    assert (w > 0.0).all() and st.total_local == counts.sum()
    res = ob.letkf_points(X, np.arange(ncol), n_var, ncol, HX, yo, rvar, off, idx, w, rho, flags)
    for v in range(n_var):
        assert rel_err(Xd[:, v * ncol:(v + 1) * ncol].cpu().numpy(), res[:, v].T) <= FP64_TOL
