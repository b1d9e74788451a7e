"""FP64 local analyses with the Cholesky square root (the reference's form)
against the oracle, at the edges of the kernel's member layouts, with and
without weights, levels, variables and the per-member update."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
CHOL, INFL, UPD, RID = _lib.MG_SQRT_CHOLESKY, _lib.MG_INFL_COMPAT, _lib.MG_UPDATE_COMPAT, _lib.MG_R_IDENTITY


@pytest.mark.parametrize("k", [2, 9, 16, 17, 31, 32, 33, 48, 64, 65, 96])
@pytest.mark.parametrize("flags,n_var,nlev", [(_lib.MG_COMPAT, 1, 1), (CHOL, 3, 3), (CHOL | INFL | UPD, 5, 2),
                                              (CHOL | _lib.MG_RTPS, 2, 3), (CHOL | RID | INFL, 1, 2)])
def test_chol_matches_oracle(dev, k, flags, n_var, nlev):
    g = np.random.default_rng(100 * k + flags)
    ncol, p = 23, 150
    n = ncol * nlev * n_var
    X = g.standard_normal((k, n)) + 3.0
    HX = g.standard_normal((p, k)) + 1.0
    yo, rvar = g.standard_normal(p) + 1.0, g.uniform(0.2, 2.0, p)
    lev = g.uniform(0.0, max(nlev - 1, 1), p)
    counts = g.integers(0, 140, ncol)
    counts[:4] = [0, 1, 128, 129]
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([np.sort(g.choice(p, c, replace=False)) for c in counts]).astype(np.int32)
    dist = g.uniform(0.0, 9.9, len(idx))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    Xd = T(X)
    mean, st = K.letkf_batched(Xd, col_base=T(np.arange(ncol, dtype=np.int64)), nlev=nlev, n_var=n_var,
                               lev_stride=ncol, var_stride=ncol * nlev, HX=T(HX), yo=T(yo), rvar=T(rvar),
                               loc_off=T(off), loc_idx=T(idx), loc_dist=T(dist), obs_lev=T(lev), hsupport=10.0,
                               vsupport=1.5, rho=1.07 if not flags & _lib.MG_RTPS else 0.9, flags=flags)
    # point lists and weights as the library forms them (no Gaspari-Cohn weights with R = I)
    want = np.empty_like(X)
    nloc = 0
    for c in range(ncol):
        for l in range(nlev):
            o, d = idx[off[c]:off[c + 1]], dist[off[c]:off[c + 1]]
            dl = np.abs(lev[o] - l)
            w = np.ones(len(o))
            if not flags & RID:
                w = np.array([ob.gaspari_cohn(a / 0.75) * ob.gaspari_cohn(b / 5.0) for a, b in zip(dl, d)])
            keep = (dl <= 1.5) & (w > 0.0)
            nloc += int(keep.sum())
            res = ob.letkf_points(X, np.array([l * ncol + c], dtype=np.int64), n_var, ncol * nlev, HX, yo, rvar,
                                  np.array([0, keep.sum()], dtype=np.int64), o[keep].astype(np.int32),
                                  np.ascontiguousarray(w[keep]), 1.07 if not flags & _lib.MG_RTPS else 0.9, flags)
            for v in range(n_var):
                want[:, (v * nlev + l) * ncol + c] = res[0, v]
    assert st.total_local == nloc
    assert rel_err(Xd.cpu().numpy(), want) <= FP64_TOL
    assert rel_err(mean.cpu().numpy(), want.mean(0)) <= FP64_TOL
