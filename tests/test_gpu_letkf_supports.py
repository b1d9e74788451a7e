"""Local analyses with an infinite localisation support: no localisation in
that direction (weight 1 at every distance), horizontally, vertically or both,
and supports whose halves or their reciprocals lie at the ends of the exponent
range, by each of the kernels, against the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

INF = float("inf")
MIXED, FP64 = _lib.MG_PREC_MIXED, _lib.MG_PREC_FP64


@pytest.mark.parametrize("hs,vs", [(INF, 1.5), (10.0, INF), (INF, INF), (1e308, 1e308), (10.0, 1e250)])
@pytest.mark.parametrize("k", [12, 40, 70])
@pytest.mark.parametrize("flags,precision,tol", [(0, FP64, 1e-10), (_lib.MG_UPDATE_COMPAT, FP64, 1e-10),
                                                 (_lib.MG_SQRT_CHOLESKY, FP64, 1e-10), (0, MIXED, 1e-5),
                                                 (_lib.MG_SOLVE_SIMT, MIXED, 1e-5)])
def test_infinite_supports(dev, flags, precision, tol, k, hs, vs):
    g = np.random.default_rng(k)
    ncol, nlev, n_var, p = 5, 4, 2, 60
    n = ncol * nlev * n_var
    X = g.standard_normal((k, n)) + 3.0
    HX = g.standard_normal((p, k)) + 1.0
    yo, rvar = g.standard_normal(p) + 1.0, g.uniform(4.0, 8.0, p)
    lev = g.uniform(0.0, nlev - 1.0, p)
    counts = np.array([0, 1, 33, 40, 60])
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([np.sort(g.choice(p, c, replace=False)) for c in counts]).astype(np.int32)
    dist = g.uniform(0.0, 9.0, len(idx))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    Xd = T(X)
    _, st = K.letkf_batched(Xd, col_base=T(np.arange(ncol, dtype=np.int64)), nlev=nlev, n_var=n_var, lev_stride=ncol,
                            var_stride=ncol * nlev, HX=T(HX), yo=T(yo), rvar=T(rvar), loc_off=T(off), loc_idx=T(idx),
                            loc_dist=T(dist), obs_lev=T(lev), hsupport=hs, vsupport=vs, rho=1.07, flags=flags,
                            precision=precision)
    want, nloc = np.empty_like(X), 0
    for c in range(ncol):
        for l in range(nlev):
            o, d = idx[off[c]:off[c + 1]], dist[off[c]:off[c + 1]]
            dl = np.abs(lev[o] - l)
            w = np.array([ob.gaspari_cohn(a / (0.5 * vs)) * ob.gaspari_cohn(b / (0.5 * hs)) for a, b in zip(dl, d)])
            keep = (dl <= vs) & (w > 0.0)
            nloc += int(keep.sum())
            res = ob.letkf_points(X, np.array([l * ncol + c], dtype=np.int64), n_var, ncol * nlev, HX, yo, rvar,
                                  np.array([0, keep.sum()], dtype=np.int64), o[keep].astype(np.int32),
                                  np.ascontiguousarray(w[keep]), 1.07, flags & ~_lib.MG_SOLVE_SIMT)
            for v in range(n_var):
                want[:, (v * nlev + l) * ncol + c] = res[0, v]
    assert st.total_local == nloc > 0
    assert rel_err(Xd.cpu().numpy(), want) <= tol
