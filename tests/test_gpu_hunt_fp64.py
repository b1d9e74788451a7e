"""FP64 symmetric square root from a corrected FP32 eigenbasis: local and
global analyses against the oracle at the edges of the member layouts, with
every combination of weights, levels, variables, inflation and update that
takes this path, from few vague obs to ill-conditioned systems (those the
correction leaves to the FP64 Jacobi included)."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
EPS = np.finfo(np.float64).eps


def _tol(kappa):
    """Any FP64 method, the oracle's Jacobi included, forms A with a backward
    error of a few eps ||A||, a relative error of a few eps kappa in its
    small eigenvalues."""
    return max(FP64_TOL, 16.0 * EPS * kappa)


def _kappa(Yw, k, rho):
    lam = np.linalg.eigvalsh(Yw.T @ Yw)
    return 1.0 + max(lam[-1], 0.0) * rho / (k - 1)

INFL, UPD, RID, RTPS = _lib.MG_INFL_COMPAT, _lib.MG_UPDATE_COMPAT, _lib.MG_R_IDENTITY, _lib.MG_RTPS


def _run(dev, k, flags, n_var, nlev, sigma, p=180, ncol=14, seed=0):
    g = np.random.default_rng(1000 * k + flags + seed)
    n = ncol * nlev * n_var
    X = g.standard_normal((k, n)) + 3.0
    HX = g.standard_normal((p, k)) + 1.0
    yo, rvar = g.standard_normal(p) + 1.0, sigma * sigma * g.uniform(0.5, 2.0, p)
    lev = g.uniform(0.0, max(nlev - 1, 1), p)
    counts = g.integers(0, p, ncol)
    counts[:5] = [0, 1, 31, 33, p]
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([np.sort(g.choice(p, c, replace=False)) for c in counts]).astype(np.int32)
    dist = g.uniform(0.0, 9.9, len(idx))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    rho = 0.9 if flags & RTPS else 1.07
    Xd = T(X)
    mean, st = K.letkf_batched(Xd, col_base=T(np.arange(ncol, dtype=np.int64)), nlev=nlev, n_var=n_var,
                               lev_stride=ncol, var_stride=ncol * nlev, HX=T(HX), yo=T(yo), rvar=T(rvar),
                               loc_off=T(off), loc_idx=T(idx), loc_dist=T(dist), obs_lev=T(lev), hsupport=10.0,
                               vsupport=1.5, rho=rho, flags=flags)
    want = np.empty_like(X)
    nloc, kappa = 0, 1.0
    Yp = HX - HX.mean(1, keepdims=True)
    for c in range(ncol):
        for l in range(nlev):
            o, d = idx[off[c]:off[c + 1]], dist[off[c]:off[c + 1]]
            dl = np.abs(lev[o] - l)
            w = np.ones(len(o))
            if not flags & RID:
                w = np.array([ob.gaspari_cohn(a / 0.75) * ob.gaspari_cohn(b / 5.0) for a, b in zip(dl, d)])
            keep = (dl <= 1.5) & (w > 0.0)
            nloc += int(keep.sum())
            if keep.any():
                wk = np.ones(keep.sum()) if flags & RID else w[keep] / rvar[o[keep]]
                kappa = max(kappa, _kappa(np.sqrt(wk)[:, None] * Yp[o[keep]], k, rho))
            res = ob.letkf_points(X, np.array([l * ncol + c], dtype=np.int64), n_var, ncol * nlev, HX, yo, rvar,
                                  np.array([0, keep.sum()], dtype=np.int64), o[keep].astype(np.int32),
                                  np.ascontiguousarray(w[keep]), rho, flags)
            for v in range(n_var):
                want[:, (v * nlev + l) * ncol + c] = res[0, v]
    assert st.total_local == nloc
    assert rel_err(Xd.cpu().numpy(), want) <= _tol(kappa)
    assert rel_err(mean.cpu().numpy(), want.mean(0)) <= _tol(kappa)
    return st


@pytest.mark.parametrize("k", [2, 3, 9, 16, 17, 31, 32, 33, 48, 63, 64, 65, 80, 96])
@pytest.mark.parametrize("flags,n_var,nlev", [(0, 1, 1), (0, 9, 2), (INFL, 3, 3), (RTPS, 4, 2), (UPD, 2, 2),
                                              (RID | INFL | UPD, 1, 1), (RID, 8, 1)])
def test_letkf_matches_oracle(dev, k, flags, n_var, nlev):
    st = _run(dev, k, flags, n_var, nlev, 1.0)
    assert st.n_fallback == 0


@pytest.mark.parametrize("k", [8, 32, 64, 90])
@pytest.mark.parametrize("sigma", [1e-3, 0.05, 30.0, 1e6])
def test_letkf_conditioning(dev, k, sigma):
    _run(dev, k, 0, 2, 2, sigma, seed=7)


@pytest.mark.parametrize("k", [2, 3, 16, 31, 32, 33, 64, 65, 99, 100, 112])
@pytest.mark.parametrize("sigma", [1e-3, 0.05, 1.0, 100.0])
def test_etkf_hunt(dev, k, sigma):
    g = np.random.default_rng(k)
    n, p = 300, 250
    X = g.standard_normal((k, n)) + 4.0
    HX = g.standard_normal((p, k)) + 4.0
    yo, rvar = g.standard_normal(p) + 4.0, sigma * sigma * g.uniform(0.5, 2.0, p)
    Xd = torch.from_numpy(X.copy()).to(dev)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    K.etkf(Xd, T(HX), T(yo), T(rvar), 1.07, flags=0)
    off = np.arange(n + 1, dtype=np.int64) * p
    idx = np.tile(np.arange(p, dtype=np.int32), n)
    pts = g.choice(n, 20, replace=False)
    want = ob.letkf_points(X, pts, 1, 0, HX, yo, rvar, off[:21], idx[: 20 * p], None, 1.07, 0)[:, 0, :].T
    kappa = _kappa((HX - HX.mean(1, keepdims=True)) / np.sqrt(rvar)[:, None], k, 1.07)
    assert rel_err(Xd.cpu().numpy()[:, pts], want) <= _tol(kappa)


@pytest.mark.parametrize("k", [33, 64, 99, 112])
@pytest.mark.parametrize("sigma", [0.5, 0.02, 1e-3])
def test_etkf_hunt_graded(dev, k, sigma):
    """Obs that span 20 directions well: most eigenvalues at the bottom, the rest far above (the second pass)."""
    g = np.random.default_rng(k)
    n, p = 300, 250
    X = g.standard_normal((k, n)) + 4.0
    HX = (g.standard_normal((p, 20)) * np.geomspace(1.0, 0.1, 20)) @ g.standard_normal((20, k)) + 4.0
    yo, rvar = g.standard_normal(p) + 4.0, sigma * sigma * g.uniform(0.5, 2.0, p)
    Xd = torch.from_numpy(X.copy()).to(dev)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    K.etkf(Xd, T(HX), T(yo), T(rvar), 1.0, flags=0)
    off = np.arange(n + 1, dtype=np.int64) * p
    idx = np.tile(np.arange(p, dtype=np.int32), n)
    pts = g.choice(n, 20, replace=False)
    want = ob.letkf_points(X, pts, 1, 0, HX, yo, rvar, off[:21], idx[: 20 * p], None, 1.0, 0)[:, 0, :].T
    kappa = _kappa((HX - HX.mean(1, keepdims=True)) / np.sqrt(rvar)[:, None], k, 1.0)
    assert rel_err(Xd.cpu().numpy()[:, pts], want) <= _tol(kappa)
