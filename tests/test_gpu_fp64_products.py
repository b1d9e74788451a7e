"""The FP64 contractions on the tensor cores (exact splitting): global ETKF
and EnKF at the edges of the member layouts and tiles, against the oracle;
members and obs of very different magnitudes, where the scaled integers'
row and column scales matter; magnitudes past their range; NaN."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10


def T(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def _case(seed, n, k, p):
    g = np.random.default_rng(seed)
    X = g.standard_normal((k, n)) + 5.0
    HX = g.standard_normal((p, k)) + 5.0
    return X, HX, g.standard_normal(p) + 5.0, g.uniform(0.3, 3.0, p), g


@pytest.mark.parametrize("k", [2, 15, 16, 17, 32, 33, 48, 49, 64, 65, 96, 97, 112])
@pytest.mark.parametrize("n,p", [(1, 1), (131, 63), (257, 64), (1000, 65), (4097, 700)])
def test_etkf_reference_form(dev, k, n, p):
    X, HX, yo, rvar, _ = _case(k * 7 + p, n, k, p)
    Xd = T(X, dev)
    mean = K.etkf(Xd, T(HX, dev), T(yo, dev), T(rvar, dev), 1.07)
    want, wmean = ob.etkf_compat(X, HX, yo, rvar, 1.07)
    assert rel_err(Xd.cpu().numpy(), want) <= FP64_TOL
    assert np.array_equal(mean.cpu().numpy(), wmean)


@pytest.mark.parametrize("k", [3, 16, 40, 64, 100])
def test_enkf(dev, k):
    X, HX, yo, rvar, g = _case(k, 333, k, 190)
    eps = np.sqrt(rvar)[:, None] * g.standard_normal((190, k))
    Xd = T(X, dev)
    mean, diag = K.enkf(Xd, T(HX, dev), T(yo, dev), T(rvar, dev), T(eps, dev), 1.05)
    want = ob.enkf(X, HX, yo, rvar, eps, 1.05)
    wX = want[0] if isinstance(want, tuple) else want
    assert rel_err(Xd.cpu().numpy(), wX) <= FP64_TOL
    assert rel_err(mean.cpu().numpy(), wX.mean(0)) <= FP64_TOL
    assert abs(diag["analysis_spread"] - np.sqrt(np.mean((wX - wX.mean(0)) ** 2))) <= 1e-10


@pytest.mark.parametrize("scale", [1e-30, 1e-6, 1e6, 1e30])
def test_scales(dev, scale):
    """One state a factor off the others, one obs that precise or vague, values on a large offset."""
    k, n, p = 20, 200, 150
    X, HX, yo, rvar, _ = _case(11, n, k, p)
    X[:, 7] *= scale
    HX[3] *= scale
    yo[3] *= scale
    rvar[3] *= scale * scale
    Xd = T(X, dev)
    K.etkf(Xd, T(HX, dev), T(yo, dev), T(rvar, dev), 1.0)
    want, _ = ob.etkf_compat(X, HX, yo, rvar, 1.0)
    got = Xd.cpu().numpy()
    for s in (slice(0, 7), 7, slice(8, n)):
        assert rel_err(got[:, s], want[:, s]) <= FP64_TOL


def test_out_of_range_states(dev):
    """States past the integers' range or not finite take the plain sum; the others are untouched by them."""
    k, n, p = 12, 300, 40
    X, HX, yo, rvar, _ = _case(12, n, k, p)
    clean, _ = ob.etkf_compat(X, HX, yo, rvar, 1.0)
    X[:, 50] *= 1e250
    X[4, 130] = np.nan
    X[5, 260] = np.inf
    Xd = T(X, dev)
    K.etkf(Xd, T(HX, dev), T(yo, dev), T(rvar, dev), 1.0)
    got = Xd.cpu().numpy()
    want, _ = ob.etkf_compat(X, HX, yo, rvar, 1.0)
    assert rel_err(got[:, 50], want[:, 50]) <= FP64_TOL
    assert np.isnan(got[:, 130]).all() and np.isnan(got[:, 260]).all()
    keep = np.setdiff1d(np.arange(n), [50, 130, 260])
    assert rel_err(got[:, keep], clean[:, keep]) <= FP64_TOL


def test_not_finite_obs_fails(dev):
    X, HX, yo, rvar, _ = _case(13, 50, 10, 30)
    HX[5, 2] = np.nan
    with pytest.raises(_lib.MgError):
        K.etkf(T(X, dev), T(HX, dev), T(yo, dev), T(rvar, dev), 1.0)
