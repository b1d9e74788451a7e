"""FP32 members: the point-major layout and back at member counts and state
sizes off every tile, and H(X) of values that do not take the integer
widening.  Without obs an analysis with rho = 1 is mean + perturbation: a
perturbation correctly rounded to FP32 is off by half an ulp of it, the sum by
half an ulp of the value, so the state comes back within 2^-23 of its largest.
H(X) is bit-identical to H of the widened members."""
import numpy as np
import pytest
import torch

from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [1, 63, 65, 129, 300])
@pytest.mark.parametrize("k", [2, 7, 8, 33, 64, 90, 91, 96])
def test_layout_round_trip(dev, k, ncol):
    g = torch.Generator(device=dev).manual_seed(k)
    X = 300.0 + torch.randn((k, ncol), generator=g, device=dev, dtype=torch.float32)
    X0 = X.clone()
    z = lambda n, t: torch.zeros(n, dtype=t, device=dev)  # noqa: E731
    K.letkf_batched(X, col_base=torch.arange(ncol, device=dev), nlev=1, n_var=1, lev_stride=ncol, var_stride=ncol,
                    HX=z((1, k), torch.float64), yo=z(1, torch.float64), rvar=z(1, torch.float64) + 1.0,
                    loc_off=z(ncol + 1, torch.int64), loc_idx=z(1, torch.int32), loc_dist=z(1, torch.float64),
                    obs_lev=z(1, torch.float64), hsupport=100.0, vsupport=2.0, rho=1.0, flags=0,
                    precision=_lib.MG_PREC_MIXED, want_mean=False)
    assert (X - X0).abs().max().item() <= 2.0 ** -23 * X0.abs().max().item()


@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("k", [1, 5, 32, 70])
def test_hx_of_fp32_members_equals_hx_of_widened(dev, k, special):
    nlon, nlat, nlev, nvar, p = 24, 12, 3, 2, 700
    r = np.random.default_rng(k)
    X = (r.normal(0, 1, (k, nvar * nlev * nlat * nlon)) * 10.0 ** r.integers(-30, 30, (k, 1))).astype(np.float32)
    X[:, ::5] = 0.0
    X[:, 1::10] = -0.0
    if special:
        X[:, 2::7] = 1e-41 * r.normal(0, 1, X[:, 2::7].shape)
        X[0, 3] = np.inf
        X[-1, 11] = np.nan
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    where = (t(r.uniform(-90, 90, p)), t(r.uniform(0, 360, p)), t(r.uniform(0, nlev - 1, p)),
             t(r.integers(0, nvar, p).astype(np.int32)))
    x = t(X)
    got = K.hx_latlon(x, nlon, nlat, nlev, *where)
    want = K.hx_latlon(x.double(), nlon, nlat, nlev, *where)
    assert torch.equal(torch.nan_to_num(got, nan=7.0), torch.nan_to_num(want, nan=7.0))
