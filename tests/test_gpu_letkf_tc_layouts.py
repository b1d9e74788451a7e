"""GPU parity of the tensor-core local analyses at the edges of their three
member-slot layouts (64, 80 and 96 slots), with few and many variables per
point (the short finish and the one that forms W), with and without RTPS, and
with variables of very different scale: the operands of the solve are scaled
FP16 pairs, and each variable's perturbations are taken in units of their
largest.  Bound: 1e-5 of each variable's own largest value, the bar of mixed
precision (FP32 Gram at the condition numbers that this path accepts)."""
import numpy as np
import pytest
import torch

from oracle.lists import point_lists

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K
from metada_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu

MIXED_TOL = 1e-5
SCALES = (1.0, 1e-6, 3e5, 1e-12, 7e9, 1.0)


@pytest.mark.parametrize("nvar,rtps", [(3, False), (4, True), (6, False), (6, True)])
@pytest.mark.parametrize("k", [2, 31, 64, 65, 71, 80, 81, 96])
def test_layout_edges_and_variable_scales(dev, k, nvar, rtps):
    c = syn.latlon_letkf_case(nlon=48, nlat=24, nlev=3, nvar=nvar, k=k, p=6_000, T=12, case=48,
                              rho=0.8 if rtps else 1.05)
    per = c.X.shape[1] // nvar
    scale = np.repeat(np.array(SCALES[:nvar]), per)  # variable-major layout
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    olat, olon, olev = t(c.obs_lat), t(c.obs_lon), t(c.obs_lev)
    HX = K.hx_latlon(t(c.X), c.nlon, c.nlat, c.nlev, olat, olon, olev, t(c.obs_var))
    clat, clon = c.col_lat_lon()
    off, idx, dist = K.select_geo(t(clat), t(clon), olat, olon, c.hsupport_km)
    Xs = c.X * scale
    Xd, yo = t(Xs), t(c.yo)
    flags = _lib.MG_RTPS if rtps else 0
    _, st = K.letkf_batched(Xd, col_base=t(c.col_base()), nlev=c.nlev, n_var=nvar, lev_stride=c.lev_stride,
                            var_stride=c.var_stride, HX=HX, yo=yo, rvar=torch.full_like(yo, c.sigma_o ** 2),
                            loc_off=off, loc_idx=idx, loc_dist=dist, obs_lev=olev, hsupport=c.hsupport_km,
                            vsupport=c.vsupport, rho=c.rho, flags=flags, precision=_lib.MG_PREC_MIXED,
                            want_mean=False)
    assert st.tensor_path == 1 and st.n_fallback <= st.n_points // 10
    pts, poff, pidx, pw = point_lists(np.arange(c.nlat * c.nlon), c.nlev, off.cpu().numpy(), idx.cpu().numpy(),
                                      dist.cpu().numpy(), c.obs_lev, c.hsupport_km, c.vsupport)
    base = c.col_base()[pts[:, 0]] + pts[:, 1] * c.lev_stride
    want = ob.letkf_points(Xs, base, nvar, c.var_stride, HX.cpu().numpy(), c.yo, c.rvar, poff, pidx, pw, c.rho,
                           ob.ORC_RTPS if rtps else 0)
    got = Xd.cpu().numpy()
    for v in range(nvar):
        g = got[:, base + v * c.var_stride].T
        assert np.abs(g - want[:, v]).max() <= MIXED_TOL * np.abs(want[:, v]).max()
