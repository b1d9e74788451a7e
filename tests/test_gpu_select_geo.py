"""The geographic search against the oracle's lists: list lengths around the
sizes where the sort changes, radii on both sides of the chord test's limit
and up to thousands of km, columns at the poles, on the date line and with
longitudes outside 0 .. 360, obs at the column itself.  Offsets and indices
are equal; distances to 1e-13 relative, as in the existing test of the search
(1e-9 km absolute near zero)."""
import numpy as np
import pytest
import torch

import oracle.bind as ob
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _check(dev, clat, clon, olat, olon, radius):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)  # noqa: E731
    off, idx, dist = K.select_geo(t(clat), t(clon), t(olat), t(olon), radius)
    woff, widx, wdist = ob.select_geo(np.asarray(clat, float), np.asarray(clon, float), olat, olon, radius)
    assert np.array_equal(off.cpu().numpy(), woff)
    assert np.array_equal(idx.cpu().numpy(), widx)
    np.testing.assert_allclose(dist.cpu().numpy(), wdist, rtol=1e-13, atol=1e-9)
    return np.diff(woff)


@pytest.mark.parametrize("n", [1, 32, 255, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 5000])
def test_list_lengths(dev, n):
    r = np.random.default_rng(n)
    olat = 10.0 + r.uniform(-1.5, 1.5, n)
    olon = 359.5 + r.uniform(-1.5, 1.5, n)
    olat[0], olon[0] = 10.0, 359.5
    counts = _check(dev, [10.0, 12.0, -50.0], [359.5, 0.5, 100.0], olat, olon, 300.0)
    assert counts[0] == n and counts[2] == 0


@pytest.mark.parametrize("radius", [0.0, 0.5, 30.0, 49.9, 50.0, 51.0, 700.0, 2500.0, 9000.0])
def test_radii_and_columns(dev, radius):
    r = np.random.default_rng(6)
    p = 3000
    olat = np.rad2deg(np.arcsin(r.uniform(-1, 1, p)))
    olon = r.uniform(-180, 400, p)
    clat = np.array([90.0, -90.0, 89.6, -89.9, 0.0, 0.0, 45.0, -30.0, 60.0])
    clon = np.array([0.0, 77.0, 180.0, -1e-9, 0.0, 359.9999, -123.0, 365.0, 180.0])
    # some obs on the columns and some close around them
    near = r.integers(0, clat.size, 600)
    olat[:600] = np.clip(clat[near] + r.normal(0, radius / 111.0, 600), -90, 90)
    olon[:600] = clon[near] + r.normal(0, radius / 111.0, 600)
    olat[:9], olon[:9] = clat, clon
    _check(dev, clat, clon, olat, olon, radius)
