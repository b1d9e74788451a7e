"""The grid search at radii on and off integer distances, against the oracle's lists."""
import numpy as np
import pytest
import torch

import oracle.bind as ob
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0.0, 0.99, 1.0, np.sqrt(2.0), np.nextafter(np.sqrt(2.0), 0.0), 5.0,
                                    np.sqrt(13.0), 7.5, 1e4, 1e8])
@pytest.mark.parametrize("nx,ny,p", [(1, 1, 3), (9, 7, 40), (33, 17, 700), (16, 8, 5000)])
def test_select_grid_radii(dev, nx, ny, p, radius):
    g = np.random.default_rng(nx + p)
    xy = np.stack([g.integers(-5, nx + 5, p), g.integers(-5, ny + 5, p)], axis=1).astype(np.int32)
    off, idx = K.select_grid(nx, ny, torch.from_numpy(xy).to(dev), float(radius))
    woff, widx = ob.select_grid(nx, ny, xy, float(radius))
    assert np.array_equal(off.cpu().numpy(), woff)
    assert np.array_equal(idx.cpu().numpy(), widx)
