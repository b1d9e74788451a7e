"""The reference-order LETKF (in place, point by point) against the oracle:
members at the edges of the kernel's layouts, obs denser and sparser than the
points, on and off the grid's border, invalid obs, points without local obs."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10


@pytest.mark.parametrize("nx,ny,k,p,radius", [(7, 5, 2, 4, 2.0), (12, 9, 6, 60, 3.0), (12, 9, 7, 90, 20.0),
                                              (10, 8, 13, 20, 2.5), (9, 6, 16, 33, 4.0), (9, 6, 17, 33, 4.0),
                                              (40, 20, 9, 200, 3.0), (8, 6, 32, 40, 3.0), (7, 6, 33, 65, 3.0),
                                              (6, 5, 64, 30, 3.0), (5, 4, 9, 0, 3.0), (1, 1, 5, 3, 1.0)])
def test_sequential_matches_oracle(dev, nx, ny, k, p, radius):
    g = np.random.default_rng(nx * 100 + k)
    X = g.standard_normal((k, nx * ny)) + 2.0
    xy = np.stack([g.integers(0, nx, p), g.integers(0, ny, p)], axis=1).astype(np.int32).reshape(p, 2)
    yo = g.standard_normal(p) + 2.0
    valid = (g.random(p) > 0.2).astype(np.uint8) if k % 2 else None
    Xd = torch.from_numpy(X.copy()).to(dev)
    T = lambda a: None if a is None else torch.from_numpy(a).to(dev)  # noqa: E731
    mean = K.letkf_compat_grid(Xd, nx, ny, T(xy), T(yo), radius, 1.08, T(valid))
    want, wmean = ob.letkf_compat_grid(X, nx, ny, xy, yo, radius, 1.08, valid)
    assert rel_err(Xd.cpu().numpy(), want) <= FP64_TOL
    assert rel_err(mean.cpu().numpy(), wmean) <= FP64_TOL
