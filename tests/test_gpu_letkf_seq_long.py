"""The reference-order LETKF where every point has hundreds of local obs, several
chunks of them a point, against the oracle."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [5, 16, 17, 40, 64])
@pytest.mark.parametrize("p", [127, 128, 500])
def test_many_obs_a_point(dev, k, p):
    nx, ny = 6, 5
    g = np.random.default_rng(p + k)
    X = g.standard_normal((k, nx * ny)) + 2.0
    xy = np.stack([g.integers(0, nx, p), g.integers(0, ny, p)], axis=1).astype(np.int32)
    yo = g.standard_normal(p) + 2.0
    Xd = torch.from_numpy(X.copy()).to(dev)
    mean = K.letkf_compat_grid(Xd, nx, ny, torch.from_numpy(xy).to(dev), torch.from_numpy(yo).to(dev), 50.0, 1.05)
    want, wmean = ob.letkf_compat_grid(X, nx, ny, xy, yo, 50.0, 1.05, None)
    assert rel_err(Xd.cpu().numpy(), want) <= 1e-10
    assert rel_err(mean.cpu().numpy(), wmean) <= 1e-10
