"""Global analyses of states whose perturbations are so small that products of
the scaled integers would fall below the normal range: alone, beside ordinary
states in the same tile, and beside states that are zero in every member."""
import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10


@pytest.mark.parametrize("scale", [1e-240, 1e-265, 1e-290, 1e-292, 1e-300, 1e-307])
@pytest.mark.parametrize("k", [9, 32, 64, 100])
@pytest.mark.parametrize("form", ["reference", "hunt", "enkf"])
def test_tiny_states(dev, form, k, scale):
    g = np.random.default_rng(k)
    n, p = 300, 60
    X = g.standard_normal((k, n)) + 3.0
    X[:, 40] *= scale      # one state of a tile
    X[:, 128:] *= scale    # whole tiles
    X[:, 41] = X[:, 200:260] = 0.0
    HX, yo, rvar = g.standard_normal((p, k)) + 1.0, g.standard_normal(p) + 1.0, g.uniform(0.5, 2.0, p)
    eps = np.sqrt(rvar)[:, None] * g.standard_normal((p, k))
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    Xd = T(X)
    if form == "enkf":
        K.enkf(Xd, T(HX), T(yo), T(rvar), T(eps), 1.05)
        want = ob.enkf(X, HX, yo, rvar, eps, 1.05)
        want = want[0] if isinstance(want, tuple) else want
    elif form == "reference":
        K.etkf(Xd, T(HX), T(yo), T(rvar), 1.05)
        want, _ = ob.etkf_compat(X, HX, yo, rvar, 1.05)
    else:
        K.etkf(Xd, T(HX), T(yo), T(rvar), 1.05, flags=0)
        # every state has all obs
        off, idx = np.arange(n + 1, dtype=np.int64) * p, np.tile(np.arange(p, dtype=np.int32), n)
        want = ob.letkf_points(X, np.arange(n), 1, 0, HX, yo, rvar, off, idx, None, 1.05, 0)[:, 0, :].T
    got = Xd.cpu().numpy()
    assert not got[:, 41].any() and not got[:, 200:260].any()
    for s in (slice(0, 40), slice(40, 41), slice(42, 128), slice(128, 200), slice(260, n)):
        assert rel_err(got[:, s], want[:, s]) <= FP64_TOL
