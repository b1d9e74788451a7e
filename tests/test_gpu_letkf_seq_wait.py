"""The bounded waits of the reference-order LETKF: where one runs out, the call
says so and the caller's members and mean stay as they were, and the next call
on the same context is right."""
import ctypes

import numpy as np
import pytest
import torch

from conftest import rel_err

import oracle.bind as ob
from metada_gb300 import _lib
from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _run(dev, X, nx, ny, xy, yo, radius, rho, wait_ns):
    """(status, members, mean) of the call with the given limit; the mean starts as -7."""
    k = X.shape[0]
    Xd, mean = torch.from_numpy(X.copy()).to(dev), torch.full((nx * ny,), -7.0, dtype=torch.float64, device=dev)
    xyd, yod = torch.from_numpy(xy).to(dev), torch.from_numpy(yo).to(dev)
    ctx = K.context(dev.index)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    rc = ctx.lib.mg_letkf_compat_grid_wait_selftest(ctx.handle, p(Xd), k, nx * ny, nx, ny, p(xyd), None, p(yod),
                                                    len(yo), radius, rho, p(mean), wait_ns)
    return rc, Xd.cpu().numpy(), mean.cpu().numpy()


def _case(nx, ny, k, p, seed):
    g = np.random.default_rng(seed)
    X = g.standard_normal((k, nx * ny)) + 2.0
    xy = np.stack([g.integers(0, nx, p), g.integers(0, ny, p)], axis=1).astype(np.int32)
    return X, xy, g.standard_normal(p) + 2.0


@pytest.mark.parametrize("k", [9, 40])
def test_members_stay_when_a_wait_gives_up(dev, k):
    nx, ny, radius, rho = 30, 20, 8.0, 1.1
    X, xy, yo = _case(nx, ny, k, 200, k)
    rc, got, mean = _run(dev, X, nx, ny, xy, yo, radius, rho, 0)
    assert rc == _lib.MG_ERR_TIMEOUT
    assert np.array_equal(got, X) and (mean == -7.0).all()
    rc, got, mean = _run(dev, X, nx, ny, xy, yo, radius, rho, 10 ** 10)
    want, wmean = ob.letkf_compat_grid(X, nx, ny, xy, yo, radius, rho, None)
    assert rc == _lib.MG_OK
    assert rel_err(got, want) <= 1e-10 and rel_err(mean, wmean) <= 1e-10


def test_a_long_chain_is_not_a_stuck_one(dev):
    """Every point reads its neighbours and takes some 0.1 ms or more: a CTA that
    starts with the last of the points in flight waits far beyond the limit, but
    never for that long without another point being finished."""
    nx, ny, k, p, radius, rho, limit_ns = 40, 16, 48, 2000, 60.0, 1.05, 10_000_000
    X, xy, yo = _case(nx, ny, k, p, 3)
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    _run(dev, X, nx, ny, xy, yo, radius, rho, 10 ** 11)
    t0.record()
    rc, want, wmean = _run(dev, X, nx, ny, xy, yo, radius, rho, 10 ** 11)
    t1.record()
    torch.cuda.synchronize()
    assert rc == _lib.MG_OK
    assert t0.elapsed_time(t1) * 1e6 > 5 * limit_ns  # the whole chain: the last wait is most of it
    rc, got, mean = _run(dev, X, nx, ny, xy, yo, radius, rho, limit_ns)
    assert rc == _lib.MG_OK
    assert np.array_equal(got, want) and np.array_equal(mean, wmean)
