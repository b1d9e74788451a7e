"""The EnKF's spread diagnostics (squares summed in fixed point) against sums
in extended precision of the members before and after, over magnitudes,
offsets, equal members, mixed exponents and values that take the FP64 sum.
Bound: 1e-12 relative; FP64 sums of n k squares against a rounded mean are
good to a few 1e-15 sqrt(n k), and the mean's rounding adds (2^-53 |x| / spread)^2
below that for the offsets here."""
import numpy as np
import pytest
import torch

from metada_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _spread(X):
    x = X.astype(np.longdouble)
    d = x - x.mean(axis=0)
    return float(np.sqrt((d * d).sum() / x.size))


@pytest.mark.parametrize("kind", ["offset", "zero_mean", "mixed", "tiny", "huge", "equal"])
@pytest.mark.parametrize("k,n", [(2, 1), (5, 300), (64, 257), (112, 4099)])
def test_spread_diagnostics(dev, k, n, kind):
    r = np.random.default_rng(k)
    X = r.normal(0, 1, (k, n))
    if kind == "offset":
        X += 280.0
    elif kind == "mixed":
        X *= 10.0 ** r.integers(-12, 13, (k, n))
    elif kind == "tiny":
        X *= 1e-140
    elif kind == "huge":
        X *= 1e140
    elif kind == "equal":
        X[:] = 2.0 - 2.0 ** -52
        X[0, 0] = 1.0
    p = 7
    HX = r.normal(0, 1, (p, k))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    Xd = t(X)
    _, diag = K.enkf(Xd, t(HX), t(r.normal(0, 1, p)), t(np.full(p, 4.0)), t(r.normal(0, 2, (p, k))), 1.0)
    after = Xd.cpu().numpy()
    np.testing.assert_allclose(diag["background_spread"], _spread(X), rtol=1e-12)
    np.testing.assert_allclose(diag["analysis_spread"], _spread(after), rtol=1e-12)


def test_spread_of_members_whose_sum_overflows(dev):
    """Finite members with an infinite sum: an infinite mean and spread, as the FP64 sums give."""
    k, n, p = 64, 40, 5
    r = np.random.default_rng(1)
    X = np.ldexp(1.0 + r.uniform(0, 1, (k, n)), 1019)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    _, diag = K.enkf(t(X), t(r.normal(0, 1, (p, k))), t(r.normal(0, 1, p)), t(np.full(p, 4.0)),
                     t(r.normal(0, 2, (p, k))), 1.0)
    assert diag["background_spread"] == np.inf
