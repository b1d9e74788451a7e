"""FP64 symmetric square root past what one FP32 eigenbasis corrects: well observed
local points are solved by the second pass (none handed back), precise ones
beyond it by the FP64 Jacobi, each with weights, inflation, relaxation and the
per-member update, against the oracle."""
import pytest

from metada_gb300 import _lib

from test_gpu_hunt_fp64 import _run

pytestmark = pytest.mark.gpu

INFL, UPD, RTPS = _lib.MG_INFL_COMPAT, _lib.MG_UPDATE_COMPAT, _lib.MG_RTPS
FORMS = [(0, 2, 2), (INFL, 1, 1), (RTPS, 4, 2), (UPD, 2, 2), (INFL | UPD, 9, 1)]


@pytest.mark.parametrize("k", [9, 16, 31, 32, 33, 63, 64, 65, 96])
@pytest.mark.parametrize("flags,n_var,nlev", FORMS)
def test_second_pass(dev, k, flags, n_var, nlev):
    st = _run(dev, k, flags, n_var, nlev, 0.03)
    assert st.n_fallback == 0


@pytest.mark.parametrize("k", [9, 32, 64, 90])
@pytest.mark.parametrize("flags,n_var,nlev", FORMS)
def test_handed_back(dev, k, flags, n_var, nlev):
    st = _run(dev, k, flags, n_var, nlev, 1e-4)
    assert 0 < st.n_fallback <= st.n_points - st.n_empty
