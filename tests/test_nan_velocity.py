"""A particle whose velocity is not a number leaves its neighbours' accelerations
alone: the viscosity asks whether two records approach, which such a pair does
not; the rates of change of rho and u take it."""
import numpy as np
import pytest

from parity import COL, run_pass
from sph_playground_b200 import abi
from test_circuit2_modes import _set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eqs", ["hydro", "magnetohydro"])
@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_COMP])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_nan_velocity(oracle_lib, engine_lib, cuda_ok, sign, prec, eqs):
    st, s = _set(3, eqs, 3)
    s[101, COL["vx"]] = np.copysign(np.nan, sign)
    par = {abi.P_NEWTON_MAXITER: 6}
    ref = run_pass(oracle_lib, st, s, "m6", abi.PREC_FP64, "iterate", par)[0]
    got = run_pass(engine_lib, st, s, "m6", prec, "iterate", par)[0]
    tol = 1e-12 if prec == abi.PREC_FP64 else 1e-5
    for f in ("ax", "ay", "az"):
        a, b = got[:, COL[f]], ref[:, COL[f]]
        assert np.isfinite(b).all() and np.abs(a - b).max() <= tol * np.abs(b).max()
    for f in ("du", "dh"):
        assert np.array_equal(np.isnan(got[:, COL[f]]), np.isnan(ref[:, COL[f]]))
