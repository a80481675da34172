"""The FP64 roots of the pair arithmetic (frsqrt, fsqrt, froot_ratio), which
start from the hardware's approximate reciprocal root: their error over the
exponent range, next to powers of two and over the mantissas, against roots in
extended precision; what they give outside their range; and the force pass
where a field's square is subnormal or overflows.

Bounds, with d the relative error of the approximation, below 2^-19 (checked
here over the leading 20 bits of the mantissa) and one ulp 2^-53 to 2^-52 of
the value: 1/sqrt leaves 5/16 (2 d)^3 < 2^-55.6 of the series (0.2 ulp), half
of x y's rounding (0.5) and the last sum's (0.5): 1.2; sqrt leaves 1.5 d^3 =
2^-56.4 (0.1) and its last rounding: 0.6; the ratio takes s b rounded as well,
half of which it keeps: 1.1.  CUDA's own: 1.5 of a root and a reciprocal, 0.5
of a root, 1 of a quotient and its root."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from parity import COL, rel_field, run_pass
from sph_playground_b200 import abi
from test_circuit2_modes import _set

pytestmark = pytest.mark.gpu
LD, LOW = np.longdouble, 2.0 ** -1010  # (the range's lower end)


@pytest.fixture(scope="module")
def roots(cuda_ok):
    so = os.path.join(ROOT, "sph_playground_b200", "_lib", "libsph_roots.so")
    if not os.path.exists(so):
        subprocess.run(["make", "-C", os.path.join(ROOT, "sph_playground_b200", "csrc"), so], check=True,
                       capture_output=True)
    f = ctypes.CDLL(so).pair_roots
    f.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_void_p]

    def call(a, b):
        a, b = (np.ascontiguousarray(x, dtype=np.float64) for x in (a, b))
        out = np.empty((7, a.size))
        assert f(a.ctypes.data, b.ctypes.data, a.size, out.ctypes.data) == 0
        return out
    return call


def _ulps(got, ref):
    return np.abs(got.astype(LD) - ref) / np.spacing(ref.astype(np.float64)).astype(LD)


def _values(n, seed, lo, hi):
    rng = np.random.default_rng(seed)
    any_ = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
    two = np.ldexp(1.0, np.arange(lo + 1, hi))
    near = [two]
    for _ in range(3):
        near += [np.nextafter(near[-1], np.inf)]
    below = [np.nextafter(two, 0.0)]
    for _ in range(2):
        below += [np.nextafter(below[-1], 0.0)]
    return np.concatenate([any_] + near + below)


def test_normal_numbers(roots):
    assert np.finfo(LD).nmant >= 63
    x = _values(1 << 20, 1, -1022, 1024)
    out = roots(x, np.ones_like(x))
    ref = np.sqrt(x.astype(LD))
    on = x >= LOW
    assert _ulps(out[1], 1 / ref).max() <= 1.2
    assert _ulps(out[3][on], ref[on]).max() <= 0.6 and not out[3][~on].any()
    assert _ulps(out[2], 1 / ref).max() <= 1.5 and _ulps(out[4], ref).max() <= 0.5  # CUDA's own


def test_mantissas(roots):
    # the approximation reads the leading mantissa bits and the exponent's parity
    for e in (0, 1):
        x = np.ldexp(1.0 + np.arange(1 << 20) / (1 << 20), e)
        x = np.concatenate([x, np.nextafter(np.ldexp(x, 0), np.inf)])
        out = roots(x, np.ones_like(x))
        ref = np.sqrt(x.astype(LD))
        assert np.abs(out[0].astype(LD) * ref - 1).max() < 2.0 ** -19
        assert _ulps(out[1], 1 / ref).max() <= 1.2 and _ulps(out[3], ref).max() <= 0.6


def test_ratios(roots):
    a, b = _values(1 << 20, 2, -511, 511), _values(1 << 20, 3, -500, 500)
    b = np.random.default_rng(4).permutation(np.resize(b, a.size))
    out = roots(a, b)
    ref = np.sqrt(a.astype(LD) / b.astype(LD))
    assert _ulps(out[5], ref).max() <= 1.1
    assert _ulps(out[6], ref).max() <= 1.0


def test_ratios_of_small_and_large(roots):
    a, b, c = _values(1 << 18, 5, -1022, -700), _values(1 << 18, 6, 700, 1024), _values(1 << 18, 7, -300, 300)
    shuffled = np.random.default_rng(8).permutation
    for p, q in ((a, shuffled(np.resize(c, a.size))), (b, shuffled(np.resize(c, b.size)))):
        out = roots(p, q)
        with np.errstate(all="ignore"):
            on = (p >= LOW) & (p * q >= LOW) & (p * q < np.inf) & (p / q < np.inf)
            below = (p < LOW) | (p * q < LOW)
        assert on.sum() > 100000
        ref = np.sqrt(p[on].astype(LD) / q[on].astype(LD))
        assert _ulps(out[5][on], ref).max() <= 1.1
        assert not out[5][below].any()


def test_edges(roots):
    x = np.array([0.0, 5e-324, np.nextafter(LOW, 0.0), LOW, np.finfo(float).max, np.nan])
    out = roots(x, np.ones_like(x))
    assert np.array_equal(out[1][:2], [np.nan, np.inf], equal_nan=True)
    assert np.array_equal(out[3][:3], np.zeros(3)) and np.array_equal(out[5][:3], np.zeros(3))
    for got, own in ((3, 4), (5, 6)):
        np.testing.assert_array_max_ulp(out[got][3:5], out[own][3:5], 2)
    assert np.isnan(out[[1, 3, 5], 5]).all()


@pytest.mark.parametrize("ddw,tensor", [("fab", 0.0), ("fab", 1.0), ("2nw_ds", 0.0)])
@pytest.mark.parametrize("scale", [1e-154, 1e150, 1e160])
def test_fields_whose_square_is_out_of_range(oracle_lib, engine_lib, cuda_ok, ddw, tensor, scale):
    # |B|^2 about 1e-309, a subnormal number of 45 bits, 1e299 and infinite:
    # the direction is that of a field of ordinary size
    from sph_playground_b200 import consts
    st, s = _set(2, "diffusion", 4, ddw=consts.esd[ddw], disotropic=0.0)
    par = {abi.P_FULL_TENSOR: tensor, abi.P_NEWTON_MAXITER: 6}
    ref = run_pass(oracle_lib, st, s, "m6", abi.PREC_FP64, "iterate", par)[0]
    s[:, COL["bx"]:COL["bz"] + 1] *= scale
    got = run_pass(engine_lib, st, s, "m6", abi.PREC_FP64, "iterate", par)[0]
    assert np.abs(ref[:, COL["ddt"]]).max() > 0
    assert rel_field(got[:, COL["ddt"]], ref[:, COL["ddt"]]) <= 1e-12
