"""sph_density_noalloc against the plain sum over all pairs in FP64 torch, at
the sizes where its paths change (a partial warp, the switch between a warp
and two lanes per particle), with coincident particles, one crowded cell and
radii that differ a hundredfold, and its refusals.

Tolerance: a sum of up to n positive terms in FP64, each within a few ulp,
differs by at most a few n eps from another order of it; 1e-12 covers n of a
few hundred neighbours, the repository's parity tolerance."""
import ctypes
import math

import numpy as np
import pytest

from sph_playground_b200 import consts

pytestmark = pytest.mark.gpu

NORM = {"m4": (2 / 3, 10 / (7 * math.pi), 1 / math.pi),
        "m6": (1 / 120, 7 / (478 * math.pi), 1 / (120 * math.pi))}
KRAD = {"m4": 2.0, "m6": 3.0}


def _call(lib, r, h, m, kernel):
    import torch
    f = lib.sph_density_noalloc
    f.argtypes = [ctypes.c_void_p] * 5 + [ctypes.c_int64, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 2
    f.restype = ctypes.c_int
    dim, n = r.shape
    dev = [torch.tensor(np.ascontiguousarray(a), device="cuda") for a in (*r, h, m)]
    rho = torch.full((n,), -1.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ptr = [dev[k].data_ptr() if k < dim else None for k in range(3)]
    rc = f(*ptr, dev[-1].data_ptr(), dev[-2].data_ptr(), n, dim, consts.KERNELS[kernel], rho.data_ptr(), None)
    return rc, rho.cpu().numpy()


def _plain(r, h, m, kernel):
    import torch
    dim = r.shape[0]
    x, h_, m_ = (torch.tensor(np.ascontiguousarray(a), device="cuda") for a in (r, h, m))
    out = torch.empty_like(h_)
    for i in range(0, h.shape[0], 512):
        d2 = sum((x[k, i:i + 512, None] - x[k, None, :]) ** 2 for k in range(dim))
        q = d2.sqrt() / h_[i:i + 512, None]
        t = lambda c: (c - q).clamp(min=0.0)  # noqa: E731
        if kernel == "m6":
            f = t(3.0) ** 5 - 6 * t(2.0) ** 5 + 15 * t(1.0) ** 5
        else:
            f = 0.25 * t(2.0) ** 3 - t(1.0) ** 3
        out[i:i + 512] = f @ m_
    return (out * NORM[kernel][dim - 1] / h_ ** dim).cpu().numpy()


def _set(n, dim, seed, spread=0.1):
    rng = np.random.default_rng(seed)
    h = 1.2 * n ** (-1.0 / dim) * rng.uniform(1.0 - spread, 1.0 + spread, n)
    return rng.uniform(0.0, 1.0, (dim, n)), h, rng.uniform(0.8, 1.2, n) / n


@pytest.mark.parametrize("kernel", ["m4", "m6"])
@pytest.mark.parametrize("dim,n", [(1, 1), (2, 2), (3, 5), (3, 33), (1, 29999), (1, 30000), (2, 29999),
                                   (2, 30000), (2, 30001), (3, 30000)])
def test_sizes(engine_lib, cuda_ok, dim, n, kernel):
    r, h, m = _set(n, dim, 31 + n)
    rc, rho = _call(engine_lib, r, h, m, kernel)
    assert rc == 0
    np.testing.assert_allclose(rho, _plain(r, h, m, kernel), rtol=1e-12)


@pytest.mark.parametrize("dim", [1, 2, 3])
@pytest.mark.parametrize("how", ["coincident", "crowded", "radii", "far"])
def test_arrangements(engine_lib, cuda_ok, dim, how):
    r, h, m = _set(2000, dim, 7)
    if how == "coincident":  # every particle twice
        r[:, 1000:] = r[:, :1000]
    elif how == "crowded":   # half of them in one cell
        r[:, 1000:] = 0.5 + 1e-3 * r[:, 1000:] * h.min()
    elif how == "radii":
        h[::7] *= 100.0
    else:                    # far from the origin: a coordinate keeps 1e-10 of the box
        r += 1e6
    rc, rho = _call(engine_lib, r, h, m, "m6")
    assert rc == 0
    # (the crowded cell sums a thousand terms per particle)
    np.testing.assert_allclose(rho, _plain(r, h, m, "m6"), rtol=4e-12)


@pytest.mark.parametrize("what,code", [("h", 9), ("x", 3), ("inf", 3)])
def test_refusals(engine_lib, cuda_ok, what, code):
    r, h, m = _set(500, 3, 3)
    if what == "h":
        h[17] = 0.0
    else:
        r[1, 17] = np.nan if what == "x" else np.inf
    rc, rho = _call(engine_lib, r, h, m, "m6")
    assert rc == code
    assert np.all(rho == -1.0)  # nothing written
