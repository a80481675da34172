"""sph_density_noalloc on smoothing lengths that are not ordinary numbers: a
NaN radius ends the call with 'q is nan' wherever its particle and the others
lie (also where no particle is near it or near the grid's first cell), and
what has a defined sum keeps it."""
import ctypes

import numpy as np
import pytest

from test_noalloc_density import _call, _plain, _set

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(1, 400), (1, 30000), (2, 500), (2, 30000), (3, 2), (3, 500), (3, 20000)])
@pytest.mark.parametrize("seed", [1, 2, 3, 4, 5, 6])
def test_nan_radius_is_refused(engine_lib, cuda_ok, dim, n, seed):
    r, h, m = _set(n, dim, seed)
    h[(7919 * seed) % n] = np.nan
    rc, _ = _call(engine_lib, r, h, m, "m6")
    assert rc == 3


def test_all_radii_nan(engine_lib, cuda_ok):
    r, h, m = _set(500, 3, 1)
    rc, _ = _call(engine_lib, r, np.full_like(h, np.nan), m, "m6")
    assert rc == 3


def test_infinite_radii(engine_lib, cuda_ok):
    # W = f(0) / inf^3: a sum of zero, for one particle or for all
    r, h, m = _set(500, 3, 2)
    h[11] = np.inf
    rc, rho = _call(engine_lib, r, h, m, "m6")
    assert rc == 0 and rho[11] == 0.0
    rest = np.arange(500) != 11
    ref = _plain(r, np.where(rest, h, 1.0), m, "m6")
    np.testing.assert_allclose(rho[rest], ref[rest], rtol=1e-12)
    rc, rho = _call(engine_lib, r, np.full_like(h, np.inf), m, "m6")
    assert rc == 0 and np.all(rho == 0.0)


@pytest.mark.parametrize("cells,code", [(5000, 0), (7000, 18)])
def test_smallest_radius(engine_lib, cuda_ok, cells, code):
    # cells start at the smallest radius (or a half or an eighth of it) and
    # are widened by 1.25 up to 401 times: where `cells` of the widest, of up
    # to 4 n + 4096, span the set, it has a grid
    n = 500
    r, h, m = _set(n, 1, 4)
    h[7] = (r.max() - r.min()) / (3.0 * 1.25 ** 401 * cells)
    rc, rho = _call(engine_lib, r, h, m, "m6")
    assert rc == code
    if code == 0:
        rest = np.arange(n) != 7
        ref = _plain(r, np.where(rest, h, 1.0), m, "m6")
        np.testing.assert_allclose(rho[rest], ref[rest], rtol=1e-12)
        # (nothing else lies within 1e-42 of it)
        assert abs(rho[7] / (m[7] * 66.0 / 120.0 / h[7]) - 1.0) < 1e-12
