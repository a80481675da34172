"""Sets with far outliers, whose other particles share one cell or a few: the
records of a crowded cell are sorted in chunks.  At the sizes where that
changes (up to 128 members counted, chunks of 1,024), against the oracle, the
device-resident step (the library's sort) and the plain sum."""
import numpy as np
import pytest

from parity import COL
from sph_playground_b200 import abi, consts, ic
from test_noalloc_density import _call, _plain

pytestmark = pytest.mark.gpu
SIZES = [127, 128, 129, 1023, 1024, 1025, 2049, 5000]


def _clump(m, dim, seed, width):
    rng = np.random.default_rng(seed)
    pos = np.zeros((m + 2, 3))
    pos[:, :dim] = 0.43 + rng.uniform(0.0, width, (m + 2, dim))
    pos[0, :dim], pos[1, :dim] = 0.95, 0.06
    return rng.permutation(pos), 1.2 * width * m ** (-1.0 / dim)


def _store(pos, h):
    n = len(pos)
    s = np.zeros((n, consts.ES_TOTAL))
    s[:, :3] = pos
    for name, v in (("m", 1.0 / n), ("den", 1.0), ("h", h), ("om", 1.0), ("u", 1.0), ("p", 0.6), ("c", 1.0),
                    ("type", consts.ept["real"])):
        s[:, COL[name]] = v
    return s


def _state(n, dim):
    st = ic._periodic_state(dim, 64, 1.2, "m6", "hydro", tfinish=1.0)
    for key, v in (("realpn", n), ("gamma", 5.0 / 3.0), ("dtprint", 1.0), ("time", 0.0)):
        ic.set_state(st, key, v)
    return st


@pytest.mark.parametrize("m", SIZES)
@pytest.mark.parametrize("dim,width", [(2, 1e-5), (3, 1e-5), (3, 1e-2)])
def test_neighbours(engine_lib, oracle_lib, cuda_ok, dim, width, m):
    pos, h = _clump(m, dim, 3, width)
    st, s = _state(len(pos), dim), _store(pos, h)
    got = []
    for lib, skin in ((engine_lib, 0.0), (engine_lib, 0.1), (oracle_lib, 0.0)):
        with abi.Engine(st, s, "m6", precision=abi.PREC_FP64, lib=lib) as e:
            if lib is engine_lib:
                e.set_param(abi.P_SKIN, skin)
            e.set_param(abi.P_NEWTON_MAXITER, 0)
            e.density()
            got.append(e.get_neighbour_digest())
    for c, d in got[:2]:
        assert np.array_equal(c, got[2][0]) and np.array_equal(d, got[2][1])


@pytest.mark.parametrize("m", [129, 1025, 5000])
def test_order_is_the_library_sorts(engine_lib, cuda_ok, m):
    # the sums of a row follow its order, which follows the records': equal bits
    pos, h = _clump(m, 3, 5, 1e-5)
    st, s = _state(len(pos), 3), _store(pos, h)
    # (cold and at rest: two steps move a particle by a part of its h)
    for name, v in (("u", 1e-30), ("p", 1e-30), ("c", 1e-15)):
        s[:, COL[name]] = v
    out = []
    for graph in (0.0, 1.0):
        with abi.Engine(st, s, "m6", precision=abi.PREC_FP64, lib=engine_lib) as e:
            e.set_param(abi.P_SKIN, 0.0)
            e.set_param(abi.P_NEWTON_MAXITER, 0)
            e.set_param(abi.P_GRAPH, graph)
            e.step(0)
            e.step(2)
            out.append((e.get_store(), e.counters()["graph_steps"]))
    assert out[0][1] == 0 and out[1][1] > 0
    assert np.array_equal(out[0][0], out[1][0])


@pytest.mark.parametrize("m", SIZES)
@pytest.mark.parametrize("dim", [1, 2, 3])
def test_noalloc(engine_lib, cuda_ok, dim, m):
    rng = np.random.default_rng(7)
    r = rng.uniform(0.0, 1e-3, (dim, m + 2))
    r[:, 0], r[:, m // 2] = 1e4, -1e4
    h = np.full(m + 2, 1.2e-3 * m ** (-1.0 / dim))
    mass = rng.uniform(0.8, 1.2, m + 2) / m
    rc, rho = _call(engine_lib, r, h, mass, "m6")
    assert rc == 0
    np.testing.assert_allclose(rho, _plain(r, h, mass, "m6"), rtol=1e-12)
    assert np.array_equal(rho, _call(engine_lib, r, h, mass, "m6")[1])


def test_noalloc_long_rows(engine_lib, cuda_ok):
    # (above 30,000 particles in 2D: two lanes a particle)
    m = 40000
    rng = np.random.default_rng(8)
    r = rng.uniform(0.0, 1e-3, (2, m))
    r[:, 0] = 1e4
    h = np.full(m, 1.2e-3 * m ** -0.5)
    mass = rng.uniform(0.8, 1.2, m) / m
    rc, rho = _call(engine_lib, r, h, mass, "m6")
    assert rc == 0
    np.testing.assert_allclose(rho, _plain(r, h, mass, "m6"), rtol=1e-12)
