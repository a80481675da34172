"""Skin lists so thin that a record counts as fast (it moved a quarter of the
skin) before it counts as moving at all: the sets stay those of a fresh
search, for neighbours that cross a sphere from just outside the skin."""
import numpy as np
import pytest

from parity import COL
from sph_playground_b200 import abi, consts, ic

pytestmark = pytest.mark.gpu
FP64, FP32 = abi.PREC_FP64, abi.PREC_FP32_COMP


@pytest.mark.parametrize("prec", [FP64, FP32])
@pytest.mark.parametrize("skin,move", [(3e-7, 5e-7), (5e-7, 8e-7), (2e-5, 3e-5), (1e-4, 2e-4)])
def test_fast_records_below_the_keeping_bound(engine_lib, oracle_lib, cuda_ok, skin, move, prec):
    n, dim = 14, 3
    pos, dx = ic.periodic_lattice(n, dim, seed=3, amp=0.1)
    N = pos.shape[0]
    st = ic._periodic_state(dim, n, 1.2, "m6", "hydro", tfinish=1.0)
    for k, v in (("realpn", N), ("gamma", 5.0 / 3.0), ("dtprint", 1.0), ("time", 0.0)):
        ic.set_state(st, k, v)
    store = np.zeros((N, consts.ES_TOTAL))
    store[:, :3] = pos
    for name, v in (("m", 1.0 / N), ("den", 1.0), ("h", 1.2 * dx), ("om", 1.0), ("u", 1.0), ("p", 1.0),
                    ("c", 1.0), ("type", consts.ept["real"])):
        store[:, COL[name]] = v
    # centres i with a record j just beyond (1 + skin) of their radius, which
    # then moves straight towards them, by `move` of the smallest radius: into
    # the sphere
    rng = np.random.default_rng(1)
    movers = rng.choice(N, 40, replace=False)
    target = pos.copy()
    h = np.full(N, 1.2 * dx)
    used = set(movers.tolist())
    for j in movers:
        d = pos[j] - pos
        d -= np.round(d / (n * dx)) * (n * dx)
        r = np.sqrt((d ** 2).sum(1))
        i = next(int(q) for q in np.argsort(np.abs(r - 3.0 * 1.25 * dx)) if q not in used)
        used.add(i)
        h[i] = r[i] / 3.0 / (1.0 + 1.25 * skin)
        target[j] -= d[i] / r[i] * 3.0 * h.min() * move
    store[:, COL["h"]] = h
    with abi.Engine(st, store, "m6", precision=prec, lib=engine_lib) as e:
        e.set_param(abi.P_SKIN, skin)
        e.set_param(abi.P_NEWTON_MAXITER, 0)  # (h stays)
        e.density()
        e.set_columns(["rx", "ry", "rz"], np.ascontiguousarray(target.T))
        e.density()
        got = e.get_neighbour_digest()
        table, state = e.get_store(), e.get_state()
    with abi.Engine(state, table, "m6", precision=FP64, lib=oracle_lib) as o:
        o.set_param(abi.P_NEWTON_MAXITER, 0)
        o.density()
        ref = o.get_neighbour_digest()
        o.set_store(store)
        o.density()
        before = o.get_neighbour_digest()
    assert np.sum(before[1] != ref[1]) >= len(movers)  # (every one of them crossed)
    assert np.array_equal(got[0], ref[0])
    assert np.array_equal(got[1], ref[1])
