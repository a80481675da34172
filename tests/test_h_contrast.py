"""Sets whose smallest radius lies far below the usual one, so that the cells
of the search outnumber the records: sets of neighbours through the sort and
through iterates served from skin lists, against the oracle."""
import numpy as np
import pytest

from parity import COL
from sph_playground_b200 import abi, consts, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 0.1])
@pytest.mark.parametrize("dim,n,ratio", [(3, 4, 30.0), (3, 9, 10.0), (3, 14, 4.0), (2, 20, 100.0), (1, 40, 1e4)])
def test_cells_outnumber_records(engine_lib, oracle_lib, cuda_ok, dim, n, ratio, skin):
    pos, dx = ic.periodic_lattice(n, dim, seed=2, amp=0.1)
    k = 5
    clump = np.zeros((k ** dim, 3))
    clump[:, :dim] = 0.5 + (ic.periodic_lattice(k, dim, seed=4, amp=0.1)[0][:, :dim] - 0.5) * k * dx / ratio
    N, M = len(pos), len(clump)
    st = ic._periodic_state(dim, n, 1.2, "m6", "hydro", tfinish=1.0)
    for key, v in (("realpn", N + M), ("gamma", 5.0 / 3.0), ("dtprint", 1.0), ("time", 0.0)):
        ic.set_state(st, key, v)
    store = np.zeros((N + M, consts.ES_TOTAL))
    store[:, :3] = np.concatenate([pos, clump])
    for name, v in (("m", 1.0 / N), ("den", 1.0), ("h", 1.2 * dx), ("om", 1.0), ("u", 1.0), ("p", 1.0),
                    ("c", 1.0), ("type", consts.ept["real"])):
        store[:, COL[name]] = v
    store[N:, COL["h"]] = 1.2 * dx / ratio
    rng = np.random.default_rng(6)
    step = np.zeros((N + M, 3))
    step[:, :dim] = rng.uniform(-1.0, 1.0, (N + M, dim)) * (1e-3 * dx / ratio)
    half = 2.0 * store[:, :3] / dx
    step[(np.abs(half - np.round(half)) < 0.02)[:, :dim].any(1)] = 0.0  # (beside the planes images are told by)
    with abi.Engine(st, store, "m6", precision=abi.PREC_FP64, lib=engine_lib) as e:
        e.set_param(abi.P_SKIN, skin)
        e.set_param(abi.P_NEWTON_MAXITER, 0)
        for j in range(3):
            e.set_columns(["rx", "ry", "rz"], np.ascontiguousarray((store[:, :3] + j * step).T))
            e.density()
        got, table, state, cnt = e.get_neighbour_digest(), e.get_store(), e.get_state(), e.counters()
    with abi.Engine(state, table, "m6", precision=abi.PREC_FP64, lib=oracle_lib) as o:
        o.set_param(abi.P_NEWTON_MAXITER, 0)
        o.density()
        ref = o.get_neighbour_digest()
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])
    # (the 1D set: its largest radius spans 25,000 cells, over the 256 up to
    # which lists serve)
    assert cnt["skin_reuses"] == (2 if skin and dim > 1 else 0)
