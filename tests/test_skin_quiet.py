"""Skin lists of a set at rest whose h the caller only guessed: the first
Newton solve moves every h away from the one the lists were made with, after
which the rows are written once more, with a gap of their own, and kept.
The sets must stay those of a fresh search, also when h is nudged by less
and by more than the gaps allow, and through a re-layout of the rows."""
import numpy as np
import pytest

from sph_playground_b200 import abi, consts, ic
from test_skin import _split_run

pytestmark = pytest.mark.gpu


def _guessed(n, dim, seed=5):
    pos, dx = ic.periodic_lattice(n, dim, seed=seed, amp=0.1)
    st = ic._periodic_state(dim, n, 1.2, "m6", "hydro", tfinish=1.0)
    N = pos.shape[0]
    for k, v in (("realpn", N), ("gamma", 5.0 / 3.0), ("dtprint", 1.0), ("time", 0.0)):
        ic.set_state(st, k, v)
    store = np.zeros((N, consts.ES_TOTAL))
    store[:, :3] = pos
    for name, v in (("m", 1.0 / N), ("den", 1.0), ("h", 1.2 * dx), ("om", 1.0), ("u", 1e-9), ("p", 1e-9),
                    ("c", 1.0), ("type", consts.ept["real"])):
        store[:, ic.col(name)] = v
    # one hot particle sets the timestep: the others move far less than eps
    store[N // 2, ic.col("u")] *= 1e8
    store[N // 2, ic.col("p")] *= 1e8
    return st, store


@pytest.mark.parametrize("prec", [abi.PREC_FP64, abi.PREC_FP32_COMP])
@pytest.mark.parametrize("dim,n", [(2, 60), (3, 32)])
def test_rows_kept_after_the_guess(engine_lib, oracle_lib, cuda_ok, dim, n, prec):
    st, store = _guessed(n, dim)
    cnt, _ = _split_run(engine_lib, oracle_lib, st, store, prec, nsteps=4)
    assert cnt["skin_reuses"] >= 4
    # 3D, 178 neighbours: few rows have a record within 4 eps of their
    # sphere plus the measuring bounds; the
    # hot particle's surroundings (14 spacings of 32) are not kept
    assert cnt["skin_kept"] > 0.6 * (cnt["skin_reuses"] - 1) * n ** dim, cnt


@pytest.mark.parametrize("nudge", [1e-6, 1e-4, 3e-3, 2e-2])
def test_h_moved_within_and_beyond_the_gaps(engine_lib, oracle_lib, cuda_ok, nudge):
    st, store = _guessed(16, 3)
    rng = np.random.default_rng(9)

    def move_h(e, step):
        if step % 2 == 1:
            h = e.get_columns(["h"])
            e.set_columns(["h"], h * (1.0 + nudge * rng.uniform(-1.0, 1.0, h.shape)))

    cnt, _ = _split_run(engine_lib, oracle_lib, st, store, abi.PREC_FP64, nsteps=8, between=move_h)
    assert cnt["skin_reuses"] >= 1
