"""A centre at a NaN position, wherever it falls in the search's groups: the
call ends with the reference's status ('q is nan'), and the search stays
inside its arrays (a NaN distance is neither inside nor outside, so such a
centre takes every candidate it is shown)."""
import pytest

from parity import COL
from sph_playground_b200 import abi, ic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("skin", [0.0, 0.1])
@pytest.mark.parametrize("axis", ["rx", "ry", "rz"])
@pytest.mark.parametrize("row", [0, 3, 77, 300, 511])
def test_nan_position(engine_lib, cuda_ok, row, axis, skin):
    st, store = ic.sedov3d(n=8)
    store[row, COL[axis]] = float("nan")
    with abi.Engine(st, store, "m6", lib=engine_lib) as e:
        e.set_param(abi.P_SKIN, skin)
        with pytest.raises(abi.SphError) as ex:
            e.iterate()
        assert ex.value.code in (3, 4)
