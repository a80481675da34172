"""sph_get_columns / sph_set_columns against the whole table, for host and
device buffers: one to all columns (four are written together), a device
buffer inside a larger allocation, and a field named twice."""
import numpy as np
import pytest
import torch

from sph_playground_b200 import abi, consts, ic

pytestmark = pytest.mark.gpu

NAMES = sorted((k for k, v in consts.es.items() if 1 <= v <= consts.ES_TOTAL), key=lambda k: consts.es[k])


@pytest.mark.parametrize("nf", [1, 3, 4, 5, 13, len(NAMES)])
@pytest.mark.parametrize("where", ["host", "device", "slice"])
def test_columns_round_trip(nf, where):
    st, store = ic.sedov3d(n=9)
    with abi.Engine(st, store, "m6") as e:
        e.step(1)  # (the rows are in cell order from here on)
        table = e.get_store()
        names = NAMES[-nf:]
        idx = [ic.col(n) for n in names]
        shape = (nf, e.n_rows)
        if where == "host":
            got = e.get_columns(names)
        else:
            big = torch.full((nf * e.n_rows + 3,), -7.0, dtype=torch.float64, device="cuda")
            buf = big[1:1 + nf * e.n_rows] if where == "slice" else big[: nf * e.n_rows]
            torch.cuda.synchronize()
            e.get_columns(names, buf.data_ptr())
            got = buf.cpu().numpy().reshape(shape)
            assert int((big == -7.0).sum()) >= 3
        assert np.array_equal(got, table[:, idx].T)
        new = np.arange(nf * e.n_rows, dtype=np.float64).reshape(shape) + 0.5
        if where == "host":
            e.set_columns(names, new)
        else:
            buf.copy_(torch.from_numpy(new.ravel()))
            torch.cuda.synchronize()
            e.set_columns(names, buf.data_ptr())
        table[:, idx] = new.T
        assert np.array_equal(e.get_store(), table)


@pytest.mark.parametrize("names", [["u", "u"], ["u", "vx", "vy", "vz", "u"], ["vx", "u", "vx", "u"]])
def test_the_last_of_a_field_named_twice_stays(names):
    st, store = ic.sedov3d(n=9)
    with abi.Engine(st, store, "m6") as e:
        e.step(1)
        table = e.get_store()
        new = np.random.default_rng(3).uniform(1.0, 2.0, (len(names), e.n_rows))
        for k, n in enumerate(names):
            table[:, ic.col(n)] = new[k]
        buf = torch.from_numpy(new).cuda()
        torch.cuda.synchronize()
        e.set_columns(names, buf.data_ptr())
        assert np.array_equal(e.get_store(), table)
        assert np.array_equal(e.get_columns(names), np.stack([table[:, ic.col(n)] for n in names]))
