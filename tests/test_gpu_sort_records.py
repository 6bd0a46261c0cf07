"""The cell sort's records: a sort, and a sort back to rows, move every word of
every slot -- state, row and RF phase -- to one place, for bunches around a
warp, a block and an unpacking tile, with and without phases, in a scratch
buffer aligned to 8 bytes only."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("phases", [False, True])
@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 256, 1000, 70001])
def test_sort_moves_whole_slots(cuda, precision, phases, n):
    torch = cuda
    dev = torch.device("cuda", 0)
    g = np.linspace(-0.05, 0.05, 9)
    df = DeviceFields(None, Field.from_arrays({"x": g, "y": g, "z": g}, {"z": np.ones((9,) * 3)}), precision, dev)
    rng = np.random.default_rng(n)
    r = torch.from_numpy(rng.uniform(-0.06, 0.06, (n, 3))).to(dev)
    v = torch.from_numpy(rng.normal(0, 1e6, (n, 3))).to(dev)
    phase = torch.arange(n, dtype=torch.float64) if phases else None
    tr = DeviceTracker("boris", 9.58e7, df, n, 10, 1e-11, 10, precision, rf_phase=phase, device=dev)
    tr.load(r, v)
    size = tr.lib.ppt_cell_sort_scratch_bytes(n)
    tr.sort_scratch = torch.empty(size + 8, dtype=torch.uint8, device=dev)[8:]
    before = tr.f64.clone() if precision == "fp64" else (tr.i32.clone(), tr.f32.clone())
    tr.sort()
    order = tr.order.cpu().numpy()
    assert np.array_equal(np.sort(order), np.arange(n))
    if n > 1000:
        assert not np.array_equal(order, np.arange(n))
    idx = tr.order
    blocks = [(tr.f64, before)] if precision == "fp64" else [(tr.i32, before[0]), (tr.f32, before[1])]
    for now, then in blocks:
        assert torch.equal(now.reshape(-1, n), then.reshape(-1, n)[:, idx])
    if phases:
        assert torch.equal(tr.rf_phase, idx.double())
    back_r, back_v = torch.empty_like(r), torch.empty_like(v)
    tr.store(back_r, back_v)
    if precision == "fp64":
        assert torch.equal(back_r, r) and torch.equal(back_v, v)
    tr.restore_order()
    for now, then in blocks:
        assert torch.equal(now, then)
