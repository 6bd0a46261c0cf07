"""The mixed Vay kernel carries 1/gamma from one step's position increment to the
next step's update.  A track in long launches against the same track in launches
of a single step, each of which forms 1/gamma of the stored u: bitwise."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 129, 1000])
@pytest.mark.parametrize("comps,rf", [("z", 0.0), ("Ex Ey Ez", 2 * np.pi * 1e8), ("Ez x y z", 0.0)])
def test_long_launches_against_single_steps(cuda, n, comps, rf):
    torch = cuda
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(n)
    g = np.linspace(-0.05, 0.05, 9)
    grid = {"x": g, "y": g, "z": g}
    names = comps.split()
    e = {c[1].lower(): 2e6 * rng.standard_normal((9,) * 3) for c in names if c[0] == "E"}
    b = {c: 0.01 * rng.standard_normal((9,) * 3) for c in names if c[0] != "E"}
    df = DeviceFields(Field.from_arrays(grid, e) if e else None, Field.from_arrays(grid, b) if b else None, "mixed",
                      dev)
    r0 = torch.from_numpy(rng.uniform(-0.07, 0.07, (n, 3))).to(dev)
    v0 = torch.from_numpy(rng.normal(0.0, 1e8, (n, 3)).clip(-1.6e8, 1.6e8)).to(dev)
    rows = []
    for chunk in (60, 1):
        tr = DeviceTracker("vay", -1.7588e11, df, n, 60, 1e-11, 15, "mixed", device=dev, rf_omega=rf,
                           rf_phase=torch.linspace(0, 6, n).double() if rf else None)
        tr.load(r0, v0)
        tr.run(60, chunk)
        rows.append((tr.r_hist.cpu().numpy(), tr.v_hist.cpu().numpy()))
    for a, b in zip(*rows):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
