"""Float64 kernels that keep a cell's corner records between field
evaluations (RK4 and Vay on a pruned record layout) against the same
algorithm on the full E / B / E+B records of the six-component kind or with
the run-time dispatch, which gather at every evaluation: the same values
enter the same operations, so the tracks must agree bit for bit.  Bunches of
1 to 129 particles (remainders of a warp and of a block), tracks that cross
cells, leave the map and come back into it, and a map of two cells."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu

LAYOUTS = {0x20: "z", 0x24: "Ez z", 0x23: "Ex Ey z", 0x38: "x y z", 0x07: "Ex Ey Ez"}


def _fields(layout, nodes):
    g = np.linspace(-0.05, 0.05, nodes)
    x, y, z = np.meshgrid(g, g, g, indexing="ij")
    rng = np.random.default_rng(layout)
    comps = {}
    for c in range(6):
        if layout & (1 << c):
            scale = 2e5 if c < 3 else 0.5
            comps[c] = scale * (1.0 + 0.3 * rng.standard_normal(x.shape))
    grid = {"x": g, "y": g, "z": g}

    def field(base):
        vals = {a: comps[base + i] for i, a in enumerate("xyz") if base + i in comps}
        return Field.from_arrays(grid, vals) if vals else None

    return field(0), field(3)


@pytest.mark.parametrize("alg", ["rk4", "rk4_rel", "vay", "vay_rel"])
@pytest.mark.parametrize("layout", sorted(LAYOUTS))
@pytest.mark.parametrize("n,nodes", [(1, 9), (33, 2), (129, 17)])
def test_kept_corners_are_bitwise_the_gathered_ones(cuda, alg, layout, n, nodes):
    import torch
    dev = torch.device("cuda", 0)
    e, b = _fields(layout, nodes)
    # two grids (the second far away, never met) take the run-time dispatch
    far = {a: np.array([50.0, 50.1]) for a in "xyz"}
    other = Field.from_arrays(far, {"z": np.ones((2, 2, 2))})
    rng = np.random.default_rng(n)
    r0 = rng.uniform(-0.06, 0.06, (n, 3))          # some start outside
    v0 = rng.normal(0.0, 2e7, (n, 3))
    nsteps = 160
    got = []
    for bf in (b, other if b is None else b + other):
        df = DeviceFields(e, bf, "fp64", dev)
        assert len(df.maps) == (1 if bf is b else 2)
        tr = DeviceTracker(alg, 9.5788e7, df, n, nsteps, 2e-11, 20, "fp64", device=dev)
        tr.load(torch.from_numpy(r0).to(dev), torch.from_numpy(v0).to(dev))
        tr.run(nsteps, 37)
        got.append((tr.r_hist.cpu().numpy(), tr.v_hist.cpu().numpy(), tr.device_status()))
    np.testing.assert_array_equal(got[0][0], got[1][0])
    np.testing.assert_array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2] == 0
