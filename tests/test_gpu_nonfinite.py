"""Velocities that are not finite: the kernels of a pruned record layout give
what the run-time dispatch gives, which forms every product."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu
LAYOUTS = {"Bz": ({}, {"z": 0.5}), "Ez Bz": ({"z": 2e5}, {"z": 0.5}), "Ex Ey Bz": ({"x": 2e5, "y": 1e5}, {"z": 0.5}),
           "B": ({}, {"x": 0.1, "y": 0.2, "z": 0.5}), "E": ({"x": 2e5, "y": 1e5, "z": 1e5}, {})}


def _field(values):
    g = np.linspace(-0.05, 0.05, 5)
    return Field.from_arrays({a: g for a in "xyz"}, {a: np.full((5, 5, 5), x) for a, x in values.items()}) if values \
        else None


@pytest.mark.parametrize("alg", ["leapfrog", "vay_rel", "rk4", "rk4_rel", "yoshida_rel", "boris_rel", "vay"])
@pytest.mark.parametrize("layout", sorted(LAYOUTS))
def test_one_step(cuda, alg, layout):
    import torch
    dev = torch.device("cuda", 0)
    rows = []
    for a in range(3):
        for x in (np.inf, -np.inf, np.nan):
            for rest in ((1e7, 2e7, -3e7), (0.0, 0.0, 0.0)):
                v = np.array(rest)
                v[a] = x
                rows.append(v)
    v0 = np.array(rows)
    n = len(v0)
    e, b = (_field(values) for values in LAYOUTS[layout])
    far = Field.from_arrays({a: np.array([50.0, 50.1]) for a in "xyz"}, {"z": np.ones((2, 2, 2))})
    got = []
    for bf in (b, far if b is None else b + far):         # two grids take the run-time dispatch
        tr = DeviceTracker(alg, 9.5788e7, DeviceFields(e, bf, "fp64", dev), n, 1, 2e-11, 1, "fp64", record=False,
                           stagger=False, device=dev)
        r, v = torch.zeros((n, 3), dtype=torch.float64, device=dev), torch.from_numpy(v0).to(dev)
        tr.load(r, v)
        tr.advance(1)
        tr.store(r, v)
        got.append(np.concatenate([r.cpu().numpy(), v.cpu().numpy()], axis=1))
    np.testing.assert_array_equal(got[0], got[1])
