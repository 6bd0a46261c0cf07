"""Mixed RK4 kernels that keep a cell's corner records between the stages of a
step.  A Bz field stored with zero Bx and By (a four-element record, kept)
against the one-element record (gathered at every stage): the same
interpolation of Bz, products with exact zeros apart, so within the float32
rounding that test_gpu_layouts allows such pairs.  And the kernel of small
bunches against that of large ones, which differ in registers alone: bitwise.
Tracks that cross cells, leave the map and come back."""
import numpy as np
import pytest

from pypatools_b200 import Field
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker

pytestmark = pytest.mark.gpu


def _track(torch, alg, df, r0, v0, nsteps, rf=None):
    n = len(r0)
    dev = torch.device("cuda", 0)
    tr = DeviceTracker(alg, 9.5788e7, df, n, nsteps, 2e-11, nsteps // 4, "mixed", device=dev,
                       rf_omega=rf or 0.0, rf_phase=None if rf is None else torch.linspace(0, 6, n).double())
    tr.load(torch.from_numpy(r0).to(dev), torch.from_numpy(v0).to(dev))
    tr.run(nsteps, 37)
    return tr.r_hist.cpu().numpy(), tr.v_hist.cpu().numpy()


def _bunch(n):
    rng = np.random.default_rng(n)
    return rng.uniform(-0.06, 0.06, (n, 3)), rng.normal(0.0, 2e7, (n, 3))


@pytest.mark.parametrize("alg", ["rk4", "rk4_rel"])
@pytest.mark.parametrize("n,nodes", [(1, 9), (33, 2), (129, 17)])
def test_kept_records_against_gathered_ones(cuda, alg, n, nodes):
    torch = cuda
    g = np.linspace(-0.05, 0.05, nodes)
    bz = 0.5 * (1.0 + 0.3 * np.random.default_rng(nodes).standard_normal((nodes,) * 3))
    zero = np.zeros_like(bz)
    field = Field.from_arrays({"x": g, "y": g, "z": g}, {"x": zero, "y": zero, "z": bz})
    r0, v0 = _bunch(n)
    got = [_track(torch, alg, DeviceFields(None, field, "mixed", torch.device("cuda", 0), prune=p), r0, v0, 160)
           for p in (True, False)]
    for k, floor in ((0, 0.05), (1, 1e6)):
        size = np.maximum(np.linalg.norm(got[0][k], axis=-1), floor)
        assert (np.linalg.norm(got[0][k] - got[1][k], axis=-1) / size).max() <= 1e-6


@pytest.mark.parametrize("alg,rf", [("rk4", None), ("rk4_rel", 2 * np.pi * 1e8)])
@pytest.mark.parametrize("comps", ["Ez z", "Ex Ey z", "x y z", "Ex Ey Ez"])
def test_small_and_large_bunches_agree_bitwise(cuda, alg, rf, comps):
    torch = cuda
    g = np.linspace(-0.05, 0.05, 17)
    rng = np.random.default_rng(len(comps))
    names = comps.split()
    e = {c[1].lower(): 2e5 * rng.standard_normal((17,) * 3) for c in names if c[0] == "E"}
    b = {c: 0.5 * rng.standard_normal((17,) * 3) for c in names if c[0] != "E"}
    grid = {"x": g, "y": g, "z": g}
    df = DeviceFields(Field.from_arrays(grid, e) if e else None, Field.from_arrays(grid, b) if b else None, "mixed",
                      torch.device("cuda", 0))
    large = 148 * 3 * 128 + 1
    r0, v0 = _bunch(large)
    whole = _track(torch, alg, df, r0, v0, 80, rf)
    if rf is None:
        small = _track(torch, alg, df, r0[:1000], v0[:1000], 80)
    else:       # the phases of the large bunch's rows
        dev = torch.device("cuda", 0)
        tr = DeviceTracker(alg, 9.5788e7, df, 1000, 80, 2e-11, 20, "mixed", device=dev, rf_omega=rf,
                           rf_phase=torch.linspace(0, 6, large).double()[:1000])
        tr.load(torch.from_numpy(r0[:1000]).to(dev), torch.from_numpy(v0[:1000]).to(dev))
        tr.run(80, 37)
        small = tr.r_hist.cpu().numpy(), tr.v_hist.cpu().numpy()
    np.testing.assert_array_equal(whole[0][:, :1000], small[0])
    np.testing.assert_array_equal(whole[1][:, :1000], small[1])
