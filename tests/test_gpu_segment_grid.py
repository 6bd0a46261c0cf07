"""The segment test's shortcuts -- the plane test in front of a triangle's, the
finer grid (``ppt_surface_refine``), and a track's clear boxes -- against the
oracle, which tests every triangle: the same hits, bit for bit.  Soups of
triangles with slivers and some without area, near the origin and far from it;
segments from a hundredth of a cell to the whole mesh, with ends within a few
ulps of triangles' planes."""
import ctypes

import numpy as np
import pytest

from pypatools_b200 import ElectrodeSurface, Field, _lib
from pypatools_b200.device_fields import DeviceFields
from pypatools_b200.pusher import DeviceTracker
from oracle import pusher_oracle as orc

pytestmark = pytest.mark.gpu


def _soup(n, offset, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1.0, 1.0, (n, 1, 3))
    v = c + rng.normal(0, 0.15, (n, 3, 3))
    v[: n // 8, 2] = v[: n // 8, 0] + 1e-9 * rng.normal(size=(n // 8, 3))      # slivers
    v[n // 8: n // 6, 1] = v[n // 8: n // 6, 0]                                 # no area
    v[n // 6: n // 3, :, 2] = np.round(v[n // 6: n // 3, :1, 2], 1)            # in planes of constant z
    return (v + offset).reshape(-1, 3), np.arange(3 * n).reshape(n, 3)


def _hits(handle, p0, p1):
    import torch
    a, b = torch.from_numpy(p0).cuda(), torch.from_numpy(p1).cuda()
    out = torch.empty(len(p0), dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().ppt_surface_segments_hit(handle, len(p0), a.data_ptr(), b.data_ptr(), out.data_ptr(),
                                                    _lib.stream_handle()))
    return out.cpu().numpy().astype(bool)


@pytest.mark.parametrize("offset", [0.0, 1000.0])
@pytest.mark.parametrize("n", [1, 7, 400])
def test_hits_with_and_without_the_finer_grid(cuda, n, offset):
    v, t = _soup(n, offset, n)
    rng = np.random.default_rng(n + 1)
    m = 20000
    p0 = rng.uniform(-1.3, 1.3, (m, 3)) + offset
    p1 = p0 + rng.normal(size=(m, 3)) * 10.0 ** rng.uniform(-3, 0.5, (m, 1))
    # ends on triangles' planes, a few ulps off
    k = rng.integers(0, n, m // 2)
    w = rng.dirichlet([1, 1, 1], m // 2)
    on = np.einsum("ij,ijk->ik", w, v[t[k]])
    p1[: m // 2] = on + rng.integers(-4, 5, on.shape) * np.spacing(on)
    p0[: m // 4] = p1[: m // 4] + rng.normal(size=(m // 4, 3)) * 10.0 ** rng.uniform(-6, -1, (m // 4, 1))
    expect = orc.segments_hit(p0, p1, v, t)
    s = ElectrodeSurface(v, t)
    plain = s.handle("cuda")
    before = s.info()["cells"]
    np.testing.assert_array_equal(_hits(plain, p0, p1), expect)
    refined = s.handle("cuda", segments=True)
    assert refined == plain and s.info()["cells"] == before
    np.testing.assert_array_equal(_hits(refined, p0, p1), expect)
    assert expect.any() or n < 400


@pytest.mark.parametrize("alg,precision", [("boris", "fp64"), ("boris", "mixed"), ("boris_rel", "fp64"),
                                           ("rk4", "fp64")])
@pytest.mark.parametrize("layout", ["z", "Exy z", "xyz"])
def test_tracks_stop_at_the_step_the_test_finds(cuda, alg, precision, layout):
    """Launches of one step begin without a clear box and test every segment;
    whole launches skip what their boxes cover and run through field-free
    stretches: the same tracks, stopped at the same steps."""
    import torch
    dev = torch.device("cuda", 0)
    g = np.linspace(-0.03, 0.03, 13)
    grid = {"x": g, "y": g, "z": g}
    one = np.ones((13,) * 3)
    b = Field.from_arrays(grid, {"x": 0.05 * one, "y": -0.1 * one, "z": 0.5 * one} if layout == "xyz"
                          else {"z": 0.5 * one})
    e = Field.from_arrays(grid, {"x": 1e5 * one, "y": -2e5 * one}) if layout == "Exy z" else None
    df = DeviceFields(e, b, precision, dev)
    surf = ElectrodeSurface.tube(0.02, -0.2, 0.25, n_phi=24, n_z=9) + \
        ElectrodeSurface.aperture_plate(0.1, 0.008, 0.02, n_phi=24, n_r=2)
    rng = np.random.default_rng(3)
    n, nsteps = 700, 260
    r0 = np.column_stack([rng.uniform(-0.012, 0.012, (n, 2)), rng.uniform(-0.02, 0.02, n)])
    v0 = np.column_stack([rng.normal(0, 1.5e6, (n, 2)), rng.normal(2e7, 1e6, n)])
    out = []
    for chunk in (1, 37, nsteps):
        tr = DeviceTracker(alg, 9.5788e7, df, n, nsteps, 5e-11, 20, precision, device=dev, surface=surf)
        tr.load(torch.from_numpy(r0).to(dev), torch.from_numpy(v0).to(dev))
        tr.run(nsteps, chunk)
        out.append((tr.r_hist.cpu().numpy(), tr.v_hist.cpu().numpy(), tr.active.cpu().numpy()))
    for a in out[1:]:
        for x, y in zip(a, out[0]):
            np.testing.assert_array_equal(x, y)
    stopped = 1.0 - out[0][2].mean()
    assert 0.1 < stopped < 0.98, stopped
