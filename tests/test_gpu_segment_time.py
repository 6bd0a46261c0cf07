"""Segments much longer than a cell of the surface's grid: the finer grid of the
short ones must not cost them time."""
import numpy as np
import pytest

from pypatools_b200 import ElectrodeSurface, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [2.0, 12.0])
def test_long_segments_are_as_fast_on_a_refined_surface(cuda, cells):
    import torch
    lib = _lib.load()
    shape = (ElectrodeSurface.aperture_plate(0.03, 0.005, 0.02, n_phi=48, n_r=3) +
             ElectrodeSurface.tube(0.012, -0.05, 0.06, n_phi=48, n_z=22))
    plain, refined = (ElectrodeSurface(shape.vertices, shape.triangles) for _ in range(2))
    handles = plain.handle("cuda"), refined.handle("cuda", segments=True)
    size = np.mean((shape.vertices.max(0) - shape.vertices.min(0)) / np.array(plain.info()["cells"]))
    rng = np.random.default_rng(0)
    m = 200000
    p0 = shape.vertices[rng.integers(0, len(shape.vertices), m)] + rng.normal(0.0, size, (m, 3))
    d = rng.normal(size=(m, 3))
    p1 = p0 + d / np.linalg.norm(d, axis=1, keepdims=True) * cells * size
    a, b = torch.from_numpy(p0).cuda(), torch.from_numpy(p1).cuda()
    took, hits = [], []
    for h in handles:
        out = torch.empty(m, dtype=torch.uint8, device="cuda")
        best = np.inf
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            _lib.check(lib.ppt_surface_segments_hit(h, m, a.data_ptr(), b.data_ptr(), out.data_ptr(),
                                                    _lib.stream_handle()))
            end.record()
            torch.cuda.synchronize()
            best = min(best, start.elapsed_time(end))
        took.append(best)
        hits.append(out.cpu().numpy())
    np.testing.assert_array_equal(hits[0], hits[1])
    # the same cells are visited: half as much again is room for the clocks (2.7 and 8 times without them)
    assert took[1] <= 1.5 * took[0], took
