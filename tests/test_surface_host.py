"""Device handles of electrode surfaces, on a stand-in for the library."""
import contextlib

import pytest

from pypatools_b200 import ElectrodeSurface, _lib, electrodes


class _FakeLib:
    def __init__(self, refine):
        self.refine = refine

    def ppt_surface_create(self, nv, v, nt, t, out):
        out.value = 1234
        return 0

    def ppt_surface_refine(self, handle):
        return self.refine

    def ppt_surface_destroy(self, handle):
        return 0

    def ppt_last_error(self):
        return b"fake"


@pytest.fixture
def surface(monkeypatch):
    import torch
    lib = _FakeLib(0)
    monkeypatch.setattr(electrodes._lib, "load", lambda: lib)
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    s = ElectrodeSurface([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.0, 1.0, 0.0]], [[0, 1, 2]])
    yield s, lib
    s._handles.clear()          # nothing of the stand-in's for the library to destroy


def test_a_segment_grid_without_memory_leaves_the_surface_usable(surface):
    s, lib = surface
    lib.refine = _lib.PPT_ERR_OOM
    assert s.handle("cuda:0", segments=True) == 1234


def test_another_error_of_it_is_raised(surface):
    s, lib = surface
    lib.refine = -3
    with pytest.raises(_lib.PptError):
        s.handle("cuda:0", segments=True)
