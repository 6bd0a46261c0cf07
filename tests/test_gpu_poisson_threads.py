"""Poisson solves from two threads at once, of meshes that take the same kernel
with different amounts of shared memory: neither's launch may be refused for
the other's."""
import ctypes
import threading

import numpy as np
import pytest

from pypatools_b200 import _lib
from test_gpu_poisson_resident import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conductors", [0.0, 0.08])
def test_two_threads_solve_different_meshes(cuda, conductors):
    import torch
    lib = _lib.load()
    errors = []

    def work(cells):
        try:
            extent, coef, rhs = _problem(cells, conductors)
            mesh = _lib.MeshDesc()
            for a in range(3):
                mesh.extent[a], mesh.cells[a] = extent[a], cells[a]
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                scratch = torch.empty(lib.ppt_poisson_coef_scratch_bytes(mesh), dtype=torch.uint8, device="cuda")
                b, c = torch.from_numpy(rhs).cuda(), torch.from_numpy(coef).cuda()
                x = torch.zeros_like(b)
                it, res = _lib.c_int64(), _lib.c_double()
                tail = (scratch.data_ptr(), 0.0, 1, ctypes.byref(it), ctypes.byref(res), stream.cuda_stream)
                for _ in range(1500):
                    if conductors:
                        _lib.check(lib.ppt_poisson_solve_coef(mesh, c.data_ptr(), b.data_ptr(), x.data_ptr(), *tail))
                    else:
                        _lib.check(lib.ppt_poisson_solve(mesh, b.data_ptr(), x.data_ptr(), *tail))
                stream.synchronize()
                assert np.isfinite(x.cpu().numpy()).all()
        except Exception as e:          # noqa: BLE001 -- shown by the assertion below
            errors.append(e)

    # four cells per thread both, 41 and 47 KB of shared memory (with conductors 225 and 229)
    threads = [threading.Thread(target=work, args=(cells,)) for cells in ((24, 24, 24), (60, 60, 60))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
