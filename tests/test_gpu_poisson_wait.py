"""The grid-wide waits of the one-kernel Poisson solves: a wait that runs out
ends the solve with PPT_ERR_TIMEOUT, and the next solve is not affected."""
import ctypes

import numpy as np
import pytest

from pypatools_b200 import _lib
from test_gpu_poisson_resident import TOL, _problem, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("conductors", [0.0, 0.08])
def test_a_wait_that_runs_out_is_an_error(cuda, conductors):
    import torch
    cells = (54, 53, 54)
    extent, coef, rhs = _problem(cells, conductors)
    lib = _lib.load()
    solve = lib.ppt_poisson_solve_polls
    solve.restype, solve.argtypes = ctypes.c_int, [ctypes.POINTER(_lib.MeshDesc)] + [ctypes.c_void_p] * 4 + [
        ctypes.c_double, ctypes.c_int64, ctypes.c_int, ctypes.c_void_p]
    mesh = _lib.MeshDesc()
    for a in range(3):
        mesh.extent[a], mesh.cells[a] = extent[a], cells[a]
    scratch = torch.empty(lib.ppt_poisson_coef_scratch_bytes(mesh), dtype=torch.uint8, device="cuda")
    b, c = torch.from_numpy(rhs).cuda(), torch.from_numpy(coef).cuda()
    x = torch.zeros_like(b)
    # one poll: no block can hold every other block's word at the first look of hundreds of waits
    rc = solve(mesh, c.data_ptr() if conductors else None, b.data_ptr(), x.data_ptr(), scratch.data_ptr(), 0.0, 400, 1,
               _lib.stream_handle())
    assert rc == -5
    torch.cuda.synchronize()
    x, it, res = _solve(cells, extent, rhs, coef if conductors else None, 2000)
    assert res <= TOL and it >= 1 and np.isfinite(x).all()
