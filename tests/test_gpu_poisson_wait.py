"""What can keep a Poisson solve from running as one kernel: a grid-wide wait
that runs out ends it with PPT_ERR_TIMEOUT, and the next solve is not affected; a
cooperative launch that the device does not take leaves the solve to the launched
iterations."""
import ctypes

import numpy as np
import pytest

from pypatools_b200 import _lib
from test_gpu_poisson_resident import SLACK, TOL, _problem, _rows_times, _solve

pytestmark = pytest.mark.gpu


def _polls(cells, extent, rhs, coef, conductors, tol, max_iter, polls):
    import torch
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
    rc = solve(mesh, c.data_ptr() if conductors else None, b.data_ptr(), x.data_ptr(), scratch.data_ptr(), tol, max_iter,
               polls, _lib.stream_handle())
    torch.cuda.synchronize()
    return rc, x.cpu().numpy()


@pytest.mark.parametrize("conductors", [0.0, 0.08])
def test_a_wait_that_runs_out_is_an_error(cuda, conductors):
    cells = (54, 53, 54)
    extent, coef, rhs = _problem(cells, conductors)
    # one poll: no block can hold every other block's word at the first look of hundreds of waits
    rc, _ = _polls(cells, extent, rhs, coef, conductors, 0.0, 400, 1)
    assert rc == -5
    x, it, res = _solve(cells, extent, rhs, coef if conductors else None, 2000)
    assert res <= TOL and it >= 1 and np.isfinite(x).all()


@pytest.mark.parametrize("conductors", [0.0, 0.08])
def test_a_refused_launch_leaves_the_launched_form(cuda, conductors):
    cells = (20, 21, 22)
    extent, coef, rhs = _problem(cells, conductors)
    rc, x = _polls(cells, extent, rhs, coef, conductors, TOL, 2000, 0)
    assert rc == 0
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert true <= SLACK * TOL
