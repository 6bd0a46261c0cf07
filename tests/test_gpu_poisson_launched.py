"""The launched BiCGSTAB (meshes past the one-kernel form, or a refused
cooperative launch) beside conductors whose surface lies close to the cells, and a
charge that is zero almost everywhere: it has to converge where the one-kernel
form does."""
import numpy as np
import pytest

from test_gpu_poisson_resident import SLACK, _rows_times, _solve
from test_gpu_poisson_wait import _polls

from pypatools_b200.space_charge import CONDUCTOR, operator_coefficients

pytestmark = pytest.mark.gpu
TOL = 1e-8


def _pipe(cells, seed):
    """A pipe with walls at 0.02 .. 1 of a cell from the cells next to it, and a
    Gaussian bunch on the axis, cut off at 3 sigma."""
    extent = (0.02, 0.02, 0.3)
    h = [e / c for e, c in zip(extent, cells)]
    x, y, z = (((np.arange(c) + 0.5) / c - 0.5) * e for c, e in zip(cells, extent))
    radius = np.hypot(x[:, None], y[None, :])[:, :, None]
    kind = np.where(np.broadcast_to((radius > 0.008) & (radius < 0.0095), cells), CONDUCTOR, 0)
    rng = np.random.default_rng(seed)
    dist = 10.0 ** rng.uniform(-3.0, 0.0, cells + (6,)) * np.repeat(h, 2)
    coef = operator_coefficients(cells, h, kind, dist)
    rhs = np.exp(-0.5 * (radius / 1e-3) ** 2) * (radius < 3e-3) * (np.abs(z) < 0.07) * rng.uniform(0.9, 1.1, cells)
    return extent, coef, rhs


@pytest.mark.parametrize("cells,seed", [((36, 59, 117), 1), ((31, 33, 40), 2), ((48, 48, 64), 3)])
def test_a_refused_launch_converges(cuda, cells, seed):
    extent, coef, rhs = _pipe(cells, seed)
    rc, x = _polls(cells, extent, rhs, coef, True, TOL, 1000, 0)
    assert rc == 0
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert true <= SLACK * TOL, true


def test_a_mesh_past_the_one_kernel_form_converges(cuda):
    cells = (72, 72, 160)
    extent, coef, rhs = _pipe(cells, 4)
    x, it, res = _solve(cells, extent, rhs, coef, 1000, tol=TOL)
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert res <= TOL and true <= SLACK * TOL and it < 1000, (it, res, true)
