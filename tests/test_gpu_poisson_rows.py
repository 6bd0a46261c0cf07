"""Rows that the one-kernel BiCGSTAB treats on their own: a zero on the diagonal,
and a step whose residual is a small difference of large sums."""
import numpy as np
import pytest

from test_gpu_poisson_resident import SLACK, _problem, _rows_times, _solve

pytestmark = pytest.mark.gpu


def test_a_row_without_a_diagonal(cuda):
    """Cells a, b side by side with the rows (0, 2) and (-1, 3): eigenvalues 1 and 2,
    so the system is a good one, and only a division by the diagonal is not."""
    cells = (4, 5, 6)
    extent, coef, rhs = _problem(cells, 0.0)
    w = coef.reshape(cells + (7,))
    a, b = (1, 2, 2), (1, 2, 3)
    w /= w[0, 0, 0, 0]
    w[a], w[b] = 0.0, 0.0
    w[a][5] = 2.0                     # +z
    w[b][0], w[b][6] = 3.0, -1.0      # -z
    x, it, res = _solve(cells, extent, rhs, coef, 400)
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert res <= 1e-9 and true <= SLACK * 1e-9


@pytest.mark.parametrize("eps", [1e-9, 2e-9, 3e-9, 5e-9, 7e-9, 1e-8])
def test_the_residual_is_summed_where_it_is_small(cuda, eps):
    """Two cells with the rows (1, eps) and (-0.7, 1): from the first column the
    half step leaves s along the second, A s is s up to eps, and the residual eps |s|
    lies below what s.s - 2 omega t.s + omega^2 t.t resolves."""
    cells = (1, 1, 2)
    coef = np.zeros((2, 7))
    coef[:, 0] = 1.0
    coef[0, 5], coef[1, 6] = eps, -0.7
    rhs = np.array([1.1, 0.0]).reshape(cells)
    x, it, res = _solve(cells, (1.0, 1.0, 2.0), rhs, coef, 50, tol=1e-11)
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert res <= 1e-11 and true <= SLACK * 1e-11, (it, res, true)
