"""Rows that the one-kernel BiCGSTAB treats on their own: a zero on the diagonal."""
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
