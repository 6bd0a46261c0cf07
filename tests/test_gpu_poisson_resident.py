"""The Poisson solves that run as one cooperative kernel (and, past its
largest mesh, as launched iterations): the residual of the returned potential,
formed on the host from the rows, must meet the requested one.  Sizes: one
cell, one block exactly and one cell more, each number of cells per thread,
ragged last blocks, axes of one cell, and a mesh past the limit."""
import ctypes

import numpy as np
import pytest

from pypatools_b200 import _lib
from pypatools_b200.space_charge import CONDUCTOR, operator_coefficients

pytestmark = pytest.mark.gpu
TOL = 1e-9
TIGHT = 1e-12
# the recurrence's residual and the true one part by about eps |A| |x| / |b| per
# iteration, 1e-13 to 1e-11 on these meshes
SLACK = 1.05


def _rows_times(coef, x):
    n = x.shape
    w = coef.reshape(n + (7,))
    y = w[..., 0] * x
    for d in range(6):
        a, up = d // 2, d % 2 == 0
        lo = [slice(None)] * 3
        hi = [slice(None)] * 3
        lo[a], hi[a] = slice(0, n[a] - 1), slice(1, n[a])
        here, there = (lo, hi) if up else (hi, lo)
        y[tuple(here)] += w[tuple(here)][..., 1 + d] * x[tuple(there)]
    return y


def _solve(mesh_cells, extent, rhs, coef, max_iter, guess=None, offset=0, tol=TOL):
    import torch
    lib = _lib.load()
    mesh = _lib.MeshDesc()
    for a in range(3):
        mesh.extent[a], mesh.cells[a] = extent[a], mesh_cells[a]
    size = lib.ppt_poisson_scratch_bytes if coef is None else lib.ppt_poisson_coef_scratch_bytes
    scratch = torch.empty(size(mesh) + 8, dtype=torch.uint8, device="cuda")[offset:]   # a caller's 8-byte alignment
    b = torch.from_numpy(rhs).cuda()
    x = torch.zeros_like(b) if guess is None else torch.from_numpy(guess).cuda()
    it, res = _lib.c_int64(), _lib.c_double()
    tail = (scratch.data_ptr(), tol, max_iter, ctypes.byref(it), ctypes.byref(res), _lib.stream_handle())
    if coef is None:
        _lib.check(lib.ppt_poisson_solve(mesh, b.data_ptr(), x.data_ptr(), *tail))
    else:
        c = torch.from_numpy(coef).cuda()
        _lib.check(lib.ppt_poisson_solve_coef(mesh, c.data_ptr(), b.data_ptr(), x.data_ptr(), *tail))
    return x.cpu().numpy(), it.value, res.value


def _problem(cells, conductors):
    rng = np.random.default_rng(sum(cells))
    extent = tuple(0.01 * c * (1.0 + 0.2 * a) for a, c in enumerate(cells))
    h = [e / c for e, c in zip(extent, cells)]
    kind = np.where(rng.random(cells) < conductors, CONDUCTOR, 0)
    dist = rng.uniform(0.2, 1.0, cells + (6,)) * np.repeat(h, 2)
    coef = operator_coefficients(cells, h, kind, dist)
    rhs = rng.normal(size=cells)
    rhs[kind == CONDUCTOR] = 0.0
    return extent, coef, rhs


CG = [(1, 1, 1), (2, 3, 5), (32, 32, 1), (5, 41, 5), (1, 1, 4000), (54, 53, 54), (64, 64, 128), (97, 90, 96),
      (112, 108, 110)]
BI = [(1, 1, 1), (3, 2, 7), (16, 1, 64), (5, 41, 5), (54, 53, 54), (64, 65, 127), (90, 88, 80)]


@pytest.mark.parametrize("cells", CG)
def test_laplacian_solve_meets_its_residual(cuda, cells):
    extent, coef, rhs = _problem(cells, 0.0)
    x, it, res = _solve(cells, extent, rhs, None, 40 * max(cells))
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert res <= TOL and true <= SLACK * TOL and it >= 1
    # from the solution nothing is left to do; the same solve gives the same bits, at any 8-byte alignment
    again, it2, _ = _solve(cells, extent, rhs, None, 40 * max(cells), offset=8)
    np.testing.assert_array_equal(x, again)
    assert it2 == it
    _, it3, _ = _solve(cells, extent, rhs, None, 1)
    assert it3 == 1


@pytest.mark.parametrize("cells", BI)
def test_coefficient_solve_meets_its_residual(cuda, cells):
    extent, coef, rhs = _problem(cells, 0.08)
    if not np.any(rhs):
        rhs[0, 0, 0] = 1.0
    x, it, res = _solve(cells, extent, rhs, coef, 40 * max(cells))
    true = np.linalg.norm(rhs - _rows_times(coef, x)) / np.linalg.norm(rhs)
    assert res <= TOL and true <= SLACK * TOL and it >= 1
    again, it2, _ = _solve(cells, extent, rhs, coef, 40 * max(cells), offset=8)
    np.testing.assert_array_equal(x, again)
    assert it2 == it


@pytest.mark.parametrize("conductors", [0.0, 0.08])
def test_an_exact_guess_and_a_zero_right_hand_side(cuda, conductors):
    cells = (9, 33, 8)
    extent, coef, rhs = _problem(cells, conductors)
    x, it, res = _solve(cells, extent, np.zeros(cells), coef if conductors else None, 100)
    assert it == 0 and res == 0.0 and not x.any()
    guess = np.random.default_rng(0).normal(size=cells)
    rhs = _rows_times(coef, guess)
    x, it, res = _solve(cells, extent, rhs, coef if conductors else None, 100, guess=guess)
    np.testing.assert_array_equal(x, guess)
    assert it == 0 and res <= TOL


def test_a_compact_charge_converges_to_a_tight_residual_every_time(cuda):
    """rhat.r of a right-hand side that lives on a few cells is a small
    difference of large terms near the end: a value of it that is carried on by
    recurrence alone drifts, and some solves then never got there.  Right-hand
    sides that differ in their last bits, as a deposition's atomics make them."""
    cells = (16, 16, 40)
    extent, coef, rhs = _problem(cells, 0.0)
    h = [e / c for e, c in zip(extent, cells)]
    x, y = (np.arange(16) + 0.5) / 16 - 0.5, (np.arange(16) + 0.5) / 16 - 0.5
    wall = np.hypot(x[:, None], y[None, :])[:, :, None] > 0.35
    kind = np.where(np.broadcast_to(wall, cells), CONDUCTOR, 0)
    dist = np.random.default_rng(5).uniform(0.01, 1.0, cells + (6,)) * np.repeat(h, 2)
    coef = operator_coefficients(cells, h, kind, dist)
    rhs = np.zeros(cells)
    rhs[6:10, 6:10, 18:24] = np.random.default_rng(6).uniform(0.5, 1.5, (4, 4, 6))
    for k in range(40):
        b = rhs * (1.0 + 2e-16 * np.random.default_rng(k).integers(-2, 3, cells))
        x, it, res = _solve(cells, extent, b, coef, 300, tol=TIGHT)
        assert res <= TIGHT and it < 150, (k, it, res)
        true = np.linalg.norm(b - _rows_times(coef, x)) / np.linalg.norm(b)
        assert true <= 1e-10, (k, true)
