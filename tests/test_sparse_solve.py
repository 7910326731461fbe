"""The sparse factor's triangular solves over the shapes of supernode that their task rules tell
apart: panels of 1 to more than 2,048 columns and rows (1, 4 and 16 warps per task, 1 and more
turns of the staged right side), in FP64 through the direct method, and the float form inside a
V-cycle whose coarsest level is factored.

The systems are diagonally dominant (each row's off-diagonal magnitudes sum to half its diagonal,
so the condition number is at most 3): a backward stable solve of n unknowns is then within
about n eps = 4200 * 2.2e-16 < 1e-12 of numpy's.
"""
import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

N = 4200  # above the largest system that takes a dense inverse


def _clique_system(width, seed=3):
    """A clique of ``width`` unknowns with the others in short chains that end in it."""
    rng = np.random.default_rng(seed)
    a = np.zeros((N, N))
    a[:width, :width] = rng.uniform(-1.0, 1.0, (width, width))
    for i in range(width, N):
        j = i + 1 if i % 7 and i + 1 < N else int(rng.integers(0, width))
        a[i, j] = rng.uniform(-1.0, 1.0)
        a[i, int(rng.integers(0, width))] = rng.uniform(-1.0, 1.0)
    a = a + a.T
    np.fill_diagonal(a, 0.0)
    np.fill_diagonal(a, 2.0 * np.abs(a).sum(axis=1) + 1.0)
    rows, cols = np.nonzero(a)
    ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=N))])
    xyz = rng.uniform(0.0, 1.0, (N, 3))
    xyz[:width, 0] = 2.0  # the clique on the far side, so that it stays together
    return a, fg.Csr.from_arrays(N, ptr, cols, a[rows, cols]), xyz


@pytest.mark.parametrize("width", [1, 5, 31, 33, 120, 130, 510, 1100, 2200])
def test_direct_solve_over_panel_sizes(width):
    a, m, xyz = _clique_system(width)
    s = fg.Solver(m, fg.Unknowns.Points(xyz), fg.Method.Direct)
    assert "sparse multifrontal factor" in s.describe()
    b = np.random.default_rng(5).standard_normal(N)
    x = np.zeros(N)
    st = s.solve(b, x)
    y = np.linalg.solve(a, b)
    assert st.true_residual <= 1e-13
    assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(y)
    # A second right side through the same factor: no state stays from the first.
    x2 = np.zeros(N)
    s.solve(-3.0 * b, x2)
    assert np.linalg.norm(x2 + 3.0 * y) <= 3e-12 * np.linalg.norm(y)


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
def test_factored_coarsest_level(precision):
    """A grid that may only coarsen along z keeps a coarsest level above the dense limit: the
    solve to 1e-10 agrees with the same system's solve by full coarsening."""
    h = mg.heat_cube(40)
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    a = k.submatrix(h.free)
    rhs = fg.reduced_rhs(k, h.load, h.values, h.free)
    u = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h)))
    xs = []
    for axes in (4, 0):
        s = fg.Solver(a, u, fg.Method.Multigrid,
                      options=fg.Options(precision=precision, degree=2, axes=axes,
                                         max_levels=2 if axes else 0, coarsest=3000))
        assert ("sparse multifrontal" in s.describe()) == (axes == 4)
        x = np.zeros(a.n)
        st = s.solve(rhs, x)
        assert st.true_residual <= 1e-10
        xs.append(x)
    # Each is within cond(A) * 1e-10 of the exact solution in the worst case; in the energy norm
    # both residuals are at 1e-10, and the solutions' difference stays below 1e-7.
    assert np.linalg.norm(xs[0] - xs[1]) <= 1e-7 * np.linalg.norm(xs[1])
