"""The solve as 1 graph, its first and last smoothing steps fused with the PCG kernels: the same
bits as a launch per kernel, over the smoother's degrees and the kernels that update d in place
(pairs, planes, tiles) or not, and the solve's edges (nothing to iterate, no iterations allowed, a
flag raised beforehand)."""
import ctypes

import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def heat():
    h = mg.heat_cube(28)
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    return (k.submatrix(h.free), fg.reduced_rhs(k, h.load, h.values, h.free),
            fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h))))


def _solve(system, **options):
    a, rhs, u = system
    s = fg.Solver(a, u, fg.Method.Multigrid, options=fg.Options(coarsest=600, **options))
    x = np.zeros(a.n)
    st = s.solve(rhs, x)
    return x, st, s


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("degree", [1, 2, 3, 4])
def test_the_same_bits_as_separate_launches(heat, degree, precision):
    x, st, s = _solve(heat, degree=degree, precision=precision, stencil=2, tiles=1)
    y, st2, _ = _solve(heat, degree=degree, precision=precision, stencil=2, tiles=1, graph=2)
    assert st.iterations == st2.iterations > 0
    assert np.array_equal(x, y)
    assert st.launches == st2.launches
    # A second solve through the same graph starts afresh.
    z = np.zeros(len(x))
    st3 = s.solve(heat[1], z)
    assert st3.iterations == st.iterations and np.array_equal(x, z)


@pytest.mark.parametrize("degree", [1, 2, 3])
@pytest.mark.parametrize("options", [{"stencil": 1}, {"stencil": 3}, {"stencil": 4},
                                     {"stencil": 2, "tiles": 2}])
def test_kernels_that_keep_d_in_place(heat, degree, options):
    """The cycles are the same bits; the dot products are summed in another order where they are
    a launch of their own, so the solutions agree to the tolerance's rounding."""
    x, st, _ = _solve(heat, degree=degree, precision=fg.MIXED, stencil=2, tiles=1)
    y, st2, _ = _solve(heat, degree=degree, precision=fg.MIXED, **options)
    assert st.iterations == st2.iterations
    assert np.linalg.norm(x - y) <= 1e-12 * np.linalg.norm(x)


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
def test_edges(heat, precision, graph):
    a, rhs, u = heat
    x, st, s = _solve(heat, degree=2, precision=precision, graph=graph)
    assert st.true_residual <= 1e-10
    # From the solution nothing is left to do, and x stays.
    y = x.copy()
    st = s.solve(rhs, y)
    assert st.iterations == 0 and np.array_equal(x, y)
    # b = 0: x = 0 without an iteration.
    y = x.copy()
    st = s.solve(np.zeros(a.n), y)
    assert st.iterations == 0 and not y.any()
    # A flag raised before the solve.
    with pytest.raises(fg.FemError) as e:
        s.solve(rhs, np.zeros(a.n), cancelled=ctypes.c_int(1))
    assert str(e.value) == "cancelled"
    # No iterations allowed; then all of them again.
    s.with_max_iter(0)
    with pytest.raises(fg.FemError) as e:
        s.solve(rhs, np.zeros(a.n))
    assert "did not converge" in str(e.value) and "after 0 iterations" in str(e.value)
    s.with_max_iter(3)
    y = np.zeros(a.n)
    with pytest.raises(fg.FemError) as e:
        s.solve(rhs, y)
    assert "after 3 iterations" in str(e.value)
    st = s.with_max_iter(500).solve(rhs, np.zeros(a.n))
    assert st.true_residual <= 1e-10
