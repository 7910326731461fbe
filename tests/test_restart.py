"""A mixed solve restarts from the residual that called for it. A stencil takes its lower triangle
from the upper one; where the matrix's own lower triangle differs a little, the stencil's residual
reaches the tolerance while the true one does not, and only a start by the exact matrix goes on."""
import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("by", [1e-7, 1e-6])
def test_a_restart_goes_on_from_the_true_residual(by, graph):
    h = mg.heat_cube(24)
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    a = k.submatrix(h.free)
    rhs = fg.reduced_rhs(k, h.load, h.values, h.free)
    ptr, idx, val = a.arrays()
    row = np.repeat(np.arange(a.n), np.diff(ptr))
    val = np.where(idx < row, val * (1.0 + by), val)
    b = fg.Csr.from_arrays(a.n, ptr, idx, val)
    s = fg.Solver(b, fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h))), fg.Method.Multigrid,
                  options=fg.Options(precision=fg.MIXED, coarsest=600, degree=2, stencil=2,
                                     tiles=1, graph=graph))
    first = None
    for _ in range(2):  # the second solve takes the restart's graph as it is
        x = np.zeros(a.n)
        st = s.solve(rhs, x)
        # Each restart leaves the difference of the triangles times the residual before it.
        assert st.residual <= 1e-10 and st.true_residual <= 1e-10
        first = x if first is None else first
        assert np.array_equal(x, first)
    r = rhs - np.bincount(row, val * x[idx], minlength=a.n)
    assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(rhs)
