"""The 3x3-block operators at the sizes where their rules change: 4, 2 and 1 threads per block
row, partial slices and windows, even rows (kept in order) and uneven ones (sorted by width).

Each solve's solution is checked by its FP64 residual, computed here from the matrix, against the
tolerance (the residual itself is computed to rounding, far below it)."""
import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _residual(a, b, x):
    return np.linalg.norm(b - a.mul(x)) / np.linalg.norm(b)


def _check(a, rhs, u, precision, tol=1e-10, **options):
    s = fg.Solver(a, u, fg.Method.Multigrid,
                  options=fg.Options(precision=precision, degree=2, **options)).with_tol(tol)
    assert "3x3-block" in s.describe()
    x = np.zeros(a.n)
    st = s.solve(rhs, x)
    # The recurrence's residual, which the FP64 form stops on; its true residual carries the
    # drift of the recurrence too (1.1e-10 on the 80,640 unknown cantilever below).
    assert st.residual <= tol
    # FP64 products of at most 243 terms per row round to 243 eps |A||x| / |b|: the beams'
    # |A||x| / |b| is below 1e5, so 1e-8 leaves room and still shows a wrong product.
    assert _residual(a, rhs, x) <= tol + 1e-8
    return x


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("dims", [(9, 3, 3), (33, 5, 4), (120, 15, 13), (100, 32, 25),
                                  (260, 32, 32)])
def test_even_rows(dims, precision):
    """Box cells: 27-block rows. 144 to 284,000 block rows; the last sizes cross the lines at
    25,000, 60,000 and 250,000."""
    prob = mg.hex_cantilever(nx=dims[0], ny=dims[1], nz=dims[2], length=dims[0] / 8.0,
                             width=dims[1] / 8.0, depth=dims[2] / 8.0, seed=3)
    k = fg.Csr.assemble(fg.HEX8_ELASTIC, prob.xyz, prob.nodes, prob.coef)
    a = k.submatrix(prob.free)
    rhs = fg.reduced_rhs(k, prob.load, prob.values, prob.free)
    u = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(prob)))
    _check(a, rhs, u, precision, coarsest=300)


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("dims", [(3, 2, 2), (21, 4, 3), (62, 8, 7)])
def test_uneven_rows(dims, precision):
    """P2 tetrahedra: rows of 10 to 65 blocks, which are sorted within their windows."""
    m = mg.box(*dims, tuple(float(d) for d in dims))
    q = fg.Quadratic.new(m.points, m.tets)
    prob = mg.beam_p2(q.edges, q.tets, mesh=m)
    k = fg.Csr.assemble(fg.P2_ELASTIC, prob.xyz, prob.nodes, prob.coef)
    a = k.submatrix(prob.free)
    rhs = fg.reduced_rhs(k, prob.load, prob.values, prob.free)
    p, coarse = fg.prolongation(prob.xyz, m.n, q.edges, prob.free)
    u = fg.Unknowns.Quadratic(prob.xyz[prob.free // 3], p, coarse)
    x = _check(a, rhs, u, precision, coarsest=100)
    if a.n <= 3000:
        ptr, idx, val = a.arrays()
        full = np.zeros((a.n, a.n))
        full[np.repeat(np.arange(a.n), np.diff(ptr)), idx] = val
        y = np.linalg.solve(full, rhs)
        assert np.linalg.norm(x - y) <= 1e-6 * np.linalg.norm(y)
