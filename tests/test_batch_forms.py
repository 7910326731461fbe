"""The batched kernels over their forms: 1, 4 and 16 right sides, FP64 and mixed, 3x3-block and SELL
levels, and the deepest levels' dense products at the edges of their tiles (64 rows of which the
last may be 32, steps of 64 columns in FP32 and 32 in FP64)."""
import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg
from femahoy_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _member(dims, nrhs, seed):
    p = mg.cantilever_p1(dims=dims, lengths=tuple(2.5 * d for d in dims))
    k = fg.Csr.assemble(fg.P1_ELASTIC, p.xyz, p.nodes, p.coef)
    a = k.submatrix(p.free)
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((a.n, nrhs))
    ptr, idx, val = a.arrays()
    d = np.zeros((a.n, a.n))
    d[np.repeat(np.arange(a.n), np.diff(ptr)), idx] = val
    return a, d, b, fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(p)))


def _check(dims, nrhs, precision, levels, **options):
    """Each pair's residual on the CPU, and its distance to numpy's solution, which the residual
    bounds by the condition number. (The stopping test is on the recurrence; 1.2 for its drift.)"""
    members = [_member(d, nrhs, k) for k, d in enumerate(dims)]
    b = Batch([m[0] for m in members], [m[3] for m in members], nrhs, precision=precision,
              options=fg.Options(precision=precision, degree=2, **options)).with_tol(1e-9)
    assert (len(b.levels()) > 1) == levels
    xs, st = b.solve([m[2] for m in members])
    assert st.not_converged == 0
    for (_, d, rhs, _), x in zip(members, xs):
        res = np.linalg.norm(rhs - d @ x, axis=0) / np.linalg.norm(rhs, axis=0)
        assert res.max() <= 1.2e-9
        y = np.linalg.solve(d, rhs)
        far = np.linalg.norm(x - y, axis=0) / np.linalg.norm(y, axis=0)
        assert far.max() <= 2e-9 * np.linalg.cond(d)


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("nrhs", [1, 4, 16])
@pytest.mark.parametrize("fmt", [0, 1])
def test_levels(nrhs, precision, fmt):
    _check([(14, 3, 2), (9, 4, 3), (21, 2, 2), (5, 1, 1)], nrhs, precision, True, coarsest=120,
           format=fmt)


@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("nrhs", [1, 4, 16])
def test_dense_tiles(nrhs, precision):
    """24, 96, 132, 192, 81, 135 and 360 rows: below a step, 32 rows over, 4 over, whole, 17 over
    and so on."""
    _check([(2, 1, 1), (8, 1, 1), (11, 1, 1), (16, 1, 1), (3, 2, 2), (5, 2, 2), (10, 3, 2)], nrhs,
           precision, False, coarsest=4096)
