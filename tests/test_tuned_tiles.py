"""The choice of the tile kernels is timed once per size class: a later solver of the class takes the
same choice without a trial, so that both take the same steps."""
import re

import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_later_solvers_of_a_class_take_the_choice_untimed():
    h = mg.heat_cube(56)  # 175,000 unknowns: above the 148 tiles of 1,024 rows
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    a = k.submatrix(h.free)
    rhs = fg.reduced_rhs(k, h.load, h.values, h.free)
    u = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h)))
    xs, finest = [], []
    for _ in range(3):
        s = fg.Solver(a, u, fg.Method.Multigrid, options=fg.Options(precision=fg.MIXED, degree=2))
        x = np.zeros(a.n)
        s.solve(rhs, x)
        xs.append(x)
        finest.append(re.findall(r"stencil K=8 (.*?) \(.*?tiles ([\d.]+)\)(.*?) nnz",
                                 s.describe()))
    assert all(finest) and [f[0][0] for f in finest[1:]] == [finest[0][0][0]] * 2
    assert [f[0][2] for f in finest[1:]] == [finest[0][0][2]] * 2
    # Another test of this process may have timed the class already.
    assert all(float(t) == 0.0 for f in finest[1:] for _, t, _ in f)
    assert np.array_equal(xs[0], xs[1]) and np.array_equal(xs[0], xs[2])
