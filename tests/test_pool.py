"""The setup buffers' pool under several host threads: solvers of different sizes built, solved and
freed side by side give the bits of the same solvers made one after another (a buffer handed to a
second user too early would show there)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

SIZES = [9, 14, 21, 26]


def _analysis(cells):
    h = mg.heat_cube(cells)
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    a = k.submatrix(h.free)
    rhs = fg.reduced_rhs(k, h.load, h.values, h.free)
    u = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h)))
    s = fg.Solver(a, u, fg.Method.Multigrid, options=fg.Options(coarsest=400, degree=2, stencil=2,
                                                                tiles=1))
    x = np.zeros(a.n)
    st = s.solve(rhs, x)
    return x, st.iterations


def test_threads_side_by_side_give_the_same_bits():
    alone = [_analysis(c) for c in SIZES]
    with ThreadPoolExecutor(max_workers=len(SIZES)) as pool:
        for _ in range(3):
            for (x, its), (y, its2) in zip(alone, pool.map(_analysis, SIZES)):
                assert its == its2 > 0
                assert np.array_equal(x, y)
