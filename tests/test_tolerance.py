"""A solver whose tolerance is changed between solves stops where a new solver of that tolerance
does (the same iterations, the same bits), and a flag raised while the device runs the PCG loop ends
that loop."""
import ctypes
import threading

import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import _lib
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def _system(cells):
    h = mg.heat_cube(cells)
    k = fg.Csr.assemble(fg.P1_HEAT, h.xyz, h.nodes, h.coef)
    return (k.submatrix(h.free), fg.reduced_rhs(k, h.load, h.values, h.free),
            fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(h))))


@pytest.fixture(scope="module")
def heat():
    return _system(24)


def _solver(system, **options):
    return fg.Solver(system[0], system[2], fg.Method.Multigrid,
                     options=fg.Options(coarsest=600, degree=2, stencil=2, tiles=1, **options))


@pytest.mark.parametrize("graph", [1, 2])
@pytest.mark.parametrize("precision", [fg.FP64, fg.MIXED])
@pytest.mark.parametrize("first,then", [(1e-10, 1e-3), (1e-3, 1e-10)])
def test_a_changed_tolerance_counts(heat, first, then, precision, graph):
    a, rhs, _ = heat
    s = _solver(heat, precision=precision, graph=graph).with_tol(first)
    s.solve(rhs, np.zeros(a.n))
    x, y = np.zeros(a.n), np.zeros(a.n)
    st = s.with_tol(then).solve(rhs, x)
    want = _solver(heat, precision=precision, graph=graph).with_tol(then).solve(rhs, y)
    assert st.iterations == want.iterations > 0
    assert st.residual <= then and np.array_equal(x, y)
    # Back again.
    st2 = s.with_tol(first).solve(rhs, x)
    assert st2.residual <= first and (st2.iterations > st.iterations) == (first < then)


@pytest.mark.parametrize("graph", [1, 2])
def test_a_start_value_within_the_new_tolerance(heat, graph):
    """Nothing is left to do at the looser tolerance, and x stays."""
    a, rhs, _ = heat
    s = _solver(heat, precision=fg.FP64, graph=graph).with_tol(1e-6)
    x = np.zeros(a.n)
    s.solve(rhs, x)
    s.with_tol(1e-12).solve(rhs, np.zeros(a.n))
    y = x.copy()
    st = s.with_tol(1e-5).solve(rhs, y)
    assert st.iterations == 0 and np.array_equal(x, y)


@pytest.mark.parametrize("graph", [1, 2])
def test_an_unreachable_tolerance_uses_the_iterations_it_has(heat, graph):
    """r.r of the FP64 recurrence underflows to 0 at r of 1e-162: that is no residual of x, which
    stays at rounding, so the solve goes on from there to its iteration limit. A tolerance of 0
    asks for just that end of the recurrence."""
    a, rhs, _ = heat
    s = _solver(heat, precision=fg.FP64, graph=graph).with_tol(0.0)
    st = s.solve(rhs, np.zeros(a.n))
    ends = st.iterations
    assert 0 < ends < 500 and st.residual == 0.0
    limit = 2 * ends + 5
    st = s.with_tol(1e-300).with_max_iter(limit).solve(rhs, np.zeros(a.n))
    assert st.iterations == limit and 0.0 < st.true_residual <= 1e-13


def test_a_flag_ends_the_device_loop():
    """The loop is 1 launch of about 50 ms and would converge; the flag is raised after 5 ms."""
    system = _system(96)
    a, rhs, _ = system
    s = _solver(system, precision=fg.FP64).with_tol(1e-140)
    whole = s.solve(rhs, np.zeros(a.n))
    flag, st = ctypes.c_int(0), _lib.Stats_t()
    x = np.zeros(a.n)
    timer = threading.Timer(0.005, lambda: setattr(flag, "value", 1))
    timer.start()
    code = fg.lib().femgpu_solver_solve(ctypes.c_void_p(s.handle), _lib.ptr(rhs), _lib.ptr(x),
                                        ctypes.byref(flag), ctypes.byref(st))
    timer.cancel()
    buf = ctypes.create_string_buffer(256)
    fg.lib().femgpu_last_error(buf, 256)
    assert code != 0 and buf.value == b"cancelled"
    assert st.iterations < whole.iterations
