"""The products with inverses (the dense one, and the sparse factor's panels) on badly conditioned
systems: stiffness jumps of 1e6 from cell to cell, and nearly incompressible material; 1 application,
without the refinement step.

The sparse factor's panels hold the inverses of its pivot blocks only: where those are well enough
conditioned a solve is backward stable as by substitution, an error of order n eps in the residual
at any condition number of the whole. The dense inverse is a product with A^-1 itself, whose
residual may be the condition number times that; its error is bounded as a solution's is, by n eps
times the condition number of the system scaled to a unit diagonal, for each of factor, inverse and
product."""
import ctypes as C

import numpy as np
import pytest

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg

pytestmark = pytest.mark.gpu

MATERIALS = [("plain", 1.0, 0.3), ("jumps", 1e6, 0.3), ("incompressible", 1.0, 0.4999),
             ("both", 1e6, 0.4999)]


def _p1(dims):
    p = mg.cantilever_p1(dims=dims, lengths=tuple(2.5 * d for d in dims))
    return p, fg.P1_ELASTIC


def _p2(dims):
    m = mg.box(*dims, tuple(5.0 * d for d in dims))
    q = fg.Quadratic.new(m.points, m.tets)
    return mg.beam_p2(q.edges, q.tets, mesh=m), fg.P2_ELASTIC


def _system(p, element, jump, nu):
    """Soft cells at random, 1 in 2."""
    soft = np.random.default_rng(1).random(len(p.nodes)) < 0.5
    coef = np.stack([np.where(soft, 200e3 / jump, 200e3), np.full(len(p.nodes), nu)], axis=1)
    k = fg.Csr.assemble(element, p.xyz, p.nodes, coef)
    return p, k, k.submatrix(p.free)


def _apply(s, b):
    import torch
    r, z = torch.from_numpy(b).cuda(), torch.empty(len(b), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    fg._lib.check(fg.lib().femgpu_solver_precondition_device(
        s.handle, C.c_void_p(r.data_ptr()), C.c_void_p(z.data_ptr())))
    return z.cpu().numpy()


@pytest.mark.parametrize("name,jump,nu", MATERIALS, ids=[m[0] for m in MATERIALS])
@pytest.mark.parametrize("make,dims", [(_p1, (60, 6, 6)), (_p2, (16, 4, 5))], ids=["p1", "p2"])
def test_sparse_panels(make, dims, name, jump, nu):
    p, k, a = _system(*make(dims), jump, nu)
    s = fg.Solver(a, fg.Unknowns.Points(p.xyz[p.free // 3]), fg.Method.Direct)
    assert "sparse multifrontal" in s.describe()
    ptr, idx, val = a.arrays()
    rng = np.random.default_rng(7)

    def mul(v, x):
        return np.add.reduceat(v.astype(np.longdouble) * x[idx], ptr[:-1])

    norm = np.sqrt((val ** 2).sum())
    smooth = np.asarray(mul(val, np.cos(np.arange(a.n) / a.n)), dtype=np.float64)
    for b in (fg.reduced_rhs(k, p.load, p.values, p.free), rng.standard_normal(a.n), smooth):
        x = _apply(s, b)
        left = np.asarray(b - mul(val, x), dtype=np.float64)
        assert np.linalg.norm(left) <= a.n * 2.2e-16 * (norm * np.linalg.norm(x)
                                                        + np.linalg.norm(b))
        # And row by row, against the magnitudes of the row's own terms.
        own = np.asarray(mul(np.abs(val), np.abs(x)), dtype=np.float64) + np.abs(b)
        assert (np.abs(left) <= a.n * 2.2e-16 * own).all()
        # The solve takes the refinement step.
        st = s.solve(b, y := np.zeros(a.n))
        left = np.asarray(b - mul(val, y), dtype=np.float64)
        own = np.asarray(mul(np.abs(val), np.abs(y)), dtype=np.float64) + np.abs(b)
        assert (np.abs(left) <= 16 * 2.2e-16 * own).all() and st.iterations == 0


@pytest.mark.parametrize("name,jump,nu", MATERIALS, ids=[m[0] for m in MATERIALS])
def test_dense_inverse(name, jump, nu):
    p, k, a = _system(*_p1((24, 4, 3)), jump, nu)
    s = fg.Solver(a, fg.Unknowns.Points(p.xyz[p.free // 3]), fg.Method.Direct)
    assert "sparse" not in s.describe()
    ptr, idx, val = a.arrays()
    d = np.zeros((a.n, a.n))
    d[np.repeat(np.arange(a.n), np.diff(ptr)), idx] = val
    scale = 1.0 / np.sqrt(np.diag(d))
    unit = d * scale[:, None] * scale[None, :]
    cond = np.linalg.cond(unit)
    inverse = np.linalg.inv(unit)
    rng = np.random.default_rng(7)
    for b in (fg.reduced_rhs(k, p.load, p.values, p.free), rng.standard_normal(a.n),
              d @ np.cos(np.arange(a.n) / a.n)):
        # The scaled solution, refined against residuals in extended precision.
        y = np.zeros(a.n, dtype=np.longdouble)
        for _ in range(6):
            left = scale * (b - np.add.reduceat(val.astype(np.longdouble) * (scale * y)[idx],
                                                ptr[:-1]))
            y = y + inverse @ np.asarray(left, dtype=np.float64)
        x = _apply(s, b) / scale
        assert np.linalg.norm(np.asarray(x - y, dtype=np.float64)) <= (
            3 * a.n * 2.2e-16 * cond * np.linalg.norm(np.asarray(y, dtype=np.float64)))
