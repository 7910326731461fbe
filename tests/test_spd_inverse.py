"""The dense SPD inverse at the edges of its 128-column blocks, 32-column sub-blocks and padding:
one product with it (no refinement) against numpy's solve of the same system."""
import ctypes as C

import numpy as np
import pytest

import femahoy_b200 as fg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 128, 129, 255, 257, 511, 1000, 4096])
def test_inverse_product(n):
    """Diagonally dominant rows (off-diagonal magnitudes half the diagonal: condition at most 3):
    factor, inverse and product each round within about n eps, so the product is within
    3 * 3 n eps of the solution (n at least 32: a few roundings are left at any size)."""
    import torch
    rng = np.random.default_rng(n)
    a = rng.uniform(-1.0, 1.0, (n, n))
    a = a + a.T
    np.fill_diagonal(a, 0.0)
    scale = 10.0 ** rng.uniform(-3, 3, n)  # a wide range of pivots
    np.fill_diagonal(a, 2.0 * np.abs(a).sum(axis=1) + 1.0)
    d = a * scale[:, None] * scale[None, :]
    ptr = np.arange(n + 1, dtype=np.int64) * n
    m = fg.Csr.from_arrays(n, ptr, np.tile(np.arange(n, dtype=np.uint32), n), d)
    s = fg.Solver(m, fg.Unknowns.Points(rng.uniform(0.0, 1.0, (n, 3))), fg.Method.Direct)
    assert "sparse" not in s.describe()
    b = rng.standard_normal(n) * scale
    r = torch.from_numpy(b).cuda()
    z = torch.empty_like(r)
    torch.cuda.synchronize()
    fg._lib.check(fg.lib().femgpu_solver_precondition_device(
        s.handle, C.c_void_p(r.data_ptr()), C.c_void_p(z.data_ptr())))
    # In the scaled unknowns the system is the well conditioned one.
    y = np.linalg.solve(a, b / scale)
    got = z.cpu().numpy() * scale
    assert np.linalg.norm(got - y) <= 9 * max(n, 32) * 2.3e-16 * np.linalg.norm(y)


@pytest.mark.parametrize("n,bad", [(40, 0), (300, 130), (300, 299), (700, 511)])
def test_first_failing_pivot(n, bad):
    """The text names the first column whose pivot is not positive, in any block."""
    a = np.eye(n) * 2.0
    a[bad, bad] = -1.0
    if bad + 1 < n:
        a[n - 1, n - 1] = -4.0
    ptr = np.arange(n + 1, dtype=np.int64) * n
    m = fg.Csr.from_arrays(n, ptr, np.tile(np.arange(n, dtype=np.uint32), n), a)
    with pytest.raises(fg.FemError) as e:
        fg.Solver(m, fg.Unknowns.Points(np.zeros((n, 3))), fg.Method.Direct)
    assert e.value.code == 3 and f"column {bad} " in str(e.value)
