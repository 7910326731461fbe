"""The work that users of this framework have it do, as cases that can be timed and compared.

Each case is one call, or one chain of calls, of the public API on inputs made from a seed. The
listed cases cover a resident solver asked for one more right side (the steady and the serving
use; small to large, P1 heat, box-cell elasticity, P2 elasticity on a box and on a prism mesh,
FP64 and mixed), the direct method, a batch, a transient run, the recovery of stresses, and two
whole analyses from the mesh to the solution. ``draw`` gives further cases of the same ranges.

The smoother's degree is given wherever a multigrid solver is made: by default it is chosen by
timing, and a program that wants the same digits from every process gives it.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

import femahoy_b200 as fg
from femahoy_b200 import meshgen as mg
from femahoy_b200 import prism
from femahoy_b200.batch import Batch
from femahoy_b200.recover import Recovery
from femahoy_b200.transient import Transient

RHS = 16  # the right sides of each system of a batch


def listed():
    return [
        # The smallest call in earnest: the 100 x 10 x 10 mm steel cantilever (3,000 unknowns),
        # FP64, host vectors in and out, to the default 1e-10.
        {"name": "solve_cantilever", "kind": "solve_p1_elastic", "nx": 40, "ny": 4, "nz": 4,
         "mixed": False, "host": True},
        # The benchmark configuration: P1 heat of the 128^3 cube to 1e-8, mixed precision.
        {"name": "solve_heat", "kind": "solve_heat", "nx": 128, "ny": 128, "nz": 128,
         "mixed": True, "tol": 1e-8},
        # A ragged plate with odd cell counts in the plain FP64 form, to the default tolerance.
        {"name": "solve_heat_fp64", "kind": "solve_heat", "nx": 131, "ny": 93, "nz": 37,
         "mixed": False},
        # The box-grid elastic model (box cells, 2 materials), the size of its benchmark.
        {"name": "solve_hex", "kind": "solve_hex", "nx": 256, "ny": 32, "nz": 32,
         "mixed": True, "tol": 1e-8},
        # P2 elasticity with p-multigrid: the 200 x 20 x 20 beam, 2.0M unknowns.
        {"name": "solve_p2", "kind": "solve_p2", "nx": 200, "ny": 20, "nz": 20, "mixed": True,
         "tol": 1e-8},
        # P2 elasticity on the mesh of a real part (extruded footprint with holes and a boss).
        {"name": "solve_prism", "kind": "solve_prism", "cell": 0.06, "mixed": True, "tol": 1e-8},
        # The direct method (a sparse factor, resident) on a P2 beam: one more right side.
        {"name": "solve_direct", "kind": "solve_direct", "nx": 50, "ny": 5, "nz": 5},
        # 256 uneven cantilevers with 16 load cases each, one batched call.
        {"name": "solve_batch", "kind": "batch", "count": 256, "mixed": True, "tol": 1e-8},
        # Transient heat on a ragged box: warm-started solves, launch-bound on its small levels.
        {"name": "transient", "kind": "transient", "nx": 50, "ny": 46, "nz": 47, "steps": 10},
        # Stresses of a solved P2 model.
        {"name": "recover", "kind": "recover", "nx": 160, "ny": 20, "nz": 20},
        # Whole analyses, from the mesh in host memory to the solution: assembly, reduction,
        # hierarchy, solve.
        {"name": "model_heat", "kind": "model_heat", "nx": 64, "ny": 64, "nz": 64, "mixed": True},
        {"name": "model_p2", "kind": "model_p2", "nx": 60, "ny": 8, "nz": 8, "mixed": True},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve_p1_elastic", "solve_heat", "solve_heat", "solve_hex", "solve_p2",
                       "solve_prism", "solve_direct", "batch", "transient", "recover",
                       "model_heat", "model_p2"])
    mixed = rng.random() < 0.6
    tol = rng.choice([1e-8, 1e-10])
    if kind == "solve_p1_elastic":
        return {"kind": kind, "nx": _size(rng, 20, 80), "ny": _size(rng, 2, 10),
                "nz": _size(rng, 2, 10), "mixed": mixed, "host": rng.random() < 0.5, "tol": tol}
    if kind in ("solve_heat", "model_heat"):
        hi = 128 if kind == "solve_heat" else 64
        return {"kind": kind, "nx": _size(rng, 24, hi), "ny": _size(rng, 20, hi),
                "nz": _size(rng, 20, hi), "mixed": mixed, "tol": tol}
    if kind == "solve_hex":
        return {"kind": kind, "nx": _size(rng, 40, 256), "ny": _size(rng, 8, 32),
                "nz": _size(rng, 8, 32), "mixed": mixed, "tol": tol}
    if kind == "solve_p2":
        return {"kind": kind, "nx": _size(rng, 40, 200), "ny": _size(rng, 6, 20),
                "nz": _size(rng, 6, 20), "mixed": mixed, "tol": tol}
    if kind == "solve_prism":
        return {"kind": kind, "cell": round(math.exp(rng.uniform(math.log(0.06),
                                                                 math.log(0.14))), 4),
                "mixed": True, "tol": tol}
    if kind == "solve_direct":
        return {"kind": kind, "nx": _size(rng, 30, 60), "ny": rng.randint(4, 5),
                "nz": rng.randint(4, 6)}
    if kind == "batch":
        return {"kind": kind, "count": _size(rng, 16, 256), "mixed": mixed, "tol": tol}
    if kind == "transient":
        return {"kind": kind, "nx": _size(rng, 36, 56), "ny": _size(rng, 36, 56),
                "nz": _size(rng, 36, 56), "steps": rng.randint(4, 10)}
    if kind == "recover":
        return {"kind": kind, "nx": _size(rng, 30, 160), "ny": _size(rng, 5, 20),
                "nz": _size(rng, 5, 20)}
    return {"kind": "model_p2", "nx": _size(rng, 30, 60), "ny": rng.randint(6, 8),
            "nz": rng.randint(6, 8), "mixed": mixed, "tol": tol}


# ------------------------------------------------------------------ the models

_HEX = ("nx", "ny", "nz")


def _dims(case):
    return tuple(int(case[k]) for k in _HEX)


@lru_cache(maxsize=4)
def _box(dims, lengths):
    """The Kuhn box mesh, and the sum at each node of V / 4 over its tetrahedra."""
    m = mg.box(*dims, lengths)
    vol = float(np.prod(lengths)) / (6.0 * float(np.prod(dims)))
    share = np.bincount(m.tets.ravel(), minlength=m.n) * (vol / 4.0)
    return m, share


def _heat(dims, seed):
    """P1 heat: lognormal conductivity per tetrahedron, a source, fixed ends."""
    h = max(dims)
    m, share = _box(dims, tuple(d / h for d in dims))
    rng = np.random.default_rng(seed)
    k = np.exp(rng.standard_normal(len(m.tets)))
    first, last = m.ijk[:, 0] == 0, m.ijk[:, 0] == dims[0]
    values = np.where(first, rng.uniform(0.5, 1.5), 0.0)
    return mg.Problem("p1_heat", m, m.tets, np.repeat(k[:, None], 3, axis=1), m.n, 1,
                      first | last, values, rng.uniform(0.5, 2.0) * share, xyz=m.points)


def _p1_elastic(dims, seed):
    """A P1 cantilever (mm, MPa), clamped at x = 0, a traction on the top face."""
    m, _ = _box(dims, tuple(2.5 * d for d in dims))
    rng = np.random.default_rng(seed)
    coef = np.tile([rng.uniform(50e3, 250e3), rng.uniform(0.25, 0.35)], (len(m.tets), 1))
    load = _top_load(dims, 2.5)[:, None] * rng.uniform(-1.0, 1.0, 3)
    return mg.Problem("p1_elastic", m, m.tets, coef, m.n, 3,
                      np.repeat(m.ijk[:, 0] == 0, 3), np.zeros(3 * m.n), load.ravel(),
                      xyz=m.points)


@lru_cache(maxsize=512)
def _top_load(dims, cell):
    """The area of the top face at each node (A / 3 to each corner of its triangles)."""
    m = mg.box(*dims, tuple(cell * d for d in dims))
    t, f = mg.boundary_faces(m, 2, 1)
    tri = m.tets[t][np.arange(len(t))[:, None], mg.FACES[f]]
    area = mg.face_area(m.points, tri)
    return np.bincount(tri.ravel(), np.repeat(area / 3.0, 3), minlength=m.n)


@lru_cache(maxsize=2)
def _hex_model(dims):
    nx, ny, nz = dims
    return mg.hex_cantilever(nx=nx, ny=ny, nz=nz, length=nx / 32.0, width=ny / 32.0,
                             depth=nz / 32.0)


def _hex(dims, seed):
    """A cantilever of box cells, about half of them orthotropic, a tip load."""
    p = _hex_model(dims)
    rng = np.random.default_rng(seed)
    e = rng.uniform(500.0, 2000.0)
    coef = np.tile(mg.orthotropic(e, rng.uniform(0.25, 0.33)), (len(p.nodes), 1))
    coef[rng.random(len(coef)) < 0.5] = mg.orthotropic(
        [e, e / 2.0, e / 4.0], [0.25, 0.3, 0.35], [0.3 * e, 0.25 * e, 0.2 * e])
    return mg.Problem("hex_elastic", p.mesh, p.nodes, coef, p.n_points, 3, p.fixed, p.values,
                      p.load * rng.uniform(0.5, 2.0), xyz=p.xyz)


@lru_cache(maxsize=2)
def _p2_mesh(dims, side):
    m = mg.box(*dims, tuple(side * d for d in dims))
    q = fg.Quadratic.new(m.points, m.tets)
    return m, q, mg.beam_p2(q.edges, q.tets, mesh=m)


def _p2(dims, seed, side=1.0):
    """A P2 beam clamped at x = 0 with random forces on the loaded points of x = L."""
    m, q, p = _p2_mesh(dims, side)
    rng = np.random.default_rng(seed)
    coef = np.tile([rng.uniform(50e3, 250e3), rng.uniform(0.25, 0.35)], (len(p.nodes), 1))
    at = p.load != 0.0
    load = np.zeros_like(p.load)
    load[at] = np.abs(p.load[at]).mean() * rng.uniform(-1.0, 1.0, int(at.sum()))
    prob = mg.Problem("p2_elastic", m, p.nodes, coef, p.n_points, 3, p.fixed, p.values, load,
                      edges=q.edges, xyz=p.xyz)
    return prob, m.n


@lru_cache(maxsize=2)
def _prism_mesh(cell):
    def hole(c, r):
        return prism.Outline.circle(c, r)
    plate = prism.Part("plate", 0, 0, (0.0, 0.0, 0.0), (0.0, 0.0, 0.25), prism.Footprint(
        prism.Outline.polygon([(0, 0), (4, 0), (4, 2), (0, 2)]),
        [hole((1.0, 1.0), 0.3), hole((2.2, 0.6), 0.2), hole((3.2, 1.3), 0.25)]))
    boss = prism.Part("boss", 1, 1, (0.0, 0.0, 0.25), (0.0, 0.0, 0.45), prism.Footprint(
        prism.Outline.polygon([(1.8, 1.1), (2.8, 1.1), (2.8, 1.8), (1.8, 1.8)]), []))
    tm = prism.mesh([plate, boss], 2, prism.Spacing(cell, 1.3, 2), 250_000,
                    "the mesh has more points than the solver takes")
    return tm, fg.Quadratic.new(tm.points, tm.tets)


def _prism(cell, seed):
    """A plate with 3 holes and a boss of another material, clamped at x = 0, pulled at x = 4."""
    tm, q = _prism_mesh(cell)
    rng = np.random.default_rng(seed)
    e = np.array([200e9, 70e9]) * rng.uniform(0.8, 1.2, 2)
    coef = np.stack([e[tm.part], np.array([0.3, 0.33])[tm.part]], axis=1)
    n = len(q.points)
    load = np.zeros((n, 3))
    at = np.nonzero(q.points[:, 0] == 4.0)[0]
    load[at] = rng.uniform(-1e3, 1e3, 3) / len(at)
    prob = mg.Problem("p2_elastic", None, q.tets, coef, n, 3,
                      np.repeat(q.points[:, 0] == 0.0, 3), np.zeros(3 * n), load.ravel(),
                      edges=q.edges, xyz=q.points)
    return prob, len(tm.points)


_ELEMENT = {"p1_heat": fg.P1_HEAT, "p1_elastic": fg.P1_ELASTIC, "p2_elastic": fg.P2_ELASTIC,
            "hex_elastic": fg.HEX8_ELASTIC}


def _problem(case, seed):
    """(problem, corner points of a P2 mesh or None)."""
    kind = case["kind"]
    if kind in ("solve_heat", "model_heat", "transient"):
        return _heat(_dims(case), seed), None
    if kind == "solve_p1_elastic":
        return _p1_elastic(_dims(case), seed), None
    if kind == "solve_hex":
        return _hex(_dims(case), seed), None
    if kind == "solve_prism":
        return _prism(float(case["cell"]), seed)
    if kind == "solve_direct":
        return _p2(_dims(case), seed, 5.0)
    return _p2(_dims(case), seed)


def _reduce(prob, corners):
    """The free system: (A, right side, unknowns), by the calls of a user's program."""
    free = prob.free
    k = fg.Csr.assemble(_ELEMENT[prob.kind], prob.xyz, prob.nodes, prob.coef)
    a = k.submatrix(free)
    rhs = fg.reduced_rhs(k, prob.load, prob.values, free)
    if corners is None:
        unknowns = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(prob)))
    else:
        p, coarse = fg.prolongation(prob.xyz, corners, prob.edges, free)
        unknowns = fg.Unknowns.Quadratic(prob.xyz[free // 3], p, coarse)
    return a, rhs, unknowns


def _solver(case, a, unknowns):
    if case["kind"] == "solve_direct":
        return fg.Solver(a, unknowns, fg.Method.Direct)
    options = fg.Options(precision=fg.MIXED if case.get("mixed") else fg.FP64, degree=2,
                         axes=4 if case["kind"] == "solve_prism" else 0)
    s = fg.Solver(a, unknowns, fg.Method.Multigrid, options=options)
    return s.with_tol(case["tol"]) if "tol" in case else s


# ------------------------------------------------------------------ the batch

@lru_cache(maxsize=2)
def _batch_dims(count):
    rng = np.random.default_rng(1234)
    lo, hi = (10, 1, 1), (80, 8, 8)
    return [tuple(int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
                  for a, b in zip(lo, hi)) for _ in range(count)]


@lru_cache(maxsize=512)
def _member(dims):
    m = mg.box(*dims, tuple(2.5 * d for d in dims))
    fixed = np.repeat(m.ijk[:, 0] == 0, 3)
    return m, fixed, _top_load(dims, 2.5)


def _batch_members(count, seed):
    """Each member's problem and its (rows, 16) right sides."""
    rng = np.random.default_rng(seed)
    for dims in _batch_dims(count):
        m, fixed, top = _member(dims)
        coef = np.tile([rng.uniform(50e3, 250e3), rng.uniform(0.25, 0.35)], (len(m.tets), 1))
        loads = (top[:, None, None] * rng.uniform(-1.0, 1.0, (3, RHS))).reshape(3 * m.n, RHS)
        p = mg.Problem("p1_elastic", m, m.tets, coef, m.n, 3, fixed, np.zeros(3 * m.n),
                       loads[:, 0], xyz=m.points)
        yield p, loads[~fixed]


# ------------------------------------------------------------------ prepare and run

def _field(xyz, seed):
    """A smooth displacement as a bent and twisted bar has it, 3 values per point."""
    rng = np.random.default_rng(seed)
    span = xyz.max(axis=0) - xyz.min(axis=0)
    s = (xyz - xyz.min(axis=0)) / span
    base = np.stack([s[:, 0], s[:, 1], s[:, 2], s[:, 0] ** 2, s[:, 0] * s[:, 1],
                     s[:, 0] * s[:, 2], s[:, 1] * s[:, 2], s[:, 0] ** 3,
                     np.sin(3.0 * s[:, 0]) * s[:, 2], s[:, 1] ** 2], axis=1)
    return np.ascontiguousarray(1e-3 * span.max() * base @ rng.uniform(-1.0, 1.0, (10, 3)))


def _cells_of(prob):
    """4 parts along the beam and the singular mask of its clamped edges."""
    ne = len(prob.nodes)
    part = (4 * np.arange(ne) // ne).astype(np.uint32)
    x = prob.xyz
    edge = np.zeros(len(x), dtype=bool)
    for d in (1, 2):
        edge |= (x[:, d] == x[:, d].min()) | (x[:, d] == x[:, d].max())
    return part, ((x[:, 0] == 0.0) & edge).astype(np.uint8)


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "batch":
        mats, unknowns, rhs = [], [], []
        for p, loads in _batch_members(int(case["count"]), seed):
            k = fg.Csr.assemble(fg.P1_ELASTIC, p.xyz, p.nodes, p.coef)
            mats.append(k.submatrix(p.free))
            unknowns.append(fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(p))))
            rhs.append(loads)
        precision = fg.MIXED if case["mixed"] else fg.FP64
        s = Batch(mats, unknowns, RHS, precision=precision).with_tol(case["tol"])
        state["solver"] = s
        state["stream"] = torch.cuda.ExternalStream(s.stream())
        state["b"] = torch.from_numpy(s.pack(rhs).ravel()).cuda()
        state["x"] = torch.zeros_like(state["b"])
        torch.cuda.synchronize()
        return state
    prob, corners = _problem(case, seed)
    if kind in ("model_heat", "model_p2"):
        state["model"] = (prob, corners)
        return state
    if kind == "transient":
        k = fg.Csr.assemble(fg.P1_HEAT, prob.xyz, prob.nodes, prob.coef)
        m = prob.mesh
        cap = _box(m.dims, m.lengths)[1]
        u = fg.Unknowns.Grid(fg.Level(*mg.grid_unknowns(prob)))
        state["loop"] = Transient(k, cap, 1e-3, prob.free, u, fg.Method.Multigrid,
                                  options=fg.Options(precision=fg.MIXED, degree=2))
        state["load"], state["t0"] = prob.load, prob.values
        return state
    if kind == "recover":
        part, singular = _cells_of(prob)
        state["recovery"] = Recovery(prob.xyz, prob.nodes, prob.coef, part=part, nparts=4,
                                     singular=singular)
        n = prob.n_points
        state["u"] = torch.from_numpy(_field(prob.xyz, seed).ravel()).cuda()
        for name, shape in (("stress", (n, 6)), ("strain", (n, 6)), ("mises", (n,)),
                            ("principal", (n, 3))):
            state[name] = torch.empty(shape, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        return state
    a, rhs, unknowns = _reduce(prob, corners)
    s = _solver(case, a, unknowns)
    state["solver"] = s
    if case.get("host"):
        state["b"], state["x"] = rhs, np.empty_like(rhs)
    else:
        state["stream"] = torch.cuda.ExternalStream(fg.lib().femgpu_solver_stream(s.handle))
        state["b"] = torch.from_numpy(rhs).cuda()
        state["x"] = torch.zeros_like(state["b"])
        torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "recover":
        peaks = state["recovery"].run_device(state["u"], state["stress"], state["strain"],
                                             mises=state["mises"], principal=state["principal"])
        return {"stress": state["stress"], "strain": state["strain"], "mises": state["mises"],
                "principal": state["principal"], "peak": [p.mises for p in peaks],
                "regular": [p.regular_mises for p in peaks]}
    if kind == "transient":
        frames, _, t, _ = state["loop"].run(int(case["steps"]), state["load"], state["t0"],
                                            output_every=2)
        return {"frames": frames, "t": t}
    if kind in ("model_heat", "model_p2"):
        a, rhs, unknowns = _reduce(*state["model"])
        x = np.empty(a.n)
        _solver(case, a, unknowns).solve_zero(rhs, x)
        return x
    s, b, x = state["solver"], state["b"], state["x"]
    if case.get("host"):
        s.solve_zero(b, x)
        return x
    with torch.cuda.stream(state["stream"]):
        x.zero_()
    if kind == "batch":
        s.solve_device(b, x)
    else:
        s.solve_device(b.data_ptr(), x.data_ptr())
    return x


# ------------------------------------------------------------------ what a pass cannot do without

def _counts(case):
    """(unknowns, stored entries of the symmetric half, elements) of a case's matrix."""
    kind = case["kind"]
    if kind == "batch":
        n = sum(3 * (a + 1) * (b + 1) * (c + 1) for a, b, c in _batch_dims(int(case["count"])))
        return n, 22 * n, 0
    if kind == "solve_prism":
        tm, q = _prism_mesh(float(case["cell"]))
        n = 3 * len(q.points)
        return n, 42 * n, len(tm.tets)
    nx, ny, nz = _dims(case)
    cells = nx * ny * nz
    points = (nx + 1) * (ny + 1) * (nz + 1)
    if kind in ("solve_heat", "model_heat", "transient"):
        return points, 8 * points, 6 * cells
    if kind == "solve_p1_elastic":
        return 3 * points, 23 * 3 * points, 6 * cells
    if kind == "solve_hex":
        return 3 * points, 41 * 3 * points, cells
    fine = (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1)
    return 3 * fine, 42 * 3 * fine, 6 * cells


def work(case):
    """Bytes and operations of one pass. A PCG iteration cannot do without the FP64 operator's
    symmetric half, the cycle's operator in its own precision (once before and once after the
    coarser levels) and about 12 vectors; the iterations are those the reference's method takes
    to the tolerance. A direct solve reads its factor twice; a recovery reads the cells and the
    displacement and writes its outputs; an analysis adds the matrix, written and read once."""
    kind = case["kind"]
    n, half, elements = _counts(case)
    if kind == "recover":
        points = n // 3
        return {"bytes": elements * 56.0 + 8.0 * points * (3 + 3 + 6 + 6 + 1 + 3),
                "flops": elements * 10 * 250.0}
    if kind == "solve_direct":
        entries = 370.0 * n
        return {"bytes": 16.0 * entries + 16.0 * n, "flops": 4.0 * entries}
    its = {"solve_p1_elastic": 2, "solve_heat": 9, "model_heat": 10, "solve_hex": 10,
           "solve_p2": 13, "model_p2": 13, "solve_prism": 20, "batch": 20,
           "transient": 5}[kind]
    if kind == "transient":
        its *= int(case["steps"])
    cycle = 4.0 if case.get("mixed") or kind == "transient" else 8.0
    columns = RHS if kind == "batch" else 1
    one = half * (8.0 + 2.0 * cycle) + n * columns * 12.0 * cycle
    total = its * one
    flops = its * columns * 3.0 * 4.0 * half
    if kind.startswith("model"):
        total += 2.0 * 24.0 * half + elements * 64.0
        flops += elements * (200.0 if kind == "model_heat" else 36_000.0)
    return {"bytes": total, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, plainly

_MAX_EXACT = 420_000  # elastic unknowns: above, plain conjugate gradients take too long


def _gradients(xyz, tets):
    """The gradients of the 4 volume coordinates (T, 4, 3) and the volumes."""
    p = xyz[tets]
    j = p[:, 1:] - p[:, :1]
    inv = torch.linalg.inv(j)
    g = inv.transpose(1, 2)
    return torch.cat([-g.sum(1, keepdim=True), g], 1), torch.linalg.det(j).abs() / 6.0


def _law(constants):
    """The stress of each strain component pair (T, 6, 6), order xx yy zz xy yz xz, of the 9
    constants Ex Ey Ez nu_xy nu_xz nu_yz G_xy G_xz G_yz."""
    e, nu, g = constants[:, :3], constants[:, 3:6], constants[:, 6:]
    s = torch.zeros(len(constants), 3, 3, dtype=torch.float64, device=constants.device)
    for d in range(3):
        s[:, d, d] = 1.0 / e[:, d]
    for (a, b), k in (((0, 1), 0), ((0, 2), 1), ((1, 2), 2)):
        s[:, a, b] = s[:, b, a] = -nu[:, k] / e[:, a]
    out = torch.zeros(len(constants), 6, 6, dtype=torch.float64, device=constants.device)
    out[:, :3, :3] = torch.linalg.inv(s)
    out[:, 3, 3], out[:, 4, 4], out[:, 5, 5] = g[:, 0], g[:, 2], g[:, 1]
    return out


def _strain_rows(g):
    """B (..., 6, 3 N) of the gradients (..., N, 3); shear rows are engineering strains."""
    n = g.shape[-2]
    b = torch.zeros(*g.shape[:-2], 6, 3 * n, dtype=torch.float64, device=g.device)
    for d in range(3):
        b[..., d, d::3] = g[..., d]
    for row, (p, q) in ((3, (0, 1)), (4, (1, 2)), (5, (0, 2))):
        b[..., row, p::3] = g[..., q]
        b[..., row, q::3] = g[..., p]
    return b


def _p2_gradients(g, at):
    """The gradients of the 10 functions at the volume coordinates ``at``."""
    out = [(4.0 * at[i] - 1.0) * g[:, i] for i in range(4)]
    out += [4.0 * (at[a] * g[:, b] + at[b] * g[:, a]) for a, b in mg.EDGES.tolist()]
    return torch.stack(out, 1)


def _isotropic(coef):
    e, nu = coef[:, :1], coef[:, 1:]
    return _law(torch.cat([e, e, e, nu, nu, nu] + [e / (2.0 * (1.0 + nu))] * 3, 1))


def _hex_matrix(size, law):
    """The 24 x 24 stiffness of box cells with the incompatible modes 1 - xi^2 condensed."""
    bits = torch.tensor(mg.HEX_BITS, dtype=torch.float64, device=size.device) * 2.0 - 1.0
    k = torch.zeros(len(size), 33, 33, dtype=torch.float64, device=size.device)
    for xi in bits / math.sqrt(3.0):
        f = 0.5 * (1.0 + bits * xi)
        g = torch.stack([bits[:, d] * f[:, (d + 1) % 3] * f[:, (d + 2) % 3] for d in range(3)],
                        1)
        g = torch.cat([g, torch.diag(-4.0 * xi)])[None] / size[:, None, :]
        b = _strain_rows(g)
        k += (size.prod(1) / 8.0)[:, None, None] * b.transpose(1, 2) @ law @ b
    mode = torch.linalg.solve(k[:, 24:, 24:], k[:, 24:, :24])
    return k[:, :24, :24] - k[:, :24, 24:] @ mode


def _element_matrices(prob):
    """(matrices (K, m, m), the class of each element or None)."""
    x = torch.from_numpy(prob.xyz).cuda()
    t = torch.from_numpy(prob.nodes.astype(np.int64)).cuda()
    c = torch.from_numpy(prob.coef).cuda()
    if prob.kind == "hex_elastic":
        keys = torch.cat([x[t[:, 6]] - x[t[:, 0]], c], 1)
        keys, cls = torch.unique(keys.round(decimals=12), dim=0, return_inverse=True)
        return _hex_matrix(keys[:, :3], _law(keys[:, 3:])), cls
    g, v = _gradients(x, t[:, :4])
    if prob.kind == "p1_heat":
        return v[:, None, None] * (g * c[:, None, :]) @ g.transpose(1, 2), None
    law = _isotropic(c)
    if prob.kind == "p1_elastic":
        b = _strain_rows(g)
        return v[:, None, None] * b.transpose(1, 2) @ law @ b, None
    lo, hi = (5.0 - math.sqrt(5.0)) / 20.0, (5.0 + 3.0 * math.sqrt(5.0)) / 20.0
    k = 0.0
    for q in range(4):
        b = _strain_rows(_p2_gradients(g, [hi if i == q else lo for i in range(4)]))
        k = k + (v / 4.0)[:, None, None] * b.transpose(1, 2) @ law @ b
    return k, None


class _Plain:
    """The full matrix as its elements, and Jacobi-preconditioned conjugate gradients."""

    def __init__(self, prob, extra=None):
        self.k, self.cls = _element_matrices(prob)
        c = prob.comps
        t = torch.from_numpy(prob.nodes.astype(np.int64)).cuda()
        self.dof = (c * t[:, :, None] + torch.arange(c, device="cuda")).reshape(len(t), -1)
        self.n = prob.n_unknowns
        self.free = torch.from_numpy(~prob.fixed).cuda()
        self.extra = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        if extra is not None:
            self.extra += torch.from_numpy(extra).cuda()
        diag = self.k.diagonal(dim1=1, dim2=2)
        diag = diag if self.cls is None else diag[self.cls]
        self.diag = self.extra.clone().index_add_(0, self.dof.ravel(), diag.ravel())

    def mul(self, x):
        u = x[self.dof]
        if self.cls is None:
            y = (self.k @ u[:, :, None])[:, :, 0]
        else:
            y = torch.empty_like(u)
            for i, k in enumerate(self.k):
                at = self.cls == i
                y[at] = u[at] @ k
        return (self.extra * x).index_add_(0, self.dof.ravel(), y.ravel())

    def solve(self, load, values, x=None):
        """The solution with the fixed ``values``, to what 64 bits hold; full vectors."""
        x = values.clone() if x is None else torch.where(self.free, x, values)
        r = torch.where(self.free, load - self.mul(x), 0.0)
        inv = torch.where(self.free, 1.0 / self.diag, 0.0)
        goal = 1e-14 * float(torch.where(self.free, load - self.mul(values), 0.0).norm())
        z = inv * r
        p, rz = z.clone(), float(r @ z)
        best, since = math.inf, 0
        for i in range(30_000):
            q = torch.where(self.free, self.mul(p), 0.0)
            a = rz / float(p @ q)
            x += a * p
            r -= a * q
            z = inv * r
            now, rz0 = float(r @ z), rz
            rz = now
            if float(r.norm()) <= goal or rz == 0.0:
                break
            p = z + (rz / rz0) * p
        return x


def _recovered(prob, seed):
    x = torch.from_numpy(prob.xyz).cuda()
    t = torch.from_numpy(prob.nodes.astype(np.int64)).cuda()
    law = _isotropic(torch.from_numpy(prob.coef).cuda())
    u = torch.from_numpy(_field(prob.xyz, seed)).cuda()[t].reshape(len(t), 30, 1)
    g, _ = _gradients(x, t[:, :4])
    corners = torch.eye(4, dtype=torch.float64).tolist()
    local = corners + [[0.5 * (corners[a][i] + corners[b][i]) for i in range(4)]
                       for a, b in mg.EDGES.tolist()]
    n = prob.n_points
    hits = torch.bincount(t.ravel(), minlength=n).double()[:, None]
    mean = torch.zeros(2, n, 6, dtype=torch.float64, device="cuda")
    part, singular = _cells_of(prob)
    part = torch.from_numpy(part.astype(np.int64)).cuda()
    bad = torch.from_numpy(singular.astype(bool)).cuda()
    bad = bad[t] | bad[t[:, :4]].any(1, keepdim=True)

    def mises(s):
        d = (s[:, 0] - s[:, 1]) ** 2 + (s[:, 1] - s[:, 2]) ** 2 + (s[:, 2] - s[:, 0]) ** 2
        return (0.5 * d + 3.0 * (s[:, 3:] ** 2).sum(1)).sqrt()

    peak = torch.full((2, 4), -math.inf, dtype=torch.float64, device="cuda")
    for i, at in enumerate(local):
        e = (_strain_rows(_p2_gradients(g, at)) @ u)[:, :, 0]
        s = (law @ e[:, :, None])[:, :, 0]
        e[:, 3:] *= 0.5
        mean[0].index_add_(0, t[:, i], s)
        mean[1].index_add_(0, t[:, i], e)
        m = mises(s)
        peak[0].index_reduce_(0, part, m, "amax")
        peak[1].index_reduce_(0, part, torch.where(bad[:, i], -math.inf, m), "amax")
    s, e = mean / hits
    full = s[:, [0, 3, 5, 3, 1, 4, 5, 4, 2]].reshape(n, 3, 3)
    eig = torch.cat([torch.linalg.eigvalsh(c) for c in full.split(16384)]).flip(1)
    return {"stress": s, "strain": e, "mises": mises(s), "principal": eig,
            "peak": peak[0].tolist(), "regular": peak[1].tolist()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        # Each member's 16 solutions, by rows; the batch's vector holds the members in order.
        out = []
        if _counts(case)[0] > 200_000:
            return None
        for p, loads in _batch_members(int(case["count"]), seed):
            free = torch.from_numpy(p.free).cuda()
            if len(free) > 12_000:
                return None
            plain = _Plain(p)
            full = torch.zeros(plain.n, plain.n, dtype=torch.float64, device="cuda")
            m = plain.dof.shape[1]
            rows = plain.dof[:, :, None].expand(-1, m, m).reshape(-1)
            cols = plain.dof[:, None, :].expand(-1, m, m).reshape(-1)
            full.view(-1).index_add_(0, rows * plain.n + cols, plain.k.reshape(-1))
            a = full[free][:, free]
            out.append(torch.linalg.solve(a, torch.from_numpy(loads).cuda()))
        return torch.cat(out).ravel()
    n = _counts(case)[0]
    if kind == "recover":
        prob, _ = _problem(case, seed)
        return _recovered(prob, seed)
    if kind not in ("solve_heat", "model_heat", "transient") and n > _MAX_EXACT:
        return None
    prob, _ = _problem(case, seed)
    load = torch.from_numpy(prob.load).cuda()
    values = torch.from_numpy(prob.values).cuda()
    if kind == "transient":
        m = prob.mesh
        rate = _box(m.dims, m.lengths)[1] / 1e-3
        plain = _Plain(prob, extra=rate)
        rate = torch.from_numpy(rate).cuda()
        frames, t, steps = [], values, int(case["steps"])
        for s in range(1, steps + 1):
            t = plain.solve(load + rate * t, values, t)
            if s % 2 == 0 or s == steps:
                frames.append(t)
        return {"frames": torch.stack(frames), "t": t}
    x = _Plain(prob).solve(load, values)
    free = torch.from_numpy(prob.free).cuda()
    return x[free].cpu().numpy() if case.get("host") or kind.startswith("model") else x[free]
