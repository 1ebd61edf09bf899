"""The solves whose speed this repository is held to: what a user's program has the library do, over the sizes,
boundary types, precision forms and directions it is used with.

A case is a dict of plain values. Its "kind" picks the entry point:

  rect         capi.Rect.solve           one or several rectangles of one shape, FP64
  rect3d       capi.Rect3D.solve         one box, FP64
  composite    capi.Composite            a tree of rectangles: FP64 solve, refined solves, adjoint
  grad         autograd.solve            forward and backward of the differentiable solve
  batch        capi.Batch                many uneven L and T problems in one captured graph
  composite3d  capi.Composite3D          a star of boxes
  stream       capi.Composite.solve_async  a stream of independent problems from page-locked host memory

Solves work in place, so a pass first puts the right-hand sides into the fields (one copy, as a program does
that keeps its source terms) and then solves. The fields of one problem are views into one buffer.
Boundary strings give one letter per face in the order x-, x+, y-, y+ (, z-, z+): D Dirichlet, N Neumann,
P periodic. Every problem has a Dirichlet face somewhere.
"""
import math

import torch

from focalors_poisson_b200 import autograd, capi
from focalors_poisson_b200 import workloads as W

BC = {"D": W.DIRICHLET, "N": W.NEUMANN, "P": W.PERIODIC}


def listed():
    return [
        # A general rectangle: sides that are no multiple of anything, a Neumann wall in each direction.
        {"name": "rect_1000x1500", "kind": "rect", "nx": 1000, "ny": 1500, "bc": "DNND", "fields": 1},
        # A plane channel: periodic along the flow, walls across it.
        {"name": "channel_2048x1024", "kind": "rect", "nx": 2048, "ny": 1024, "bc": "PPDD", "fields": 1},
        # The 3D rectangle solve at the size its throughput is quoted on.
        {"name": "box_256", "kind": "rect3d", "nx": 256, "ny": 256, "nz": 256, "bc": "DDDDDD"},
        # A turbulent-channel box: periodic in the two wall-parallel directions, uneven sides.
        {"name": "channel3d_96x80x144", "kind": "rect3d", "nx": 96, "ny": 80, "nz": 144, "bc": "PPDDPP"},
        # The smallest composite solve: five 128 x 128 rectangles, one FP64 solve per call.
        {"name": "cross_128", "kind": "composite", "shape": "cross", "n": 128, "tips": "D", "form": "f64"},
        # The largest single composite solve, refined to 1e-11 by FP32 corrections of the FP64 solve.
        {"name": "cross_2048_mixed", "kind": "composite", "shape": "cross", "n": 2048, "tips": "N", "form": "mixed"},
        # A tree of depth two with periodic arms and Neumann faces: the Schur-complement GMRES.
        {"name": "tree9_384", "kind": "composite", "shape": "tree9", "n": 384, "tips": "N", "form": "f64"},
        # Source inversion: gradients with respect to the right-hand side and a per-cell source scale.
        {"name": "grad_512", "kind": "grad", "n": 512},
        # Many uneven problems at once, FP64.
        {"name": "batch_48_f64", "kind": "batch", "count": 48, "first": 2024, "precision": "f64", "steps": 0},
        # Many uneven problems at once, FP32 solves in FP64 refinement.
        {"name": "batch_24_f32ir", "kind": "batch", "count": 24, "first": 3024, "precision": "f32", "steps": 2},
        # The 3D composite: a root box with four children on x, y and z faces.
        {"name": "star3d_48", "kind": "composite3d", "n": 48, "arm": 40, "leaves": 4},
        # Problems that arrive in host memory and whose solutions go back there, one after the other.
        {"name": "stream_768", "kind": "stream", "n": 768, "calls": 4},
    ]


def draw(rng):
    def size(lo, hi, step=1):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return max(lo, int(round(v / step)) * step)

    kind = rng.choice(["rect", "rect", "rect", "rect3d", "rect3d", "composite", "composite", "composite", "grad", "batch",
                       "batch", "composite3d", "stream"])
    if kind == "rect":
        bx = rng.choice(["DD", "DN", "ND", "NN", "PP", "DD"])
        by = rng.choice(["DD", "DN", "ND", "NN", "PP", "DD"])
        if "D" not in bx + by:
            bx = "DN"
        nx, ny = size(40, 2048), size(40, 2048)
        ny += ny % 2 if by == "PP" else 0
        most = max(1, min(8, (1 << 21) // (nx * ny)))
        return {"kind": kind, "nx": nx, "ny": ny, "bc": bx + by, "fields": rng.randint(1, most)}
    if kind == "rect3d":
        b = [rng.choice(["DD", "DN", "NN", "PP", "DD"]) for _ in range(3)]
        if "D" not in "".join(b):
            b[1] = "DD"
        n = [size(24, 224) for _ in range(3)]
        n = [n[0]] + [v + (v % 2 if p == "PP" else 0) for v, p in zip(n[1:], b[1:])]
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "bc": "".join(b)}
    if kind == "composite":
        shape = rng.choice(["cross", "cross", "lt", "ragged", "tree9"])
        form = rng.choice(["f64", "f64", "mixed", "f32", "adjoint"])
        if shape == "cross":
            return {"kind": kind, "shape": shape, "n": size(64, 1536, 32), "tips": rng.choice("DN"), "form": form}
        if shape == "lt":
            return {"kind": kind, "shape": shape, "n": rng.randint(1, 1 << 20), "tips": "D", "form": form}
        if shape == "ragged":  # sides that are no multiple of 32: the Schur-complement GMRES
            return {"kind": kind, "shape": "cross", "n": size(41, 300) | 1, "tips": rng.choice("DN"), "form": "f64"}
        return {"kind": kind, "shape": shape, "n": size(64, 256, 32), "tips": "N", "form": "f64"}
    if kind == "grad":
        return {"kind": kind, "n": size(96, 640, 32)}
    if kind == "batch":
        f32 = rng.random() < 0.5
        return {"kind": kind, "count": rng.randint(4, 24), "first": rng.randint(1, 1 << 20),
                "precision": "f32" if f32 else "f64", "steps": 2 if f32 else 0}
    if kind == "composite3d":
        return {"kind": kind, "n": size(16, 44), "arm": size(12, 40), "leaves": rng.randint(2, 4)}
    return {"kind": kind, "n": size(128, 704, 32), "calls": rng.randint(2, 6)}


# ---------------------------------------------------------------------------------------------------------
# Problems
# ---------------------------------------------------------------------------------------------------------
def _steps(case):
    """Grid steps of a rectangle or box of unit height (a general aspect ratio of the cells in 3D)."""
    h = 1.0 / case["ny"]
    return h, h, 1.25 * h


def _geometry(case):
    if case.get("shape", "cross") == "lt":
        return W.lt_problem(case["n"])
    if case.get("shape") == "tree9":
        return W.tree9(case["n"])
    return W.cross(case["n"], neumann_tips=case.get("tips") == "N")


def _star3d(case):
    """A cube of n^3 cells with children of `arm` cells along their axis on the faces x-, x+, y+, z-."""
    n, arm, k = case["n"], case["arm"], case["leaves"]
    h = 1.0 / n
    faces = [0, 1, 3, 4][:k]
    shapes = [(n, n, n)] + [tuple(arm if f // 2 == a else n for a in range(3)) for f in faces]
    bc = [[W.DIRICHLET] * 6 for _ in shapes]
    bc[1][faces[0]] = W.NEUMANN  # the first child's far face
    return shapes, h, bc, [(0, f, i + 1) for i, f in enumerate(faces)]


def _shapes(case):
    """The shape of every field of the case, problems back to back."""
    kind = case["kind"]
    if kind == "rect":
        return [(case["fields"], case["nx"], case["ny"])]
    if kind == "rect3d":
        return [(case["nx"], case["ny"], case["nz"])]
    if kind == "composite3d":
        return _star3d(case)[0]
    if kind == "batch":
        return [s for p in range(case["count"]) for s in _pairs(W.lt_problem(case["first"] + p))]
    return _pairs(_geometry(case))


def _pairs(g):
    return [(int(a), int(b)) for a, b in zip(g.nx, g.ny)]


def _flat(shapes, device="cuda", **kw):
    """One buffer for fields of these shapes, each on a 512-byte boundary, and the fields as views of it."""
    starts, at = [], 0
    for s in shapes:
        starts.append(at)
        at += -(-math.prod(s) // 64) * 64
    flat = torch.zeros(at, dtype=torch.float64, device=device, **kw)
    return flat, [flat[o:o + math.prod(s)].view(s) for o, s in zip(starts, shapes)]


def _sources(case, seed, count=1):
    """`count` sets of right-hand sides: seeded N(0,1) values per cell."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
    out = []
    for _ in range(count):
        flat, fields = _flat(_shapes(case))
        for f in fields:
            f.normal_(generator=gen)
        out.append((flat, fields))
    return out


def _inversion(case, seed):
    """Source, per-cell scale in [0.5, 1.5) and target of the differentiable solve."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 29)
    rhs, scale, target = [], [], []
    for s in _shapes(case):
        rhs.append(torch.randn(s, generator=gen, dtype=torch.float64, device="cuda"))
        scale.append(torch.rand(s, generator=gen, dtype=torch.float64, device="cuda") + 0.5)
        target.append(torch.randn(s, generator=gen, dtype=torch.float64, device="cuda") * 1e-2)
    return rhs, scale, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        rhs, scale, target = _inversion(case, seed)
        for t in rhs + scale:
            t.requires_grad_(True)
        return {"kind": kind, "solver": capi.Composite(_geometry(case), m=20, tol=1e-12, max_iter=100), "rhs": rhs,
                "scale": scale, "target": target}
    if kind == "stream":
        rhs = []
        for flat, _ in _sources(case, seed, case["calls"]):
            host, fields = _flat(_shapes(case), device="cpu", pin_memory=True)
            host.copy_(flat)
            rhs.append(fields)
        outs = [_flat(_shapes(case), device="cpu", pin_memory=True) for _ in range(case["calls"])]
        return {"kind": kind, "solver": capi.Composite(_geometry(case), m=20, tol=1e-12, max_iter=100), "rhs": rhs,
                "out": [f for _, f in outs], "flat": [h for h, _ in outs]}
    (rhs, _), = _sources(case, seed)
    flat, fields = _flat(_shapes(case))
    state = {"kind": kind, "form": case.get("form"), "rhs": rhs, "flat": flat, "fields": fields}
    if kind == "rect":
        hx, hy, _ = _steps(case)
        state["solver"] = capi.Rect(case["nx"], case["ny"], hx, hy, [BC[c] for c in case["bc"]])
    elif kind == "rect3d":
        hx, hy, hz = _steps(case)
        state["solver"] = capi.Rect3D(case["nx"], case["ny"], case["nz"], hx, hy, hz, [BC[c] for c in case["bc"]])
    elif kind == "batch":
        problems = [W.lt_problem(case["first"] + p) for p in range(case["count"])]
        state["solver"] = capi.Batch(problems, precision=case["precision"])
        state["steps"] = case["steps"]
    elif kind == "composite3d":
        shapes, h, bc, conns = _star3d(case)
        state["solver"] = capi.Composite3D([s + (h, h, h) for s in shapes], conns, bc, m=20, tol=1e-12, max_iter=100)
    else:
        state["solver"] = capi.Composite(_geometry(case), m=20, tol=1e-12, max_iter=100)
    return state


def run(state):
    kind, solver = state["kind"], state["solver"]
    if kind == "grad":
        u = autograd.solve(solver, state["rhs"], state["scale"], form="f32ir", rel_tol=1e-11)
        grads = torch.autograd.grad(u, state["rhs"] + state["scale"], [a.detach() - b for a, b in zip(u, state["target"])])
        return [a.detach() for a in u], list(grads)
    if kind == "stream":
        for rhs, out in zip(state["rhs"], state["out"]):
            solver.solve_async(rhs, out, form="mixedir", rel_tol=1e-11)
        solver.wait()
        return state["flat"]
    flat, fields = state["flat"], state["fields"]
    flat.copy_(state["rhs"])
    if kind in ("rect", "rect3d"):
        solver.solve(fields[0])
    elif kind == "batch":
        solver.solve(fields, steps=state["steps"], graph=True)
    elif kind == "composite3d" or state["form"] == "f64":
        solver.solve(fields)
    elif state["form"] == "adjoint":
        solver.adjoint(fields)
    else:
        solver.solve_ir(fields, rel_tol=1e-11, inner=state["form"])
    return flat


def work(case):
    """Each right-hand side read once and each solution written once; per cell one forward and one inverse fast
    transform (2.5 log2 n operations each) along every transformed axis and an 8-operation tridiagonal solve."""
    cells, ops, axes = 0, 0.0, 2 if case["kind"] in ("rect3d", "composite3d") else 1
    for s in _shapes(case):
        n = math.prod(s)
        cells += n
        ops += n * (8 + sum(5.0 * math.log2(v) for v in s[-axes:]))
    if case["kind"] == "stream":
        return {"bytes": 16 * cells * case["calls"], "flops": ops * case["calls"]}
    if case["kind"] == "grad":  # rhs, scale and target read, solution and two gradients written; two solves
        return {"bytes": 48 * cells, "flops": 2 * ops}
    return {"bytes": 16 * cells, "flops": ops}


# ---------------------------------------------------------------------------------------------------------
# The answers in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------------------
def _line(n, lo, hi, seen):
    """Eigenvalues and eigenvectors of the 1D second difference on n cells (Neumann mirrors the end cell,
    Dirichlet and connected faces leave it out, periodic wraps)."""
    key = (n, lo, hi)
    if key not in seen:
        t = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        t.diagonal().fill_(-2.0)
        t.diagonal(1).fill_(1.0)
        t.diagonal(-1).fill_(1.0)
        t[0, 0] += 1.0 if lo == W.NEUMANN else 0.0
        t[-1, -1] += 1.0 if hi == W.NEUMANN else 0.0
        if lo == W.PERIODIC:
            t[0, -1] += 1.0
            t[-1, 0] += 1.0
        seen[key] = torch.linalg.eigh(t)
    return seen[key]


class _Box:
    """The constant-coefficient operator of one rectangle or box, inverted in its eigenbasis."""

    def __init__(self, shape, weights, bc, seen):
        self.lines = [_line(n, bc[2 * a], bc[2 * a + 1], seen) for a, n in enumerate(shape)]
        self.weights, self.bc = weights, bc
        eig = 0.0
        for a, ((w, _), c) in enumerate(zip(self.lines, weights)):
            eig = eig + (c * w).view([-1 if b == a else 1 for b in range(len(shape))])
        self.eig = eig

    def _basis(self, f, transpose):
        for a, (_, v) in enumerate(self.lines):
            g = f.movedim(a, -1)
            f = (g @ (v if transpose else v.T)).movedim(-1, a)
        return f

    def inverse(self, f):
        return self._basis(self._basis(f, True) / self.eig, False)

    def apply(self, u):
        r = torch.zeros_like(u)
        for a, c in enumerate(self.weights):
            n = u.shape[a]
            r.narrow(a, 0, n - 1).add_(u.narrow(a, 1, n - 1), alpha=c)
            r.narrow(a, 1, n - 1).add_(u.narrow(a, 0, n - 1), alpha=c)
            r.add_(u, alpha=-2.0 * c)
            lo, hi = self.bc[2 * a], self.bc[2 * a + 1]
            if lo == W.NEUMANN:
                r.select(a, 0).add_(u.select(a, 0), alpha=c)
            if hi == W.NEUMANN:
                r.select(a, n - 1).add_(u.select(a, n - 1), alpha=c)
            if lo == W.PERIODIC:
                r.select(a, 0).add_(u.select(a, n - 1), alpha=c)
                r.select(a, n - 1).add_(u.select(a, 0), alpha=c)
        return r


def _tree_solve(boxes, conns, rhs):
    """The coupled problem (adjacent cells of connected faces coupled with coefficient 1) by conjugate gradients
    preconditioned with the single boxes' inverses, restarted twice on the true residual."""
    def edge(u, face):
        return u.select(face // 2, u.shape[face // 2] - 1 if face % 2 else 0)

    def apply(u):
        r = [b.apply(v) for b, v in zip(boxes, u)]
        for a, face, b in conns:
            edge(r[a], face).add_(edge(u[b], face ^ 1))
            edge(r[b], face ^ 1).add_(edge(u[a], face))
        return r

    def dot(p, q):
        return sum((x * y).sum() for x, y in zip(p, q))

    u = [torch.zeros_like(f) for f in rhs]
    if not conns:
        return [b.inverse(f) for b, f in zip(boxes, rhs)]
    for _ in range(3):
        r = [f - v for f, v in zip(rhs, apply(u))]
        z = [b.inverse(v) for b, v in zip(boxes, r)]
        p, rz = [v.clone() for v in z], dot(r, z)
        begun = abs(float(rz))
        for k in range(2000):
            ap = apply(p)
            alpha = rz / dot(p, ap)
            for x, y, s, t in zip(u, r, p, ap):
                x.add_(alpha * s)
                y.sub_(alpha * t)
            z = [b.inverse(v) for b, v in zip(boxes, r)]
            new = dot(r, z)
            if k % 8 == 7 and abs(float(new)) <= 1e-26 * begun:
                break
            p = [v.add_((new / rz) * s) for v, s in zip(z, p)]
            rz = new
    return u


def _composite_answer(g, rhs, seen):
    """A u = hx^2 rhs on the tree g of rectangles."""
    boxes = [_Box((g.nx[d], g.ny[d]), [1.0, (g.hx[d] / g.hy[d]) ** 2], g.bc[d], seen) for d in range(g.n_domains)]
    return _tree_solve(boxes, g.connections, [f * (h * h) for f, h in zip(rhs, g.hx)])


def exact(case, seed):
    kind, seen = case["kind"], {}
    if kind == "grad":
        rhs, scale, target = _inversion(case, seed)
        g = _geometry(case)
        u = _composite_answer(g, [a * b for a, b in zip(rhs, scale)], seen)
        v = _composite_answer(g, [a - b for a, b in zip(u, target)], seen)
        return u, [a * b for a, b in zip(v, scale)] + [a * b for a, b in zip(v, rhs)]
    if kind == "stream":
        g, out = _geometry(case), []
        for _, rhs in _sources(case, seed, case["calls"]):
            flat, fields = _flat(_shapes(case))
            for a, b in zip(fields, _composite_answer(g, rhs, seen)):
                a.copy_(b)
            out.append(flat)
        return out
    (_, rhs), = _sources(case, seed)
    flat, fields = _flat(_shapes(case))
    if kind in ("rect", "rect3d"):
        hx, hy, hz = _steps(case)
        weights = [1.0, (hx / hy) ** 2] + ([(hx / hz) ** 2] if kind == "rect3d" else [])
        shape = _shapes(case)[0][-len(weights):]
        box = _Box(shape, weights, [BC[c] for c in case["bc"]], seen)
        for a, b in zip(fields[0].view((-1,) + shape), rhs[0].view((-1,) + shape)):
            a.copy_(box.inverse(b))
        return flat
    if kind == "composite3d":
        shapes, h, bc, conns = _star3d(case)
        boxes = []
        for d, s in enumerate(shapes):
            joined = {f for a, f, b in conns if a == d} | {f ^ 1 for a, f, b in conns if b == d}
            boxes.append(_Box(s, [1.0] * 3, [W.ADJACENTED if f in joined else bc[d][f] for f in range(6)], seen))
        answer = _tree_solve(boxes, conns, [f * (h * h) for f in rhs])
    elif kind == "batch":
        answer, at = [], 0
        for p in range(case["count"]):
            g = W.lt_problem(case["first"] + p)
            answer += _composite_answer(g, rhs[at:at + g.n_domains], seen)
            at += g.n_domains
    else:
        answer = _composite_answer(_geometry(case), rhs, seen)
    for a, b in zip(fields, answer):
        a.copy_(b)
    return flat
