"""The spectral solvers' work lists over the caller's fields: other pointers on the same stream only refill the lists'
records, other streams, ghost patterns or kinds of call build them again. Every call must give what a solver that
never saw another buffer gives, bit for bit (fixed-order sums). And the batched one-pass chase at the sizes where its
launch classes change, against the Schur GMRES path."""
import numpy as np
import pytest

from gpu_util import rel_max, torch_cuda
from focalors_poisson_b200 import capi
from focalors_poisson_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _rhs(torch, g, seed):
    return [torch.tensor(f, device="cuda") for f in W.gaussian_rhs(g, seed, zero_mean=False)]


def _ghosts(torch, g, seed, doms):
    rng = np.random.default_rng(seed)
    return [[torch.tensor(rng.standard_normal(g.ny[d] if f < 2 else g.nx[d]), device="cuda") if g.bc[d][f] != 3 else None
             for f in range(4)] if d in doms else None for d in range(g.n_domains)]


@pytest.mark.parametrize("n", [64, 96])
def test_other_buffers_streams_and_ghosts(n):
    torch = torch_cuda()
    g = W.cross(n, neumann_tips=True)
    one = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
    side = torch.cuda.Stream()
    calls = [("f64", None, False), ("f64", None, False), ("f64", (1, 3), False), ("f64", (1, 3), False), ("f64", (2,), False),
             ("f64", None, True), ("mixed", None, False), ("mixed", (4,), False), ("f32", None, True), ("f32", None, False),
             ("adjoint", None, False), ("f64", None, False)]

    def run(solver, form, f, gh):
        if form == "f64":
            solver.solve(f, gh)
        elif form == "adjoint":
            solver.adjoint(f)
        else:
            solver.solve_ir(f, gh, rel_tol=1e-11, inner=form)

    kept = []  # every call gets buffers of its own
    for k, (form, doms, other) in enumerate(calls):
        f, gh = _rhs(torch, g, k), None if doms is None else _ghosts(torch, g, k, doms)
        want = [x.clone() for x in f]
        run(capi.Composite(g, m=20, tol=1e-12, max_iter=100), form, want, gh)
        torch.cuda.synchronize()
        with torch.cuda.stream(side if other else torch.cuda.current_stream()):
            run(one, form, f, gh)
        torch.cuda.synchronize()
        kept.append((f, gh))
        for a, b in zip(f, want):
            assert torch.equal(a, b), (k, form, doms, other)


@pytest.mark.parametrize("sides", [(64, 64, 64, 64), (128, 160, 512, 96), (544, 64, 96, 128), (1024, 64, 1056, 64),
                                   (64, 96, 2080, 64), (96, 65, 4096, 33)])
def test_batched_chase_classes_match_gmres(sides):
    """An L of a x b, c x b and a x d cells: rows per chunk, tile width and CTA size all follow from nx."""
    torch = torch_cuda()
    a, b, c, d = sides
    h = 1.0 / max(a, b)
    g = W.Geometry([a, c, a], [b, b, d], [h] * 3, [h] * 3, [[0] * 4 for _ in range(3)], [(0, W.XPOS, 1), (0, W.YPOS, 2)])
    f = _rhs(torch, g, 7)
    want = [x.clone() for x in f]
    capi.Composite(g, m=40, tol=1e-15, max_iter=200, spectral=False).solve(want)
    scale = max(float(x.abs().max()) for x in want)
    for precision, steps, bound in (("f64", 0, 1e-10), ("f32", 3, 1e-10)):
        got = [x.clone() for x in f]
        capi.Batch([g], precision=precision).solve(got, steps=steps, sync=True)
        for x, y in zip(got, want):
            assert float((x - y).abs().max()) <= bound * scale, (sides, precision)
