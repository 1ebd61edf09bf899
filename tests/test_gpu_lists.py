"""The spectral solvers' work lists over the caller's fields where a call cannot finish, follows unfinished work or is
recorded: every solve must still be one of its own fields."""
import pytest

from gpu_util import torch_cuda
from focalors_poisson_b200 import capi
from focalors_poisson_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _rhs(torch, g, seed):
    return [torch.tensor(f, device="cuda") for f in W.gaussian_rhs(g, seed, zero_mean=False)]


def _solved(torch, solve, f):
    want = [x.clone() for x in f]
    solve(want)
    torch.cuda.synchronize()
    return want


def _same(torch, f, want):
    return all(torch.equal(a, b) for a, b in zip(f, want))


@pytest.mark.parametrize("retry", ["same", "other"])
def test_no_lists_left_by_a_call_out_of_memory(retry):
    """The first refined solve allocates its buffers (94 MB each here): with 64 MB left on the device it fails, and
    afterwards the same solver solves the same fields, and others, as one that never failed."""
    torch = torch_cuda()
    g = W.cross(1536)
    f, other = _rhs(torch, g, 1), _rhs(torch, g, 2)
    want = _solved(torch, lambda x: capi.Batch([g]).solve(x, steps=2), f if retry == "same" else other)
    one = capi.Batch([g])
    one.solve([x.clone() for x in f])
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    hog = torch.empty(free - (64 << 20), dtype=torch.uint8, device="cuda")
    with pytest.raises(capi.FpError):
        one.solve(f, steps=2)
    del hog
    torch.cuda.empty_cache()
    got = f if retry == "same" else other
    one.solve(got, steps=2)
    torch.cuda.synchronize()
    assert _same(torch, got, want)


def test_calls_queued_on_one_stream_and_on_two():
    """Calls on other fields follow each other without a wait of the host: the lists of a solve still running must not
    change. On two streams ordered by nothing else the solver orders its own calls."""
    torch = torch_cuda()
    g = W.cross(512, neumann_tips=True)
    one = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
    batch = capi.Batch([g, W.cross(256)], precision="f32")
    sets = [_rhs(torch, g, k) for k in range(6)]
    more = [_rhs(torch, g, k) + _rhs(torch, W.cross(256), k) for k in range(6)]
    fresh = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
    calls = [(fresh.solve, one.solve), (fresh.adjoint, one.adjoint)] * 3
    want = [_solved(torch, c[0], f) for c, f in zip(calls, sets)]
    same = capi.Batch([g, W.cross(256)], precision="f32")
    bwant = [_solved(torch, lambda x: same.solve(x, steps=2), f) for f in more]
    for streams in (1, 2):
        lanes = [torch.cuda.Stream() for _ in range(streams)]
        got, bgot = [[x.clone() for x in f] for f in sets], [[x.clone() for x in f] for f in more]
        torch.cuda.synchronize()
        for k in range(6):
            with torch.cuda.stream(lanes[k % streams]):
                calls[k][1](got[k])
                batch.solve(bgot[k], steps=2, graph=True)
        torch.cuda.synchronize()
        for k in range(6):
            assert _same(torch, got[k], want[k]) and _same(torch, bgot[k], bwant[k]), (streams, k)


def test_stream_handle_given_out_again():
    """A stream is destroyed with a solve still queued on it, and the next stream may get its handle: a solve of other
    fields there must leave the queued one its lists."""
    import ctypes

    torch = torch_cuda()
    g = W.cross(64)
    one = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
    a, b = _rhs(torch, g, 1), _rhs(torch, g, 2)
    rhs = [x.clone() for x in a]
    fresh = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
    want_a, want_b = _solved(torch, fresh.solve, a), _solved(torch, fresh.solve, b)
    rt = torch.cuda.cudart()

    def stream():
        h = ctypes.c_void_p()
        assert int(rt.cudaStreamCreate(ctypes.addressof(h))) == 0
        return h.value

    first = stream()
    with torch.cuda.stream(torch.cuda.ExternalStream(first)):
        one.solve(a)
        one.solve(a)
        for x, y in zip(a, rhs):
            x.copy_(y)
        torch.cuda._sleep(400_000_000)  # 0.2 s
        one.solve(a)
    assert int(rt.cudaStreamDestroy(first)) == 0
    second = stream()
    with torch.cuda.stream(torch.cuda.ExternalStream(second)):
        one.solve(b)
    torch.cuda.synchronize()
    assert _same(torch, a, want_a) and _same(torch, b, want_b), second == first
    assert int(rt.cudaStreamDestroy(second)) == 0


@pytest.mark.parametrize("form", ["solve", "adjoint", "batch", "batch_graph"])
def test_captured_solve_keeps_its_fields(form):
    """A caller's graph solves the fields it was captured with, also after calls on other fields, a second graph and the
    end of the first; fields the solver has not seen cannot be captured."""
    torch = torch_cuda()
    g = W.cross(64, neumann_tips=True)

    def make():
        if form.startswith("batch"):
            b = capi.Batch([g])
            return lambda x: b.solve(x, steps=2, graph=form == "batch_graph")
        c = capi.Composite(g, m=20, tol=1e-12, max_iter=100)
        return getattr(c, form)

    one, fresh = make(), make()
    rhs = [_rhs(torch, g, k) for k in range(3)]
    want = [_solved(torch, fresh, f) for f in rhs]
    f = [[x.clone() for x in r] for r in rhs]

    def refill():
        for a, b in zip(f, rhs):
            for x, y in zip(a, b):
                x.copy_(y)

    def captured(k):
        one(f[k])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            one(f[k])
        return graph

    first = captured(0)
    one(f[1])
    one(f[1])
    refill()
    one(f[2])
    first.replay()
    torch.cuda.synchronize()
    assert _same(torch, f[0], want[0]) and _same(torch, f[1], rhs[1]) and _same(torch, f[2], want[2])
    second = captured(1)
    refill()
    second.replay()
    first.replay()
    one(f[2])
    torch.cuda.synchronize()
    assert all(_same(torch, a, b) for a, b in zip(f, want))
    refused = torch.cuda.CUDAGraph()
    with torch.cuda.graph(refused):
        with pytest.raises(capi.FpError):
            one([x.clone() for x in f[0]])
    torch.cuda.synchronize()
    del first, refused
    for k in (0, 2, 0, 2):
        refill()
        one(f[k])
        second.replay()
        torch.cuda.synchronize()
        assert _same(torch, f[k], want[k]) and _same(torch, f[1], want[1])
