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
