"""Calls at the sizes and values where the library changes the way it takes: both ways must give the same."""
import pytest

from gpu_util import torch_cuda
from focalors_poisson_b200 import capi
from focalors_poisson_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_fp32_rows_are_scaled_before_they_are_rounded():
    """A right-hand side of 1e38 has transforms beyond the FP32 range; times hx^2 they, and the solution's, are inside
    it. Against the solve of the constant 1: the same FP32 arithmetic up to the rounding of the scaled values, 1e-4."""
    torch = torch_cuda()
    g = W.cross(64)
    one = capi.Batch([g], precision="f32")
    got, want = ([torch.full((a, b), v, dtype=torch.float64, device="cuda") for a, b in zip(g.nx, g.ny)] for v in (1e38, 1.0))
    one.solve(got, sync=True)
    one.solve(want, sync=True)
    top = max(float(y.abs().max()) for y in want)
    for x, y in zip(got, want):
        assert float((x / 1e38 - y).abs().max()) <= 1e-4 * top
