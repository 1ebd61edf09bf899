"""The dense y-transforms (fp_dense.cuh) at the edges of their tiles and of their range, against the oracle: row
lengths around the column tiles (32, 48, 64, 80 columns of half a row), the last length of each family and the first
one beyond it, row counts around the row tiles and around the change of launch shape (100 tiles of 32 rows)."""
import numpy as np
import pytest

from gpu_util import rel_max, torch_cuda
from oracle import fp_oracle as O
from focalors_poisson_b200 import capi

pytestmark = pytest.mark.gpu
PAIRS = {"DD": (0, 0), "NN": (1, 1), "ND": (1, 0), "DN": (0, 1), "PP": (2, 2)}


@pytest.mark.parametrize("kind", list(PAIRS))
@pytest.mark.parametrize("ny", [2, 3, 5, 16, 31, 33, 63, 64, 65, 80, 95, 96, 97, 129, 144, 146, 160, 193, 224, 225, 256, 258])
def test_dense_transforms_vs_oracle(kind, ny):
    """In place on the device, forward and inverse; FP64 at the other transforms' 1e-13, FP32 rows at 2e-5."""
    if kind == "PP" and ny % 2:
        ny += 1
    torch = torch_cuda()
    rng = np.random.default_rng(ny)
    for rows in (1, 7, 33, 3199, 3217):
        f = rng.standard_normal((rows, ny))
        for inv in (False, True):
            ref = (O.transform_inverse if inv else O.transform_forward)(kind, f)
            t = torch.tensor(f, device="cuda")
            capi.transform(*PAIRS[kind], t, inverse=inv, out=t)
            assert rel_max(t.cpu().numpy(), ref) <= 1e-13, (kind, ny, rows, inv)
            t = torch.tensor(f, device="cuda", dtype=torch.float32)
            capi.transform(*PAIRS[kind], t, inverse=inv, out=t)
            assert rel_max(t.double().cpu().numpy(), ref) <= 2e-5, (kind, ny, rows, inv, "f32")


@pytest.mark.parametrize("shape,bc", [((33, 64, 31), (0, 0, 0, 0, 0, 0)), ((17, 97, 70), (1, 0, 1, 0, 0, 1)),
                                      ((40, 66, 34), (2, 2, 2, 2, 0, 0)), ((16, 95, 8), (0, 0, 1, 1, 2, 2)),
                                      ((24, 50, 40), (1, 1, 1, 1, 1, 1)), ((24, 34, 36), (2, 2, 1, 1, 2, 2))])
def test_rect3d_middle_axis_vs_oracle(shape, bc):
    """The y-transform on the middle axis of a 3D field (no transposes), two fields in one call; the last two have no
    Dirichlet face (the last one keeps the transposed layout). 1e-11 as for the other 3D solves."""
    torch = torch_cuda()
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + ny + nz)
    f = rng.standard_normal((2, nx, ny, nz))
    h = (0.1, 0.07, 0.09)
    ref = np.stack([O.PoissonSolver3D(nx, ny, nz, *h, bc).solve(f[b]) for b in range(2)])
    t = torch.tensor(f, device="cuda")
    capi.Rect3D(nx, ny, nz, *h, bc).solve(t)
    assert rel_max(t.cpu().numpy(), ref) <= 1e-11, (shape, bc)
