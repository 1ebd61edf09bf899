"""The chase along x at the sizes where its chunk layout changes (fp_chase_tile.cuh: chunks of R and R - 1 rows,
R = 16, 8 or 4; two sizes no R divides; beyond 4096 rows another kernel), against the oracle's sequential solve."""
import numpy as np
import pytest

from gpu_util import rel_max, torch_cuda
from oracle import fp_oracle as O
from focalors_poisson_b200 import capi

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 4, 5, 7, 8, 9, 12, 13, 31, 32, 33, 49, 57, 100, 255, 256, 257, 511, 512, 513, 527, 528, 1000, 2047, 2048,
         2049, 4095, 4096, 4097, 4128]
X_PAIRS = [(0, 0), (1, 0), (0, 1), (1, 1), (2, 2)]


@pytest.mark.parametrize("nx", SIZES)
def test_chase_layouts_vs_oracle(nx):
    """Every x boundary pair, with a width of one tile, a tile and one lane, and a whole number of tiles. Dirichlet
    walls across keep every system well conditioned: 1e-11 as for the other rectangle solves."""
    torch = torch_cuda()
    rng = np.random.default_rng(nx)
    for ny in (6, 9, 16):
        for x in X_PAIRS:
            bc = x + (0, 0)
            f = rng.standard_normal((2, nx, ny))
            ref = np.stack([O.PoissonSolver2D(nx, ny, 0.05, 0.07, bc).solve(f[b]) for b in range(2)])
            t = torch.tensor(f, device="cuda")
            capi.Rect(nx, ny, 0.05, 0.07, bc).solve(t)
            assert rel_max(t.cpu().numpy(), ref) <= 1e-11, (nx, ny, bc)


@pytest.mark.parametrize("nx,bc", [(100, (1, 1, 1, 1)), (100, (2, 2, 2, 2)), (57, (1, 1, 2, 2)), (96, (2, 2, 1, 1))])
def test_chase_singular_mode_vs_oracle(nx, bc):
    """No Dirichlet face: the last wavenumber takes the reference's singular recursion next to the tiles."""
    torch = torch_cuda()
    rng = np.random.default_rng(nx + 1)
    f = rng.standard_normal((2, nx, 34))
    ref = np.stack([O.PoissonSolver2D(nx, 34, 0.05, 0.07, bc).solve(f[b]) for b in range(2)])
    t = torch.tensor(f, device="cuda")
    capi.Rect(nx, 34, 0.05, 0.07, bc).solve(t)
    assert rel_max(t.cpu().numpy(), ref) <= 1e-11, bc
