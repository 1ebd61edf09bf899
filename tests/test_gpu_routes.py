"""Calls at the sizes and values where the library changes the way it takes: both ways must give the same."""
import numpy as np
import pytest

from gpu_util import rel_max, torch_cuda
from oracle import fp_oracle as O
from focalors_poisson_b200 import capi
from focalors_poisson_b200 import workloads as W

pytestmark = pytest.mark.gpu
PAIRS = {"DD": (0, 0), "NN": (1, 1), "ND": (1, 0), "DN": (0, 1), "PP": (2, 2)}


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


@pytest.mark.parametrize("kind,ny", [("DD", 63), ("DD", 95), ("DD", 127), ("DD", 128), ("DD", 134), ("DD", 199), ("DD", 224),
                                     ("DD", 256), ("NN", 64), ("NN", 96), ("NN", 95), ("PP", 60), ("PP", 64), ("PP", 126),
                                     ("PP", 128), ("PP", 144), ("ND", 67), ("ND", 122), ("ND", 157), ("ND", 224),
                                     ("DN", 94), ("DN", 175), ("DN", 192), ("DN", 200)])
def test_product_and_fft_rows_vs_oracle(kind, ny):
    """Row counts on both sides of every line between the dense product and the FFT, and of the change of launch shape;
    row lengths at the ends of the bands. In place, FP64 at 1e-13 and FP32 rows at 2e-5 as for the other transforms."""
    torch = torch_cuda()
    f = np.random.default_rng(ny).standard_normal((12288, ny))
    for inv in (False, True):
        ref = (O.transform_inverse if inv else O.transform_forward)(kind, f)
        for rows in (1535, 1536, 2047, 2048, 2559, 2560, 3072, 3200, 3584, 5632, 7167, 7168, 12287, 12288):
            for dtype, bound in ((torch.float64, 1e-13), (torch.float32, 2e-5)):
                t = torch.tensor(f[:rows], device="cuda", dtype=dtype)
                capi.transform(*PAIRS[kind], t, inverse=inv, out=t)
                assert rel_max(t.double().cpu().numpy(), ref[:rows]) <= bound, (kind, ny, rows, inv, dtype)


def test_batched_lists_by_product_and_by_fft():
    """1, 2 and 10 crosses of 256 x 256 are 1280, 2560 and 12800 rows a launch: product, FFT, product. Every problem's
    solution against the others' (1e-11 as for the other composite solves; FP32 in three refinement steps 1e-10)."""
    torch = torch_cuda()
    g = W.cross(256)
    f = [torch.tensor(x, device="cuda") for x in W.gaussian_rhs(g, 3)]
    for precision, steps, bound in (("f64", 0, 1e-11), ("f32", 3, 1e-10)):
        want = None
        for count in (1, 2, 10):
            got = [x.clone() for _ in range(count) for x in f]
            capi.Batch([g] * count, precision=precision).solve(got, steps=steps, sync=True)
            want = want or got
            top = max(float(x.abs().max()) for x in want)
            for k, x in enumerate(got):
                assert float((x - want[k % 5]).abs().max()) <= bound * top, (precision, count, k)


@pytest.mark.parametrize("nx", [3, 4, 7, 8, 13, 16, 20, 24, 27, 34, 41])
def test_one_pass_and_sequential_columns(nx):
    """Many short columns take one thread each, few the one-pass chase: field counts on both sides of every line between
    them, against the same fields solved 32 at a time. Every x pair, and systems without a Dirichlet face. 1e-11 as for the
    other rectangle solves."""
    torch = torch_cuda()
    ny = 64
    f = torch.tensor(np.random.default_rng(nx).standard_normal((3072, nx, ny)), device="cuda")
    for bc in ((0, 0, 0, 0), (1, 0, 0, 0), (0, 1, 0, 0), (1, 1, 0, 0), (2, 2, 0, 0), (1, 1, 1, 1), (2, 2, 1, 1)):
        one = capi.Rect(nx, ny, 0.05, 0.07, bc)
        want = f.clone()
        for part in want.split(32):
            one.solve(part)
        top = float(want.abs().max())
        for columns in (8192, 24576, 32768, 49152, 65536, 98304, 131072, 196608):
            for fields in (columns // ny - 1, columns // ny):
                got = f[:fields].clone()
                one.solve(got)
                assert float((got - want[:fields]).abs().max()) <= 1e-11 * top, (bc, columns, fields)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_bad_value_stays_in_its_row_field_and_problem(bad):
    """One bad value spoils its own row of a dense transform (tiles of 32 and of 8 rows), its own field of a rectangle or
    box solve and its own problem of a batch; everything else is what it is without it, bit for bit."""
    torch = torch_cuda()
    gen = torch.Generator(device="cuda").manual_seed(1)

    def check(run, shape, item):
        f = torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")
        g = f.clone()
        g[item].view(-1)[g[item].numel() // 3] = bad
        run(f)
        run(g)
        torch.cuda.synchronize()
        keep = torch.ones(shape[0], dtype=torch.bool, device="cuda")
        keep[item] = False
        assert torch.equal(f[keep], g[keep]) and bool(torch.isfinite(f).all()) and not bool(torch.isfinite(g[item]).all())

    for kind, ny, rows in (("DD", 128, 4000), ("NN", 64, 100), ("PP", 144, 8000), ("ND", 96, 37)):
        for inv in (False, True):
            check(lambda x: capi.transform(*PAIRS[kind], x, inverse=inv, out=x), (rows, ny), rows // 2)
    for nx, ny, bc in ((64, 96, (0, 0, 0, 0)), (600, 40, (1, 0, 0, 0)), (100, 64, (2, 2, 0, 0)), (8, 64, (0, 0, 0, 0))):
        check(capi.Rect(nx, ny, 0.05, 0.07, bc).solve, (3, nx, ny), 1)
    check(capi.Rect3D(16, 32, 24, 0.05, 0.07, 0.06, (0, 0, 0, 0, 2, 2)).solve, (3, 16, 32, 24), 1)
    g = W.cross(64)
    b = capi.Batch([g] * 3)
    check(lambda x: b.solve([x[p, d] for p in range(3) for d in range(5)], sync=True), (3, 5, 64, 64), 1)
