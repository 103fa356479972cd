"""The persistent CG on grids cut into boxes, at the cuts' edges: fewer points
than CTAs, axes of one or a few points, unequal boxes, runs of one to twelve
points, orders with narrower halos, and the sizes above which the flat ranges
take over.  The reference is the oracle's CG, run for a fixed number of
iterations.

Bound: two runs of the same recurrences in another order of summation differ
by the rounding of each step, grown by at most the condition number of the
operator, about (4 n / pi)^2 < 2e4 for n <= 100, per step taken: 30 x 2e4 x
2^-53 = 7e-11 of the iterate's norm; 1e-9 allows for the constant."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
CASES = [((1, 1, 1), 2, 1), ((5, 3, 2), 8, 4), ((3, 40, 1), 4, 6), ((7, 11, 13), 6, 12), ((25, 24, 26), 2, 30),
         ((61, 55, 67), 8, 30), ((130, 8, 96), 8, 30), ((10, 200, 30), 4, 30), ((84, 83, 82), 8, 12),
         ((92, 90, 91), 8, 12)]


@pytest.mark.parametrize("shape,order,maxit", CASES, ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_box_cg_matches_oracle(shape, order, maxit):
    nx, ny, nz = shape
    dom = {"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 0.17 * (nx - 1)}
    ctx = gpu.GridContext(dom, order)
    rng = np.random.default_rng(sum(shape) + order)
    rhs, x0 = rng.standard_normal(ctx.n), 0.1 * rng.standard_normal(ctx.n)
    x, its = gpu.pcg(gpu.Laplacian(ctx), torch.from_numpy(rhs).to(DEV), torch.from_numpy(x0).to(DEV), maxit, 1e-9)
    xo, its_o = O.pcg(O.laplacian(dom, order), rhs, x0, maxit, 1e-9)
    assert its == its_o
    assert np.linalg.norm(x.cpu().numpy() - xo) <= 1e-9 * np.linalg.norm(xo)
    ctx.check_status()


@pytest.mark.parametrize("n", [12, 40, 52])
def test_repeated_solves_are_identical(n):
    """Thousands of grid-wide reductions, in which fast CTAs run ahead of slow
    ones: every solve ends, with the same bits."""
    ctx = gpu.GridContext({"nx": n, "ny": n, "nz": n, "h": 0.34, "radius": 0.17 * (n - 1)}, 8)
    g = torch.Generator(device="cuda").manual_seed(n)
    rhs = torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=g)
    x0, A = torch.zeros_like(rhs), gpu.Laplacian(ctx)
    first, its = gpu.pcg(A, rhs, x0, 50, 1e-30)
    for _ in range(150):
        x, i = gpu.pcg(A, rhs, x0, 50, 1e-30)
        assert i == its and torch.equal(x, first)
    ctx.check_status()
