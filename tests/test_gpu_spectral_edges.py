"""The spectral preconditioner at the edges of its tiles: axes of one to a few
points (no odd modes, fewer rows than a fragment), around the 8-row fragment
and the 32-line tile, the longest axis it takes, and unequal x and y axes
(each with its own matrix).

Bound: three forward and three backward passes of at most 128 products, each
within 128 units of 2^-53 of the line's norm, through 1 / Lambda; relative to
the largest entry 1e-12 covers 6 x 128 x 2^-53 = 9e-14 with the growth of a
maximum against a norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
SHAPES = [((1, 1, 1), 2), ((2, 3, 1), 2), ((5, 1, 4), 2), ((7, 9, 8), 4), ((16, 15, 17), 6), ((31, 33, 2), 8),
          ((65, 64, 63), 8), ((128, 127, 5), 8), ((9, 128, 128), 8), ((127, 8, 121), 8)]


@pytest.mark.parametrize("shape,order", SHAPES)
def test_preconditioner_at_tile_edges(shape, order):
    nx, ny, nz = shape
    dom = {"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 0.17 * (nx - 1)}
    ctx = gpu.GridContext(dom, order)
    r = np.random.default_rng(sum(shape) + order).standard_normal(ctx.n)
    rd = torch.from_numpy(r).to(DEV)
    z = gpu.poisson_precond(ctx, rd).cpu().numpy()
    ref = O.spectral_preconditioner(dom, order)(r)
    assert np.abs(z - ref).max() <= 1e-12 * np.abs(ref).max()
    assert np.array_equal(rd.cpu().numpy(), r)          # the input is only read


@pytest.mark.parametrize("maxit,tol", [(0, 1e-5), (1, 1e-5), (2, 1e-30), (4, 1e-30), (60, 1e-5)])
def test_device_side_stop(maxit, tol):
    """Iteration limits inside, at and past the batches queued ahead: the
    oracle's count and its iterate (a solve past its stop changes nothing)."""
    dom, order = {"nx": 20, "ny": 17, "nz": 22, "h": 0.34, "radius": 3.2}, 8
    ctx = gpu.GridContext(dom, order)
    rng = np.random.default_rng(5)
    rhs, x0 = rng.standard_normal(ctx.n), 0.1 * rng.standard_normal(ctx.n)
    x, its = gpu.pcg(gpu.Laplacian(ctx), torch.from_numpy(rhs).to(DEV), torch.from_numpy(x0).to(DEV), maxit, tol,
                     "spectral", "precLU")
    xo, its_o = O.pcg_prec(O.laplacian(dom, order), rhs, x0, maxit, tol, O.spectral_preconditioner(dom, order))
    assert its == its_o if maxit <= 4 else abs(its - its_o) <= 1
    assert np.linalg.norm(x.cpu().numpy() - xo) <= 1e-8 * np.linalg.norm(xo)
