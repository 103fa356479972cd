"""The sphere mask where its edge meets the grid: odd and unequal sides, radii
that end exactly on a plane, a point or between points, spheres that cut the
box, hold all of it, one point or none, and orders with other halos.  Spacing and
radii are multiples of 1/8, so whether a point is inside is exact arithmetic.

Reference: the operator assembled in 64 bits from the values each precision
starts from (FP32: X, the potential and the weights are rounded first, which
moves each of the 27 terms by 3 x 2^-24).  Bounds of the largest result, whose
terms add up to less than eight times as much: FP64 27 x 2^-53 x 8 = 2.4e-14,
FP32 (27 + 3) x 2^-24 x 8 = 1.43e-5."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
CASES = [
    # sides, order, columns, radius in units of h = 1/2 (points of an odd side lie
    # at whole numbers from the centre, those of an even side at halves)
    ((40, 36, 38), 8, 5, 16.5),
    ((42, 34, 33), 8, 3, 16.0),
    ((41, 36, 35), 4, 4, 17.0),
    ((41, 34, 52), 8, 3, 16.5),
    ((33, 35, 31), 8, 5, 15.0),
    ((46, 44, 21), 6, 2, 40.0),
    ((37, 36, 9), 2, 3, 4.0),
    ((28, 26, 24), 8, 2, 200.0),
    ((29, 28, 27), 8, 2, 0.5),
    ((28, 28, 28), 8, 2, 0.5),
    ((61, 55, 67), 8, 31, 27.0),
    ((62, 54, 66), 8, 31, 26.5),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-o{c[1]}-r{c[3]}")
@pytest.mark.parametrize("impl", [0, 1])
def test_mask_is_exact(case, impl):
    (nx, ny, nz), order, k, r = case
    h = 0.5
    dom = {"nx": nx, "ny": ny, "nz": nz, "h": h, "radius": 0.5 * h * (nx - 1)}
    n = nx * ny * nz
    x, y, z = ((np.arange(m) - 0.5 * (m - 1)) for m in (nx, ny, nz))
    inside = (((x[None, None, :] ** 2 + y[None, :, None] ** 2) + z[:, None, None] ** 2) <= r * r).ravel()
    rng = np.random.default_rng(n + k)
    pot = rng.standard_normal(n)
    X = rng.uniform(0.5, 1.5, (k, n)) * inside
    ctx = gpu.GridContext(dom, order)
    ctx.call("psc_set_stencil_impl", impl)
    ctx.set_sphere_mask(r * h)
    assert ctx.inside_count() == int(inside.sum())
    H = gpu.Hamiltonian(ctx, torch.from_numpy(pot).to(DEV))
    L = 0.5 * O.laplacian(dom, order)
    for dt, tol in ((torch.float64, 2.4e-14), (torch.float32, 1.43e-5)):
        Xd = torch.from_numpy(X).to(DEV, dt)
        Xr = Xd.double().cpu().numpy()
        ref = ((L @ Xr.T).T + pot * Xr) * inside
        Y = (H @ Xd).double().cpu().numpy()
        assert not Y[:, ~inside].any()
        assert np.abs(Y - ref).max() <= tol * max(np.abs(ref).max(), 1.0)
    ctx.check_status()
