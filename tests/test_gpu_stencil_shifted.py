"""The bulk-copy stencil with shifted windows where the shift changes from plane
to plane or only from column to column (odd, 2-mod-4 and aligned planes with
odd leading dimensions), just above the sizes it starts at, and the smaller
grids it leaves to the register-queue kernel.  With no poll allowed only the
bulk-copy pipelines report a wait, which shows the route of each call.

Reference: the operator assembled in 64 bits from the values each precision
starts from (the FP32 potential and weights are rounded first, which moves each
of the 29 terms by 3 x 2^-24 more).  Bounds of the largest result, whose terms
add up to less than four times as much: FP64 29 x 2^-53 x 4 = 1.3e-14, FP32
(29 + 3) x 2^-24 x 4 = 7.6e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import F32, F64  # noqa: E402

DEV = torch.device("cuda", 0)
CASES = [
    # sides, order, precision, columns, ld - n, whether the bulk-copy kernel takes it
    ((61, 54, 67), 8, "f32", 31, 0, True),      # planes of 2 mod 4 elements
    ((61, 54, 67), 8, "f32", 31, 1, True),
    ((62, 54, 67), 8, "f64", 31, 1, True),      # even planes, columns at odd addresses
    ((64, 52, 50), 4, "f32", 31, 1, True),      # aligned planes, columns at every remainder
    ((64, 52, 50), 2, "f32", 31, 2, True),
    ((45, 47, 49), 8, "f64", 8, 0, True),       # 0.83 M points, slabs 83 % full
    ((45, 47, 49), 8, "f64", 7, 0, False),      # 0.73 M
    ((61, 55, 67), 8, "f32", 9, 3, True),       # 2.0 M points
    ((61, 55, 67), 8, "f32", 8, 3, False),      # 1.798 M
    ((33, 35, 31), 8, "f64", 64, 0, False),     # slabs 75 % full
    ((45, 23, 30), 8, "f64", 3, 0, False),
    ((3, 3, 3), 8, "f32", 5, 0, False),
    ((1, 1, 9), 8, "f64", 3, 1, False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-{c[2]}-k{c[3]}-ld{c[4]}")
def test_against_the_assembled_operator(case):
    (nx, ny, nz), order, dt, k, extra, bulk = case
    dom = {"nx": nx, "ny": ny, "nz": nz, "h": 0.5, "radius": 0.25 * (nx - 1)}
    ctx = gpu.GridContext(dom, order)
    n, ld = ctx.n, ctx.n + extra
    tdt, code, tol = (torch.float64, F64, 1.3e-14) if dt == "f64" else (torch.float32, F32, 7.6e-6)
    rng = np.random.default_rng(nx + k)
    pot = rng.standard_normal(n)
    gpu.Hamiltonian(ctx, torch.from_numpy(pot).to(DEV))

    def columns():
        """k columns of the block, NaN in the gaps; the last column ends the buffer."""
        buf = torch.full(((k - 1) * ld + n,), float("nan"), dtype=tdt, device=DEV)
        rows = torch.from_numpy(rng.standard_normal((k, n))).to(DEV, tdt)
        for j in range(k):
            buf[j * ld:j * ld + n] = rows[j]
        return buf, rows.double().cpu().numpy()

    (X, xr), (P, pr) = columns(), columns()
    Y = torch.full_like(X, float("nan"))

    def step():
        ctx.call("psc_apply_h_axpby", code, gpu._p(X), ld, gpu._p(P), ld, gpu._p(Y), ld, k, 0.75, -0.25, -0.875,
                 gpu._stream())

    step()
    ctx.check_status()
    got = np.stack([Y[j * ld:j * ld + n].double().cpu().numpy() for j in range(k)])
    for j in range(k - 1):
        assert bool(torch.isnan(Y[j * ld + n:(j + 1) * ld]).all())
    w = (0.5 * O.laplacian(dom, order) @ xr.T).T + pot * xr
    ref = 0.75 * w - 0.25 * xr - 0.875 * pr
    assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    ctx.call("psc_set_wait_limit", 0)
    step()
    assert bool(ctx.status()[3]) == bulk
    ctx.call("psc_set_wait_limit", -1)
    step()
    again = np.stack([Y[j * ld:j * ld + n].double().cpu().numpy() for j in range(k)])
    assert np.array_equal(again, got)
