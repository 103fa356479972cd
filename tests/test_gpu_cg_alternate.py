"""The box CG after one to six iterations: r alternates between two arrays and
the partial sums between four sets, so every turn of both is compared with the
kernels that run one launch per step (psc_set_use_graphs 0).

Bound: the two add the same terms in other orders; the rounding of a step,
2^-53 of the vectors' norms times the terms of a sum (27), grows by at most the
condition number per step, below 2e4 at these sizes: 6 x 27 x 2e4 x 2^-53 =
4e-10 of the iterate's norm."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dims", [(9, 7, 5), (40, 41, 42), (78, 77, 79)])
def test_every_turn_of_the_arrays(dims):
    nx, ny, nz = dims
    ctx = gpu.GridContext({"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 1.0}, 8)
    A = gpu.Laplacian(ctx)
    g = torch.Generator(device="cuda").manual_seed(nx)
    rhs, x0 = (torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=g) for _ in range(2))
    for maxit in range(1, 7):
        ctx.call("psc_set_use_graphs", 2)
        x, its = gpu.pcg(A, rhs, x0, maxit, 1e-12)
        ctx.call("psc_set_use_graphs", 0)
        ref, its_ref = gpu.pcg(A, rhs, x0, maxit, 1e-12)
        assert its == its_ref == maxit
        assert float((x - ref).norm()) <= 4e-10 * float(ref.norm())
    ctx.check_status()
