"""A CG solve of no iterations leaves x as it was and reports none, also after
another solve on the same context, on each of its paths."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("mode", [0, 1, 2])
def test_no_iterations_after_a_solve(mode):
    ctx = gpu.GridContext({"nx": 18, "ny": 18, "nz": 18, "h": 0.34, "radius": 1.0}, 8)
    ctx.call("psc_set_use_graphs", mode)
    A = gpu.Laplacian(ctx)
    g = torch.Generator(device="cuda").manual_seed(3)
    rhs, x0 = (torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=g) for _ in range(2))
    assert gpu.pcg(A, rhs, x0, 5, 1e-12)[1] == 5
    x, its = gpu.pcg(A, rhs, x0, 0, 1e-12)
    assert its == 0 and torch.equal(x, x0)
