"""The widest rows whose windows fit the shared memory of a CTA, and the first
that do not: the register-queue stencil (two windows of 512 points and 2 x 4
rows of the order-8 stencil) and the CG that runs one launch per step (256
points).  Bounds as in tests/test_gpu_stencil_shifted.py; three CG steps within
3 x 27 x 2e4 x 2^-53 of the oracle's iterate (condition number below 2e4 for
order 8 in a box two points high)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import PscError  # noqa: E402

DEV = torch.device("cuda", 0)


def _ctx(nx, ny, nz):
    dom = {"nx": nx, "ny": ny, "nz": nz, "h": 0.5, "radius": 0.25 * (nx - 1)}
    return dom, gpu.GridContext(dom, 8)


@pytest.mark.parametrize("nx, fits", [(1751, True), (1752, False)])
def test_widest_stencil_rows(nx, fits):
    dom, ctx = _ctx(nx, 2, 3)
    ctx.call("psc_set_stencil_impl", 1)
    rng = np.random.default_rng(nx)
    pot, X = rng.standard_normal(ctx.n), rng.standard_normal((2, ctx.n))
    H = gpu.Hamiltonian(ctx, torch.from_numpy(pot).to(DEV))
    Xd = torch.from_numpy(X).to(DEV)
    if not fits:
        with pytest.raises(PscError):
            H @ Xd
        return
    ref = (0.5 * O.laplacian(dom, 8) @ X.T).T + pot * X
    assert np.abs((H @ Xd).cpu().numpy() - ref).max() <= 1.3e-14 * np.abs(ref).max()


@pytest.mark.parametrize("nx, fits", [(1783, True), (1784, False)])
def test_widest_cg_rows(nx, fits):
    dom, ctx = _ctx(nx, 1, 2)
    ctx.call("psc_set_use_graphs", 0)
    # (the residual that starts a solve takes the register-queue stencil)
    ctx.call("psc_set_stencil_impl", 1)
    rng = np.random.default_rng(nx)
    rhs, x0 = rng.standard_normal(ctx.n), rng.standard_normal(ctx.n)
    args = gpu.Laplacian(ctx), torch.from_numpy(rhs).to(DEV), torch.from_numpy(x0).to(DEV), 3, 1e-12
    if not fits:
        with pytest.raises(PscError):
            gpu.pcg(*args)
        return
    x, its = gpu.pcg(*args)
    ref, its_ref = O.pcg(O.laplacian(dom, 8), rhs, x0, 3, 1e-12)
    assert its == its_ref
    assert np.linalg.norm(x.cpu().numpy() - ref) <= 1.8e-10 * np.linalg.norm(ref)
