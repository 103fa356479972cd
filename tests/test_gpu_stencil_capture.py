"""H X on grids with odd sides as part of a stream capture: the first call of a
context may be the captured one, and a captured graph stays good.

Both kernels add the same terms in the same order with contractions of their
own: 1e-14 (FP64) and 4e-6 (FP32) of the largest result cover the rounding of
26 terms, as in tests/test_gpu_stencil_odd.py."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import F32, F64  # noqa: E402

DEV = torch.device("cuda", 0)
DIMS, K = (61, 55, 67), 31


def _setup(dt):
    nx, ny, nz = DIMS
    ctx = gpu.GridContext({"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 0.17 * (nx - 1)}, 8)
    g = torch.Generator(device="cuda").manual_seed(9)
    gpu.Hamiltonian(ctx, torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=g))
    X = torch.randn(K, ctx.n, dtype=torch.float64, device=DEV, generator=g).to(
        torch.float64 if dt == "f64" else torch.float32)
    return ctx, X, torch.empty_like(X), F64 if dt == "f64" else F32


def _apply(ctx, code, X, Y):
    ctx.call("psc_apply_h", code, gpu._p(X), ctx.n, gpu._p(Y), ctx.n, K, gpu._stream())


def _capture(ctx, code, X, Y):
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.capture_begin()
        _apply(ctx, code, X, Y)
        graph.capture_end()
    return graph


def _close(Y, ref):
    tol = 1e-14 if Y.dtype == torch.float64 else 4e-6
    assert float((Y - ref).abs().max()) <= tol * float(ref.abs().max())


@pytest.mark.parametrize("dt", ["f64", "f32"])
def test_first_call_in_a_capture(dt):
    ctx, X, Y, code = _setup(dt)
    graph = _capture(ctx, code, X, Y)
    Y.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    ref = torch.empty_like(Y)
    _apply(ctx, code, X, ref)
    _close(Y, ref)
    ctx.check_status()


def test_captured_graph_outlives_a_sphere_mask():
    """Setting and clearing the sphere mask leaves the tables of unmasked
    launches where the captured graph holds them."""
    ctx, X, Y, code = _setup("f64")
    ref = torch.empty_like(Y)
    _apply(ctx, code, X, ref)               # builds the table
    graph = _capture(ctx, code, X, Y)
    ctx.set_sphere_mask(8.0)
    ctx.set_sphere_mask(0.0)
    other = [_setup("f32") for _ in range(3)]   # takes freed memory, if any was
    for c, x, y, cd in other:
        _apply(c, cd, x, y)
    Y.fill_(float("nan"))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(Y, ref)
    ctx.check_status()
