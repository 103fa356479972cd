"""A context destroyed while a stream still has its work queued: the work ends
before the context's memory can serve another context."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import F64  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("n", [24, 61])
def test_destroy_waits_for_every_stream(n):
    dom = {"nx": n, "ny": n, "nz": n, "h": 0.4, "radius": 0.2 * (n - 1)}
    g = torch.Generator(device="cuda").manual_seed(n)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device=DEV, generator=g)  # noqa: E731
    pot, X = r(n ** 3), r(9, n ** 3)

    def apply(ctx, y):
        ctx.call("psc_apply_h", F64, gpu._p(X), ctx.n, gpu._p(y), ctx.n, 9, gpu._stream())

    ctx = gpu.GridContext(dom, 8)
    gpu.Hamiltonian(ctx, pot)
    ref, Y = torch.empty_like(X), torch.empty_like(X)
    apply(ctx, ref)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        torch.cuda._sleep(20_000_000)
        apply(ctx, Y)
    assert not s.query()
    del ctx
    assert s.query()
    other = gpu.GridContext(dom, 8)          # its memory is the first one's
    gpu.Hamiltonian(other, -pot)
    torch.cuda.synchronize()
    assert torch.equal(Y, ref)
