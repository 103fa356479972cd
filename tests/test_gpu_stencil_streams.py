"""H X on two streams of one context right after another, the first of which
builds the work table behind other work of its stream: the second does not
wait for that stream, and finds the table.  On grids of every path that has
one; X and Y of the streams are their own, and there are no projectors, so the
calls share nothing else."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import F32, F64  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("dims", [(61, 55, 67), (52, 52, 52)], ids=["odd", "even"])
@pytest.mark.parametrize("dt", ["f64", "f32"])
def test_second_stream_finds_the_table(dims, dt):
    nx, ny, nz = dims
    tdt, code = (torch.float64, F64) if dt == "f64" else (torch.float32, F32)
    g = torch.Generator(device="cuda").manual_seed(nx)
    X = [torch.randn(31, nx * ny * nz, dtype=tdt, device=DEV, generator=g) for _ in range(2)]
    pot = torch.randn(nx * ny * nz, dtype=torch.float64, device=DEV, generator=g)
    results = []
    for overlap in (False, True):
        ctx = gpu.GridContext({"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 0.17 * (nx - 1)}, 8)
        gpu.Hamiltonian(ctx, pot)
        streams = [torch.cuda.Stream(), torch.cuda.Stream()]
        Y = [torch.full_like(x, float("nan")) for x in X]
        torch.cuda.synchronize()
        for x, y, s in zip(X, Y, streams):
            with torch.cuda.stream(s):
                if overlap and s is streams[0]:
                    torch.cuda._sleep(50_000_000)
                ctx.call("psc_apply_h", code, gpu._p(x), ctx.n, gpu._p(y), ctx.n, 31, gpu._stream())
            if not overlap:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        ctx.check_status()
        results.append(Y)
    for a, b in zip(*results):
        assert bool(torch.isfinite(a).all()) and torch.equal(a, b)
