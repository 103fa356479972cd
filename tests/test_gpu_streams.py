"""Reductions that end in their launch's last CTA, queued on two streams of one
context at once: dot products on one, mixer steps on the other (neither
touches the other's partial sums), and more launches than there are arrival
counters.  Every result has the bits of the same calls on one stream."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
DIMS, STEPS, DOTS = (61, 70, 80), 12, 120


def _run(overlap):
    nx, ny, nz = DIMS
    ctx = gpu.GridContext({"nx": nx, "ny": ny, "nz": nz, "h": 0.4, "radius": 1.0}, 2)
    g = torch.Generator(device="cuda").manual_seed(5)
    a, b = (torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=g) for _ in range(2))
    x = torch.randn(STEPS, ctx.n, dtype=torch.float64, device=DEV, generator=g)
    f = torch.randn(STEPS, ctx.n, dtype=torch.float64, device=DEV, generator=g)
    dots = torch.full((STEPS * DOTS,), float("nan"), dtype=torch.float64, device=DEV)
    mixer, mixed = gpu.Mixer(ctx, 40), []
    sa, sb = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for i in range(STEPS):
        with torch.cuda.stream(sa):
            for j in range(DOTS):
                # lengths from one CTA to all of them
                n = 1 + (ctx.n - 1) * (j % 7) // 6
                ctx.call("psc_dot", gpu._p(a), gpu._p(b), n, gpu._p(dots[i * DOTS + j:]), gpu._stream())
        if not overlap:
            torch.cuda.synchronize()
        with torch.cuda.stream(sb):
            mixed.append(mixer(x[i], f[i])[0])
        if not overlap:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    return dots, torch.stack(mixed)


def test_two_streams_do_not_share_arrival_counters():
    dots, mixed = _run(False)       # 1440 dot products and 36 launches of the mixer: the ring of counters wraps
    assert bool(torch.isfinite(dots).all()) and bool(torch.isfinite(mixed).all())
    assert torch.equal(dots[:DOTS], dots[-DOTS:])
    for _ in range(3):
        d, m = _run(True)
        assert torch.equal(d, dots) and torch.equal(m, mixed)
