"""The network's backward needs scratch for a layer's input gradient only where
the gradient is split or pooled: with dvin = dA elsewhere the gradients keep
their bits, and dvin is left alone."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)


@pytest.mark.parametrize("stride, acc", [(1, 0), (1, 1), (2, 0), (2, 1)])
def test_dvin_may_be_dA(stride, acc):
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    g = torch.Generator(device="cuda").manual_seed(stride)
    f32 = dict(dtype=torch.float32, device=DEV)
    n, cin, cout = 11, 16, 24
    m = (n + stride - 1) // stride
    r = lambda *s: torch.randn(*s, generator=g, **f32)  # noqa: E731
    a, w, gout = r(n ** 3, cin).bfloat16(), r(27, cin, cout).bfloat16(), r(m ** 3, cout)
    start, work = r(n ** 3, cin), torch.empty(1 << 20, **f32)
    geom = (ctypes.c_int * 15)(n, n, n, n, n, n, 0, cin, 0, m, m, m, stride, 3, cout)
    out = []
    for own in (True, False):
        dA, gm = start.clone(), torch.empty(m ** 3, cout, **f32)
        dW, dB = torch.empty(27, cin, cout, **f32), torch.empty(cout, **f32)
        dvin = torch.full((n ** 3, cin), 7.0, **f32) if own else dA
        ctx.call("psc_conv3d_bwd", geom, gpu._p(a), None, gpu._p(w), gpu._p(gout), None, 0, gpu._p(gm), gpu._p(dvin),
                 gpu._p(dA), acc, None, 0, gpu._p(dW), gpu._p(dB), gpu._p(work), work.numel(), gpu._stream())
        if own:
            assert bool((dvin == 7.0).all())
        out.append((dA, dW, dB))
    for x, y in zip(*out):
        assert torch.equal(x, y)
