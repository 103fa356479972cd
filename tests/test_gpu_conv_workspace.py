"""The convolution backward works in its caller's memory alone: its first call
on a context may be part of a stream capture, calls on two streams of one
context do not meet, gm receives the gradient through the activation, and the
input gradient may be written over gm or gout.  Every result has the bits of
an ordinary call."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
F32 = dict(dtype=torch.float32, device=DEV)


def _ctx():
    return gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)


class Layer:
    def __init__(self, n, cin, cout, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        r = lambda *s: torch.randn(*s, generator=g, **F32)  # noqa: E731
        self.n, self.cin, self.cout, self.nv = n, cin, cout, n ** 3
        self.geom = (ctypes.c_int * 15)(n, n, n, n, n, n, 0, cin, 0, n, n, n, 1, 3, cout)
        self.a, self.w, self.y = r(self.nv, cin).bfloat16(), r(27, cin, cout).bfloat16(), r(self.nv, cout).bfloat16()
        self.gout = r(self.nv, cout)
        self.dvin, self.work = torch.empty(self.nv, cin, **F32), torch.empty(1 << 20, **F32)
        self.dW, self.dB = torch.empty(27, cin, cout, **F32), torch.empty(cout, **F32)

    def run(self, ctx, gout, gm, dA, act=2):
        ctx.call("psc_conv3d_bwd", self.geom, gpu._p(self.a), None, gpu._p(self.w), gpu._p(gout), gpu._p(self.y), act,
                 gpu._p(gm), gpu._p(self.dvin), gpu._p(dA), 0, None, 0, gpu._p(self.dW), gpu._p(self.dB),
                 gpu._p(self.work), self.work.numel(), gpu._stream())
        return dA, self.dW, self.dB

    def empty(self):
        return torch.empty(self.nv, self.cout, **F32), torch.empty(self.nv, self.cin, **F32)

    def want(self, act=2):
        return [t.clone() for t in self.run(_ctx(), self.gout, *self.empty(), act)]


def _equal(got, want):
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_first_call_in_a_capture():
    layer = Layer(12, 16, 8, 1)
    want, ctx, (gm, dA) = layer.want(), _ctx(), layer.empty()
    for t in (layer.dW, layer.dB, dA):
        t.zero_()
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        graph.capture_begin()
        layer.run(ctx, layer.gout, gm, dA)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    _equal((dA, layer.dW, layer.dB), want)


def test_two_streams():
    layers = [Layer(24, 16, 24, 2), Layer(22, 24, 16, 3)]
    wants, bufs, ctx = [x.want() for x in layers], [x.empty() for x in layers], _ctx()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(20):
        for layer, (gm, dA), s in zip(layers, bufs, streams):
            with torch.cuda.stream(s):
                layer.run(ctx, layer.gout, gm, dA)
        torch.cuda.synchronize()
        for layer, (_, dA), want in zip(layers, bufs, wants):
            _equal((dA, layer.dW, layer.dB), want)


@pytest.mark.parametrize("act", [0, 1, 2])
def test_gm_and_gradients_in_place(act):
    layer = Layer(13, 16, 16, 4)
    want, ctx = layer.want(act), _ctx()
    below = {0: 1.0, 1: 0.0, 2: 0.0625}[act]
    masked = torch.where(layer.y.float() > 0, layer.gout, below * layer.gout)
    gm, dA = layer.empty()
    _equal(layer.run(ctx, layer.gout, gm, dA, act), want)
    assert torch.equal(gm, masked)
    g = layer.gout.clone()
    _equal(layer.run(ctx, g, g, dA, act), want)         # gm over gout
    assert torch.equal(g, masked)
    g, (gm, _) = layer.gout.clone(), layer.empty()
    _equal(layer.run(ctx, g, gm, g, act), want)         # dA over gout
    g = layer.gout.clone()
    _equal(layer.run(ctx, g, gm, gm, act), want)        # dA over gm
    g = layer.gout.clone()
    _equal(layer.run(ctx, g, g, g, act), want)          # all three
