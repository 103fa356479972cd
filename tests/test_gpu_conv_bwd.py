"""Convolution backward at the edges of its tiles: grids around the 8 x 4 x 4
and 8 x 8 x 4 bricks, channel counts around the octet, column and unit
blocks, both strides, unaligned caller pointers, and the exact split of the
gradient (an entry far below its neighbours keeps its bits).

Bound per entry: the products are exact; each 16-entry step passes through
three tensor-core accumulations that may drop up to a unit in the last place
each (3 x 2^-23 of the step's absolute sum), and every later FP32 add rounds
to nearest (2^-24 of at most the whole absolute sum)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

import torch.nn.functional as F  # noqa: E402

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)

CASES = [
    # grid_in, up, Ca, Cs, Cout, stride, ksize, act, elements the W / gradient pointers are off 16-byte alignment
    ((1, 1, 1), 0, 8, 0, 8, 1, 3, 0, 0),
    ((8, 4, 4), 0, 8, 0, 16, 1, 3, 2, 0),
    ((9, 5, 5), 0, 40, 0, 8, 1, 3, 2, 1),
    ((17, 9, 3), 0, 24, 0, 24, 1, 3, 1, 0),
    ((16, 8, 8), 0, 8, 0, 40, 2, 3, 2, 0),
    ((17, 16, 9), 0, 16, 0, 72, 2, 3, 0, 1),
    ((13, 9, 10), 1, 32, 8, 8, 1, 3, 2, 0),
    ((7, 6, 5), 1, 64, 40, 32, 1, 3, 2, 0),
    ((9, 9, 9), 0, 72, 0, 8, 1, 1, 0, 0),
    ((5, 4, 3), 0, 264, 0, 256, 1, 1, 2, 0),
]


def _ncdhw(t, grid, c):
    nx, ny, nz = grid
    return t.reshape(nz, ny, nx, c).permute(3, 0, 1, 2).unsqueeze(0)


def _flat(t):
    return t[0].permute(1, 2, 3, 0).reshape(-1, t.shape[1])


def _off(t, k):
    """t at an address k elements past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 16, dtype=t.dtype, device=DEV)
    v = buf[k:k + t.numel()]
    v.copy_(t.reshape(-1))
    return v


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-{c[2]}+{c[3]}-{c[4]}")
def test_conv_backward_within_the_rounding_bound(case):
    gi, up, ca, cs, cout, stride, k, act, off = case
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    rng = np.random.default_rng(ca * 1000 + cout)
    ga = tuple((v + 1) // 2 for v in gi) if up else gi
    go = gi if stride == 1 else tuple((v + 1) // 2 for v in gi)
    nva, nvi, nvo = (int(np.prod(v)) for v in (ga, gi, go))
    cin, bf = ca + cs, torch.bfloat16
    a = torch.from_numpy(rng.standard_normal((nva, ca)).astype(np.float32)).to(bf)
    s = torch.from_numpy(rng.standard_normal((nvi, cs)).astype(np.float32)).to(bf) if cs else None
    w = torch.from_numpy(rng.standard_normal((k ** 3, cin, cout)).astype(np.float32)).to(bf)
    y = torch.from_numpy(rng.standard_normal((nvo, cout)).astype(np.float32)).to(bf)
    R = rng.standard_normal((nvo, cout)).astype(np.float32)
    R[rng.random((nvo, cout)) < 0.3] *= np.float32(1.7e-6)
    R = torch.from_numpy(R)
    below = {0: 1.0, 1: 0.0, 2: 0.0625}[act]
    mask = torch.where(y.float() > 0, 1.0, below) if act else torch.ones(nvo, cout)
    gm = (R * mask).double()                   # exact in FP32: the slope is a power of two or zero
    A = _ncdhw(a.double(), ga, ca)
    S = _ncdhw(s.double(), gi, cs) if cs else None
    W = w.double().reshape(k, k, k, cin, cout).permute(4, 3, 0, 1, 2)

    def grads(A, S, W, G):
        A, W = A.clone().requires_grad_(True), W.clone().requires_grad_(True)
        x = A
        if up:
            for ax, n in ((2, gi[2]), (3, gi[1]), (4, gi[0])):
                x = x.repeat_interleave(2, ax).narrow(ax, 0, n)
        if cs:
            S = S.clone().requires_grad_(True)
            x = torch.cat([x, S], 1)
        F.conv3d(x, W, stride=stride, padding=k // 2).backward(_ncdhw(G, go, cout))
        return W.grad, A.grad, S.grad if cs else None

    ref = grads(A, S, W, gm)
    mag = grads(A.abs(), S.abs() if cs else None, W.abs(), gm.abs())
    ad, sd = a.to(DEV), s.to(DEV) if cs else None
    wd, Rd, yd = _off(w, off), _off(R, off), y.to(DEV)
    f32 = dict(dtype=torch.float32, device=DEV)
    scratch, dvin, work = torch.empty(nvo, cout, **f32), torch.empty(nvi, cin, **f32), torch.empty(4 << 20, **f32)
    dA, dS = _off(torch.full((nva, ca), 0.5), off), torch.empty(nvi, cs, **f32) if cs else None
    dW, dB = torch.empty(k ** 3 * cin * cout, **f32), torch.empty(cout, **f32)
    geom = (ctypes.c_int * 15)(*gi, *ga, up, ca, cs, *go, stride, k, cout)
    ctx.call("psc_conv3d_bwd", geom, gpu._p(ad), gpu._p(sd), gpu._p(wd), gpu._p(Rd), gpu._p(yd if act else None), act,
             gpu._p(scratch), gpu._p(dvin), gpu._p(dA), 1, gpu._p(dS), 0, gpu._p(dW), gpu._p(dB), gpu._p(work),
             work.numel(), gpu._stream())

    def within(got, exact, mag, adds, extra=0.0):
        got = got.double().cpu()
        tol = (3 * 2.0 ** -23 + adds * 2.0 ** -24) * mag + extra
        assert bool(((got - exact).abs() <= tol).all()), float(((got - exact).abs() / tol.clamp_min(1e-300)).max())

    within(dW.reshape(k, k, k, cin, cout).permute(4, 3, 0, 1, 2).cpu(), ref[0], mag[0], nvo / 16 + 200)
    within(dB, gm.sum(0), gm.abs().sum(0), nvo)
    # accumulated into 0.5: one more rounding at that magnitude
    within(dA.reshape(nva, ca) - 0.5, _flat(ref[1]), _flat(mag[1]), k ** 3 * cout / 16 + 10,
           2.0 ** -23 * (0.5 + _flat(ref[1]).abs()))
    if cs:
        within(dS, _flat(ref[2]), _flat(mag[2]), k ** 3 * cout / 16 + 2)
