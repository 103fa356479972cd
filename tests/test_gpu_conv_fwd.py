"""Convolution forward at the edges of its tiles: grids around the 32 x 4 x 4
voxel brick of the eight-channel kernel and the 128 voxels of a tensor-core
tile, one to many reduction stages around the ring's depth, channel counts
around the octet and the 32-channel chunk, both strides, up-sampling with a
skip tensor, and results at addresses off 16-byte alignment.

Bound per entry: the products of two BF16 numbers are exact in FP32.  The
CUDA-core sum rounds once per term (2^-24 of at most the whole absolute sum);
the tensor cores pass 16 terms at a time through three accumulations that may
drop up to a unit in the last place each (3 x 2^-23).  Both activations keep
distances (slopes 1, 0 and 1/16); the BF16 result is the FP32 one rounded."""
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
    # grid_in, up, Ca, Cs, Cout, stride, ksize, act, implementation, elements the results are off alignment
    ((1, 1, 1), 0, 8, 0, 8, 1, 3, 0, 1, 0),
    ((32, 4, 4), 0, 8, 0, 8, 1, 3, 2, 1, 0),
    ((33, 5, 5), 0, 40, 0, 8, 1, 3, 2, 1, 1),
    ((31, 3, 9), 0, 24, 0, 24, 1, 3, 1, 1, 0),
    ((34, 9, 4), 0, 72, 0, 8, 1, 1, 0, 1, 3),
    ((13, 9, 10), 1, 32, 8, 8, 1, 3, 2, 1, 0),
    ((16, 7, 5), 0, 16, 0, 40, 1, 3, 2, 0, 0),
    ((17, 7, 5), 0, 16, 0, 8, 2, 3, 2, 1, 0),
    ((4, 4, 8), 0, 64, 0, 32, 1, 1, 0, 1, 0),
    ((5, 5, 5), 0, 128, 0, 32, 1, 1, 2, 1, 0),
    ((43, 3, 1), 0, 192, 0, 40, 1, 1, 2, 1, 0),
    ((5, 5, 6), 0, 264, 0, 32, 1, 1, 1, 1, 0),
    ((7, 6, 5), 0, 8, 0, 32, 1, 3, 2, 1, 0),
    ((7, 6, 5), 1, 64, 40, 256, 1, 3, 2, 1, 0),
    ((17, 16, 9), 0, 24, 0, 72, 2, 3, 0, 1, 0),
    ((9, 5, 5), 0, 40, 0, 8, 1, 3, 2, 2, 0),
]


def _ncdhw(t, grid, c):
    nx, ny, nz = grid
    return t.reshape(nz, ny, nx, c).permute(3, 0, 1, 2).unsqueeze(0)


def _flat(t):
    return t[0].permute(1, 2, 3, 0).reshape(-1, t.shape[1])


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-{c[2]}+{c[3]}-{c[4]}-i{c[8]}")
def test_conv_forward_within_the_rounding_bound(case):
    gi, up, ca, cs, cout, stride, k, act, impl, off = case
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    rng = np.random.default_rng(ca * 1000 + cout)
    ga = tuple((v + 1) // 2 for v in gi) if up else gi
    go = gi if stride == 1 else tuple((v + 1) // 2 for v in gi)
    nva, nvi, nvo = (int(np.prod(v)) for v in (ga, gi, go))
    cin, bf = ca + cs, torch.bfloat16
    a = torch.from_numpy(rng.standard_normal((nva, ca)).astype(np.float32)).to(bf)
    s = torch.from_numpy(rng.standard_normal((nvi, cs)).astype(np.float32)).to(bf) if cs else None
    w = torch.from_numpy(rng.standard_normal((k ** 3, cin, cout)).astype(np.float32)).to(bf)
    bias = torch.from_numpy(rng.standard_normal(cout).astype(np.float32))
    A = _ncdhw(a.double(), ga, ca)
    S = _ncdhw(s.double(), gi, cs) if cs else None
    W = w.double().reshape(k, k, k, cin, cout).permute(4, 3, 0, 1, 2)

    def conv(A, S, W, b):
        x = A
        if up:
            for ax, n in ((2, gi[2]), (3, gi[1]), (4, gi[0])):
                x = x.repeat_interleave(2, ax).narrow(ax, 0, n)
        if cs:
            x = torch.cat([x, S], 1)
        return _flat(F.conv3d(x, W, b.double(), stride=stride, padding=k // 2))

    ref = conv(A, S, W, bias)
    mag = conv(A.abs(), S.abs() if cs else None, W.abs(), bias.abs())
    below = {0: 1.0, 1: 0.0, 2: 0.0625}[act]
    ref = torch.where(ref > 0, ref, below * ref)
    ad, sd, wd, bd = a.to(DEV), s.to(DEV) if cs else None, w.to(DEV), bias.to(DEV)
    out = torch.full((nvo * cout + 16,), 7.0, dtype=bf, device=DEV)
    out32 = torch.full((nvo * cout + 16,), 7.0, dtype=torch.float32, device=DEV)
    o, o32 = out[off:off + nvo * cout], out32[off:off + nvo * cout]
    geom = (ctypes.c_int * 15)(*gi, *ga, up, ca, cs, *go, stride, k, cout)
    ctx.call("psc_set_conv_impl", impl)
    ctx.call("psc_conv3d_fwd", geom, gpu._p(ad), gpu._p(sd), gpu._p(wd), gpu._p(bd), act, gpu._p(o), gpu._p(o32),
             gpu._stream())
    got = o32.double().cpu().reshape(nvo, cout)
    K = k ** 3 * cin
    tol = (3 * 2.0 ** -23 * (K / 16 + 1) + (K + 2) * 2.0 ** -24) * mag
    assert bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() / tol).max())
    assert torch.equal(o.cpu(), o32.cpu().to(bf))
    for buf in (out, out32):               # nothing is written outside the result
        assert bool((buf[:off] == 7.0).all()) and bool((buf[off + nvo * cout:] == 7.0).all())
