"""Convolutions with infinite and NaN entries: a tap outside the grid is not
there, so it must not turn 0 x infinity into a NaN at the edge, and each entry
reaches the outputs that use it and no others.  The reference adds the taps
that lie in the grid one by one in 64 bits; a result is finite, an infinity of
that sign, or NaN where the reference is."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402

DEV = torch.device("cuda", 0)
BF = torch.bfloat16


def _data(gi, cin, cout, stride, ksize, seed):
    """Input [z, y, x, cin], weights [dz, dy, dx, cin, cout] (BF16 values, none
    zero) and the pairs of slices (output, input) of each tap."""
    rng = np.random.default_rng(seed)
    r = lambda *s: torch.from_numpy((rng.choice([-1.0, 1.0], s) * rng.uniform(0.5, 2, s)).astype(np.float32)).to(BF)  # noqa: E731
    nx, ny, nz = gi
    go = tuple((v + stride - 1) // stride for v in gi)
    a, w = r(nz, ny, nx, cin), r(ksize, ksize, ksize, cin, cout)

    def axis(n, no, d):
        o = [i for i in range(no) if 0 <= i * stride + d - ksize // 2 < n]
        return slice(o[0], o[-1] + 1) if o else slice(0, 0), \
            slice(o[0] * stride + d - ksize // 2, o[-1] * stride + d - ksize // 2 + 1, stride) if o else slice(0, 0)

    taps = []
    for dz in range(ksize):
        for dy in range(ksize):
            for dx in range(ksize):
                (zo, zi), (yo, yi), (xo, xi) = axis(nz, go[2], dz), axis(ny, go[1], dy), axis(nx, go[0], dx)
                taps.append(((dz, dy, dx), (zo, yo, xo), (zi, yi, xi)))
    return a, w, go, taps


def _same(got, ref, bound):
    got, ref = got.double().cpu().numpy().reshape(ref.shape), ref.numpy() if torch.is_tensor(ref) else ref
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    inf = np.isinf(ref)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], ref[inf])
    fin = np.isfinite(ref)
    assert not fin.any() or np.abs(got[fin] - ref[fin]).max() <= bound


@pytest.mark.parametrize("gi, cin, cout, ksize", [((5, 4, 3), 8, 8, 3), ((35, 6, 5), 40, 24, 3), ((33, 5, 4), 16, 8, 1)],
                         ids=["small", "blocks", "1x1x1"])
def test_forward_skips_taps_outside(gi, cin, cout, ksize):
    a, w, go, taps = _data(gi, cin, cout, 1, ksize, cin)
    w[0, 0, 0, 1, 2] = float("inf")
    w[-1, 0, -1, cin - 1, 5] = float("-inf")
    w[0, -1, 0, 3, cout - 1] = float("nan")
    a[0, 0, -1, 4] = float("inf")
    bias = torch.arange(cout, dtype=torch.float32) / 8
    ref = np.zeros((go[2], go[1], go[0], cout)) + bias.double().numpy()
    with np.errstate(invalid="ignore"):
        for t, o, i in taps:
            for c in range(cin):
                ref[o] += a.double().numpy()[i][..., c, None] * w.double().numpy()[t][c]
    assert np.isfinite(ref).any() and np.isinf(ref).any() and np.isnan(ref).any()
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    geom = (ctypes.c_int * 15)(*gi, *gi, 0, cin, 0, *go, 1, ksize, cout)
    ad, wd, bd = a.to(DEV), w.to(DEV), bias.to(DEV)
    out = torch.empty(ref.size, dtype=BF, device=DEV)
    out32 = torch.empty(ref.size, dtype=torch.float32, device=DEV)
    ctx.call("psc_set_conv_impl", 0)
    ctx.call("psc_conv3d_fwd", geom, gpu._p(ad), None, gpu._p(wd), gpu._p(bd), 0, gpu._p(out), gpu._p(out32),
             gpu._stream())
    # up to 27 cin + 1 terms below 4, each rounded at the size of the whole sum
    terms = ksize ** 3 * cin + 1
    _same(out32, ref, terms * terms * 4 * 2.0 ** -24)


@pytest.mark.parametrize("gi, cin, cout, stride", [((5, 4, 3), 8, 8, 1), ((9, 6, 5), 40, 24, 1), ((13, 9, 6), 16, 40, 2),
                                                   ((8, 5, 4), 24, 16, 2)],
                         ids=["small", "blocks", "stride-2", "stride-2-even"])
@pytest.mark.parametrize("where", ["weights", "input", "gradient", "all"])
def test_backward_keeps_to_the_terms_there_are(gi, cin, cout, stride, where):
    a, w, go, taps = _data(gi, cin, cout, stride, 3, cin + stride)
    rng = np.random.default_rng(7)
    G = torch.from_numpy((rng.choice([-1.0, 1.0], (go[2], go[1], go[0], cout)) *
                          rng.uniform(0.5, 2, (go[2], go[1], go[0], cout))).astype(np.float32))
    G[0, 0, 0, 3] = 1.0                      # one bit: its two lower planes are zero
    inf, nan = float("inf"), float("nan")
    if where in ("weights", "all"):
        w[0, 0, 0, 1, 2], w[-1, 1, -1, cin - 1, 5], w[1, -1, 0, 3, cout - 1], w[1, 1, 1, 2, 3] = inf, -inf, nan, inf
    if where in ("input", "all"):
        a[0, 0, -1, 4], a[-1, -1, 0, 1], a[1, 1, 1, 6] = inf, -inf, nan
    if where in ("gradient", "all"):
        G[-1, 0, 0, 1], G[0, -1, -1, 4], G[0, 1, 1, cout - 2] = inf, -inf, nan
    an, wn, gn = (t.double().numpy() for t in (a, w, G))
    dA, dW, dB = np.zeros(an.shape), np.zeros(wn.shape), np.zeros(cout)
    with np.errstate(invalid="ignore"):
        dB += gn.sum((0, 1, 2))
        for t, o, i in taps:
            for c in range(cin):
                dA[i][..., c] += (gn[o] * wn[t][c]).sum(-1)
                dW[t][c] += (an[i][..., c, None] * gn[o]).sum((0, 1, 2))
    for ref in (dA, dW):
        assert np.isfinite(ref).any()
    nvi, nvo = int(np.prod(gi)), int(np.prod(go))
    f32 = dict(dtype=torch.float32, device=DEV)
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    geom = (ctypes.c_int * 15)(*gi, *gi, 0, cin, 0, *go, stride, 3, cout)
    ad, wd, gd = a.to(DEV), w.to(DEV), G.to(DEV)
    gm, dv, da, work = (torch.empty(k, **f32) for k in (nvo * cout, nvi * cin, nvi * cin, 1 << 20))
    dw, db = torch.empty(27 * cin * cout, **f32), torch.empty(cout, **f32)
    ctx.call("psc_conv3d_bwd", geom, gpu._p(ad), None, gpu._p(wd), gpu._p(gd), None, 0, gpu._p(gm), gpu._p(dv),
             gpu._p(da), 0, None, 0, gpu._p(dw), gpu._p(db), gpu._p(work), work.numel(), gpu._stream())
    # terms below 4, each rounded at the size of the whole sum
    for got, ref, terms in ((dw, dW, nvo), (da, dA, 27 * cout), (db, dB, nvo)):
        _same(got, ref, terms * terms * 4 * 2.0 ** -24)
