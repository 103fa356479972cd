"""The stencil step on grids whose planes do not start on 16-byte boundaries:
the bulk-copy kernel with shifted windows against the register-queue kernel
(which tests/test_gpu_kernels.py holds against the oracle), over orders,
slabs that end inside a row, calls below its sizes, leading
dimensions of every remainder, blocks that start off a boundary (left to the
register-queue kernel), Prev in place, absent or separate, and the last
column's end (nothing past it is read, nothing outside the columns written).

Both kernels add 2 + 6 R products per point in FP64 or FP32; their difference
is at most the rounding of that many terms, 26 x 2^-53 or 2^-24 of the sum of
their magnitudes, which the bounds 1e-14 and 4e-6 of the largest result
cover (weights of alternating signs: the sum is at most 1.6 times c0)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from parsec_python_b200 import gpu  # noqa: E402
from parsec_python_b200._lib import F32, F64  # noqa: E402

DEV = torch.device("cuda", 0)

CASES = [
    # grid, order, columns, ld - n, elements X starts past a 16-byte boundary, Prev
    ((1, 1, 9), 8, 3, 1, 0, "in place"),
    ((3, 3, 3), 8, 5, 0, 0, "in place"),
    ((45, 23, 30), 8, 3, 0, 1, "separate"),
    ((71, 57, 61), 2, 9, 1, 0, "none"),
    ((63, 65, 31), 4, 16, 2, 0, "separate"),
    ((91, 45, 29), 6, 17, 3, 0, "in place"),
    ((61, 55, 67), 8, 31, 0, 0, "in place"),
    ((125, 41, 37), 8, 11, 1, 0, "separate"),
    ((125, 41, 37), 8, 11, 0, 1, "none"),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(map(str, c[0])) + f"-o{c[1]}-ld{c[3]}-off{c[4]}")
@pytest.mark.parametrize("dt", ["f64", "f32"])
def test_odd_planes_match_register_kernel(case, dt):
    (nx, ny, nz), order, k, extra, off, prev = case
    ctx = gpu.GridContext({"nx": nx, "ny": ny, "nz": nz, "h": 0.34, "radius": 0.17 * (nx - 1)}, order)
    n, ld = ctx.n, ctx.n + extra
    tdt, code, tol = (torch.float64, F64, 1e-14) if dt == "f64" else (torch.float32, F32, 4e-6)
    g = torch.Generator(device="cuda").manual_seed(nx + k)
    gpu.Hamiltonian(ctx, torch.randn(n, dtype=torch.float64, device=DEV, generator=g))

    def columns(fill):
        """k columns of the block, NaN in the gaps; the last column ends the buffer."""
        buf = torch.full((off + (k - 1) * ld + n,), float("nan"), dtype=tdt, device=DEV)
        for j in range(k):
            buf[off + j * ld:off + j * ld + n] = fill[j]
        return buf

    X = columns(torch.randn(k, n, dtype=tdt, device=DEV, generator=g))
    P = columns(torch.randn(k, n, dtype=tdt, device=DEV, generator=g))
    outs = []
    for impl in (1, 0):
        ctx.call("psc_set_stencil_impl", impl)
        Y = P.clone() if prev == "in place" else torch.full_like(P, float("nan"))
        p = {"in place": Y, "separate": P, "none": None}[prev]
        ctx.call("psc_apply_h_axpby", code, gpu._p(X[off:]), ld, gpu._p(p[off:] if p is not None else None), ld,
                 gpu._p(Y[off:]), ld, k, 0.7, -0.2, -0.9 if p is not None else 0.0, gpu._stream())
        cols = np.stack([Y[off + j * ld:off + j * ld + n].double().cpu().numpy() for j in range(k)])
        for j in range(k - 1):
            assert bool(torch.isnan(Y[off + j * ld + n:off + (j + 1) * ld]).all())
        outs.append(cols)
    assert np.isfinite(outs[1]).all()
    assert np.abs(outs[1] - outs[0]).max() <= tol * np.abs(outs[0]).max()
    ctx.check_status()
