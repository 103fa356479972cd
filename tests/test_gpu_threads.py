"""Two host threads, each with a context and a stream of its own, whose calls
need different amounts of shared memory of the same kernels: no launch is
refused, and every result has the bits of the same call alone.  The limit that
a call sets for a kernel holds for the whole process, so no call may lower it
(the threads alone rarely meet in the few instructions where that would show)."""
import ctypes
import re
import subprocess
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from parsec_python_b200 import _lib, gpu  # noqa: E402
from parsec_python_b200.inputs import ElementTable, pseudo_tables  # noqa: E402

DEV = torch.device("cuda", 0)


def _conv(cin, cout):
    """Forward and backward of a 3x3x3 layer on an 8^3 grid."""
    ctx = gpu.GridContext({"nx": 8, "ny": 8, "nz": 8, "h": 0.5, "radius": 1.75}, 8)
    g = torch.Generator(device="cuda").manual_seed(cin)
    f32 = dict(dtype=torch.float32, device=DEV)
    r = lambda *s: torch.randn(*s, generator=g, **f32)  # noqa: E731
    a, w, b = r(512, cin).bfloat16(), r(27, cin, cout).bfloat16(), r(cout)
    gout, work = r(512, cout), torch.empty(1 << 20, **f32)
    geom = (ctypes.c_int * 15)(8, 8, 8, 8, 8, 8, 0, cin, 0, 8, 8, 8, 1, 3, cout)

    def run():
        y, y32 = torch.empty(512, cout, dtype=torch.bfloat16, device=DEV), torch.empty(512, cout, **f32)
        gm, dv, dA = (torch.empty(512, c, **f32) for c in (cout, cin, cin))
        dW, dB = torch.empty(27, cin, cout, **f32), torch.empty(cout, **f32)
        ctx.call("psc_conv3d_fwd", geom, gpu._p(a), None, gpu._p(w), gpu._p(b), 2, gpu._p(y), gpu._p(y32),
                 gpu._stream())
        ctx.call("psc_conv3d_bwd", geom, gpu._p(a), None, gpu._p(w), gpu._p(gout), gpu._p(y), 2, gpu._p(gm),
                 gpu._p(dv), gpu._p(dA), 0, None, 0, gpu._p(dW), gpu._p(dB), gpu._p(work), work.numel(),
                 gpu._stream())
        return torch.cat([t.flatten() for t in (y32, dA, dW, dB)])

    return run


def _precond(n):
    ctx = gpu.GridContext({"nx": n, "ny": n + 1, "nz": n, "h": 0.4, "radius": 1.0}, 8)
    v = torch.randn(ctx.n, dtype=torch.float64, device=DEV, generator=torch.Generator(device="cuda").manual_seed(n))
    return lambda: gpu.poisson_precond(ctx, v)


def _sad(symbol):
    ctx = gpu.GridContext(O.build_system([{"typ": symbol, "coord": np.zeros((1, 3))}], h=0.6, radius=5.0), 8)
    atoms = [{"typ": symbol, "coord": np.zeros((1, 3))}]
    return lambda: torch.cat(gpu.sad_setup(ctx, atoms, ElementTable(), pseudo_tables())[:3])


CASES = pytest.mark.parametrize("make, args", [(_conv, ((8, 8), (64, 8))), (_conv, ((16, 32), (128, 32))),
                                               (_precond, (24, 90)), (_sad, ("H", "Si"))],
                                ids=["conv-8", "conv-32", "precond", "sad"])


class _FuncAttributes(ctypes.Structure):   # cudaFuncAttributes up to the limit
    _fields_ = [("sizes", ctypes.c_size_t * 3), ("ints", ctypes.c_int * 5), ("max_dynamic", ctypes.c_int),
                ("rest", ctypes.c_int * 64)]


def _limits():
    """Dynamic shared memory allowed for each kernel of the library."""
    lib = ctypes.CDLL(str(_lib.LIB_PATH))
    names = subprocess.run(["nm", "-D", "--defined-only", str(_lib.LIB_PATH)], capture_output=True, text=True,
                           check=True).stdout.split()
    out = {}
    for name in names:
        if re.match(r"_Z\d+k_", name):
            a = _FuncAttributes()
            if lib.cudaFuncGetAttributes(ctypes.byref(a), ctypes.cast(getattr(lib, name), ctypes.c_void_p)) == 0:
                out[name] = a.max_dynamic
    return out


@CASES
def test_no_call_lowers_a_kernels_limit(make, args):
    runs = [make(*a) if isinstance(a, tuple) else make(a) for a in args]
    runs[1]()
    before = _limits()
    assert len(before) > 20
    runs[0]()
    after = _limits()
    assert all(after[k] >= v for k, v in before.items()), {k: (v, after[k]) for k, v in before.items() if after[k] < v}


@CASES
def test_threads_with_different_sizes(make, args):
    runs = [make(*a) if isinstance(a, tuple) else make(a) for a in args]
    want = [r() for r in runs]
    torch.cuda.synchronize()
    bad, start = [], threading.Barrier(2)

    def loop(run, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(30)
                for _ in range(150):
                    got = run()
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(got, ref):
                        raise AssertionError("another result")
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            bad.append(e)

    ts = [threading.Thread(target=loop, args=p) for p in zip(runs, want)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
