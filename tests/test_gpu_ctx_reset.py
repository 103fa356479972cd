"""Contexts created after others were destroyed, and after cudaDeviceReset: the
pinned scratch of the earlier ones is used again only while it is still pinned,
and it starts zeroed.  A process of its own without torch, which would not
survive the reset."""
import subprocess
import sys

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA device", allow_module_level=True)

CHILD = r"""
import ctypes, sys
from ctypes import byref, c_double, c_int, c_long, c_void_p
import numpy as np
rt = ctypes.CDLL(sys.argv[2], ctypes.RTLD_GLOBAL)     # the runtime that libpsc then uses
psc = ctypes.CDLL(sys.argv[1])
N = 24 * 24 * 24

def ok(rc):
    assert rc == 0, rc

def up(a):
    p = c_void_p()
    ok(rt.cudaMalloc(byref(p), c_long(a.nbytes)))
    ok(rt.cudaMemcpy(p, a.ctypes.data_as(c_void_p), c_long(a.nbytes), 1))
    return p

def ctxs(count):
    out = []
    for _ in range(count):
        p = c_void_p()
        ok(psc.psc_ctx_create(24, 24, 24, c_double(0.4), 8, byref(p)))
        out.append(p)
    return out

def work(ctx):
    # mixer steps (norms read on the host) and a Hartree solve (state read on the host)
    rng = np.random.default_rng(1)
    res = []
    ok(psc.psc_mixer_reset(ctx, 20))
    for i in range(6):
        x, f = up(rng.standard_normal(N)), up(0.5 ** i * rng.standard_normal(N))
        o, m = up(np.zeros(N)), c_int()
        ok(psc.psc_mixer_step(ctx, x, f, c_double(0.5), c_double(0.1), o, byref(m), None))
        assert m.value == i
        h = np.empty(N)
        ok(rt.cudaMemcpy(h.ctypes.data_as(c_void_p), o, c_long(h.nbytes), 2))
        res.append(h)
    its = c_int()
    b, s = up(rng.standard_normal(N)), up(np.zeros(N))
    ok(psc.psc_pcg_poisson_prec(ctx, b, s, 50, c_double(1e-8), byref(its), None))
    h = np.empty(N)
    ok(rt.cudaMemcpy(h.ctypes.data_as(c_void_p), s, c_long(h.nbytes), 2))
    return its.value, np.array(res + [h])

def no_steps(ctx):
    # a fresh context's solve of no iterations has none to report
    its, b, s = c_int(-1), up(np.ones(N)), up(np.zeros(N))
    ok(psc.psc_set_use_graphs(ctx, 0))
    ok(psc.psc_pcg_poisson(ctx, b, s, 0, c_double(1e-8), byref(its), None))
    assert its.value == 0, its.value
    ok(psc.psc_pcg_poisson(ctx, b, s, 3, c_double(1e-8), byref(its), None))
    ok(psc.psc_set_use_graphs(ctx, 2))

first = None
for round_ in range(3):
    many = ctxs(20)                     # more than are kept
    for c in many[:2] + many[-1:]:
        no_steps(c)
        got = work(c)
        first = first or got
        assert got[0] == first[0] and np.array_equal(got[1], first[1])
    for c in many:
        ok(psc.psc_ctx_destroy(c))
    ok(rt.cudaDeviceSynchronize())
    if round_:
        ok(rt.cudaDeviceReset())
print("ok")
"""


def test_contexts_after_a_device_reset():
    from parsec_python_b200 import _lib

    _lib.load()
    with open("/proc/self/maps") as f:
        cudart = next(line.split()[-1] for line in f if "libcudart.so" in line)
    r = subprocess.run([sys.executable, "-c", CHILD, str(_lib.LIB_PATH), cudart], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stderr[-2000:]
