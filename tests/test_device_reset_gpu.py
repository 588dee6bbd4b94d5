"""A program may reset its device between calls (cudaDeviceReset ends the process's own context only): what the
library has set up in the old context is gone, and it must not rely on it.  Each case runs in a process of its
own, with another copy of the CUDA runtime than the library's, as a program that links against it has one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C
import sys

import numpy as np

sys.path.insert(0, %(root)r)
import openfish_b200 as of
from openfish_b200 import synth

for name in ("libcudart.so.12", "/usr/local/cuda/lib64/libcudart.so", "libcudart.so"):
    try:
        rt = C.CDLL(name)
        break
    except OSError:
        rt = None
assert rt is not None, "no CUDA runtime"
lib = of.lib()
vp = C.c_void_p
rt.cudaMalloc.argtypes = [C.POINTER(vp), C.c_size_t]
rt.cudaMemcpy.argtypes = [vp, vp, C.c_size_t, C.c_int]


def ok(rc):
    assert rc == 0, rc


def to_device(a):
    p = vp()
    ok(rt.cudaMalloc(C.byref(p), a.nbytes))
    ok(rt.cudaMemcpy(p, a.ctypes.data, a.nbytes, 1))
    return p


def from_device(p, like):
    out = np.empty_like(like)
    ok(rt.cudaMemcpy(out.ctypes.data, p, out.nbytes, 2))
    return out


T, N, SL = 60, 5, 5  # (kernels with more shared memory than a context grants by default)
scores = np.ascontiguousarray(synth.make_scores(T, N, SL, 61))
opt = of.decoder_init()


def decode():
    d = to_device(scores)
    gb = of.gpubuf_init(T, N, SL)
    out = [C.c_void_p() for _ in range(3)]
    lib.openfish_decode_gpu(T, N, 4 * 4 ** SL, d, SL, C.byref(opt), gb.ptr, *[C.byref(o) for o in out])
    of._check()
    got = [C.string_at(o, T * N) for o in out]
    gb.free()
    return got


def static():
    n = 1  # (of the 1024-state model, what the array holds at this length)
    out = [to_device(np.zeros((n, T), np.uint8)) for _ in range(3)]
    d = to_device(np.ascontiguousarray(scores[:, :n]))
    ok(lib.openfish_b200_decode_static(T, n, 4 * 4 ** SL, d, SL, C.byref(opt), *out))
    return [from_device(o, np.zeros((n, T), np.uint8)).tobytes() for o in out]


def rotary():
    B, S, H, D, half = 2, 33, 4, 32, 16
    rng = np.random.default_rng(62)
    x = rng.standard_normal((B, S, H, D)).astype(np.float16)
    angle = rng.standard_normal((S, half))
    p = to_device(x)
    args = (p, to_device(np.sin(angle).astype(np.float32)), to_device(np.cos(angle).astype(np.float32)), B, S, H, D, half,
            S * H * D, H * D, D)
    lib.openfish_rotary_emb_gpu(*args)
    of._check()
    return from_device(p, x).tobytes()


first = %(case)s()
ok(rt.cudaDeviceReset())
assert %(case)s() == first
ok(rt.cudaDeviceReset())
assert %(case)s() == first
print("the same after a reset")
"""


@pytest.mark.parametrize("case", ["decode", "rotary", "static"])
def test_calls_before_and_after_a_reset(native_lib, case):
    r = subprocess.run([sys.executable, "-c", CHILD % {"root": ROOT, "case": case}], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "the same after a reset" in r.stdout, r.stdout + r.stderr
