"""State the library keeps between calls belongs to the CUDA context it was
made in: kernel attributes, idle streams, kept buffers, page-locked staging.  A
second context on the GPU (what a second GPU is to them) gets its own, and the
first one's stay usable.  In a child process, whose main thread changes its
current context through the driver API."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes, sys
sys.path.insert(0, {root!r})
from libpt_b200 import ffi, synth
cu = ctypes.CDLL("libcuda.so.1")
first, second, dev = ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_int()

def new_context():
    assert cu.cuCtxGetCurrent(ctypes.byref(first)) == 0 and first.value
    assert cu.cuDeviceGet(ctypes.byref(dev), 0) == 0
    assert cu.cuCtxCreate_v2(ctypes.byref(second), 0, dev) == 0   # now current

def use(ctx):
    assert cu.cuCtxSetCurrent(ctx) == 0
"""

KERNELS = """
forms = [(ffi.PREC_FP64, 0), (ffi.PREC_FP64, 1), (ffi.PREC_TF32X3, 0),
         (ffi.PREC_EMU64 | (5 << 8), 0)]
bars = [1e-14, 1e-14, 5e-5, 2.0 ** -29]

def check():
    for (prec, variant), bar in zip(forms, bars):
        for device_maps in (False, True):
            e = ffi.selftest(prec, 130, 260, 37, variant,
                             device_maps=device_maps)
            assert e < bar, (prec, variant, device_maps, e)

check()
new_context()
check()
use(first)
check()
print("ok")
"""

SOLVES = """
cases = [synth.make(k, o, v, seed=7 + v, fock=1e-3) for k, o, v in
         (("rpt", 4, 50), ("rft", 3, 21), ("rpt", 5, 13))]
cases.append(synth.make("upt", 4, 17, 3, 19, seed=5))
alone = [ffi.solve_host(c) for c in cases]
new_context()
for ctx in (second, first, second, first):
    use(ctx)
    for c, e in zip(cases, alone):
        assert ffi.solve_host(c) == e
print("ok")
"""


def child(code):
    r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT) + code],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr


def test_every_contraction_kernel_launches_in_a_second_context():
    child(KERNELS)


def test_host_solves_alternate_between_contexts():
    child(SOLVES)
