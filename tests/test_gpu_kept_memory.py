"""Device memory kept between solves is not in another allocation's way: a
server's pool, the device producer and the caller can have it."""
import os
import subprocess
import sys

import pytest

from libpt_b200 import ffi, synth

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def keep_a_gibibyte():
    """A solve whose round workspace (1 GiB) stays in the cache."""
    import torch
    case, dev = synth.case_device("rpt", 12, 150, seed=1)
    ffi.solve_device(case, dev)
    del dev
    torch.cuda.empty_cache()


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_release_gives_everything_back():
    keep_a_gibibyte()
    before = free_bytes()
    ffi.release_device_memory()
    assert free_bytes() - before >= 1 << 30
    ffi.release_device_memory()      # nothing left: no effect
    case = synth.make("rpt", 4, 30, seed=2)
    assert ffi.solve_host(case) == ffi.solve_host(case)


def test_server_pool_is_sized_without_the_kept_memory():
    """0.9 of the free memory: the kept buffers count as free.  (The first solve
    also loads the library's kernels and its static array.)"""
    keep_a_gibibyte()
    ffi.release_device_memory()
    s = ffi.Server()
    whole = s.stats()["pool_bytes"]
    s.close()
    keep_a_gibibyte()
    s = ffi.Server()
    after = s.stats()["pool_bytes"]
    s.close()
    assert after >= whole - (64 << 20)


FULL = """
import sys
sys.path.insert(0, {root!r})
import torch
from libpt_b200 import ffi
from tests.test_gpu_kept_memory import keep_a_gibibyte, free_bytes
o, v, q = 1, 500, 8                      # 1 GB of scratch
f = [torch.randn(q, a, b, dtype=torch.float64, device="cuda")
     for a, b in ((o, o), (o, v), (v, v))]
ref = ffi.rpt_inputs_df(*f)              # cuBLAS is loaded, outputs exist
out = {{n: torch.empty_like(t) for n, t in ref.items()}}
torch.cuda.empty_cache()
keep_a_gibibyte()
fill = torch.empty(free_bytes() - (700 << 20), dtype=torch.uint8,
                   device="cuda")
code = ffi.lib().libpt_rpt_inputs_df(
    o, v, q, *[t.data_ptr() for t in f], None, None,
    out["i_oovo"].data_ptr(), out["i_oovv"].data_ptr(),
    out["i_ovvv"].data_ptr(), None)
torch.cuda.synchronize()
assert code == 0, ffi.lib().libpt_last_error()
for n in ref:
    assert torch.equal(out[n], ref[n]), n
print("ok")
"""


def test_producer_takes_the_kept_memory_when_the_device_is_full():
    r = subprocess.run([sys.executable, "-c", FULL.format(root=ROOT)],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr
