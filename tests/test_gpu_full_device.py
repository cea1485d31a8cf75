"""A device that holds a solve's operands and one triple's outputs but not a
closed-shell group's: the solve still runs, with the general jobs."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys
sys.path.insert(0, {root!r})
import torch
from libpt_b200 import ffi, synth
from tests.test_gpu_closed import plan_energy
from tests.test_gpu_kept_memory import free_bytes
from tests.test_gpu_parity import to_dev
o, v = 3, 240            # a group's outputs: 663 MB; a triple's: at most 553
case = synth.make("rft", o, v, seed=1)
dev = to_dev(case)
general = plan_energy(case, dev)
grouped = ffi.solve_device(case, dev)
assert grouped != general            # groups ran: the same products, other sums
for host in (False, True):           # host arrays of this size are streamed
    solve = (lambda: ffi.solve_host(case)) if host else (
        lambda: ffi.solve_device(case, dev))
    assert solve() == grouped
    ffi.release_device_memory()
    torch.cuda.empty_cache()
    need = ffi.footprint("rft", (o, v), host=host, round_triples=1)
    fill = torch.empty(free_bytes() - need - (60 << 20), dtype=torch.uint8,
                       device="cuda")
    assert solve() == general
    del fill
    torch.cuda.empty_cache()
    assert solve() == grouped
print("ok")
"""


def test_general_jobs_when_a_group_does_not_fit():
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT)],
                       capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and r.stdout.strip().endswith("ok"), r.stderr
