"""The autotuner's saved choices, and which one-call solves it tunes.  Tune files
of a version with other kernel variants: a choice this one has no kernel for is
measured anew (and then reused), not read as another variant or as a reason to
keep the defaults."""
import os
import subprocess
import sys

import pytest

from tests.test_gpu_tune import ROOT, solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,key,old,new,marker", [
    # an INT8 tile by its place in a former list; its widths are saved now
    (2 | (6 << 8), "k0 o20,20 v40,40 p2 s6 d0", "2", {"48", "64", "80"},
     "INT8 tile"),
    # 128-row DMMA tiles; fewer spin cases than the plan has
    (0, "k0 o20,20 v40,40 p0 s0 d0", "128 128", {"48", "96"},
     "DMMA tile rows"),
    (0, "k0 o20,20 v40,40 p0 s0 d0", "96", {"48", "96"}, "DMMA tile rows")])
def test_unknown_choices_are_measured_anew(tmp_path, prec, key, old, new,
                                           marker):
    f = tmp_path / "tune.txt"
    f.write_text(f"{key}: {old}\n")
    e1, err1 = solve(20, 40, prec, {"LIBPT_TUNE_FILE": str(f)})
    assert marker in err1
    lines = f.read_text().splitlines()
    assert len(lines) == 2 and lines[1].startswith(key + ":")
    assert set(lines[1].split(":")[1].split()) <= new
    e2, err2 = solve(20, 40, prec, {"LIBPT_TUNE_FILE": str(f)})
    assert marker not in err2 and f.read_text().splitlines() == lines
    assert e1 == e2


ONE_CALL = """
import sys
sys.path.insert(0, {root!r})
from libpt_b200 import ffi, synth
from tests.test_gpu_closed import plan_energy
from tests.test_gpu_parity import to_dev
case = synth.make("rpt", 20, 50, seed=3)
x = case["i_ovvv"] = case["i_ovvv"].copy()
x[:20 * 50 * 1225] *= 1.0 + 1e-9          # no row keeps the relation
dev = to_dev(case)
e = ffi.solve_device(case, dev)
sys.stderr.write("one call done\\n")
assert e == plan_energy(case, dev)
"""


def test_a_solve_without_closed_shell_rows_is_tuned():
    """The amplitudes alone satisfy the closed-shell relations: nothing can be
    grouped, and the solve is tuned like any other general one."""
    env = dict(os.environ, LIBPT_TUNE_VERBOSE="1")
    env.pop("LIBPT_TUNE_FILE", None)
    env.pop("LIBPT_AUTOTUNE", None)
    r = subprocess.run([sys.executable, "-c", ONE_CALL.format(root=ROOT)],
                       capture_output=True, text=True, timeout=300, env=env,
                       cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert "DMMA tile rows" in r.stderr.split("one call done")[0]
