"""Tune files of a version with other kernel variants: a choice this one has no
kernel for is measured anew (and then reused), not read as another variant or
as a reason to keep the defaults."""
import pytest

from tests.test_gpu_tune import solve

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
