"""What closed-shell groups may read: same-spin blocks that differ from the
antisymmetrised mixed-spin ones at all, by one unit in the last place of one
element or by a common factor far below FP64 noise of real integrals, are read
as they were passed (the general jobs of a plan, bitwise), unless the caller
names a tolerance."""
import numpy as np
import pytest

from libpt_b200 import ffi, synth
from tests.test_gpu_closed import plan_energy
from tests.test_gpu_parity import to_dev

pytestmark = pytest.mark.gpu

O, V = 4, 50
SAME = {"t2": O * O * V * V, "l2": O * O * V * V, "i_oovv": O * O * V * V,
        "oovo": O * O * V * O, "ovvv": O * V * (V * (V - 1) // 2)}
BLOCKS = [("rpt", "t2"), ("rpt", "i_oovo"), ("rpt", "i_oovv"),
          ("rpt", "i_ovvv"), ("rft", "t2"), ("rft", "l2"),
          ("rft", "i2_t2f2_oovo"), ("rft", "i3_ovvv"), ("rft", "i6_oovo"),
          ("rft", "i7_ovvv")]


def same_count(name):
    return SAME.get(name) or SAME[name[-4:]]


def changed(case, name, how):
    x = case[name].copy()
    same = x[:same_count(name)]
    if how == "factor":
        same *= 1.0 + 2.0 ** -46
    elif how == "random":
        rng = np.random.default_rng(1)
        same += 2.0 ** -46 * np.abs(x).max() * rng.uniform(-1, 1, same.size)
    else:   # one unit in the last place of a small element; of OVVV, which is
        # looked at by occupied index, in each of them
        for part in np.split(same, O if name.endswith("ovvv") else 1):
            n = np.flatnonzero(part)[np.argmin(np.abs(part[part != 0.0]))]
            part[n] = np.nextafter(part[n], np.inf)
    return dict(case, **{name: x})


@pytest.mark.parametrize("how", ["ulp", "factor", "random"])
@pytest.mark.parametrize("kind,name", BLOCKS)
def test_blocks_that_differ_are_read(kind, name, how):
    case = synth.make(kind, O, V, seed=17, fock=1e-3)
    other = changed(case, name, how)
    dev = to_dev(other)
    e = ffi.solve_device(other, dev)
    assert e == plan_energy(other, dev)
    assert e == ffi.solve_host(other)


@pytest.mark.parametrize("kind,name", BLOCKS)
def test_a_named_tolerance_reads_the_mixed_spin_blocks(kind, name,
                                                       monkeypatch):
    case = synth.make(kind, O, V, seed=17, fock=1e-3)
    exact = ffi.solve_device(case, to_dev(case))
    other = changed(case, name, "factor")
    dev = to_dev(other)
    monkeypatch.setenv("LIBPT_CLOSED_TOL", "1e-13")
    assert ffi.solve_device(other, dev) == exact
    monkeypatch.setenv("LIBPT_CLOSED_TOL", "1e-15")   # below 2^-46
    assert ffi.solve_device(other, dev) == plan_energy(other, dev)
