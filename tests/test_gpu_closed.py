"""Restricted one-call solves whose same-spin blocks are the antisymmetrised
mixed-spin ones run closed-shell groups (one set of products for the four
triples of i < j < k); others keep the general jobs of a plan.

Against a plan of the same inputs, whose per-triple energies the parity tests
hold to the oracle, at the FP64 bar of those tests: both add the same products
in FP64, in another order."""
import numpy as np
import pytest

from libpt_b200 import ffi, synth
from tests.test_gpu_parity import to_dev

pytestmark = pytest.mark.gpu

REL = 1e-12


def plan_energy(case, dev):
    p = ffi.Plan(case, dev)
    p.run()
    e = p.energy()
    p.close()
    return e


# v around the 8-wide index blocks, the 8 x 16 column tiles, the 16-row
# fragments and 96- / 128-row tiles; o from the smallest group up
@pytest.mark.parametrize("kind,o,v,fock", [
    ("rpt", 2, 50, 0.0), ("rft", 2, 61, 1e-3),
    ("rpt", 3, 48, 0.0), ("rpt", 4, 49, 1e-3), ("rpt", 5, 50, 0.0),
    ("rpt", 3, 51, 1e-3), ("rpt", 4, 52, 0.0), ("rpt", 3, 55, 0.0),
    ("rpt", 9, 57, 1e-3), ("rpt", 4, 63, 0.0), ("rpt", 17, 64, 0.0),
    ("rpt", 3, 65, 1e-3), ("rpt", 4, 96, 0.0), ("rpt", 3, 97, 0.0),
    ("rpt", 4, 113, 1e-3), ("rpt", 3, 129, 0.0),
    ("rft", 3, 48, 0.0), ("rft", 4, 53, 1e-3), ("rft", 6, 71, 0.0),
    ("rft", 3, 99, 1e-3)])
def test_closed_shell_solve_equals_the_plan(kind, o, v, fock):
    case = synth.make(kind, o, v, seed=o + v, fock=fock)
    dev = to_dev(case)
    ref = plan_energy(case, dev)
    e = ffi.solve_device(case, dev)
    # (fT) energies cancel between triples: the bar is on their magnitudes
    p = ffi.Plan(case, dev)
    p.run()
    scale = 2.0 * float(p.energy_slots().abs().sum())
    p.close()
    assert abs(e - ref) <= REL * scale
    assert ffi.solve_host(case) == e


@pytest.mark.parametrize("kind,name,part", [
    ("rpt", "t2", "same"), ("rpt", "t2", "mixed"), ("rpt", "i_oovo", "same"),
    ("rpt", "i_oovv", "same"), ("rft", "l2", "same"),
    ("rft", "i6_oovo", "same"), ("rft", "i2_t2f2_oovo", "same")])
def test_other_inputs_keep_the_general_jobs(kind, name, part):
    """One element off by 1e-9: the plan's energy, bitwise."""
    case = synth.make(kind, 4, 50, seed=3, fock=1e-3)
    x = case[name].copy()
    x[5 if part == "same" else x.size // 2 + 5] += 1e-9
    case[name] = x
    dev = to_dev(case)
    assert ffi.solve_device(case, dev) == plan_energy(case, dev)


@pytest.mark.parametrize("kind,name,index", [
    ("rpt", "i_ovvv", 0), ("rpt", "i_ovvv", 4), ("rft", "i7_ovvv", 2),
    ("rft", "i3_ovvv", 1)])
def test_integrals_are_checked_by_occupied_index(kind, name, index):
    """An OVVV block that breaks the relation at one occupied index: the
    groups without it run, the rest is general."""
    o, v = 5, 50
    case = synth.make(kind, o, v, seed=4)
    x = case[name].copy()
    x[index * v * (v * (v - 1) // 2) + 77] += 1e-3
    case[name] = x
    dev = to_dev(case)
    ref = plan_energy(case, dev)
    e = ffi.solve_device(case, dev)
    assert abs(e - ref) <= 1e-12 * max(abs(ref), 1e-2)
    assert ffi.solve_host(case) == e


def test_not_a_number_takes_the_general_jobs():
    case = synth.make("rpt", 3, 50, seed=5)
    x = case["i_ovvv"].copy()
    x[:] = np.nan
    case["i_ovvv"] = x
    assert np.isnan(ffi.solve_device(case, to_dev(case)))


@pytest.mark.parametrize("broken", [None, 1])
def test_streamed_upload_checks_rows_as_they_arrive(broken):
    """OVVV blocks over two staging buffers (137 MB) are streamed by occupied
    index: the device-input energy bitwise, whether or not an index breaks
    the relation."""
    o, v = 4, 142
    case = synth.make("rpt", o, v, seed=6)
    if broken is not None:
        x = case["i_ovvv"].copy()
        x[broken * v * (v * (v - 1) // 2) + 1234] += 1e-3
        case["i_ovvv"] = x
    assert ffi.solve_host(case) == ffi.solve_device(case, to_dev(case))
