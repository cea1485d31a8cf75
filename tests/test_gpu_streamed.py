"""Restricted FP64 host-array solves whose OVVV blocks fill both staging
buffers (128 MiB and more) copy them by occupied index beside the triples that
need them: the energy is the device-input energy bitwise.  (T) and (fT), zero
and nonzero f_ov, first indices that own no triple (o = 2, 3), and inputs of
which all, some or none of the triples run as closed-shell groups."""
import pytest

from libpt_b200 import ffi, synth
from tests.test_gpu_closed import plan_energy
from tests.test_gpu_parity import to_dev

pytestmark = pytest.mark.gpu

STREAMED = 128 << 20


def streamed_case(kind, o, v, fock, broken=None):
    assert 1.5 * o * v ** 3 * 8 >= STREAMED
    case = synth.make(kind, o, v, seed=o + v, fock=fock)
    if broken is not None:
        name, part = broken
        x = case[name].copy()
        n = part * v * (v * (v - 1) // 2) if name.endswith("ovvv") else 0
        x[n + 1234] += 1e-3
        case[name] = x
    return case


@pytest.mark.parametrize("kind,o,v,fock", [
    ("rpt", 2, 178, 0.0), ("rpt", 3, 156, 1e-3), ("rpt", 6, 125, 0.0),
    ("rft", 2, 179, 1e-3), ("rft", 3, 157, 0.0), ("rft", 4, 142, 1e-3)])
def test_streamed_host_solve_equals_device_inputs(kind, o, v, fock):
    case = streamed_case(kind, o, v, fock)
    assert ffi.solve_host(case) == ffi.solve_device(case, to_dev(case))


@pytest.mark.parametrize("kind,o,v,fock,broken", [
    # no relation at all: general jobs from the first row on
    ("rpt", 3, 156, 1e-3, ("t2", 0)), ("rpt", 2, 178, 0.0, ("i_oovv", 0)),
    ("rft", 3, 157, 1e-3, ("l2", 0)), ("rft", 2, 179, 0.0, ("i6_oovo", 0))])
def test_streamed_general_jobs(kind, o, v, fock, broken):
    case = streamed_case(kind, o, v, fock, broken)
    dev = to_dev(case)
    e = ffi.solve_host(case)
    assert e == ffi.solve_device(case, dev)
    assert e == plan_energy(case, dev)


@pytest.mark.parametrize("kind,o,v,fock,broken", [
    # the first, a middle and the last row of OVVV off: groups and pairs of
    # the others, general jobs for the rest
    ("rpt", 4, 142, 1e-3, ("i_ovvv", 0)), ("rpt", 4, 142, 0.0, ("i_ovvv", 3)),
    ("rft", 4, 142, 1e-3, ("i7_ovvv", 2)), ("rft", 4, 142, 0.0, ("i3_ovvv", 0)),
    ("rft", 2, 179, 1e-3, ("i3_ovvv", 1))])
def test_streamed_rows_that_are_off(kind, o, v, fock, broken):
    case = streamed_case(kind, o, v, fock, broken)
    assert ffi.solve_host(case) == ffi.solve_device(case, to_dev(case))
