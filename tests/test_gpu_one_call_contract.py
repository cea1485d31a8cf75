"""What one solve's energy is through each entry point, v >= 48: a plan, its
shards and a served solve agree bitwise always; a one-call solve joins them
bitwise when its inputs do not satisfy the closed-shell relations or when
LIBPT_CLOSED_TOL is negative, and agrees to rounding (the FP64 parity bar on
the magnitudes that are summed) when it shares its triples' products."""
import pytest

from libpt_b200 import ffi, synth
from tests.test_gpu_closed import REL
from tests.test_gpu_parity import to_dev

pytestmark = pytest.mark.gpu


def energies(case, dev):
    """Energy of the whole plan, of its two shards, of a served solve, and
    the sum of the triples' magnitudes."""
    p = ffi.Plan(case, dev)
    p.run()
    whole = p.energy()
    slots = p.energy_slots().clone()
    scale = 2.0 * float(slots.abs().sum())
    parts = 0.0
    for rank in range(2):
        p.run_shard(rank, 2)
        parts = parts + p.energy_slots().clone()
    p.energy_slots().copy_(parts)
    shards = p.energy()
    p.close()
    s = ffi.Server(mem_budget=2 << 30)
    served = s.wait(s.submit(case))[0]
    s.close()
    return whole, shards, served, scale


@pytest.mark.parametrize("kind,o,v", [("rpt", 4, 49), ("rpt", 3, 97),
                                      ("rft", 4, 53)])
@pytest.mark.parametrize("exact", [True, False])
def test_entry_points_agree(kind, o, v, exact, monkeypatch):
    case = synth.make(kind, o, v, seed=o * v, fock=1e-3)
    if not exact:
        case["t2"] = case["t2"].copy()
        case["t2"][5] += 1e-9
    dev = to_dev(case)
    whole, shards, served, scale = energies(case, dev)
    assert shards == whole and served == whole
    one = ffi.solve_device(case, dev)
    assert ffi.solve_host(case) == one
    if exact:
        assert abs(one - whole) <= REL * scale
    else:
        assert one == whole
    monkeypatch.setenv("LIBPT_CLOSED_TOL", "-1")
    assert ffi.solve_device(case, dev) == whole
    assert ffi.solve_host(case) == whole
