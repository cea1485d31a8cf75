"""Device buffers kept between solves: solves of different sizes and precisions,
one after another and from several threads at once, give the energies they give
alone, and what stays allocated is bounded."""
import threading

import pytest

from libpt_b200 import ffi, synth
from tests.test_gpu_parity import to_dev

pytestmark = pytest.mark.gpu

SIZES = [("rpt", 4, 49), ("upt", 4, 23), ("rpt", 3, 97), ("rft", 3, 50),
         ("uft", 3, 17), ("rpt", 5, 13)]


def test_solves_share_kept_buffers_from_any_thread():
    import torch
    cases = [synth.make(k, o, v, seed=40 + i, fock=1e-3)
             for i, (k, o, v) in enumerate(SIZES)]
    devs = [to_dev(c) for c in cases]
    alone = [ffi.solve_device(c, d) for c, d in zip(cases, devs)]
    bad = []

    def work(n):
        stream = torch.cuda.Stream()
        for r in range(3):
            for i in range(len(cases)):
                x = (i + n + r) % len(cases)
                e = (ffi.solve_host(cases[x]) if (i + n) % 2 else
                     ffi.solve_device(cases[x], devs[x],
                                      stream=stream.cuda_stream))
                if e != alone[x]:
                    bad.append((n, r, SIZES[x], e, alone[x]))

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(n,)) for n in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:3]


def test_kept_buffers_are_bounded():
    import torch
    ffi.solve_device(*_case(5, 13))
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    for v in range(100, 180, 8):        # workspaces and blocks of many sizes
        case, dev = _case(6, v)
        ffi.solve_device(case, dev)
        del dev
        torch.cuda.empty_cache()
    torch.cuda.synchronize()
    after, _ = torch.cuda.mem_get_info()
    # 2 GiB, and the driver's own rounding of up to 2 MiB a buffer
    assert before - after <= (2 << 30) + (256 << 20)


def _case(o, v):
    return synth.case_device("rpt", o, v, seed=v)
