"""The FP64 contraction kernel on row counts around its 16-row fragments and
its 96- / 48-row tiles, and on contraction lengths around the fours of its
16-deep K steps: a job's last tile multiplies only the fragments that hold
rows, a segment's last step only the fours that hold columns.  Against an FP64 product on the device, at the kernel self-test's
bar (1e-14 of the dot products' magnitude)."""
import pytest

from libpt_b200 import ffi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])          # 96-, 48-row tiles
@pytest.mark.parametrize("m", [1, 15, 16, 17, 33, 47, 48, 49, 63, 64, 65, 79,
                               80, 81, 95, 96, 97, 112, 113, 127, 128, 129,
                               143, 144, 145, 193, 209, 256, 257])
def test_rows_at_fragment_and_tile_edges(m, variant):
    assert ffi.selftest(ffi.PREC_FP64, m, 132, 37, variant) < 1e-14


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 9, 12, 13, 16, 17, 21, 32, 96,
                               97])
def test_contraction_lengths_at_step_edges(k, variant):
    for m in (20, 50, 96, 130):
        assert ffi.selftest(ffi.PREC_FP64, m, 260, k, variant) < 1e-14
