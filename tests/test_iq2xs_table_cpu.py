"""The nibble form of the IQ2_XS codebook that the warp-level GEMM builds (pb_h_fill_tabs), restated on the CPU for all 512 entries: nibble j is the number of
the magnitude in byte j (8, 25, 43), and the selector turns it back into the byte."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "pyre_b200" / "csrc"


def _prmt(a, b, sel):
    src = [(a >> (8 * i)) & 0xFF for i in range(4)] + [(b >> (8 * i)) & 0xFF for i in range(4)]
    return sum(src[(sel >> (4 * i)) & 7] << (8 * i) for i in range(4))


def test_nibbles_number_the_magnitudes():
    text = (CSRC / "pb_iq_tables.h").read_text()
    body = re.search(r"PB_IQ2XS_GRID\s*\[512\]\s*=\s*\{(.*?)\}", text, re.S).group(1)
    grid = [int(x, 16) for x in re.findall(r"0x[0-9a-fA-F]+", body)]
    assert len(grid) == 512
    for e in grid:
        lo, hi = (e >> 4) & 0x0F0F0F0F, (e >> 36) & 0x0F0F0F0F
        lo, hi = (lo | lo >> 4) & 0x00FF00FF, (hi | hi >> 4) & 0x00FF00FF
        v = _prmt(lo, hi, 0x6420)
        mags = [(e >> (8 * j)) & 0xFF for j in range(8)]
        assert [(v >> (4 * j)) & 0xF for j in range(8)] == [{8: 0, 25: 1, 43: 2}[m] for m in mags]
        assert [(_prmt(0x002B1908, 0, (v >> s) & 0xFFFF) >> (8 * j)) & 0xFF for s in (0, 16) for j in range(4)] == mags
