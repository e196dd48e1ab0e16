"""Waits of the tcgen05 kernels, by reading their source (no GPU): a wait that runs out must end for the whole warp, because what follows it -- tcgen05.ld / st,
the arrival of a warp -- takes a converged warp.  Only the one lane that brings the activation tiles of the GEMM waits by itself."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "pyre_b200" / "csrc"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_a_warp_wait_votes():
    body = re.search(r"bool tc_warp_wait\([^)]*\)\s*\{(.*?)\}", _code("pb_tc.cuh"), re.S).group(1)
    assert re.fullmatch(r"\s*return __all_sync\(0xffffffffu, pb_mbar_wait\(.*\)\) != 0;\s*", body)


@pytest.mark.parametrize("name", ["pb_gemmtc.cu", "pb_moetc.cu"])
def test_warps_wait_as_warps(name):
    code = _code(name)
    if name == "pb_gemmtc.cu":
        one_lane = re.search(r"if \(warp == TC_DECODERS\) \{.*?if \(lane == 0\) \{(.*?)\} else if \(warp == TC_DECODERS \+ 1\)", code, re.S)
        assert "pb_mbar_wait(" in one_lane.group(1) and "__syncwarp" not in one_lane.group(1)
        code = code[:one_lane.start(1)] + code[one_lane.end(1):]
    assert "pb_mbar_wait(" not in code
    assert code.count("tc_warp_wait(") >= 5
