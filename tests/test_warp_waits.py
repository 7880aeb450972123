"""Waits that whole warps make must end the same way on every lane. They are bounded by a cycle count, so lanes of one warp can
disagree about whether one ran out; behind it stand warp-collective instructions (tcgen05.ld, barriers of the warp), which hang
where a lane has left. So a wait stands where one elected thread is at work, or it is the warp's joined one."""
import re
from pathlib import Path

import pytest

CAM = Path(__file__).resolve().parent.parent / "csrc" / "cam"


def single_lane_waits_of_warps(text):
    """Lines with a wait of single lanes outside of the blocks that one elected thread runs."""
    text = re.sub(r"//[^\n]*", "", text)
    found, blocks, head = [], [], 0
    for m in re.finditer(r"[{};]|\bmbar_wait(?:_cluster)?\(", text):
        if m[0] == "{":
            blocks.append(text[head:m.start()])
        elif m[0] == "}":
            blocks.pop()
        elif m[0] != ";":
            if not any("elect_one()" in b for b in blocks):
                found.append(text.count("\n", 0, m.start()) + 1)
            continue
        head = m.end()
    assert not blocks
    return found


@pytest.mark.parametrize("name", [
    "moe_gemm_pair.cu", "moe_fused.cu", "moe_gemm.cu", "tp_gemm.cu", "tp_gemm_2sm.cu", "gemm_bf16.cu", "gemm_bf16_2sm.cu"])
def test_waits_of_warps_are_joined(name):
    assert single_lane_waits_of_warps((CAM / name).read_text()) == []


def test_the_check_sees_a_single_lane_wait():
    text = "void f() {\n if (w == 0) { if (elect_one()) { for (;;) { mbar_wait(a, 0); } } } else {\n ok = mbar_wait(b, 0); g(); }\n}"
    assert single_lane_waits_of_warps(text) == [3]
