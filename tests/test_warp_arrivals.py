"""A lane that arrives on a barrier for its whole warp does so behind a __syncwarp(): without one the stage could be handed back while other lanes
still read it or poll its barrier (a check of the sources; no GPU)."""
import os
import re

from yasakani_b200 import build


def test_every_arrival_for_a_warp_stands_behind_a_syncwarp():
    code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(build.CSRC, "kv4_decode_mma.cu")).read(), flags=re.S)
    arrivals = [m.start() for m in re.finditer(r"if \(lane == 0\) mbar_arrive\(", code)]
    assert len(arrivals) >= 2
    for at in arrivals:
        assert code[:at].rstrip().endswith("__syncwarp();"), code[max(0, at - 120):at + 60]


def test_lanes_that_went_apart_are_joined_ahead_of_the_next_warp_wide_instruction():
    """tcgen05.ld and .st are instructions of the whole warp: where its lanes have polled or divided for themselves, an instruction that joins them, and
    that no condition guards, stands in between."""
    code = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(build.CSRC, "kv4_tc.cu")).read(), flags=re.S)
    finish = code[code.index("tc_finish_row("):]
    loop = finish[finish.index("for (int c = hf;"):]
    assert "__syncwarp();" in loop[:loop.index("tmem_ld32")]
    for after in ("swap_with_partner(tmax", "if (mown != m)"):
        rest = code[code.index(after):]
        assert "if (__any_sync(0xffffffffu, bump && i > 0)) {" in rest[:rest.index("tmem_")], after
