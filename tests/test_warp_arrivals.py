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
