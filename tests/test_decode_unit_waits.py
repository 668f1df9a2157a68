"""The ring of the decode kernel under copies that come in late and warps that fall behind: every group is read from the unit it belongs to, and nobody
waits for good.  A model of producer, barriers and consumer warps with the source's constants and the source's wait (no GPU)."""
import os
import random
import re

import pytest

from yasakani_b200 import build

CODE = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(build.CSRC, "kv4_decode_mma.cu")).read(), flags=re.S)
NCW, UG, NSTAGE = (int(re.search(p, CODE)[1]) for p in (r"KV4_DECODE_NCW\s+(\d+)", r"int UG = (\d+)", r"NSTAGE = (\d+)"))
# the producer names the unit before it arms the stage, and a consumer has seen that name before its wait
NAMED = bool(re.search(r"s_tag\[s\] = k;\s*if \(lane == 0\) mbar_expect_tx\(bar,", CODE)) and \
    bool(re.search(r"while \(s_tag\[s\] != k && .*?mbar_try_wait\(full, parity\);\s*if \([^;]*!mbar_wait\(full, parity\)\)", CODE))


def _run(units, rng):
    """Random order of all that may happen next; a copy may be late by any number of steps.  Returns None, or what went wrong."""
    done, tag, free, flying = [0] * NSTAGE, [-1] * NSTAGE, [0] * NSTAGE, {}      # phases ended, unit named, arrivals, unit -> steps to go
    issued, slot = 0, list(range(NCW))                                           # next unit; next slot of each warp
    for _ in range(400 * units + 4000):
        if all(kk >= units * UG for kk in slot):
            return None
        for u in [u for u, t in flying.items() if t == 0]:
            done[u % NSTAGE] += 1
            del flying[u]
        for u in flying:
            flying[u] -= 1
        who = rng.randrange(NCW + 1)
        if who == NCW:                                                           # producer: a stage is free after UG arrivals a unit
            s = issued % NSTAGE
            if issued < units and (issued < NSTAGE or free[s] >= UG * (issued // NSTAGE)):
                tag[s], flying[issued] = issued, rng.choice([0, 1, 3, 400])
                issued += 1
            continue
        kk = slot[who]
        if kk >= units * UG:
            continue
        k = kk // UG
        s = k % NSTAGE
        if NAMED and tag[s] != k:
            continue
        if (done[s] & 1) == ((k // NSTAGE) & 1):                                 # try_wait(parity): true when the phase in progress has the other parity
            continue
        if k in flying or tag[s] != k:
            return f"warp {who} reads unit {k} before it is there"
        free[s] += 1
        slot[who] += NCW
    return "stuck"


@pytest.mark.parametrize("units", [4, 6, 11, 36])
def test_every_group_is_read_from_its_own_unit(units):
    for seed in range(60):
        assert _run(units, random.Random(seed)) is None, seed
