"""Every consumer warp of the decode kernel waits for every unit of the ring: a stage's phases differ by parity, so a warp that never saw a unit arrive
would take the stage's next one for there while the unit itself is still on its way.  A model of the loop with the source's constants and condition (no GPU)."""
import os
import re

import pytest

from yasakani_b200 import build

CODE = re.sub(r"//[^\n]*|/\*.*?\*/", "", open(os.path.join(build.CSRC, "kv4_decode_mma.cu")).read(), flags=re.S)


def _constant(name):
    return int(re.search(rf"{name}\s*=?\s+(\d+)", CODE)[1])


def _also_before():
    """The condition under which a warp waits for the unit before its slot's too, as a function of (sub, u, u0)."""
    m = re.search(r"if \(([^()]*)\) here = mbar_wait\(bar_full \+ 8 \* \(\(k - 1\) % NSTAGE\), \(\(k - 1\) / NSTAGE\) & 1\) && here;", CODE)
    if not m:
        return lambda sub, u, u0: False
    expr = m[1].replace("&&", "and").replace("NCW", str(_constant("KV4_DECODE_NCW"))).replace("L::UG", str(_constant("int UG")))
    return lambda sub, u, u0: eval(expr, {}, dict(sub=sub, u=u, u0=u0))


@pytest.mark.parametrize("units", [1, 2, 5, 6, 7, 36, 56])
def test_every_warp_waits_for_every_unit_before_its_stage_comes_again(units):
    ncw, ug, nstage, also = _constant("KV4_DECODE_NCW"), _constant("int UG"), _constant("NSTAGE"), _also_before()
    for warp in range(ncw):
        seen = set()
        for kk in range(warp, units * ug, ncw):
            sub, u = kk % ug, kk // ug
            assert u < nstage or u - nstage in seen, (warp, u)   # else the wait for u returns on the phase before u - nstage
            seen.add(u)
            if also(sub, u, 0):
                seen.add(u - 1)
