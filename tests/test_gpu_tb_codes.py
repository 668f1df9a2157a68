"""The trellis search on both sides of the line between its two key widths: code tables whose largest code is 1,400 (32-bit keys), one
more, and twice the usual (64-bit keys), every step width, against the oracle bit for bit."""
import os
import struct
import sys

import numpy as np
import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
from make_kvqp_blob import make_blob  # noqa: E402

pytestmark = pytest.mark.gpu


def _with_largest_code(blob, top):
    b = bytearray(blob)
    nt, = struct.unpack_from("<H", b, 22)
    off_t, = struct.unpack_from("<I", b, 36)
    for t in range(nt):
        o, = struct.unpack_from("<I", b, off_t + 4 * t)
        code = np.frombuffer(bytes(b[o + 12:o + 524]), "<i2").astype(np.float64)
        b[o + 12:o + 524] = np.rint(code * top / np.abs(code).max()).astype("<i2").tobytes()
    return bytes(b)


@pytest.mark.parametrize("top", [1400, 1401, 2200])
def test_encoder_key_widths(oracle, top):
    from yasakani_b200 import kvx
    blob = _with_largest_code(make_blob(nm=3), top)
    rng = np.random.default_rng(top)
    n = 40                                                       # records 0 .. 39 hold every step width and a flat one
    x = (rng.standard_normal((n, 256)) * np.exp(rng.standard_normal((n, 1)))).astype(np.float32)
    x[7, ::3] *= 40.0                                            # values that clamp at +-2048
    grp, pos = np.arange(n, dtype=np.int32), np.full(n, 9, np.int32)
    want = oracle.tb_encode(blob, x, grp, pos)
    y, pay, side = kvx.tb_encode(kvx.TrellisProfile(blob), *(torch.from_numpy(a).cuda() for a in (x, grp, pos)), pay_stride=164)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want["y"].view(np.uint32))
    got = pay.cpu().numpy().view(np.uint32).reshape(n, 41)
    assert np.array_equal(got[:, :40], want["pay"]) and not got[:, 40].any()      # what a row does not use is zero
    assert np.array_equal(side.cpu().numpy().view(np.uint32), want["side"])
