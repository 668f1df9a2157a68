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


def _plain_groups(blob):
    """The profile without mean rows, low-rank rows and guards."""
    b = bytearray(blob)
    off_g, = struct.unpack_from("<I", b, 40)
    for g in range(128):
        o, = struct.unpack_from("<I", b, off_g + 4 * g)
        b[o + 3:o + 6] = bytes(3)
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


@pytest.mark.parametrize("nm", [1, 2, 5])
# Costs of the oracle are 32-bit numbers below its infinity of 2^30 while three steps from the only state that exists at first cost less:
# 3 (10,000 + 2,048)^2 = 4.4e8.  (The largest code that a table holds, 32,767, does not: 3.6e9.)
@pytest.mark.parametrize("top", [1400, 2200, 10000])
def test_key_widths_in_every_block_size(oracle, top, nm):
    """One multiplier, few rows and many rows take blocks of their own, and the 64-bit search a warp per chain in two of them: the same rows through all."""
    from yasakani_b200 import kvx
    blob = _with_largest_code(make_blob(nm=nm), top)
    rng = np.random.default_rng(top + nm)
    x = (rng.standard_normal((40, 256)) * np.exp(rng.standard_normal((40, 1)))).astype(np.float32)
    x[7, ::3] *= 40.0
    grp, pos = np.arange(40, dtype=np.int32), np.full(40, 9, np.int32)
    want = oracle.tb_encode(blob, x, grp, pos)
    prof = kvx.TrellisProfile(blob)
    for n in (40, 593):
        rep = np.arange(n) % 40
        y, pay, side = kvx.tb_encode(prof, *(torch.from_numpy(np.ascontiguousarray(a[rep])).cuda() for a in (x, grp, pos)))
        assert np.array_equal(y.cpu().numpy().view(np.uint32), want["y"].view(np.uint32)[rep]), n
        assert np.array_equal(pay.cpu().numpy().view(np.uint32).reshape(n, 40), want["pay"][rep]) and np.array_equal(side.cpu().numpy().view(np.uint32), want["side"][rep]), n


@pytest.mark.parametrize("with_payload", [True, False])
def test_encoder_leaves_the_callers_other_words_alone(oracle, with_payload):
    """The C entry writes a packed row's payload words and its side words, nothing else: rows of records that hold other data behind the
    payload, and rows that are not packed, keep their bytes."""
    from yasakani_b200 import _lib, kvx
    prof, n, stride = kvx.TrellisProfile(make_blob()), 48, 320
    rng = np.random.default_rng(4)
    x, grp, pos = rng.standard_normal((n, 256)).astype(np.float32), np.arange(n, dtype=np.int32), (np.arange(n) % 6).astype(np.int32)
    want = oracle.tb_encode(make_blob(), x, grp, pos)
    assert (want["kb"] == 0).any() and (want["kb"] == 5).any()
    dx, dg, dp = (torch.from_numpy(a).cuda() for a in (x, grp, pos))
    y, pay, side = torch.empty_like(dx), torch.full((n, stride), 0xAB, dtype=torch.uint8, device="cuda"), torch.full((n, 2), 0x5A5A5A5A, dtype=torch.int32, device="cuda")
    assert _lib.load().yskn_tb_encode(prof.dev.data_ptr(), prof.nm, dx.data_ptr(), dg.data_ptr(), dp.data_ptr(), n, y.data_ptr(),
                                      pay.data_ptr() if with_payload else None, stride, side.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream) == 0
    got, gs = pay.cpu().numpy().view(np.uint32), side.cpu().numpy().view(np.uint32)
    for r in range(n):
        words = 8 * want["kb"][r] if with_payload else 0
        assert np.array_equal(got[r, :words], want["pay"][r, :words]) and (got[r, words:] == 0xABABABAB).all(), r
        assert np.array_equal(gs[r], want["side"][r] if words else np.full(2, 0x5A5A5A5A, np.uint32)), r
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want["y"].view(np.uint32))


@pytest.mark.parametrize("top,ctx,M,splits,stride", [
    (1100, 1000, 1, 3, 160), (1100, 1000, 2, 1, 164),               # many tiles per warp, rows that are not 16-byte aligned
    (1100, 40, 1, 37, 160), (1100, 15, 1, 1, 176),                  # splits of one or two tokens, a single ragged tile
    (2048, 200, 1, 2, 160), (2500, 200, 1, 2, 160),                 # the last table the tile path takes, the first it does not
])
def test_attention_tiles(oracle, top, ctx, M, splits, stride):
    """Attention over packed rows against the exact oracle over the oracle's unpacked rows; every code width for keys and values."""
    from yasakani_b200 import kvx
    blob = _with_largest_code(make_blob(), top)
    prof, kvh, nh, n = kvx.TrellisProfile(blob), 4, 32, ctx + M
    max_ctx = (n + 63) // 64 * 64
    rng = np.random.default_rng(top + ctx)
    x = np.zeros((2, kvh, max_ctx, 256), np.float32)
    x[:, :, :n] = rng.standard_normal((2, kvh, n, 256))
    grp = np.array([[10, 8, 0, 15], [3, 9, 5, 31]], np.int32)       # 3 / 4 / 5 bits and flat records, ranks 0 - 2
    rows_pos = np.tile(np.arange(max_ctx, dtype=np.int32), kvh)
    dev, rows = [], []
    for i in range(2):
        gr = np.repeat(grp[i], max_ctx).astype(np.int32)
        _, pay, side = kvx.tb_encode(prof, *(torch.from_numpy(a).cuda() for a in (x[i].reshape(-1, 256), gr, rows_pos)), pay_stride=stride)
        p40 = np.ascontiguousarray(pay.cpu().numpy().view(np.uint32).reshape(-1, stride // 4)[:, :40])
        rows.append(oracle.tb_unpack(blob, gr, rows_pos, p40, side.cpu().numpy().view(np.uint32), x[i].reshape(-1, 256)).reshape(kvh, max_ctx, 256))
        dev += [pay.view(kvh, max_ctx, stride), side.view(kvh, max_ctx, 2)]
    q = torch.from_numpy(rng.standard_normal((M, nh, 256)).astype(np.float32)).half()
    pm = torch.full((M, splits, nh), float("nan"), device="cuda"); pl = pm.clone(); pacc = torch.full((M, splits, nh, 256), float("nan"), device="cuda")
    kvx.launch_tb_attention(prof, q.cuda(), *dev, *(torch.from_numpy(a).cuda() for a in grp), M, torch.tensor([ctx], dtype=torch.int32, device="cuda"), splits,
                            pm, pl, pacc, nh, *(torch.from_numpy(a).cuda() for a in x))
    o16 = torch.empty((M, nh, 256), dtype=torch.float16, device="cuda")
    kvx.launch_kv8_combine(pm, pl, pacc, splits, M, nh, o16, inverse_rotate=False)
    want = oracle.rows_attention_exact(q.float().numpy(), rows[0], rows[1], ctx)
    err = np.abs(o16.float().cpu().numpy() - want)
    # queries and weights in fp32 accuracy: what remains is fp32 sums (2e-5 here) and the fp16 rounding of the row (2^-11)
    assert (err <= 5e-5 + 2.0 ** -10 * np.abs(want)).all(), err.max()


def _packed_case(oracle, blob, scale, grp, ctx, M, q, seed, stride=160):
    """Encoded rows (values times `scale`, an array that broadcasts over [key | value][kv-head][token]) with the oracle's unpacked rows; the
    kernel's partials merged in 64 bits and the exact rows."""
    from yasakani_b200 import kvx
    prof, kvh, nh, n, splits = kvx.TrellisProfile(blob), 4, q.shape[1], ctx + M, 3
    max_ctx = (n + 63) // 64 * 64
    rng = np.random.default_rng(seed)
    x = np.zeros((2, kvh, max_ctx, 256), np.float32)
    x[:, :, :n] = rng.standard_normal((2, kvh, n, 256)) * np.broadcast_to(scale, (2, kvh, n))[..., None]
    rows_pos = np.tile(np.arange(max_ctx, dtype=np.int32), kvh)
    dev, rows = [], []
    for i in range(2):
        gr = np.repeat(grp[i], max_ctx).astype(np.int32)
        _, pay, side = kvx.tb_encode(prof, *(torch.from_numpy(a).cuda() for a in (x[i].reshape(-1, 256), gr, rows_pos)), pay_stride=stride)
        p40 = np.ascontiguousarray(pay.cpu().numpy().view(np.uint32).reshape(-1, stride // 4)[:, :40])
        rows.append(oracle.tb_unpack(blob, gr, rows_pos, p40, side.cpu().numpy().view(np.uint32), x[i].reshape(-1, 256)).reshape(kvh, max_ctx, 256))
        dev += [pay.view(kvh, max_ctx, stride), side.view(kvh, max_ctx, 2)]
    pm = torch.full((M, splits, nh), float("nan"), device="cuda"); pl = pm.clone(); pacc = torch.full((M, splits, nh, 256), float("nan"), device="cuda")
    kvx.launch_tb_attention(prof, q.cuda(), *dev, *(torch.from_numpy(a).cuda() for a in grp), M, torch.tensor([ctx], dtype=torch.int32, device="cuda"), splits,
                            pm, pl, pacc, nh, *(torch.from_numpy(a).cuda() for a in x))
    m, l, o = (t.double().cpu().numpy() for t in (pm, pl, pacc))
    w = np.exp(m - m.max(1, keepdims=True))
    got = (w[..., None] * o).sum(1) / (w * l).sum(1)[..., None]
    return got, oracle.rows_attention_exact(q.float().numpy(), rows[0], rows[1], ctx).astype(np.float64)


@pytest.mark.parametrize("values", [1e-6, 1e-3, 1e-2, 1.0, 1e3, "flat 1e6", "mixed", "outlier"])
def test_attention_is_fp32_at_every_scale_of_the_values(oracle, values):
    """Weights (probability x row scale x gain) and queries keep fp32 accuracy and range whatever the rows' scale: tiny and large values, scales
    that differ by 2^30 inside a sequence, a large row that the softmax leaves out, and large flat rows (whose gain is 1, not 1 / 256)."""
    ctx, M, nh = 900, 1, 24
    rng = np.random.default_rng(7)
    scale = np.ones((2, 1, ctx + M), np.float32)
    grp = np.array([[10, 8, 0, 12], [3, 9, 5, 7]], np.int32)        # value groups of 5 / 3 / 5 / 4 bits, no flat one
    q = torch.from_numpy(rng.standard_normal((M, nh, 256)).astype(np.float32)).bfloat16()
    if values == "flat 1e6":
        grp[1] = [15, 31, 47, 63]
        scale[1] = 1e6
    elif values == "mixed":
        scale[1] = 2.0 ** rng.integers(-20, 11, ctx + M)
    elif values == "outlier":                                       # a large value under a weight of about 2^-38
        q = q * 8
        scale[1, 0, 5], scale[0, 0, 5] = 2.0 ** 12, 1e-3
    else:
        scale[1] = values
    # a profile without mean rows or low-rank rows: they do not scale with the values and would hide the codes' part
    got, want = _packed_case(oracle, _plain_groups(make_blob()), scale, grp, ctx, M, q, 3)
    rel = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    # An fp32 sum of 900 terms in runs of 16 (8 of them per warp) and 25 partial sums: at most 16 + 33 roundings of 2^-23 of the sum of
    # magnitudes, which is up to 8 times the result here; scores of up to 2^5 carry 2^-24 x 24 roundings of the dot product.
    assert (rel < 2e-5).all(), rel.max()


@pytest.mark.parametrize("size", [1e-6, 1.0, 1e6])
def test_attention_queries_of_any_size(oracle, size):
    """bf16 queries beyond the range of fp16 and far below it, against keys that bring the scores back to ordinary size."""
    ctx, M, nh = 300, 2, 32
    scale = np.ones((2, 1, ctx + M), np.float32)
    scale[0] = 1.0 / size if size > 1 else 1.0
    q = torch.from_numpy((np.random.default_rng(11).standard_normal((M, nh, 256)) * size).astype(np.float32)).bfloat16()
    got, want = _packed_case(oracle, _plain_groups(make_blob()), scale, np.array([[10, 8, 0, 12], [3, 9, 5, 7]], np.int32), ctx, M, q, 5)
    rel = np.linalg.norm(got - want, axis=-1) / np.linalg.norm(want, axis=-1)
    assert (rel < 2e-5).all(), rel.max()


@pytest.mark.parametrize("tables", [3, 0])
def test_flat_groups_have_no_table(oracle, tables):
    """The loader does not check a flat group's table index: profiles whose flat groups name a table that does not exist, with and without tables."""
    from yasakani_b200 import kvx
    b = bytearray(_plain_groups(make_blob()))
    off_g, = struct.unpack_from("<I", b, 40)
    for g in range(128):
        o, = struct.unpack_from("<I", b, off_g + 4 * g)
        if tables == 0 or b[o] == 1:
            b[o:o + 3] = bytes((1, 200, 255))                       # flat, no step width, table 255
    if tables == 0:
        struct.pack_into("<H", b, 22, 0)
        struct.pack_into("<I", b, 36, len(b))                       # the list of tables is empty: it ends with the blob
    blob = bytes(b)
    assert oracle.tb_check_blob(blob) == 0
    ctx, M, nh = 100, 1, 32
    q = torch.from_numpy(np.random.default_rng(2).standard_normal((M, nh, 256)).astype(np.float32)).half()
    got, want = _packed_case(oracle, blob, np.ones((2, 1, ctx + M), np.float32), np.array([[15, 31, 47, 63], [79, 15, 95, 31]], np.int32), ctx, M, q, 5)
    assert (np.linalg.norm(got - want, axis=-1) < 2e-5 * np.linalg.norm(want, axis=-1)).all()
    x = np.random.default_rng(3).standard_normal((8, 256)).astype(np.float32)
    grp, pos = np.full(8, 15, np.int32), np.arange(8, dtype=np.int32)
    want = oracle.tb_encode(blob, x, grp, pos)
    dev = [torch.from_numpy(a).cuda() for a in (x, grp, pos)]
    y, pay, side = kvx.tb_encode(kvx.TrellisProfile(blob), *dev)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want["y"].view(np.uint32))
    assert np.array_equal(kvx.tb_decode(kvx.TrellisProfile(blob), pay, side, dev[1], dev[2]).cpu().numpy(), want["y"])      # (by value: -0 decodes to +0)
