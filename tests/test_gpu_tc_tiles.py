"""The shares of a pass's tokens over CTA pairs, where they can go wrong: an odd number of tokens, one more than fill a pair, a last CTA with fewer than the
others, one to four occupied quadrants of 32 rows; splits without keys; a cache that ends half way through a tile of keys."""
import pytest

from tests.helpers import assert_close
from tests.test_gpu_tc import _run_tc
from yasakani_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True], ids=["workspace", "fused"])
@pytest.mark.parametrize("shape,ctx,M,splits", [
    (synth.C2, 90, 9, 3),                                  # 5 + 4 tokens: 30 and 24 rows; the cache ends at 192
    (synth.C2, 64, 11, 9),                                 # 36 rows: a second quadrant of four rows; more splits than tiles
    (synth.C2, 190, 43, 2),                                # two pairs of 11 tokens a CTA, the last one 10
    (synth.C1, 33, 33, 2),                                 # hd 128, eight heads: one row more than a pair holds
    (synth.Shape(4, 4, 256, 64, 1e4), 130, 33, 1),         # one head per kv-head: 17 rows in a tile of 128
    (synth.Shape(4, 4, 128, 32, 1e4), 5, 257, 2),          # the same over more than one pair
])
def test_token_shares_match_exact_oracle(oracle, shape, ctx, M, splits, fused):
    from yasakani_b200 import kv4
    got, want = _run_tc(kv4, oracle, shape, ctx, M, splits, seed=77, fused=fused)
    assert_close(got, want, f"{shape} ctx {ctx} M {M} splits {splits} fused {fused}")


@pytest.mark.parametrize("workspace", [True, False], ids=["workspace", "converting"])
@pytest.mark.parametrize("bf16", [False, True], ids=["fp16", "bf16"])
def test_finished_rows_are_the_rounded_quotients(workspace, bf16):
    """Rows of one split against the same pass in partials and the merge kernel, which divides: equal bits, whatever the values are (ordinary, tiny and
    zero values of both signs, infinities in a cached row), with a bias."""
    import torch
    from yasakani_b200 import kv4
    M, hq, hkv, hd, max_ctx = 70, 8, 2, 128, 128
    dt = torch.bfloat16 if bf16 else torch.float16
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    k, v, q = rnd(M, hkv, hd).to(dt), rnd(M, hkv, hd).to(dt), rnd(M, hq, hd).to(dt)
    v[:20] *= 1e-6
    v[20:24] = 0.0
    v[24:26] = -0.0
    layer = kv4.KvLayer(hkv, hd, max_ctx)
    pos = torch.zeros(1, dtype=torch.int32, device="cuda")
    kv4.launch_kv_append(layer, k, v, pos, M)
    layer.vzero[0, 60:] = float("inf")                            # rows from 60 on sum infinities in the first kv-head
    rope = torch.empty((max_ctx, hd // 2, 2), dtype=torch.float32, device="cuda")
    kv4.launch_rope_table_g(rope, max_ctx, 1e4, hd)
    bv = rnd(hkv, hd).to(dt)
    pm, pl, pacc = kv4.attn_scratch(M, 1, hq, hd)
    ws = kv4.tc_workspace(layer, M) if workspace else None
    a, b = (torch.empty((M, hq, hd), dtype=dt, device="cuda") for _ in range(2))
    kv4.launch_attention_prefill_tc(q, layer, M, pos, 1, pm, pl, pacc, rope, hq, kv4.default_qscale(hd), hd, a, ws, bv=bv)
    kv4.launch_attention_tc(q, layer, M, pos, 1, pm, pl, pacc, rope, hq, kv4.default_qscale(hd), hd, ws)
    kv4.launch_attn_combine_gqa(pm, pl, pacc, 1, M, b, hq, hq // hkv, bv=bv)
    torch.cuda.synchronize()
    assert kv4.device_status() == 0
    same = (a.view(torch.int16) == b.view(torch.int16)) | (torch.isnan(a) & torch.isnan(b))
    assert bool(same.all()), int((~same).sum())


def _same_rows_in_passes_of(widths, ctx, S, workspace, dt, hq, hkv, hd, rd):
    import torch
    from yasakani_b200 import kv4
    top = widths[-1]
    max_ctx = (ctx + top + 63) // 64 * 64
    g = torch.Generator(device="cuda").manual_seed(ctx + S)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16).to(dt)
    k, v, q = rnd(ctx + top, hkv, hd), rnd(ctx + top, hkv, hd), rnd(top, hq, hd)
    layer = kv4.KvLayer(hkv, hd, max_ctx)
    kv4.launch_kv_append(layer, k, v, torch.zeros(1, dtype=torch.int32, device="cuda"), ctx + top)
    rope = torch.empty((max_ctx, rd // 2, 2), dtype=torch.float32, device="cuda")
    kv4.launch_rope_table_g(rope, max_ctx, 1e4, rd)
    pos, first = torch.tensor([ctx], dtype=torch.int32, device="cuda"), None
    for M in widths:
        out = kv4.attn_scratch(M, S, hq, hd)
        kv4.launch_attention_tc(q[:M].contiguous(), layer, M, pos, S, *out, rope, hq, kv4.default_qscale(hd), rd, kv4.tc_workspace(layer, M) if workspace else None)
        torch.cuda.synchronize()
        assert kv4.device_status() == 0
        # the last split ends with the pass, so rows of a narrower pass see its last tiles masked
        bits = [t[:widths[0]].view(torch.int32) for t in out]
        first = first or bits
        for name, a, b in zip(("m", "l", "o"), first, bits):
            assert torch.equal(a, b), f"{name} of {int((a != b).flatten(1).any(1).sum())} of {widths[0]} rows in a pass of {M}"


# Rows 0 .. 49 of a pass from position 246: a wider pass ends behind another key tile, and its pairs of CTAs hold other tokens where they share a pass out evenly.
@pytest.mark.parametrize("workspace,bf16", [(True, False), (True, True), (False, False)], ids=["fp16", "bf16", "converting"])
@pytest.mark.parametrize("ctx,S", [(246, 1), (246, 3), (2030, 5)])
def test_rows_are_the_same_bits_in_passes_of_other_widths(ctx, S, workspace, bf16):
    import torch
    _same_rows_in_passes_of((50, 64, 85, 130), ctx, S, workspace, torch.bfloat16 if bf16 else torch.float16, 24, 4, 256, 64)


@pytest.mark.parametrize("hq,hkv,hd,rd", [(16, 2, 128, 128), (8, 4, 128, 64), (16, 4, 128, 32), (8, 4, 256, 64)])      # eight, two, four heads a kv-head; 256 channels
@pytest.mark.parametrize("ctx", [0, 100])
def test_rows_are_the_same_bits_on_both_sides_of_the_even_shares(ctx, hq, hkv, hd, rd):
    """Converting passes of up to 128 rows share their tokens out evenly, longer ones of 128 channels fill their pairs where a pair is part of a key tile."""
    import torch
    _same_rows_in_passes_of((40, 128, 129, 300), ctx, 2, False, torch.float16, hq, hkv, hd, rd)


@pytest.mark.parametrize("pos", [-200, -16, -9, -3, 190])
@pytest.mark.parametrize("int8", [False, True], ids=["int4", "int8"])
def test_positions_outside_the_cache_are_read_nowhere(int8, pos):
    """A converting pass that begins below position 0, or ends behind the cache: rows without keys leave empty partials, the others equal those of the same
    positions in a pass that lies inside."""
    import torch
    from yasakani_b200 import kv4, kvx
    M, S, nh, kvh, hd, max_ctx = 16, 2, 24, 4, 256, 192
    g = torch.Generator(device="cuda").manual_seed(9)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").half()
    q, k, v = rnd(M, nh, hd), rnd(max_ctx, kvh, hd), rnd(max_ctx, kvh, hd)
    zero = torch.zeros(1, dtype=torch.int32, device="cuda")

    def attend(rows, at, out):
        qq, p = q[rows].contiguous(), torch.tensor([at], dtype=torch.int32, device="cuda")
        m = qq.shape[0]
        if int8:
            kvx.launch_kv8_attention_tc(qq, *arrays, m, p, S, *out, nh)
        else:
            kv4.launch_attention_tc(qq, layer, m, p, S, *out, rope, nh, kv4.default_qscale(hd), 64, None)
    if int8:
        (k8, ks), (v8, vs) = (kvx.encode(x.transpose(0, 1).reshape(-1, hd).float()) for x in (k, v))
        arrays = k8.view(kvh, max_ctx, hd), v8.view(kvh, max_ctx, hd), ks.view(kvh, max_ctx), vs.view(kvh, max_ctx)
    else:
        layer = kv4.KvLayer(kvh, hd, max_ctx)
        kv4.launch_kv_append(layer, k, v, zero, max_ctx)
        rope = torch.empty((max_ctx, 32, 2), dtype=torch.float32, device="cuda")
        kv4.launch_rope_table_g(rope, max_ctx, 1e4, 64)
    out = kv4.attn_scratch(M, S, nh, hd)
    attend(slice(None), pos, out)
    torch.cuda.synchronize()
    assert kv4.device_status() == 0
    empty = [r for r in range(M) if pos + r < 0]
    if empty:
        assert (out[0][empty] == -1e30).all() and (out[1][empty] == 0).all() and (out[2][empty] == 0).all()
    inside = [r for r in range(M) if 0 <= pos + r < max_ctx]
    if inside:
        want = kv4.attn_scratch(len(inside), S, nh, hd)
        attend(slice(inside[0], inside[-1] + 1), max(pos, 0), want)
        torch.cuda.synchronize()
        for a, b in zip(out, want):
            assert torch.isfinite(b).all() and torch.equal(a[inside].view(torch.int32), b.view(torch.int32))
