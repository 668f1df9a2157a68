"""Decode grids of more blocks than the GPU holds at once run as a queue of items: every (row, split, head) has to come out as in a launch
that fits, bit for bit, whatever block computed it -- items without keys, with the open group only, with one unit and with more units
than the ring holds; rows of one sequence and rows of several, in any order of length."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cache(kv4, hkv, hd, n, max_ctx, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    layer = kv4.KvLayer(hkv, hd, max_ctx)
    rows = [torch.randn((n, hkv, hd), generator=g, device="cuda").to(torch.float16) for _ in range(2)]
    kv4.launch_kv_append(layer, *rows, torch.zeros(1, dtype=torch.int32, device="cuda"), n)
    return layer


def _shape(kv4, hd, max_ctx):
    hq, hkv, rd = (24, 4, 64) if hd == 256 else (16, 2, 128)
    rope = torch.empty((max_ctx, rd // 2, 2), dtype=torch.float32, device="cuda")
    kv4.launch_rope_table_g(rope, max_ctx, 1e6, rd)
    return hq, hkv, rd, rope


def _bits(pm, pl, pacc):
    return [t.view(torch.int32) for t in (pm, pl, pacc)]


@pytest.mark.parametrize("hd,dtype", [(256, torch.float16), (256, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("pos,M,S", [(0, 8, 37), (31, 5, 37), (126, 4, 37), (700, 2, 74), (2049, 8, 19), (9000, 8, 37), (9000, 3, 30), (9000, 1, 160)])
def test_rows_of_one_sequence_equal_their_own_launches(hd, dtype, pos, M, S):
    from yasakani_b200 import kv4
    max_ctx = 9088
    hq, hkv, rd, rope = _shape(kv4, hd, max_ctx)
    layer = _cache(kv4, hkv, hd, pos + M, max_ctx, seed=pos + M)
    q = torch.randn((M, hq, hd), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda").to(dtype)
    kv4.set_algo(2)                                                # one row and S > 148 / hkv splits: the tensor-core kernel as well
    try:
        def launch(qr, m, p, s):
            out = [torch.full_like(t, float("nan")) for t in kv4.attn_scratch(m, s, hq, hd)]
            kv4.launch_attention_gqa(qr, layer, m, torch.tensor([p], dtype=torch.int32, device="cuda"), s, *out, rope, hq, kv4.default_qscale(hd), rd)
            return out
        got = launch(q, M, pos, S)
        assert torch.isfinite(got[2]).all()
        again = launch(q, M, pos, S)
        assert all(torch.equal(a, b) for a, b in zip(_bits(*got), _bits(*again)))
        if S * hkv <= 148:
            for r in range(M):
                one = launch(q[r:r + 1].contiguous(), 1, pos + r, S)
                assert all(torch.equal(a[r], b[0]) for a, b in zip(_bits(*got), _bits(*one))), f"row {r}"
        else:                                                       # no launch of this split count fits: the merged row against one that does
            o = [torch.empty((M, hq, hd), dtype=dtype, device="cuda") for _ in range(2)]
            kv4.launch_attn_combine_gqa(*got, S, M, o[0], hq, hq // hkv)
            kv4.launch_attn_combine_gqa(*launch(q, M, pos, 37), 37, M, o[1], hq, hq // hkv)
            # the split count changes the grouping of fp32 sums and the lag of the running maximum (fp16 weights, 2^-11 each way)
            assert torch.allclose(o[0].float(), o[1].float(), rtol=2 ** -7, atol=2e-3)
    finally:
        kv4.set_algo(0)
    assert kv4.device_status() == 0


@pytest.mark.parametrize("hd", [256, 128])
@pytest.mark.parametrize("ctxs,S", [((5000, 1, 128, 3000, 5000, 33, 700, 9000), 19), (tuple(range(1, 641, 10)), 7), ((9000,) * 9, 5)])
def test_rows_of_several_sequences_equal_their_own_launches(hd, ctxs, S):
    from yasakani_b200 import kv4
    max_ctx = 9088
    hq, hkv, rd, rope = _shape(kv4, hd, max_ctx)
    kinds = sorted(set(ctxs))[:12]
    layers = {n: _cache(kv4, hkv, hd, n, max_ctx, seed=n) for n in kinds}
    ctxs = [n if n in layers else kinds[i % len(kinds)] for i, n in enumerate(ctxs)]
    M = len(ctxs)
    slots = kv4.MsSlots([layers[n] for n in kinds])
    pos = torch.tensor([n - 1 for n in ctxs], dtype=torch.int32, device="cuda")
    slot = torch.tensor([kinds.index(n) for n in ctxs], dtype=torch.int32, device="cuda")
    q = torch.randn((M, hq, hd), generator=torch.Generator(device="cuda").manual_seed(9), device="cuda").to(torch.float16)
    got = [torch.full_like(t, float("nan")) for t in kv4.attn_scratch(M, S, hq, hd)]
    kv4.launch_attention_ms(q, slots, M, pos, slot, S, *got, rope, hq, kv4.default_qscale(hd), rd)
    for r in {0, 1, M // 2, M - 2, M - 1}:
        one = kv4.attn_scratch(1, S, hq, hd)
        kv4.launch_attention_gqa(q[r:r + 1].contiguous(), layers[ctxs[r]], 1, pos[r:r + 1].contiguous(), S, *one, rope, hq, kv4.default_qscale(hd), rd)
        assert all(torch.equal(a[r], b[0]) for a, b in zip(_bits(*got), _bits(*one))), f"row {r} of {M}"
    assert torch.isfinite(got[2]).all() and kv4.device_status() == 0
