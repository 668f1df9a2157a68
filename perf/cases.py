"""Performance cases: what a program that uses this library has it do, from one decode step of a small layer to a full prefill.

Every pass goes through the public Python entry points (`yasakani_b200.kv4`, `yasakani_b200.kvx`), eagerly, on the current
stream.  The shapes are those of the repository's own configurations, tests and benchmark; cache contents are seeded N(0, 1)
rows with log-uniform key channel scales, quantised by the library's own codecs.

  kinds   decode    append M rows (1 .. 8) to the packed int4 cache, attend with them, merge          (token generation, short drafts)
          verify    the same with 9 .. 64 rows                                                          (speculative / wide-copy verification)
          prefill   append M rows, dequantise into the kept workspace, attend                           (a prompt, or a chunk of one)
          batch     one row of each of several sequences in one launch, merge                           (batched token generation)
          int8      row epilogue (norm, RoPE, rotation, INT8 append), attention over INT8 rows, merge   (Family B: decode and prefill chunks)
          packed    attention straight over trellis-packed rows, merge                                  (Family B, packed cache)
          trellis   pack rows (trellis search) and unpack them again                                    (Family B, packed cache: both directions)
"""
import math

import torch

from yasakani_b200 import kv4, kvx

SMS = 148                                   # one block per SM when splits * kv-heads = 148
INT8_SHAPE = dict(hq=24, hkv=4, hd=256, rd=64, theta=1e7)
BLOB = "tests/golden/kvqp_synthetic.bin"    # synthetic trellis profile of the repository


def _kv4(kind, name, ctx, rows, dtype, hq=24, hkv=4, hd=256, rd=64, theta=1e7, bias=False):
    c = dict(kind=kind, ctx=ctx, rows=rows, dtype=dtype, hq=hq, hkv=hkv, hd=hd, rd=rd, theta=theta, bias=bias)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one token of a small layer (head_dim 128, with a value bias) at a short context: latency and launches
        _kv4("decode", "decode_hd128_4k", 4096, 1, "f16", hq=16, hkv=2, hd=128, rd=128, theta=1e6, bias=True),
        # one token of the 27B-class layer at an everyday context, with that engine's bf16 activations
        _kv4("decode", "decode_27b_32k", 32768, 1, "bf16"),
        # one token at the longest context: the packed cache is streamed once
        _kv4("decode", "decode_27b_262k", 262144, 1, "f16"),
        # a short draft checked in one pass, at a position that is on no boundary
        _kv4("decode", "draft_5_rows_20k", 20011, 5, "bf16"),
        # speculative verification, narrow and wide
        _kv4("verify", "verify_16_rows_32k", 32768, 16, "f16"),
        _kv4("verify", "verify_64_rows_32k", 32768, 64, "bf16"),
        # a whole prompt: codec, dequantisation, causal attention
        _kv4("prefill", "prefill_8192_rows", 0, 8192, "f16"),
        # token generation for eight users at mixed contexts, one launch
        dict(kind="batch", name="decode_batch_8", contexts="2048,4096,8192,16384,32768,65536,98304,131072", dtype="f16"),
        # Family B: one token over an INT8 cache, gated output
        dict(kind="int8", name="int8_decode_32k", ctx=32768, rows=1),
        # Family B: a ragged chunk of a prompt behind a cached prefix
        dict(kind="int8", name="int8_prefill_1000_rows", ctx=3001, rows=1000),
        # Family B, packed cache: one token, odd length
        dict(kind="packed", name="packed_decode_30k", ctx=30011, rows=1, layer=0),
        # Family B, packed cache: rows of a prompt chunk go in and come back
        dict(kind="trellis", name="trellis_rows_4096", rows=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "verify", "prefill", "batch", "int8", "int8", "packed", "trellis"])
    dtype = rng.choice(["f16", "bf16"])
    if kind == "decode":
        rows = rng.choice([1, 1, 1, 2, 3, 4, 6, 8])
        ctx = _log(rng, 500, 262144) // rows + 1
        if rng.random() < 0.3:
            hq, hkv = rng.choice([(16, 2), (28, 4)])
            return _kv4(kind, None, ctx, rows, dtype, hq=hq, hkv=hkv, hd=128, rd=128, theta=1e6, bias=rng.random() < 0.5)
        return _kv4(kind, None, ctx, rows, dtype)
    if kind == "verify":
        return _kv4(kind, None, _log(rng, 500, 32768), rng.randint(9, 64), dtype)
    if kind == "prefill":
        ctx = rng.choice([0, rng.randint(1, 6000)])
        return _kv4(kind, None, ctx, _log(rng, 100, 8192 - ctx), dtype)
    if kind == "batch":
        return dict(kind=kind, contexts=",".join(str(_log(rng, 500, 60000)) for _ in range(rng.randint(2, 12))), dtype=dtype)
    if kind == "int8":
        if rng.random() < 0.5:
            rows = rng.choice([1, 1, 2, 4])
            return dict(kind=kind, ctx=_log(rng, 500, 131072) // rows + 1, rows=rows)
        return dict(kind=kind, ctx=rng.randint(0, 6000), rows=_log(rng, 16, 1500))
    if kind == "packed":
        return dict(kind=kind, ctx=_log(rng, 500, 32768), rows=rng.choice([1, 1, 2]), layer=rng.randrange(16))
    return dict(kind=kind, rows=_log(rng, 8, 4096))


# ---------------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _dtype(case):
    return torch.float16 if case["dtype"] == "f16" else torch.bfloat16


def _rows(g, n, heads, hd, dtype, scale=None):
    x = torch.randn((n, heads, hd), generator=g, device="cuda")
    return (x if scale is None else x * scale).to(torch.bfloat16).to(dtype)


def _channel_scale(g, heads, hd):
    lo, hi = math.log(0.5), math.log(4.0)
    return torch.exp(torch.rand((heads, hd), generator=g, device="cuda") * (hi - lo) + lo)


def _splits(rows, hq, hkv):
    """How many ways a caller cuts the keys: one block per SM for a few rows, one block pair per SM pair for many."""
    if rows <= 8:
        return SMS // hkv
    tokens = 128 // (hq // hkv)                                  # tokens of one 128-row tile
    pairs = (-(-rows // tokens) + 1) // 2
    return max(1, SMS // 2 // (pairs * hkv))


def _pos(p):
    return torch.tensor([p], dtype=torch.int32, device="cuda")


def _rope(max_ctx, theta, rd):
    rope = torch.empty((max_ctx, rd // 2, 2), dtype=torch.float32, device="cuda")
    kv4.launch_rope_table_g(rope, max_ctx, theta, rd)
    return rope


def _cache(g, hkv, hd, n, max_ctx, scale, chunk=16384):
    layer = kv4.KvLayer(hkv, hd, max_ctx)
    for p in range(0, n, chunk):
        m = min(chunk, n - p)
        kv4.launch_kv_append(layer, _rows(g, m, hkv, hd, torch.float16, scale), _rows(g, m, hkv, hd, torch.float16), _pos(p), m)
    return layer


def _prepare_kv4(case, seed):
    g, dt = _gen(seed), _dtype(case)
    ctx, M, hq, hkv, hd, rd = (case[k] for k in ("ctx", "rows", "hq", "hkv", "hd", "rd"))
    max_ctx = (ctx + M + 127) // 64 * 64
    scale = _channel_scale(g, hkv, hd)
    s = dict(kind=case["kind"], M=M, nh=hq, rd=rd, qscale=kv4.default_qscale(hd), splits=_splits(M, hq, hkv), pos=_pos(ctx), ctx=ctx)
    s["layer"] = _cache(g, hkv, hd, ctx, max_ctx, scale)
    s["k"], s["v"], s["q"] = _rows(g, M, hkv, hd, dt, scale), _rows(g, M, hkv, hd, dt), _rows(g, M, hq, hd, dt)
    s["bv"] = torch.randn((hkv, hd), generator=g, device="cuda").to(dt) if case["bias"] else None
    s["rope"] = _rope(max_ctx, case["theta"], rd)
    s["pm"], s["pl"], s["pacc"] = kv4.attn_scratch(M, s["splits"], hq, hd)
    s["o16"] = torch.empty((M, hq, hd), dtype=dt, device="cuda")
    if case["kind"] == "prefill":
        s["ws"] = kv4.tc_workspace(s["layer"], M)
        if ctx:                                                  # the prefix was dequantised when it was appended
            kv4.launch_kv_append(s["layer"], s["k"], s["v"], s["pos"], M)
            _prefill(s, 0)
    return s


def _prepare_batch(case, seed):
    g, dt = _gen(seed), _dtype(case)
    ctxs = [int(x) for x in case["contexts"].split(",")]
    hq, hkv, hd, rd, theta = (INT8_SHAPE[k] for k in ("hq", "hkv", "hd", "rd", "theta"))
    max_ctx, M, splits = (max(ctxs) + 127) // 64 * 64, len(ctxs), 19
    layers = [_cache(g, hkv, hd, n, max_ctx, _channel_scale(g, hkv, hd)) for n in ctxs]
    s = dict(kind="batch", M=M, nh=hq, g=hq // hkv, rd=rd, qscale=kv4.default_qscale(hd), splits=splits, slots=kv4.MsSlots(layers),
             pos=torch.tensor([n - 1 for n in ctxs], dtype=torch.int32, device="cuda"), slot=torch.arange(M, dtype=torch.int32, device="cuda"),
             q=_rows(g, M, hq, hd, dt), rope=_rope(max_ctx, theta, rd), o16=torch.empty((M, hq, hd), dtype=dt, device="cuda"))
    s["pm"], s["pl"], s["pacc"] = kv4.attn_scratch(M, splits, hq, hd)
    return s


def _prepare_int8(case, seed):
    g, bf = _gen(seed), torch.bfloat16
    ctx, M = case["ctx"], case["rows"]
    nh, kvh, rd = INT8_SHAPE["hq"], INT8_SHAPE["hkv"], INT8_SHAPE["rd"]
    max_ctx = (ctx + M + 127) // 64 * 64
    s = dict(kind="int8", M=M, nh=nh, rd=rd, splits=_splits(M, nh, kvh), pos=_pos(ctx), rope=_rope(max_ctx, INT8_SHAPE["theta"], rd))
    s["q_rows"] = _rows(g, M, nh, 512, bf)
    s["k_rows"], s["v_rows"] = _rows(g, M, kvh, 256, bf, _channel_scale(g, kvh, 256)), _rows(g, M, kvh, 256, bf)
    s["qn_w"], s["kn_w"] = ((torch.randn(256, generator=g, device="cuda") * 0.2 + b).to(bf) for b in (0.0, 0.5))
    for n, sc in (("k", _channel_scale(g, kvh, 256)[:, None]), ("v", None)):
        x = torch.randn((kvh, max_ctx, 256), generator=g, device="cuda")
        q8, scales = kvx.encode((x if sc is None else x * sc).view(-1, 256))
        s[n + "8"], s[n + "s"] = q8.view(kvh, max_ctx, 256), scales.view(kvh, max_ctx)
    s["q16"], s["gate16"], s["o16"] = (torch.empty((M, nh, 256), dtype=bf, device="cuda") for _ in range(3))
    s["pm"], s["pl"], s["pacc"] = kv4.attn_scratch(M, s["splits"], nh, 256)
    return s


def _profile():
    with open(BLOB, "rb") as f:
        return kvx.TrellisProfile(f.read())


def _prepare_packed(case, seed):
    g, ctx, M = _gen(seed), case["ctx"], case["rows"]
    nh, kvh = INT8_SHAPE["hq"], INT8_SHAPE["hkv"]
    max_ctx = (ctx + M + 127) // 64 * 64
    s = dict(kind="packed", M=M, nh=nh, splits=SMS // kvh, pos=_pos(ctx), prof=_profile())
    first = 8 * case["layer"]                                    # the profile's records of one layer: (key, value) of four kv-heads
    rows_pos = torch.arange(max_ctx, dtype=torch.int32, device="cuda").repeat(kvh)
    for n, kind in (("k", 0), ("v", 1)):
        x = torch.randn((kvh * max_ctx, 256), generator=g, device="cuda")
        s["grp_" + n] = first + 2 * torch.arange(kvh, dtype=torch.int32, device="cuda") + kind
        _, pay, side = kvx.tb_encode(s["prof"], x, s["grp_" + n].repeat_interleave(max_ctx).contiguous(), rows_pos)
        s[n + "_pay"], s[n + "_side"], s[n + "_plain"] = pay.view(kvh, max_ctx, -1), side.view(kvh, max_ctx, 2), x.view(kvh, max_ctx, 256)
    s["q"] = _rows(g, M, nh, 256, torch.bfloat16)
    s["o16"] = torch.empty((M, nh, 256), dtype=torch.bfloat16, device="cuda")
    s["pm"], s["pl"], s["pacc"] = kv4.attn_scratch(M, s["splits"], nh, 256)
    return s


def _prepare_trellis(case, seed):
    g, n = _gen(seed), case["rows"]
    x = torch.randn((n, 256), generator=g, device="cuda") * torch.exp(0.5 * torch.randn((n, 1), generator=g, device="cuda"))
    return dict(kind="trellis", prof=_profile(), x=x, grp=torch.randint(0, 128, (n,), generator=g, device="cuda", dtype=torch.int32),
                pos=torch.arange(n, dtype=torch.int32, device="cuda"))


def prepare(case, seed):
    f = {"batch": _prepare_batch, "int8": _prepare_int8, "packed": _prepare_packed, "trellis": _prepare_trellis}
    return f.get(case["kind"], _prepare_kv4)(case, seed)


# ---------------------------------------------------------------------------------------------------------------- one pass
def _prefill(s, valid):
    kv4.launch_attention_prefill_tc(s["q"], s["layer"], s["M"], s["pos"], s["splits"], s["pm"], s["pl"], s["pacc"], s["rope"], s["nh"], s["qscale"],
                                    s["rd"], s["o16"], s["ws"], bv=s["bv"], valid_tokens=valid)


def run(s):
    kind = s["kind"]
    if kind in ("decode", "verify", "prefill"):
        kv4.launch_kv_append(s["layer"], s["k"], s["v"], s["pos"], s["M"])
        if kind == "prefill":
            _prefill(s, s["ctx"])
        else:
            kv4.launch_decode(s["q"], s["layer"], s["M"], s["pos"], s["splits"], s["pm"], s["pl"], s["pacc"], s["rope"], s["nh"], s["qscale"], s["rd"],
                              s["o16"], bv=s["bv"])
        return [s["o16"]] + s["layer"].tensors()
    if kind == "batch":
        kv4.launch_attention_ms(s["q"], s["slots"], s["M"], s["pos"], s["slot"], s["splits"], s["pm"], s["pl"], s["pacc"], s["rope"], s["nh"],
                                s["qscale"], s["rd"])
        kv4.launch_attn_combine_gqa(s["pm"], s["pl"], s["pacc"], s["splits"], s["M"], s["o16"], s["nh"], s["g"])
        return s["o16"]
    if kind == "int8":
        kvx.launch_attn_post(s["q_rows"], s["k_rows"], s["v_rows"], s["qn_w"], s["kn_w"], 1e-6, s["pos"], s["rope"], s["rd"], s["q16"], s["gate16"],
                             s["k8"], s["ks"], s["v8"], s["vs"])
        kvx.launch_kv8_attention(s["q16"], s["k8"], s["v8"], s["ks"], s["vs"], s["M"], s["pos"], s["splits"], s["pm"], s["pl"], s["pacc"], s["nh"])
        kvx.launch_kv8_combine(s["pm"], s["pl"], s["pacc"], s["splits"], s["M"], s["nh"], s["o16"], gate=s["gate16"])
        return [s[k] for k in ("o16", "q16", "gate16", "k8", "ks", "v8", "vs")]
    if kind == "packed":
        kvx.launch_tb_attention(s["prof"], s["q"], s["k_pay"], s["k_side"], s["v_pay"], s["v_side"], s["grp_k"], s["grp_v"], s["M"], s["pos"],
                                s["splits"], s["pm"], s["pl"], s["pacc"], s["nh"], k_plain=s["k_plain"], v_plain=s["v_plain"])
        kvx.launch_kv8_combine(s["pm"], s["pl"], s["pacc"], s["splits"], s["M"], s["nh"], s["o16"])
        return s["o16"]
    y, pay, side = kvx.tb_encode(s["prof"], s["x"], s["grp"], s["pos"])
    return [y, pay, side, kvx.tb_decode(s["prof"], pay, side, s["grp"], s["pos"], yin=s["x"])]


# ---------------------------------------------------------------------------------------------------------------- what a pass cannot do without
def _kv4_bytes(keys, hkv, hd):
    """Packed keys and values of `keys` tokens: int4 codes, value scale and zero per token, key scales and zeros per 32-token group."""
    return hkv * (keys * (hd + 4) + (keys + 31) // 32 * hd * 4)


def work(case):
    kind = case["kind"]
    if kind == "trellis":
        n = case["rows"]
        # fp32 row in (twice: packing, and the rows that stay unpacked), row out twice, payload and side words; the search: 5 scale
        # multipliers x 256 values x 256 states, one squared difference and one addition each
        return {"bytes": n * (3 * 1024 + 2 * (128 + 8)), "flops": n * 5 * 256 * 256 * 3}
    hq, hkv, hd = (case.get(k, INT8_SHAPE[k]) for k in ("hq", "hkv", "hd"))
    if kind == "batch":
        ctxs = [int(x) for x in case["contexts"].split(",")]
        return {"bytes": sum(_kv4_bytes(n, hkv, hd) for n in ctxs) + 4 * len(ctxs) * hq * hd, "flops": 4 * hd * hq * sum(ctxs)}
    M, ctx = case["rows"], case["ctx"]
    pairs = M * ctx + M * (M + 1) // 2                           # (row, visible key)
    io = M * 4 * hq * hd                                         # queries in, rows out, 16 bits each
    if kind == "int8":
        # key and value rows with their scales; projection rows in, rotated queries and gates out
        return {"bytes": 2 * hkv * (ctx + M) * 260 + M * (hq * (1024 + 512 + 512 + 512) + 2 * hkv * 512), "flops": 4 * hd * hq * pairs}
    if kind == "packed":
        return {"bytes": 2 * hkv * (ctx + M) * (128 + 8) + io, "flops": 4 * hd * hq * pairs}
    # the cached prefix, the new rows in (keys, values) and their fp16 shadow out
    return {"bytes": _kv4_bytes(ctx + M, hkv, hd) + M * hkv * hd * 6 + io, "flops": 4 * hd * hq * pairs}


def tolerance(case):
    kind = case["kind"]
    if kind == "trellis":
        return "exact"                                           # a search over integers: every byte
    if kind in ("int8", "packed") or case["dtype"] == "bf16":
        return {"rel": 1e-2}                                     # bf16 rows out; bytes of the cache stay equal
    return {"rel": 5e-3}                                         # fp16 operands and rows
