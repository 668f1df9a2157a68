"""Steps back to back without a synchronisation against the same steps with one behind every launch, bit for bit: every launch of a chain may start
while the one in front of it still writes, so positions, rows, scales, group codes, workspaces and partials are all read close behind their writer."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NH, KVH, HD, RD = 24, 4, 256, 64


def _positions(first, steps, rows):
    return [torch.tensor([first + s * rows], dtype=torch.int32, device="cuda") for s in range(steps)]


def _rope(max_ctx):
    from yasakani_b200 import kv4
    rope = torch.empty((max_ctx, RD // 2, 2), dtype=torch.float32, device="cuda")
    kv4.launch_rope_table_g(rope, max_ctx, 1e7, RD)
    return rope


def _same(run):
    """run(sync) -> list of tensors; sync() is called behind every launch."""
    want = run(torch.cuda.synchronize)
    for _ in range(3):
        got = run(lambda: None)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(want, got))


@pytest.mark.parametrize("first,rows,steps,splits", [(0, 1, 80, 37), (700, 1, 40, 37), (200, 12, 20, 6), (64, 400, 4, 1)])
def test_int8_steps(first, rows, steps, splits):
    from yasakani_b200 import kv4, kvx
    max_ctx, bf = (first + rows * steps + 63) // 64 * 64, torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(first + rows)
    rnd = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(bf)
    q, k, v, w = rnd(steps, rows, NH, 512), rnd(steps, rows, KVH, 256), rnd(steps, rows, KVH, 256), rnd(2, 256)
    k0, v0 = (torch.randint(-127, 128, (KVH, max_ctx, 256), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    s0 = torch.rand((2, KVH, max_ctx), generator=g, device="cuda") * 0.02 + 1e-3
    pos, rope = _positions(first, steps, rows), _rope(max_ctx)
    q16, gate = (torch.empty((rows, NH, 256), dtype=bf, device="cuda") for _ in range(2))
    pm, pl, pacc = kv4.attn_scratch(rows, splits, NH, 256)

    def run(sync):
        k8, v8, (ks, vs) = k0.clone(), v0.clone(), s0.clone()
        out = torch.zeros((steps, rows, NH, 256), dtype=bf, device="cuda")
        torch.cuda.synchronize()
        for s in range(steps):
            kvx.launch_attn_post(q[s], k[s], v[s], w[0], w[1], 1e-6, pos[s], rope, RD, q16, gate, k8, ks, v8, vs)
            sync()
            kvx.launch_kv8_attention(q16, k8, v8, ks, vs, rows, pos[s], splits, pm, pl, pacc, NH)
            sync()
            kvx.launch_kv8_combine(pm, pl, pacc, splits, rows, NH, out[s], gate=gate)
            sync()
        return [out, k8, v8, ks, vs]

    _same(run)


@pytest.mark.parametrize("first,rows,steps,splits,form", [(0, 1, 100, 37, "decode"), (5000, 1, 70, 37, "early"), (90, 5, 20, 37, "decode"), (300, 24, 10, 6, "decode"),
                                                          (100, 70, 6, 3, "workspace"), (0, 300, 3, 1, "workspace")])
def test_int4_steps(first, rows, steps, splits, form):
    from yasakani_b200 import kv4
    max_ctx = (first + rows * steps + 127) // 64 * 64
    g = torch.Generator(device="cuda").manual_seed(first + rows)
    rnd = lambda *shape: torch.randn(shape, generator=g, device="cuda").half()
    q, k, v = rnd(steps, rows, NH, HD), rnd(steps, rows, KVH, HD), rnd(steps, rows, KVH, HD)
    pos, rope, qscale = _positions(first, steps, rows), _rope(max_ctx), kv4.default_qscale(HD)
    prefix = rnd(2, max(first, 1), KVH, HD)
    ext = kv4.attn_ext(early=True) if form == "early" else None
    pm, pl, pacc = kv4.attn_scratch(rows, splits, NH, HD)

    def run(sync):
        layer = kv4.KvLayer(KVH, HD, max_ctx)
        if first:
            kv4.launch_kv_append(layer, prefix[0], prefix[1], torch.zeros(1, dtype=torch.int32, device="cuda"), first)
        ws = kv4.tc_workspace(layer, rows) if form == "workspace" else None
        out = torch.zeros((steps, rows, NH, HD), dtype=torch.float16, device="cuda")
        torch.cuda.synchronize()
        for s in range(steps):
            kv4.launch_kv_append(layer, k[s], v[s], pos[s], rows)
            sync()
            if form == "workspace":
                kv4.launch_attention_prefill_tc(q[s], layer, rows, pos[s], splits, pm, pl, pacc, rope, NH, qscale, RD, out[s], ws,
                                                valid_tokens=first + s * rows if s else 0)
            else:
                kv4.launch_decode(q[s], layer, rows, pos[s], splits, pm, pl, pacc, rope, NH, qscale, RD, out[s], ext=ext)
            sync()
        assert kv4.device_status() == 0
        return [out] + layer.tensors()

    _same(run)
