"""Long passes over INT8 rows from fp16 rows written once (yskn_kv8_attention_ws) against the converting form: equal maxima and sums of
values bit for bit (the sums of weights are grouped differently), at the edges of the row tiles and key tiles, and where no memory may be taken (a stream under capture)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
NH, KVH = 24, 4


def _case(ctx, M, dtype, seed, max_ctx=None):
    g = torch.Generator(device="cuda").manual_seed(seed)
    max_ctx = max_ctx or (ctx + M + 63) // 64 * 64
    k8, v8 = (torch.randint(-127, 128, (KVH, max_ctx, 256), generator=g, device="cuda", dtype=torch.int8) for _ in range(2))
    ks, vs = (torch.rand((KVH, max_ctx), generator=g, device="cuda") * 0.02 + 1e-3 for _ in range(2))
    ks[:, ctx + M:], vs[:, ctx + M:] = float("nan"), float("nan")          # rows that do not exist yet
    q = torch.randn((M, NH, 256), generator=g, device="cuda").to(dtype)
    return q, k8, v8, ks, vs, torch.tensor([ctx], dtype=torch.int32, device="cuda")


def _entry(c, M, S, out, ws=None):
    """The C entries: over a workspace, or converting without one."""
    import ctypes as C
    from yasakani_b200 import _lib
    lib = _lib.load()
    q, k8, v8, ks, vs, pos = c
    a = _lib.Kv8AttnArgsC(q.data_ptr(), k8.data_ptr(), v8.data_ptr(), ks.data_ptr(), vs.data_ptr(), k8.shape[1], M, pos.data_ptr(), S, *(t.data_ptr() for t in out),
                          KVH, NH, 0.0625)
    dt, st = {torch.float16: 0, torch.bfloat16: 1}[q.dtype], torch.cuda.current_stream().cuda_stream
    need = 1024 * KVH * k8.shape[1]
    assert lib.yskn_kv8_workspace_bytes(C.byref(a)) == (need if M >= 384 and need <= 1 << 28 else 0)
    if ws is None:
        return lib.yskn_kv8_attention_tc(C.byref(a), dt, st)
    return lib.yskn_kv8_attention_ws(C.byref(a), dt, ws.data_ptr(), ws.numel(), st)


def _assert_same(a, b, keys):
    (m0, l0, o0), (m1, l1, o1) = a, b
    assert torch.equal(m0.view(torch.int32), m1.view(torch.int32)) and torch.equal(o0.view(torch.int32), o1.view(torch.int32))
    # l: the same positive fp32 weights, added in another order: at most one rounding of 2^-24 per addition on either side
    assert ((l0 - l1).abs() <= 2 * keys * 2.0 ** -24 * l1).all()


# max_ctx None: the cache is full.  Otherwise capacities that the rows leave mostly empty (more and fewer runs of 16 rows than the preparation has
# blocks), and an odd multiple of 64 that ends inside the last key tile.
@pytest.mark.parametrize("ctx,M,S,max_ctx", [(0, 65, 1, None), (0, 128, 2, None), (63, 65, 3, None), (127, 85, 1, None), (1000, 169, 1, None), (3001, 400, 2, None),
                                             (4096, 64, 5, None), (640, 8, 3, None), (100, 400, 1, 65536), (20000, 384, 1, 32832), (0, 384, 1, 448),
                                             (5, 400, 1, 65600)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_partials_equal_the_converting_form(ctx, M, S, max_ctx, dtype):
    from yasakani_b200 import kv4
    c = _case(ctx, M, dtype, seed=ctx + M, max_ctx=max_ctx)
    ws = torch.full((1024 * KVH * c[1].shape[1],), 0xFF, dtype=torch.uint8, device="cuda")     # fp16 NaN wherever nothing is written
    outs = []
    for w in (ws, None):
        out = [torch.full_like(t, float("nan")) for t in kv4.attn_scratch(M, S, NH, 256)]
        assert _entry(c, M, S, out, w) == 0
        outs.append(out)
    assert torch.isfinite(outs[0][2]).all() and kv4.device_status() == 0
    _assert_same(*outs, ctx + M)
    assert _entry(c, M, S, outs[0], ws[:-16]) == -1 and _entry(c, M, S, outs[0], ws[8:]) == -1


def test_other_stream_and_capture_give_the_same_rows():
    from yasakani_b200 import kv4, kvx
    M, S, c = 400, 1, _case(500, 400, torch.bfloat16, seed=3)
    want = kv4.attn_scratch(M, S, NH, 256)
    kvx.launch_kv8_attention(*c[:5], M, c[5], S, *want, NH)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    got = kv4.attn_scratch(M, S, NH, 256)
    kvx.launch_kv8_attention(*c[:5], M, c[5], S, *got, NH, stream=side)
    side.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    graphed = kv4.attn_scratch(M, S, NH, 256)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        kvx.launch_kv8_attention(*c[:5], M, c[5], S, *graphed, NH)
    graph.replay()
    torch.cuda.synchronize()
    _assert_same(want, graphed, 900)                                       # the converting form


def test_cost_does_not_grow_with_the_capacity():
    """400 rows at the start of a cache: time over a workspace in a cache of 65,536 tokens against one that is full (before the preparation's grid was
    bounded 52 against 19 us), and no memory taken for a cache whose workspace would be larger than 256 MiB."""
    from yasakani_b200 import kv4, kvx
    M, times = 400, []
    for max_ctx in (448, 65536):
        c = _case(0, M, torch.bfloat16, seed=1, max_ctx=max_ctx)
        out, ws = kv4.attn_scratch(M, 1, NH, 256), torch.empty(1024 * KVH * max_ctx, dtype=torch.uint8, device="cuda")
        best = float("inf")
        for _ in range(10):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(20):
                _entry(c, M, 1, out, ws)
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b) / 20)
        times.append(best)
    assert times[1] < 1.4 * times[0], times
    del ws
    for max_ctx, most in ((65536, 1 << 28), (131072, 0)):
        c, out = _case(0, M, torch.bfloat16, seed=1, max_ctx=max_ctx), kv4.attn_scratch(M, 1, NH, 256)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        kvx.launch_kv8_attention(*c[:5], M, c[5], 1, *out, NH)
        assert torch.cuda.max_memory_allocated() - before <= most
        assert torch.cuda.memory_allocated() == before                     # given back when the call returns


def test_scratch_is_no_tensor_and_no_part_of_another_streams_capture():
    """The scratch of a launch is seen by no dispatch mode (nor filled in deterministic mode), and it may be taken while another stream is under
    capture in global mode, where an ordinary allocation would end the capture with an error."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from yasakani_b200 import kv4, kvx

    class Ops(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(func)
            return func(*args, **(kwargs or {}))

    M, c = 400, _case(300, 400, torch.bfloat16, seed=5)
    want, got, x = kv4.attn_scratch(M, 1, NH, 256), kv4.attn_scratch(M, 1, NH, 256), torch.ones(1000, device="cuda")
    with Ops():
        kvx.launch_kv8_attention(*c[:5], M, c[5], 1, *want, NH)
    assert not Ops.seen, Ops.seen
    torch.cuda.synchronize()
    torch.cuda.empty_cache()                                               # the next scratch is not in the cache
    other, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):                                          # global mode: the strictest
        x *= 2
        kvx.launch_kv8_attention(*c[:5], M, c[5], 1, *got, NH, stream=other)
    other.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(want, got)) and kv4.device_status() == 0
    graph.replay()
    torch.cuda.synchronize()
    assert (x == 2).all()


@pytest.mark.parametrize("ctx,S", [(246, 1), (246, 3), (2030, 5)])
@pytest.mark.parametrize("written", [True, False], ids=["written", "converting"])
def test_rows_are_the_same_bits_in_passes_of_other_widths(written, ctx, S):
    """Rows 0 .. 49 of passes that end behind other key tiles and share their rows out over other pairs of CTAs."""
    from yasakani_b200 import kv4
    q, k8, v8, ks, vs, pos = _case(ctx, 130, torch.bfloat16, seed=5)
    ws = torch.full((1024 * KVH * k8.shape[1],), 0xFF, dtype=torch.uint8, device="cuda") if written else None
    first = None
    for M in (50, 64, 85, 130):
        out = kv4.attn_scratch(M, S, NH, 256)
        assert _entry((q[:M].contiguous(), k8, v8, ks, vs, pos), M, S, out, ws) == 0
        torch.cuda.synchronize()
        bits = [t[:50].view(torch.int32) for t in out]
        first = first or bits
        assert kv4.device_status() == 0 and all(torch.equal(a, b) for a, b in zip(first, bits)), M
