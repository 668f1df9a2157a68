"""The KV4 merge against double precision on both sides of the line between its two forms (many rows x heads take a warp each): one split,
the edges of a batch of loads and of a warp's lanes of weights, empty splits, bias and gate, a partial buffer that is aligned for no wide load."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,nh,g,hd", [(12, 24, 6, 256), (13, 24, 6, 256), (64, 24, 6, 256), (300, 16, 8, 128), (80, 4, 2, 64)])
@pytest.mark.parametrize("S", [1, 7, 8, 9, 18, 32, 33, 41])
@pytest.mark.parametrize("dtype,shift", [(torch.bfloat16, 0), (torch.float16, 0), (torch.float16, 1)])
def test_merge_matches_double_precision(M, nh, g, hd, S, dtype, shift):
    from yasakani_b200 import kv4
    gen = torch.Generator(device="cuda").manual_seed(M * 100 + S)
    pm = torch.randn((M, S, nh), generator=gen, device="cuda") * 3
    if S > 1:
        pm[:, S // 2] = -1e30                                  # an empty split
    pl = torch.rand((M, S, nh), generator=gen, device="cuda") * 50 + 1
    pacc = torch.randn((M, S, nh, hd), generator=gen, device="cuda") * pl[..., None]
    gate, bv = (torch.randn(s, generator=gen, device="cuda").to(dtype) for s in ((M, nh, hd), (nh // g, hd)))
    buf = torch.empty(pacc.numel() + shift, device="cuda")
    buf[shift:] = pacc.view(-1)
    o16 = torch.empty((M, nh, hd), dtype=dtype, device="cuda")
    kv4.launch_attn_combine_gqa(pm, pl, buf[shift:].view(pacc.shape), S, M, o16, nh, g, bv=bv, gate=gate)
    w = torch.exp(pm.double() - pm.double().amax(1, keepdim=True)) * (pm > -1e29)
    bare = ((w[..., None] * pacc.double()).sum(1) / (w * pl.double()).sum(1)[..., None]).to(torch.float16).double()
    want = (bare + bv.double().repeat_interleave(g, 0)) * torch.sigmoid(gate.double())
    # the row before the bias may fall to the other side of an fp16 tie: one ulp, 2^-10 of it (2^-24 among subnormals); the result is rounded to its own
    # type: half an ulp, 2^-11 or 2^-8 of the value; fp32 arithmetic between the two is far below either
    bound = bare.abs() * 2.0 ** -10 + want.abs() * (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01 + 1e-6
    assert ((o16.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("M", [19, 37, 38])                       # 304, 592 and 608 rows x heads: with more than 20 splits a warp each from 593 on
@pytest.mark.parametrize("S", [20, 21, 37])
def test_merge_on_both_sides_of_the_line_for_128_channels(M, S):
    test_merge_matches_double_precision(M, 16, 8, 128, S, torch.float16, 0)


@pytest.mark.parametrize("M", [6, 7])                             # 144 and 168 rows x heads: with up to 20 splits a warp each from 149 on
@pytest.mark.parametrize("S", [1, 20, 21, 37])
def test_merge_on_both_sides_of_the_line_for_256_channels(M, S):
    test_merge_matches_double_precision(M, 24, 6, 256, S, torch.bfloat16, 0)


@pytest.mark.parametrize("M,nh", [(1, 16), (9, 16), (10, 16)])    # 16, 144 and 160 rows x heads: eight runs of splits up to 148
@pytest.mark.parametrize("S", [40, 41, 74, 81, 160])
def test_merge_of_many_splits_in_eight_runs(M, nh, S):
    test_merge_matches_double_precision(M, nh, 8, 128, S, torch.float16, 0)


@pytest.mark.parametrize("M,nh", [(1, 16), (9, 16)])
@pytest.mark.parametrize("S", [37, 41, 74, 160])
def test_a_shards_triple_is_the_same_by_either_exchange(M, nh, S):
    """The triple that is gathered and the one that is pushed hold the same bits, at the sizes where the merge of a whole sequence takes eight runs of
    splits, and are the fold in double precision to the rounding of S additions."""
    from yasakani_b200 import kv4
    hd, gen = 128, torch.Generator(device="cuda").manual_seed(S)
    pm = torch.randn((M, S, nh), generator=gen, device="cuda") * 3
    pm[:, S // 2] = -1e30                                          # an empty split
    pl = torch.rand((M, S, nh), generator=gen, device="cuda") * 50 + 1
    pacc = torch.randn((M, S, nh, hd), generator=gen, device="cuda") * pl[..., None]
    triple = torch.empty((M, nh, hd + 2), device="cuda")
    kv4.launch_local_triple(pm, pl, pacc, S, M, nh, hd, triple)
    buf = torch.zeros((kv4.exchange_bytes(1, M, nh, hd) + 3) // 4, device="cuda")
    x, o16 = kv4.peer_exchange([buf.data_ptr()], 0), torch.empty((M, nh, hd), dtype=torch.float16, device="cuda")
    kv4.launch_push_triple(pm, pl, pacc, S, M, nh, hd, x)
    kv4.launch_merge_pushed(x, M, nh, 8, hd, o16)
    torch.cuda.synchronize()
    assert kv4.device_status() == 0
    pushed = buf[:2 * triple.numel()].view(M, nh, hd + 2, 2)[..., 0]      # the first step's half: a value and the number of its step
    assert torch.equal(pushed.view(torch.int32), triple.view(torch.int32)), int((pushed != triple).sum())
    w = torch.exp(pm.double() - pm.double().amax(1, keepdim=True)) * (pm > -1e29)
    o, l, mag = (w[..., None] * pacc.double()).sum(1), (w * pl.double()).sum(1), (w[..., None] * pacc.double().abs()).sum(1)
    # a weight is within 8 units (its argument, below 32, is rounded by the subtraction; expf within two), and every sum adds at most S terms
    assert ((triple[..., 2:].double() - o).abs() <= (S + 40) * 2.0 ** -24 * mag).all() and ((triple[..., 1].double() - l).abs() <= (S + 40) * 2.0 ** -24 * l).all()
    assert torch.equal(triple[..., 0], pm.amax(1))
