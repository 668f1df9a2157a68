"""The two forms of the INT8-row merge against a double-precision reference: the edges of their ranges (one split, the last split
count of the row form, more splits than one batch of loads, the most splits), ragged row counts, gate, both types."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inverse_rotation(y):
    h = np.array([[1.0]])
    while h.shape[0] < 256:
        h = np.block([[h, h], [h, -h]])
    d = np.arange(256, dtype=np.uint32) + np.uint32(1)
    x = d.astype(np.uint64)
    for m in (0x7feb352d, 0x846ca68b):
        x ^= x >> 16 if m == 0x7feb352d else x >> 15
        x = (x * m) & 0xFFFFFFFF
    x ^= x >> 16
    return (y @ h / 16.0) * np.where(x & 1, -1.0, 1.0)


@pytest.mark.parametrize("M,nh,S", [(1, 24, 1), (1, 24, 37), (3, 8, 41), (2, 24, 64), (86, 24, 1), (87, 24, 4), (700, 3, 2), (86, 24, 5)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_merge_matches_double_precision(M, nh, S, dtype):
    from yasakani_b200 import kvx
    g = torch.Generator().manual_seed(M * 100 + S)
    pm = torch.randn((M, S, nh), generator=g) * 3
    pm[:, S // 2] = -1e30 if S > 1 else 0.5                       # an empty split
    pl = torch.rand((M, S, nh), generator=g) * 50 + 1
    pacc = torch.randn((M, S, nh, 256), generator=g) * pl[..., None]
    gate = torch.randn((M, nh, 256), generator=g).to(dtype)
    o16 = torch.empty((M, nh, 256), dtype=dtype, device="cuda")
    kvx.launch_kv8_combine(pm.cuda(), pl.cuda(), pacc.cuda(), S, M, nh, o16, gate=gate.cuda())
    w = torch.exp((pm.double() - pm.double().amax(1, keepdim=True))) * (pm > -1e29)
    y = _inverse_rotation(((w[..., None] * pacc.double()).sum(1) / (w * pl.double()).sum(1)[..., None]).numpy())
    sg = torch.sigmoid(gate.double()).to(dtype).double().numpy()
    want = torch.from_numpy(y).to(dtype).double().numpy() * sg
    # an ulp of a type with p significant bits is at most 2^(1-p) of the value (bf16: p = 8, fp16: p = 11).  The value and the sigmoid may
    # each fall to the other side of a tie by the error of their fp32 arithmetic (one ulp each), the product is rounded (half an ulp)
    ulp = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
    err = np.abs(o16.double().cpu().numpy() - want)
    assert (err <= 2.5 * ulp * np.abs(want) + 1e-6).all(), err.max()


@pytest.mark.parametrize("M,nh,S", [(37, 4, 3), (149, 1, 1), (50, 3, 8), (25, 6, 9), (19, 8, 32), (19, 8, 33), (10, 24, 64)])
def test_row_form_edges(M, nh, S):
    """Both sides of the line between the forms, whole and broken batches of eight splits, one and two weights a lane."""
    test_merge_matches_double_precision(M, nh, S, torch.bfloat16)


@pytest.mark.parametrize("M,nh", [(37, 8), (27, 11)])             # 296 and 297 rows: with more than 32 splits a warp each from 297 on
@pytest.mark.parametrize("S", [32, 33, 37, 64])
def test_both_sides_of_the_line_for_many_splits(M, nh, S):
    test_merge_matches_double_precision(M, nh, S, torch.float16)
