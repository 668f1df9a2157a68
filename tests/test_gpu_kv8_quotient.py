"""The quotient of the INT8-row merge's form for many rows, bit for bit against fp32 division: values on and beside the ties of the output type, so
that the last bit of the quotient shows; sums of weights and values on both sides of the range of its short way; zeros of both signs, infinities, NaN, rows without keys."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
M, NH = 128, 24
N = M * NH


def _ties(rng, n, bits):
    """fp32 (v, l) whose quotient lies within an ulp of halfway between two values of a type with `bits` significant bits."""
    l = (rng.uniform(1.0, 2.0, (n, 1)) * 2.0 ** rng.integers(0, 4, (n, 1))).astype(np.float32)
    tie = (2.0 ** (bits - 1) + rng.integers(0, 2 ** (bits - 1), (n, 256)) + 0.5) * 2.0 ** (1 - bits) * rng.choice([-1.0, 1.0], (n, 256))
    return (tie * l.astype(np.float64)).astype(np.float32), l


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quotient_is_the_rounded_one(dtype):
    from yasakani_b200 import kvx
    rng = np.random.default_rng(5)
    v, l = _ties(rng, N, 8 if dtype == torch.bfloat16 else 11)
    ev, el = np.zeros((N, 1)), np.zeros((N, 1))                   # powers of two on v and on l, by row
    third = N // 3
    ev[third:2 * third] = rng.integers(-110, 110, (third, 1))
    el[third:2 * third] = rng.choice([-21, -20, -19, 0, 55, 56, 59, 60, 61, -59, -60, -61], (third, 1))
    with np.errstate(all="ignore"):
        v, l = (v * 2.0 ** ev).astype(np.float32), (l * 2.0 ** el).astype(np.float32)
    v[2 * third:2 * third + 200] *= np.float32(2.0) ** rng.integers(-126, 100, (200, 256)).astype(np.float32)   # every size in one row
    rows = iter(range(2 * third + 200, N))
    for value, weight in ((3e38, 0.5), (np.inf, 3.0), (-np.inf, 1e30), (np.nan, 2.0), (0.0, 3.0), (1e-44, 0.7), (1.5, 0.0), (-1.0, 1e-38), (3e38, 1e38)):
        r = next(rows)
        v[r, ::3], l[r] = value, weight
    S = 2                                                         # split 0 is far below split 1: its weight turns a zero's sign, no more
    pacc, pl, pm = np.zeros((M, S, NH, 256), np.float32), np.zeros((M, S, NH), np.float32), np.zeros((M, S, NH), np.float32)
    pm[:, 0] = -100.0
    r = next(rows)
    minus = slice(7, 60)
    pacc[r // NH, 0, r % NH, minus], v[r, minus] = -1e-10, -0.0   # exp(-100) * -1e-10 rounds to -0
    pacc[:, 1], pl[:, 1] = v.reshape(M, NH, 256), l.reshape(M, NH)
    empty = next(rows)
    pm[empty // NH, :, empty % NH] = -1e30
    o16 = torch.empty((M, NH, 256), dtype=dtype, device="cuda")
    kvx.launch_kv8_combine(*(torch.from_numpy(x).cuda() for x in (pm, pl, pacc)), S, M, NH, o16, inverse_rotate=False)
    with np.errstate(all="ignore"):
        q = v / l
    plus = v == 0                                                 # a zero of either sign is +0 after its sum with split 0's +0
    plus[r, minus] = False
    with np.errstate(all="ignore"):
        q[plus] = np.float32(0) / np.broadcast_to(l, v.shape)[plus]
    q[empty] = np.nan
    want = torch.from_numpy(q).to(dtype).view(M, NH, 256)
    got = o16.cpu()
    nan = torch.isnan(want)
    assert bool((torch.isnan(got) == nan).all())
    bad = (got.view(torch.int16) != want.view(torch.int16)) & ~nan
    assert not bool(bad.any()), (int(bad.sum()), got[bad][:4], want[bad][:4])
