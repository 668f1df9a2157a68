"""The append kernel outside its cache: rows before position 0 and behind the capacity, positions at the ends of 32 bits; all seven arrays
whole, with what lay in them before."""
import numpy as np
import pytest
import torch

from tests.helpers import f16_bits
from yasakani_b200 import synth

pytestmark = pytest.mark.gpu
FILL = 0x5A                                                       # as an fp16 number 203.25


def _filled(kv4, hkv, hd, max_ctx):
    layer = kv4.KvLayer(hkv, hd, max_ctx)
    for t in layer.tensors():
        t.view(torch.uint8).fill_(FILL)
    return layer


def _append(kv4, layer, pos, k, v):
    kv4.launch_kv_append(layer, k.cuda(), v.cuda(), torch.tensor([pos], dtype=torch.int32, device="cuda"), k.shape[0])
    torch.cuda.synchronize()


def _same(layer, okv):
    got = layer.to_numpy()
    for name, want in okv.arrays().items():
        assert np.array_equal(got[name].reshape(want.shape).view(np.uint8), want.view(np.uint8)), name


@pytest.mark.parametrize("hd", [64, 128, 256])
@pytest.mark.parametrize("passes", [[(-8, 40), (32, 24), (56, 40)], [(-5, 5), (-31, 33)], [(60, 4), (62, 200)], [(40, 8), (48, 300)]])
def test_only_rows_inside_the_cache_are_stored(oracle, hd, passes):
    from yasakani_b200 import kv4
    layer, okv = _filled(kv4, 2, hd, 64), oracle.KvCache(2, hd, 64)
    for a in okv.arrays().values():
        a.view(np.uint8)[...] = FILL
    for i, (pos, m) in enumerate(passes):
        k, v = synth.make_kv(synth.Shape(4, 2, hd, 64, 1e4), m, seed=17 + i)
        _append(kv4, layer, pos, k, v)
        lo, hi = max(0, -pos), min(m, 64 - pos)                   # rows inside
        if hi > lo:
            oracle.append(okv, pos + lo, f16_bits(k[lo:hi]), f16_bits(v[lo:hi]))
    _same(layer, okv)


@pytest.mark.parametrize("pos", [64, 65, 96, 2 ** 31 - 1, 2 ** 31 - 6, 2 ** 31 - 33, 2 ** 31 - 64, -2 ** 31, -2 ** 31 + 31, -40, -41, -1000])
@pytest.mark.parametrize("m", [1, 8, 40])
def test_positions_far_outside_store_nothing(pos, m):
    from yasakani_b200 import kv4
    layer = _filled(kv4, 2, 128, 64)
    k, v = synth.make_kv(synth.Shape(4, 2, 128, 64, 1e4), m, seed=3)
    _append(kv4, layer, pos, k, v)
    d_pos = torch.tensor([pos], dtype=torch.int32, device="cuda")
    kv4.launch_kv_group_quant_g(layer, d_pos, m)
    torch.cuda.synchronize()
    for t in layer.tensors():
        assert bool((t.view(torch.uint8) == FILL).all())
