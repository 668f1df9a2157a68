"""The append kernel at the edges of its warps' shares: passes that start and end inside groups, rows per launch on both sides of its block
sizes, rows that are aligned for no wide load, every element type; packed cache byte for byte against the oracle."""
import numpy as np
import pytest
import torch

from tests.helpers import f16_bits
from yasakani_b200 import synth

pytestmark = pytest.mark.gpu

SHAPES = {256: synth.C2, 128: synth.C1, 64: synth.Shape(4, 2, 64, 64, 1e4)}


@pytest.mark.parametrize("hd", sorted(SHAPES))
@pytest.mark.parametrize("dtype,shift", [(torch.float16, 0), (torch.float16, 1), (torch.bfloat16, 2), (torch.bfloat16, 3), (torch.float32, 1)])
@pytest.mark.parametrize("passes", [[1, 2, 7, 8, 9, 4, 1, 32, 64], [31, 33, 65, 1], [63, 1, 64], [5, 90, 97]])
def test_passes_of_every_size_leave_the_oracles_bytes(oracle, hd, dtype, shift, passes):
    from yasakani_b200 import kv4
    shape, n = SHAPES[hd], sum(passes)
    k, v = synth.make_kv(shape, n, seed=n + hd)
    v[2, 1, 7:9] = -0.0
    okv = oracle.KvCache(shape.hkv, hd, 256)
    layer = kv4.KvLayer(shape.hkv, hd, 256)

    def shifted(x):                                            # the same rows `shift` elements behind an aligned address
        buf = torch.zeros(x.numel() + shift, dtype=dtype, device="cuda")
        buf[shift:] = x.to(dtype).cuda().view(-1)
        return buf[shift:].view(x.shape)

    p, pos = 0, torch.zeros(1, dtype=torch.int32, device="cuda")
    for m in passes:
        rk, rv = shifted(k[p:p + m]), shifted(v[p:p + m])
        oracle.append(okv, p, f16_bits(rk.to(torch.float16).cpu()), f16_bits(rv.to(torch.float16).cpu()))
        pos.fill_(p)
        kv4.launch_kv_append(layer, rk, rv, pos, m)
        p += m
    torch.cuda.synchronize()
    got = layer.to_numpy()
    for name, want in okv.arrays().items():
        assert np.array_equal(got[name].reshape(want.shape), want), name


def test_rows_before_the_cache_and_behind_it_are_left_out():
    from yasakani_b200 import kv4
    layer = kv4.KvLayer(2, 128, 64)
    for t in layer.tensors():
        t.zero_()
    rows = torch.ones((40, 2, 128), dtype=torch.float16, device="cuda")
    for pos in (-8, 56):
        kv4.launch_kv_append(layer, rows, rows, torch.tensor([pos], dtype=torch.int32, device="cuda"), 40)
    torch.cuda.synchronize()
    have = (layer.kshadow.view(2, 64, 128).float().amax((0, 2)) > 0).cpu().numpy()
    assert np.array_equal(np.nonzero(have)[0], np.r_[0:32, 56:64])
