"""The table of tensor maps of a multi-request pass has the size its header gives, two maps of 128 bytes a slot: a caller may size it by either."""
import re

import pytest
import torch

from yasakani_b200 import _lib, build


@pytest.mark.parametrize("n", [1, 2, 63, 64])
def test_size_is_the_documented_layout(n):
    doc = re.search(r"maps\s+\[n_slots\]\[(\d+)\].*?(\d+) bytes each", open(build.ABI).read())
    assert (int(doc[1]), int(doc[2])) == (2, 128)
    assert _lib.load().yskn_kv4_ms_maps_bytes(n) == n * 256


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 3])
def test_prepare_writes_nothing_behind_the_table(n):
    from yasakani_b200 import kv4
    layers = [kv4.KvLayer(2, 128, 128) for _ in range(n)]
    slots = kv4.MsSlots(layers)                                   # for its host-side array of descriptors
    buf = torch.full((n * 1024 + 128,), 0x5A, dtype=torch.uint8, device="cuda")
    off = -buf.data_ptr() % 128
    host = (_lib.KvLayerC * n)(*[l.struct() for l in layers])
    assert _lib.load().yskn_kv4_ms_prepare(host, n, 2, 128, 128, slots.d_layers.data_ptr(), buf.data_ptr() + off, 0) == 0
    torch.cuda.synchronize()
    assert bool((buf[:off] == 0x5A).all()) and bool((buf[off + n * 256:] == 0x5A).all())
