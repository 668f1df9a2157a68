"""The append kernel on numbers that are not finite: infinities, NaN of several forms and zeros of both signs in keys and values, byte for byte
against the reference's fp32 steps."""
import numpy as np
import pytest
import torch

from yasakani_b200 import synth

pytestmark = pytest.mark.gpu


def _quant(x, lo, hi, axis):
    """Codes, scale and zero bits of fp32 values between lo and hi (the reference's fp32 steps)."""
    with np.errstate(all="ignore"):
        d = (hi - lo).astype(np.float32)
        inv = np.where(hi > lo, np.float32(15) / d, np.float32(0)).astype(np.float32)
        t = ((x - np.expand_dims(lo, axis)).astype(np.float32) * np.expand_dims(inv, axis)).astype(np.float32)
        q = np.where(np.isnan(t), 0, np.clip(np.rint(t), 0, 15)).astype(np.uint8)
        sc, z = (d / np.float32(15)).astype(np.float16), lo.astype(np.float16)
    return q, *(np.where(np.isnan(a), np.uint16(0x7FFF), a.view(np.uint16)) for a in (sc, z))


def _bounds(x, axis, lo0, hi0):
    """Minimum and maximum past NaN, -0 below +0, from the starting values."""
    neg0, pos0 = ((x == 0) & np.signbit(x)).any(axis), ((x == 0) & ~np.signbit(x)).any(axis)
    lo, hi = np.fmin.reduce(x, axis=axis), np.fmax.reduce(x, axis=axis)
    if lo0 is not None:
        lo, hi = np.fmin(lo, np.float32(lo0)), np.fmax(hi, np.float32(hi0))
    lo = np.where(lo == 0, np.where(neg0, np.float32(-0.0), np.float32(0.0)), lo)
    return lo.astype(np.float32), np.where(hi == 0, np.where(pos0, np.float32(0.0), np.float32(-0.0)), hi).astype(np.float32)


@pytest.mark.parametrize("hd", [128, 256])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("passes", [[32], [31, 1], [5, 20, 7]])
def test_values_that_are_not_finite(hd, dtype, passes):
    from yasakani_b200 import kv4
    inf, nan = float("inf"), float("nan")
    k, v = (t.to(dtype) for t in synth.make_kv(synth.Shape(4, 2, hd, 64, 1e4), 32, seed=9))
    for c, column in enumerate([[inf], [-inf], [nan], [inf, -inf], [nan, inf], [nan, -inf, 1.0], [0.0], [-0.0], [0.0, -0.0], [-0.0, 0.0], [-0.0, 3.0], [0.0, -3.0]]):
        k[:, 0, 3 * c] = torch.tensor(column * 32)[:32].to(dtype)  # every row of the group
        k[c::7, 1, 2 * c] = torch.tensor(column[0]).to(dtype)      # some rows of it
        v[c, 0, c::5] = torch.tensor(column[-1]).to(dtype)
        v[c, 1] = torch.tensor(column * hd)[:hd].to(dtype)
    bits = {torch.float16: torch.int16, torch.bfloat16: torch.int16, torch.float32: torch.int32}[dtype]
    for i, payload in enumerate({2: (0x7F81, 0xFFC0, -1) if dtype == torch.bfloat16 else (0x7C01, 0xFE00, -1), 4: (0x7F800001, 0xFFC00000, -1)}[k.element_size()]):
        n = np.array([payload], np.int64).astype(np.int32 if k.element_size() == 4 else np.int16)
        k.view(bits)[4 + i, 1, 40 + i] = torch.from_numpy(n)[0]
        v.view(bits)[20 + i, 1, 9] = torch.from_numpy(n)[0]
    layer, p = kv4.KvLayer(2, hd, 64), 0
    for m in passes:
        kv4.launch_kv_append(layer, k[p:p + m].cuda(), v[p:p + m].cuda(), torch.tensor([p], dtype=torch.int32, device="cuda"), m)
        p += m
    got = layer.to_numpy()
    x, y = (t.float().numpy().astype(np.float16).astype(np.float32).transpose(1, 0, 2) for t in (k, v))       # [head][row][channel]
    shadow = np.where(np.isnan(x), np.uint16(0x7FFF), x.astype(np.float16).view(np.uint16))
    assert np.array_equal(got["kshadow"].reshape(2, 64, hd)[:, :32].view(np.uint16), shadow)
    pack = lambda q: q[..., 0::2] | (q[..., 1::2] << 4)
    q, sc, z = _quant(x, *_bounds(x, 1, 1e30, -1e30), 1)
    assert np.array_equal(got["kq"].reshape(2, 2, 32, hd // 2)[:, 0], pack(q))
    assert np.array_equal(got["kscale"].reshape(2, 2, hd)[:, 0].view(np.uint16), sc)
    assert np.array_equal(got["kzero"].reshape(2, 2, hd)[:, 0].view(np.uint16), z)
    q, sc, z = _quant(y, *_bounds(y, 2, None, None), 2)
    assert np.array_equal(got["vq"].reshape(2, 64, hd // 2)[:, :32], pack(q))
    assert np.array_equal(got["vscale"].reshape(2, 64)[:, :32].view(np.uint16), sc)
    assert np.array_equal(got["vzero"].reshape(2, 64)[:, :32].view(np.uint16), z)
