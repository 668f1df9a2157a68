"""The native argument marshalling of the launchers refuses what the Python signature promises to refuse, before the library is
called (no GPU needed: nothing here gets as far as a launch)."""
import pytest
import torch

from yasakani_b200 import Kv4Error, kv4, kvx


def _decode_args(**change):
    kv = kv4.KvLayer(2, 128, 64, device="cpu")
    pm, pl, pacc = kv4.attn_scratch(1, 2, 16, 128, device="cpu")
    a = dict(q16=torch.zeros((1, 16, 128), dtype=torch.float16), kv=kv, M=1, d_pos=torch.zeros(1, dtype=torch.int32), splits=2, pm=pm, pl=pl, pacc=pacc,
             rope=None, nh=16, qscale=0.1, rd=0, o16=torch.zeros((1, 16, 128), dtype=torch.float16))
    return dict(a, **change)


@pytest.mark.parametrize("change,error", [
    (dict(), AssertionError),                                            # host tensors
    (dict(q16=None), TypeError),
    (dict(M=1.5), TypeError),
    (dict(M=1 << 40), OverflowError),
    (dict(kv=object()), AttributeError),
])
def test_decode_rejects(change, error):
    with pytest.raises(error):
        kv4.launch_decode(**_decode_args(**change))


def test_append_and_merge_reject():
    kv = kv4.KvLayer(2, 128, 64, device="cpu")
    k = torch.zeros((1, 2, 128), dtype=torch.float16)
    with pytest.raises(AssertionError):
        kv4.launch_kv_append(kv, k, k.float(), torch.zeros(1, dtype=torch.int32), 1)
    with pytest.raises(AssertionError):
        kv4.launch_kv_append(kv, k, k, torch.zeros(1, dtype=torch.int32), 1)
    with pytest.raises(TypeError):
        kvx.launch_attn_post(*(torch.zeros((1, 24, 512)) for _ in range(5)), 1e-6, *(torch.zeros((4, 64, 256)) for _ in range(2)), 64,
                             *(torch.zeros((4, 64, 256)) for _ in range(6)))


def test_a_call_the_library_refuses_carries_its_message():
    pm = torch.zeros((1, 2, 16))
    with pytest.raises(Kv4Error, match="unsupported head_dim 24"):
        kv4.launch_attn_combine_gqa(pm, pm, pm, 2, 1, torch.zeros((1, 16, 24), dtype=torch.float16), 16, 8, stream=type("S", (), {"cuda_stream": 0})())


@pytest.mark.parametrize("name", ["q16", "d_pos", "pm", "pl", "pacc"])
@pytest.mark.parametrize("value", [None, 3])
def test_what_is_no_tensor_raises_attribute_error(name, value):
    with pytest.raises(AttributeError):
        kv4.launch_decode(**_decode_args(**{name: value}))


@pytest.mark.gpu
def test_a_missing_buffer_is_the_librarys_to_refuse():
    o16 = torch.zeros((1, 16, 256), dtype=torch.float16, device="cuda")
    with pytest.raises(Kv4Error, match="null buffer"):
        kvx.launch_kv8_combine(None, None, None, 2, 1, 16, o16)
    with pytest.raises(AttributeError):
        kvx.launch_kv8_combine(None, None, None, 2, 1, 16, None)
