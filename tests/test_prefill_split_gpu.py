"""Prefill of a tile or two of queries behind a long past, where several CTAs share the keys of an item, exchange their
partial tiles and write a share of the columns each: shares of unequal length, tiles with few live rows, the line between
two and four shares (eight key blocks), pairs of heads and single ones, both activation types."""
import numpy as np
import pytest
import torch

from oracle import bindings as ob
from raftinfer_b200 import kernels as K
from raftinfer_b200 import synth

from gpu_util import act_tensor, cache_bits_of, cache_to_device, compare, dev, gate_bf16_outputs, to_numpy_f32

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("hq,hkv", [(16, 4), (2, 1), (3, 3)])
@pytest.mark.parametrize("tokens,past", [(2, 892), (2, 896), (5, 1150), (17, 2688), (128, 900), (127, 1031), (150, 1300)])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_shared_keys(tokens, past, hq, hkv, dtype):
    seed, rows = 0xB2005000 + tokens + past + hq, past + tokens + 7
    q = synth.round_bf16(synth.normal(seed, 0, (tokens, hq, D)))
    gate = synth.round_bf16(synth.normal(seed, 1, (tokens, hq, D)))
    k = synth.round_bf16(synth.normal(seed, 2, (past + tokens, hkv, D)))
    v = synth.round_bf16(synth.normal(seed, 3, (past + tokens, hkv, D)))
    bits = np.full((2, hkv, rows, D), 0x7FC1, dtype=np.uint16)
    bits[0, :, :past] = synth.bf16_bits(k[:past]).transpose(1, 0, 2)
    bits[1, :, :past] = synth.bf16_bits(v[:past]).transpose(1, 0, 2)
    cache = cache_to_device(bits)
    out = torch.full((tokens + 1, hq, D), 5.0, device=dev(),
                     dtype=torch.float32 if dtype == K.DTYPE_F32 else torch.bfloat16)
    shape = K.Qwen35AttentionShape(tokens, hq, hkv, D, rows, past)
    stream = torch.cuda.current_stream()
    K.qwen35_online_attention_prefill(act_tensor(q, dtype), act_tensor(k[past:], dtype), act_tensor(v[past:], dtype),
                                      act_tensor(gate, dtype), out, cache, cache.numel() * 2, shape, dtype, K.KV_BF16,
                                      K.HEAD_MAJOR, stream)
    torch.cuda.synchronize()
    assert K.device_status(stream) == 0
    gate_bf16_outputs(compare(to_numpy_f32(out[:tokens]), ob.attention_core(q, k, v, gate, past=past)))
    assert bool((out[tokens] == 5.0).all())  # nothing past the last row
    bits[0, :, past:past + tokens] = synth.bf16_bits(k[past:]).transpose(1, 0, 2)
    bits[1, :, past:past + tokens] = synth.bf16_bits(v[past:]).transpose(1, 0, 2)
    assert np.array_equal(cache_bits_of(cache).reshape(bits.shape), bits)
