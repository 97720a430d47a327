"""The launchers as native Python functions: argument counts, refusals and the way of every field into the call."""
import ctypes

import pytest

from raftinfer_b200 import _call, _lib
from raftinfer_b200 import kernels as K


@pytest.mark.parametrize("name", [n for n in dir(_call) if n.startswith("rib200_")])
def test_native_launchers_take_the_declared_arguments_and_refuse_what_ctypes_refused(name):
    call, count = getattr(_call, name), len(_lib.PROTOTYPES[name])
    for wrong in (count - 1, count + 1):
        with pytest.raises(TypeError):
            call(*[None] * wrong)
    floats = [1.5] * count  # no pointer, no size, no shape
    with pytest.raises((AttributeError, ctypes.ArgumentError)):
        call(*floats)


def test_native_launchers_pass_every_field_on():
    """Each refusal of the library names the argument it read; only the one that is off is off."""
    good = dict(tokens=2, query_heads=16, kv_heads=4, head_dim=256, max_context_tokens=256, past_tokens=0)
    call = lambda shape, dtype=K.DTYPE_BF16, policy=K.Qwen35AttentionLaunchPolicy(), cache_bytes=1 << 30, stream=16: \
        K.qwen35_causal_attention(16, 16, 16, 16, 16, 16, cache_bytes, None, 0, K.Qwen35AttentionShape(**shape), dtype,
                                  policy, stream)
    attempts = [lambda f=f, v=v: call({**good, f: v}) for f, v in
                [("tokens", 0), ("query_heads", 15), ("kv_heads", 0), ("head_dim", 255), ("max_context_tokens", 1),
                 ("past_tokens", 255)]]
    attempts += [lambda: call(good, dtype=9), lambda: call(good, cache_bytes=16), lambda: call(good, stream=None),
                 lambda: call(good, policy=K.Qwen35AttentionLaunchPolicy(7, 1, 1)),
                 lambda: call(good, policy=K.Qwen35AttentionLaunchPolicy(1, 1, 9))]
    for attempt in attempts:
        with pytest.raises(K.Qwen35PrimitiveError):
            attempt()
    delta = dict(tokens=2, hidden_size=256, key_heads=1, value_heads=2, key_dim=128, value_dim=128, conv_width=4,
                 epsilon=1.0e-6)
    for field, value in [("tokens", 0), ("hidden_size", 255), ("key_heads", 3), ("value_heads", 3), ("key_dim", 0),
                         ("value_dim", 64), ("conv_width", 0), ("epsilon", -1.0)]:
        with pytest.raises(K.Qwen35DeltaError):
            K.qwen35_gated_delta(16, 16, 16, 16, 16, 16, 16, 16, 16, 1 << 30, K.GatedDeltaShape(**{**delta, field: value}),
                                 K.DTYPE_F32, K.DTYPE_F32, 16, K.GatedDeltaLaunchPolicy())
    for policy in (K.GatedDeltaLaunchPolicy(9, 4, False), K.GatedDeltaLaunchPolicy(0, 3, False),
                   K.GatedDeltaLaunchPolicy(0, 4, True)):
        with pytest.raises(K.Qwen35DeltaError):
            K.qwen35_gated_delta(16, 16, 16, 16, 16, 16, 16, 16, 16, 1 << 30, K.GatedDeltaShape(**delta), K.DTYPE_F32,
                                 K.DTYPE_F32, 16, policy)
