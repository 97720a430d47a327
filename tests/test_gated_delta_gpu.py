"""Gated delta-rule kernels on the GPU against the CPU oracle, through the C ABI.

Cases follow cpp/tests/qwen35_cuda_delta_test.cu (T in {1,2,4,17}, decode after prefill, continued prefill, launches
sharing device state without a sync, saturation edges, mixed weight dtypes, the dk = dv = 128 model shape) with
N(0,1) operands.  Operands are quantised identically on both sides (cpp/tests/qwen35_cuda_delta_test.cu:257-270).
Tolerances: outputs max abs <= 3e-2 and relative L2 <= 1e-2; FP32 state relative L2 <= 1e-3."""
import numpy as np
import pytest
import torch

from oracle import bindings as ob
from raftinfer_b200 import kernels as K
from raftinfer_b200 import synth

from gpu_util import act_tensor, bf16_tensor, compare, dev, to_numpy_f32

pytestmark = pytest.mark.gpu
HK, HV, DK = 16, 32, 128


def core_operands(seed, tokens, hk=HK, hv=HV, quantise=True):
    q = synth.round_bf16(synth.normal(seed, 0, (tokens, hk, DK)))
    k = synth.round_bf16(synth.normal(seed, 1, (tokens, hk, DK)))
    v = synth.round_bf16(synth.normal(seed, 2, (tokens, hv, DK)))
    q = q / np.sqrt((q.astype(np.float64) ** 2).sum(-1, keepdims=True) + 1e-6) / np.sqrt(DK)
    k = k / np.sqrt((k.astype(np.float64) ** 2).sum(-1, keepdims=True) + 1e-6)
    q, k = q.astype(np.float32), k.astype(np.float32)
    if quantise:
        q, k = synth.round_bf16(q), synth.round_bf16(k)
    beta = synth.sigmoid(synth.normal(seed, 3, (tokens, hv)))
    g = (-synth.softplus(synth.normal(seed, 4, (tokens, hv)))).astype(np.float32)
    return q, k, v, beta, g


def run_core(tokens, dtype, seed, hk=HK, hv=HV, state0=None):
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv, quantise=dtype == K.DTYPE_BF16)
    if state0 is None:
        state0 = (0.05 * synth.normal(seed, 5, (hv, DK, DK))).astype(np.float32)
    state = torch.from_numpy(state0.copy()).to(dev())
    out = torch.zeros(tokens, hv, DK, device=dev())
    ws_bytes = K.gdn_core_workspace_bytes(tokens, hk, hv, DK, DK)
    ws = torch.zeros(max(ws_bytes // 4, 4), device=dev())
    K.gdn_core(act_tensor(q, dtype), act_tensor(k, dtype), act_tensor(v, dtype),
               torch.from_numpy(beta).to(dev()), torch.from_numpy(g).to(dev()), state, out, ws, ws_bytes, tokens, hk, hv,
               DK, DK, dtype, torch.cuda.current_stream())
    torch.cuda.synchronize()
    want_out, want_state = ob.gdn_core(q, k, v, beta, np.exp(g), state0)
    m_out = compare(to_numpy_f32(out), want_out)
    m_state = compare(to_numpy_f32(state), want_state)
    return m_out, m_state


@pytest.mark.parametrize("tokens", [1, 2, 4, 17, 63])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_recurrent_core(tokens, dtype):
    m_out, m_state = run_core(tokens, dtype, seed=0xB2001000 + tokens)
    assert m_out["nonfinite"] == 0 and m_out["max_abs"] <= 1.0e-4 and m_out["rel_l2"] <= 1.0e-4, m_out
    assert m_state["nonfinite"] == 0 and m_state["rel_l2"] <= 1.0e-5, m_state


@pytest.mark.parametrize("tokens", [64, 65, 100, 128, 257, 1024])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_chunked_core_matches_the_sequential_recurrence(tokens, dtype):
    """Runs of 64 tokens or more take the chunk-64 WY-form kernels; the ground truth stays the token-sequential
    recurrence.  Outputs: max abs <= 3e-2, relative L2 <= 1e-2 (held to 2e-3); FP32 state relative L2 <= 1e-3."""
    m_out, m_state = run_core(tokens, dtype, seed=0xB2001300 + tokens)
    assert m_out["nonfinite"] == 0 and m_out["max_abs"] <= 3.0e-2 and m_out["rel_l2"] <= 2.0e-3, m_out
    assert m_state["nonfinite"] == 0 and m_state["rel_l2"] <= 1.0e-3, m_state


@pytest.mark.parametrize("hk,hv", [(16, 32), (4, 8)])
def test_chunked_core_long_run_equals_the_same_run_in_pieces(hk, hv):
    """A run of 9 297 tokens (146 chunks, ragged tail) in one call and the same tokens in three calls that split on
    chunk boundaries walk the same chunks with the same arithmetic: outputs and final state are bit-identical.  It
    also takes the barrier phases and the staging rings of the chunk kernels well past their first wrap-arounds."""
    tokens, cuts = 9297, (0, 4096, 4096 + 64, 9297)
    gen = torch.Generator(device=dev()).manual_seed(0xB2001500 + hv)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q = (unit(torch.randn(tokens, hk, DK, device=dev(), generator=gen)) / DK ** 0.5).to(torch.bfloat16)
    k = unit(torch.randn(tokens, hk, DK, device=dev(), generator=gen)).to(torch.bfloat16)
    v = torch.randn(tokens, hv, DK, device=dev(), generator=gen).to(torch.bfloat16)
    beta = torch.sigmoid(torch.randn(tokens, hv, device=dev(), generator=gen))
    g = -torch.nn.functional.softplus(torch.randn(tokens, hv, device=dev(), generator=gen))
    state0 = 0.05 * torch.randn(hv, DK, DK, device=dev(), generator=gen)
    stream = torch.cuda.current_stream()

    def run(pieces):
        state = state0.clone()
        out = torch.zeros(tokens, hv, DK, device=dev())
        for lo, hi in pieces:
            n = hi - lo
            ws_bytes = K.gdn_core_workspace_bytes(n, hk, hv, DK, DK)
            ws = torch.zeros(max(ws_bytes // 4, 4), device=dev())
            K.gdn_core(q[lo:hi], k[lo:hi], v[lo:hi], beta[lo:hi], g[lo:hi], state, out[lo:hi], ws, ws_bytes, n, hk, hv,
                       DK, DK, K.DTYPE_BF16, stream)
        torch.cuda.synchronize()
        return out, state

    whole_out, whole_state = run([(0, tokens)])
    parts_out, parts_state = run(list(zip(cuts[:-1], cuts[1:])))
    assert K.device_status(stream) == 0
    assert torch.isfinite(whole_out).all() and torch.isfinite(whole_state).all()
    assert torch.equal(whole_out, parts_out) and torch.equal(whole_state, parts_state)


def test_chunked_prefill_4096_then_128_decode_steps():
    """The benchmark's gated-delta configuration: zero state, 4096-token chunked prefill, then 128 recurrent steps."""
    tokens, steps, seed = 4096, 128, 0xB2001400
    q, k, v, beta, g = core_operands(seed, tokens + steps)
    state0 = np.zeros((HV, DK, DK), dtype=np.float32)
    state = torch.zeros(HV, DK, DK, device=dev())
    out = torch.zeros(tokens + steps, HV, DK, device=dev())
    dq, dk, dv = bf16_tensor(q), bf16_tensor(k), bf16_tensor(v)
    dbeta, dg = torch.from_numpy(beta).to(dev()), torch.from_numpy(g).to(dev())
    ws_bytes = K.gdn_core_workspace_bytes(tokens, HK, HV, DK, DK)
    ws = torch.zeros(ws_bytes // 4, device=dev())
    stream = torch.cuda.current_stream()
    K.gdn_core(dq, dk, dv, dbeta, dg, state, out, ws, ws_bytes, tokens, HK, HV, DK, DK, K.DTYPE_BF16, stream)
    for t in range(tokens, tokens + steps):
        K.gdn_core(dq[t], dk[t], dv[t], dbeta[t], dg[t], state, out[t], None, 0, 1, HK, HV, DK, DK, K.DTYPE_BF16, stream)
    torch.cuda.synchronize()
    want_out, want_state = ob.gdn_core(q, k, v, beta, np.exp(g), state0)
    m_out = compare(to_numpy_f32(out), want_out)
    m_state = compare(to_numpy_f32(state), want_state)
    assert m_out["nonfinite"] == 0 and m_out["max_abs"] <= 3.0e-2 and m_out["rel_l2"] <= 1.0e-2, m_out
    assert m_state["nonfinite"] == 0 and m_state["rel_l2"] <= 1.0e-3, m_state


@pytest.mark.parametrize("hk,hv", [(2, 2), (1, 3), (3, 6)])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_chunked_core_other_head_counts(hk, hv, dtype):
    """Key heads equal to value heads, one key head for three value heads, odd counts: fewer (chunk, head) items than
    SMs, a ragged last chunk (200 tokens), the key head of a value head is head % key_heads."""
    m_out, m_state = run_core(200, dtype, seed=0xB2001900 + 16 * hk + hv, hk=hk, hv=hv)
    assert m_out["nonfinite"] == 0 and m_out["max_abs"] <= 3.0e-2 and m_out["rel_l2"] <= 2.0e-3, m_out
    assert m_state["nonfinite"] == 0 and m_state["rel_l2"] <= 1.0e-3, m_state


@pytest.mark.parametrize("hk,hv,tokens", [(HK, HV, 600), (11, 33, 640), (31, 31, 650), (9, 18, 1100)])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_chunked_core_several_items_a_cta(hk, hv, tokens, dtype):
    """More (chunk, value head) items than the prepare kernel has CTAs: shares of one to three neighbouring items, which
    begin with the first, the second or the third value head of a key head, so that its image is loaded again, kept, or the
    only one; a ragged last chunk."""
    m_out, m_state = run_core(tokens, dtype, seed=0xB2001A00 + 16 * hk + hv, hk=hk, hv=hv)
    assert m_out["nonfinite"] == 0 and m_out["max_abs"] <= 3.0e-2 and m_out["rel_l2"] <= 2.0e-3, m_out
    assert m_state["nonfinite"] == 0 and m_state["rel_l2"] <= 1.0e-3, m_state
    assert K.device_status(torch.cuda.current_stream()) == 0


def test_recurrent_core_small_head_counts():
    m_out, m_state = run_core(3, K.DTYPE_F32, seed=0xB2001100, hk=2, hv=4)
    assert m_out["rel_l2"] <= 1.0e-4 and m_state["rel_l2"] <= 1.0e-5


def test_batched_decode_step():
    batch = 6
    seed = 0xB2001200
    q, k, v, beta, g = core_operands(seed, batch)  # one token per sequence
    states0 = [(0.05 * synth.normal(seed, 10 + i, (HV, DK, DK))).astype(np.float32) for i in range(batch)]
    states = [torch.from_numpy(s.copy()).to(dev()) for s in states0]
    ptrs = torch.tensor([s.data_ptr() for s in states], device=dev(), dtype=torch.int64)
    out = torch.zeros(batch, HV, DK, device=dev())
    K.batched_gdn_decode(bf16_tensor(q), bf16_tensor(k), bf16_tensor(v), torch.from_numpy(beta).to(dev()),
                         torch.from_numpy(g).to(dev()), ptrs, out, batch, HK, HV, torch.cuda.current_stream())
    torch.cuda.synchronize()
    got = to_numpy_f32(out)
    for i in range(batch):
        want_out, want_state = ob.gdn_core(q[i:i + 1], k[i:i + 1], v[i:i + 1], beta[i:i + 1], np.exp(g[i:i + 1]),
                                           states0[i])
        assert compare(got[i], want_out[0])["rel_l2"] <= 1.0e-4
        assert compare(to_numpy_f32(states[i]), want_state)["rel_l2"] <= 1.0e-5


# ---- whole layer (packed input) -------------------------------------------------------------------
def layer_operands(seed, tokens, hk, hv, width, scale=1.0):
    hidden = hv * DK
    conv_dim = 2 * hk * DK + hidden
    stride = conv_dim + 2 * hv + hidden
    inp = synth.round_bf16(scale * synth.normal(seed, 0, (tokens, stride)))
    conv_w = synth.round_bf16(0.3 * synth.normal(seed, 1, (conv_dim, width)))
    rec_a = (-np.exp(0.3 * synth.normal(seed, 2, (hv,)))).astype(np.float32)
    dt_bias = (0.5 * synth.normal(seed, 3, (hv,))).astype(np.float32)
    norm_w = (1.0 + 0.1 * synth.normal(seed, 4, (DK,))).astype(np.float32)
    conv_state = (0.5 * synth.normal(seed, 5, (conv_dim, width - 1))).astype(np.float32)
    rec_state = (0.05 * synth.normal(seed, 6, (hv, DK, DK))).astype(np.float32)
    return inp, conv_w, rec_a, dt_bias, norm_w, conv_state, rec_state


class LayerRun:
    """Device-side layer state carried across calls, with the oracle run in lock step."""

    def __init__(self, seed, hk, hv, width, dtype, wdtype, tokens_total, scale=1.0):
        self.hk, self.hv, self.width, self.dtype, self.wdtype = hk, hv, width, dtype, wdtype
        ops = layer_operands(seed, tokens_total, hk, hv, width, scale)
        self.inp, self.conv_w, self.rec_a, self.dt_bias, self.norm_w, self.cs, self.rs = ops
        if wdtype != K.DTYPE_F32:
            self.rec_a, self.dt_bias, self.norm_w = (synth.round_bf16(x) for x in (self.rec_a, self.dt_bias, self.norm_w))
        self.d_conv_w = act_tensor(self.conv_w, wdtype)
        self.d_rec_a = act_tensor(self.rec_a, wdtype)
        self.d_dt = act_tensor(self.dt_bias, wdtype)
        self.d_norm = act_tensor(self.norm_w, wdtype)
        self.d_cs = torch.from_numpy(self.cs.copy()).to(dev())
        self.d_rs = torch.from_numpy(self.rs.copy()).to(dev())
        self.done = 0

    def step(self, tokens, sync=True):
        hidden = self.hv * DK
        shape = K.GatedDeltaShape(tokens, hidden, self.hk, self.hv, DK, DK, self.width, 1.0e-6)
        chunk = self.inp[self.done:self.done + tokens]
        self.done += tokens
        ws_bytes = K.qwen35_gated_delta_workspace_bytes(shape)
        ws = torch.zeros(ws_bytes // 4, device=dev())
        out = torch.zeros(tokens, hidden, device=dev(),
                          dtype={K.DTYPE_F32: torch.float32, K.DTYPE_F16: torch.float16}.get(self.dtype, torch.bfloat16))
        d_in = act_tensor(chunk, self.dtype)
        K.qwen35_gated_delta(d_in, self.d_conv_w, self.d_rec_a, self.d_dt, self.d_norm, out, self.d_cs, self.d_rs, ws,
                             ws_bytes, shape, self.dtype, self.wdtype, torch.cuda.current_stream())
        if sync:
            torch.cuda.synchronize()
        want, self.cs, self.rs = ob.gated_delta_layer(chunk, self.conv_w, self.rec_a, self.dt_bias, self.norm_w, self.cs,
                                                      self.rs, (tokens, hidden, self.hk, self.hv, DK, DK, self.width,
                                                                1.0e-6))
        return out, want, (d_in, ws)

    def check(self, out, want, chunked=False):
        m = compare(to_numpy_f32(out), want)
        assert m["nonfinite"] == 0 and m["max_abs"] <= 3.0e-2 and m["rel_l2"] <= 1.0e-2, m
        if self.dtype == K.DTYPE_F32 and not chunked:
            assert m["max_abs"] <= 2.0e-3 and m["rel_l2"] <= 2.0e-4, m  # FP32 recurrent path
        if self.dtype == K.DTYPE_F32 and chunked:
            assert m["max_abs"] <= 1.5e-2 and m["rel_l2"] <= 2.0e-3, m  # products of ten-bit mantissas
        cs = compare(to_numpy_f32(self.d_cs).reshape(-1), self.cs.reshape(-1))
        assert cs["max_abs"] == 0.0, cs
        rs = compare(to_numpy_f32(self.d_rs).reshape(-1), self.rs.reshape(-1))
        assert rs["nonfinite"] == 0 and rs["rel_l2"] <= 1.0e-3, rs


@pytest.mark.parametrize("tokens", [1, 2, 4, 17])
@pytest.mark.parametrize("dtype,wdtype", [(K.DTYPE_BF16, K.DTYPE_F32), (K.DTYPE_F32, K.DTYPE_F32),
                                          (K.DTYPE_BF16, K.DTYPE_BF16), (K.DTYPE_F32, K.DTYPE_BF16)])
def test_layer_small_heads(tokens, dtype, wdtype):
    run = LayerRun(0xB2002000 + tokens, 2, 4, 3, dtype, wdtype, tokens)
    out, want, _ = run.step(tokens)
    run.check(out, want)


@pytest.mark.parametrize("tokens", [3, 150])
@pytest.mark.parametrize("wdtype", [K.DTYPE_F32, K.DTYPE_F16])
def test_layer_f16_activations(tokens, wdtype):
    """FP16 input and output (the reference's delta launcher takes F32, F16 and BF16, cpp/kernels/qwen35_delta.cu:
    811-897): operands that FP16 holds exactly on both sides, the recurrent kernel (3 tokens) and the chunked one."""
    run = LayerRun(0xB2002600 + tokens, 2, 4, 4, K.DTYPE_F16, wdtype, tokens)
    half = lambda x: x.astype(np.float16).astype(np.float32)
    run.inp = half(run.inp)
    if wdtype == K.DTYPE_F16:
        run.conv_w, run.rec_a, run.dt_bias, run.norm_w = (half(x) for x in (run.conv_w, run.rec_a, run.dt_bias,
                                                                             run.norm_w))
        run.d_conv_w, run.d_rec_a = act_tensor(run.conv_w, wdtype), act_tensor(run.rec_a, wdtype)
        run.d_dt, run.d_norm = act_tensor(run.dt_bias, wdtype), act_tensor(run.norm_w, wdtype)
    out, want, _ = run.step(tokens)
    m = compare(to_numpy_f32(out), want)
    assert m["nonfinite"] == 0 and m["max_abs"] <= 3.0e-2 and m["rel_l2"] <= 1.0e-2, m
    assert compare(to_numpy_f32(run.d_cs).reshape(-1), run.cs.reshape(-1))["max_abs"] == 0.0
    assert compare(to_numpy_f32(run.d_rs).reshape(-1), run.rs.reshape(-1))["rel_l2"] <= 1.0e-3


def test_layer_model_shape_prefill_then_decode_then_continued_prefill():
    run = LayerRun(0xB2002100, HK, HV, 4, K.DTYPE_BF16, K.DTYPE_F32, 3 + 1 + 1 + 5)
    for tokens in (3, 1, 1, 5):
        out, want, _ = run.step(tokens)
        run.check(out, want)


@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_layer_chunked_prefill_then_decode(dtype):
    """A 150-token call takes the chunked kernels inside the layer; a one-token call follows on the same states."""
    run = LayerRun(0xB2002500, 4, 8, 4, dtype, K.DTYPE_F32, 151)
    for tokens in (150, 1):
        out, want, _ = run.step(tokens)
        run.check(out, want, chunked=True)


@pytest.mark.parametrize("hk,hv", [(1, 1), (2, 4), (1, 3), (HK, HV)])
@pytest.mark.parametrize("dtype,wdtype", [(K.DTYPE_BF16, K.DTYPE_F32), (K.DTYPE_F32, K.DTYPE_F32),
                                          (K.DTYPE_BF16, K.DTYPE_BF16), (K.DTYPE_F32, K.DTYPE_BF16)])
def test_layer_single_tokens(hk, hv, dtype, wdtype):
    """One-token calls back to back on the same states: one launch where a key head has one or two value heads (one
    cluster each), the general path for three.  FP32 activations are held to the recurrence's FP32 tolerance."""
    run = LayerRun(0xB2002700 + 8 * hk + hv, hk, hv, 4, dtype, wdtype, 3)
    for _ in range(3):
        out, want, _ = run.step(1)
        run.check(out, want)
    assert K.device_status(torch.cuda.current_stream()) == 0


@pytest.mark.parametrize("calls", [(2, 3), (31, 2), (32, 1), (33, 17), (63,)])
@pytest.mark.parametrize("hk,hv", [(1, 1), (2, 4), (1, 3)])
@pytest.mark.parametrize("dtype,wdtype", [(K.DTYPE_BF16, K.DTYPE_BF16), (K.DTYPE_F32, K.DTYPE_F32)])
def test_layer_short_calls(calls, hk, hv, dtype, wdtype):
    """Calls of 2 to 63 tokens, whole groups of four and ragged ones, each on the states the one before left: one launch
    where a key head has one or two value heads, the general path for three."""
    run = LayerRun(0xB2002900 + 8 * hk + hv, hk, hv, 4, dtype, wdtype, sum(calls))
    for tokens in calls:
        out, want, _ = run.step(tokens)
        run.check(out, want)
    assert K.device_status(torch.cuda.current_stream()) == 0


@pytest.mark.parametrize("tokens", [2, 3, 5, 6, 7, 8, 47, 48, 49, 62])
@pytest.mark.parametrize("hv", [1, 2])
@pytest.mark.parametrize("dtype", [K.DTYPE_F32, K.DTYPE_F16])
@pytest.mark.parametrize("aligned", [True, False])
def test_layer_short_calls_in_groups(tokens, hv, dtype, aligned):
    """The one-launch form folds tokens into the state four at a time and loads rows four elements at a time where they are
    aligned: every remainder of a group, either side of a round of loads and of a round of groups, with one and two value
    heads, and an input that starts one element off.  FP32 against the bound of the recurrence's FP32 path; FP16 operands
    are exact on both sides, so that only the output's rounding (2^-11) remains."""
    half = lambda x: x.astype(np.float16).astype(np.float32)
    run = LayerRun(0xB2002A00 + tokens, 1, hv, 4, dtype, K.DTYPE_F32, tokens)
    run.inp = half(run.inp)
    shape = K.GatedDeltaShape(tokens, hv * DK, 1, hv, DK, DK, 4, 1.0e-6)
    ws_bytes = K.qwen35_gated_delta_workspace_bytes(shape)
    ws = torch.zeros(ws_bytes // 4, device=dev())
    element = act_tensor(run.inp, dtype)
    buffer = torch.zeros(element.numel() + 1, device=dev(), dtype=element.dtype)
    d_in = buffer[:-1] if aligned else buffer[1:]
    d_in.copy_(element.reshape(-1))
    out = torch.zeros(tokens, hv * DK, device=dev(), dtype=element.dtype)
    K.qwen35_gated_delta(d_in, run.d_conv_w, run.d_rec_a, run.d_dt, run.d_norm, out, run.d_cs, run.d_rs, ws, ws_bytes, shape,
                         dtype, K.DTYPE_F32, torch.cuda.current_stream())
    torch.cuda.synchronize()
    want, run.cs, run.rs = ob.gated_delta_layer(run.inp, run.conv_w, run.rec_a, run.dt_bias, run.norm_w, run.cs, run.rs,
                                                (tokens, hv * DK, 1, hv, DK, DK, 4, 1.0e-6))
    m = compare(to_numpy_f32(out), want)
    assert m["nonfinite"] == 0 and m["rel_l2"] <= (2.0e-6 if dtype == K.DTYPE_F32 else 2.0 ** -11), m
    assert compare(to_numpy_f32(run.d_cs).reshape(-1), run.cs.reshape(-1))["max_abs"] == 0.0
    assert compare(to_numpy_f32(run.d_rs).reshape(-1), run.rs.reshape(-1))["rel_l2"] <= 2.0e-6
    assert K.device_status(torch.cuda.current_stream()) == 0


@pytest.mark.parametrize("tokens,first", [(4, 0), (5, 0), (6, 2), (8, 4), (9, 0), (9, 2), (9, 5)])
@pytest.mark.parametrize("hv", [1, 2])
@pytest.mark.parametrize("state", ["zero", "tiny", "mild"])
def test_layer_short_calls_with_growing_decays(tokens, first, hv, state):
    """A positive coefficient, for which a decay is above 1: the head goes token by token.  Four consecutive tokens from `first` on grow by e^22 to e^25
    each, so that the product of their decays overflows FP32 while every state along the way is finite: it is zero (no values
    before the growth is over) or starts at 1e-30.  `mild`: decays of up to e^0.5 on an ordinary state.  The second value head
    decays as usual.  Log decays are exact on both sides, so that 4 e^x of two ulp (1e-6) and the FP32 recurrence (2e-6, as in
    the ordinary short calls) bound the difference."""
    run = LayerRun(0xB2002B00 + 16 * tokens + first, 1, hv, 4, K.DTYPE_F32, K.DTYPE_F32, tokens)
    conv_dim = 2 * DK + hv * DK
    grown = range(first, first + 4)
    run.rec_a = np.array([1.0, -1.0][:hv], dtype=np.float32)
    run.dt_bias = np.zeros(hv, dtype=np.float32)
    log_decay = synth.normal(0xB2002B01, 0, (tokens,))
    if state == "mild":  # softplus(a) of -2 to 0.5
        run.inp[:, conv_dim + hv] = np.clip(log_decay, -2.0, 0.5) - 1.0
    else:
        run.inp[:, conv_dim + hv] = -40.0  # a decay of 1 + 4e-18
        for t in grown:
            run.inp[t, conv_dim + hv] = 22.0 + (3 * t % 4)
        run.rs[0] = 0.0 if state == "zero" else 1.0e-30 / 0.05 * run.rs[0]
        value = slice(2 * DK, 3 * DK)
        run.inp[:first + 4, value] = 0.0
        run.cs[value] = 0.0
    run.d_rec_a, run.d_dt = act_tensor(run.rec_a, K.DTYPE_F32), act_tensor(run.dt_bias, K.DTYPE_F32)
    run.d_cs, run.d_rs = torch.from_numpy(run.cs.copy()).to(dev()), torch.from_numpy(run.rs.copy()).to(dev())
    out, want, _ = run.step(tokens)
    assert np.isfinite(want).all() and np.isfinite(run.rs).all()
    m = compare(to_numpy_f32(out), want)
    assert m["nonfinite"] == 0 and m["rel_l2"] <= 3.0e-6, m
    for head in range(hv):
        rs = compare(to_numpy_f32(run.d_rs)[head].reshape(-1), run.rs.reshape(hv, -1)[head])
        assert rs["nonfinite"] == 0 and rs["rel_l2"] <= 3.0e-6, (head, rs)
    assert K.device_status(torch.cuda.current_stream()) == 0


FAR_GATES = np.concatenate([np.linspace(-88.7, -80.0, 100), [-95.0, -104.0, -200.0, np.inf, np.nan, -30.0, -1.0e-3, 0.0, 1.0e-3],
                            np.linspace(1.0, 100.0, 19)]).astype(np.float32)


@pytest.mark.parametrize("tokens,width", [(1, 4), (5, 4), (3, 3)])
def test_layer_gates_of_any_size(tokens, width):
    """SiLU of output gates down to where 1 + e^-z overflows, of an infinite one and of one that is not a number, in the
    one-launch forms and the general path: the output over that of the same call with gates of 20, whose SiLU is 20.  e^x of
    two ulp and five roundings bound the difference; below -88.72 the sum is infinite and the result zero."""
    hidden, conv_dim = DK, 3 * DK
    outs = []
    for z in (FAR_GATES, np.full(DK, 20.0, dtype=np.float32)):
        run = LayerRun(0xB2002D00 + tokens, 1, 1, width, K.DTYPE_F32, K.DTYPE_F32, tokens)
        run.inp[:, conv_dim + 2:] = z
        run.d_norm = torch.ones(DK, device=dev())
        outs.append(to_numpy_f32(run.step(tokens)[0]).astype(np.float64))
    got = outs[0] / outs[1] * 20.0
    z = FAR_GATES.astype(np.float64)
    with np.errstate(over="ignore", invalid="ignore", divide="ignore"):
        want = np.where(z < -88.72, 0.0, z / (1.0 + np.exp(-z)))
        got_error = np.abs(got / want - 1.0)
    finite = np.isfinite(want) & (want != 0.0)
    assert (got_error[:, finite] <= 7 * 2.0 ** -23).all(), got_error[:, finite].max()
    assert (got[:, want == 0.0] == 0.0).all()
    assert np.isinf(got[:, np.isinf(want)]).all() and np.isnan(got[:, np.isnan(want)]).all()


@pytest.mark.parametrize("tokens,width", [(1, 4), (5, 4), (3, 3)])
@pytest.mark.parametrize("b", [-87.0, -87.5, -88.5])
def test_layer_write_strength_near_the_smallest_float(tokens, width, b):
    """A sigmoid of 1.6e-38 and below puts subnormal numbers into a zero state; a few units of the last place (2^-149) for
    e^x of two ulp (4.6 units of a result of 2^-126), the product with the value and the sum over the tokens."""
    run = LayerRun(0xB2002D80 + tokens, 1, 1, width, K.DTYPE_F32, K.DTYPE_F32, tokens)
    run.inp[:, 3 * DK] = b
    run.rs[:] = 0.0
    run.d_rs = torch.zeros_like(run.d_rs)
    run.step(tokens)
    want = run.rs.reshape(-1).astype(np.float64)
    got = to_numpy_f32(run.d_rs).reshape(-1).astype(np.float64)
    assert np.abs(want).max() >= 2.0 ** -135
    assert np.abs(got - want).max() <= 8 * tokens * 2.0 ** -149, np.abs(got - want).max() / 2.0 ** -149


def layer_in_64_bits(inp, conv_w, rec_a, dt_bias, norm_w, conv_state, rec_state):
    """A layer call of HK and HV heads in plain torch: (output, state)."""
    inp, conv_w, rec_a, dt_bias, norm_w, conv_state, state = (
        x.double() for x in (inp, conv_w, rec_a, dt_bias, norm_w, conv_state, rec_state))
    tokens, conv_dim, width = inp.shape[0], conv_w.shape[0], conv_w.shape[1]
    rows = torch.cat([conv_state.t(), inp[:, :conv_dim]])
    mixed = torch.nn.functional.silu(sum(rows[i:i + tokens] * conv_w[:, i] for i in range(width)))
    q, k, v = (x.view(tokens, -1, DK) for x in mixed.split([HK * DK, HK * DK, HV * DK], dim=1))
    q, k = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1.0e-6) for x in (q, k))
    q, k = (x.repeat(1, HV // HK, 1) for x in (q / DK ** 0.5, k))
    beta = torch.sigmoid(inp[:, conv_dim:conv_dim + HV])
    decay = torch.exp(rec_a * torch.nn.functional.softplus(inp[:, conv_dim + HV:conv_dim + 2 * HV] + dt_bias))
    out = []
    for t in range(tokens):
        state = state * decay[t][:, None, None]
        delta = beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", state, k[t]))
        state = state + k[t][:, :, None] * delta[:, None, :]
        out.append(torch.einsum("hkv,hk->hv", state, q[t]))
    out = torch.stack(out)
    out = out * torch.rsqrt((out * out).mean(-1, keepdim=True) + 1.0e-6) * norm_w
    return (out * torch.nn.functional.silu(inp[:, conv_dim + 2 * HV:].view(tokens, HV, DK))).view(tokens, -1), state


@pytest.mark.parametrize("tokens", [4, 17, 63])
def test_layer_short_calls_are_no_further_from_64_bits_than_single_tokens(tokens):
    """Folding four tokens into the state at a time rounds less often than going token by token: the mean distance from 64
    bits over four seeds, decays spread as such layers are trained, against that of the same tokens as one-token calls.  The
    ratios are 0.92 to 0.96, and 0.98 to 1.02 where products of decays, corrections and terms of the state are each rounded."""
    gen = torch.Generator(device=dev()).manual_seed(0xB2002C00 + tokens)
    normal = lambda *s: torch.randn(*s, device=dev(), generator=gen)
    uniform = lambda low, high: low + (high - low) * torch.rand(HV, device=dev(), generator=gen)
    conv_dim, hidden = 2 * HK * DK + HV * DK, HV * DK
    distances = []
    for _ in range(4):
        inp, conv_w = normal(tokens, conv_dim + 2 * HV + hidden), 0.3 * normal(conv_dim, 4)
        step = torch.exp(uniform(np.log(1.0e-3), np.log(1.0e-1)))
        rec_a, dt_bias = -uniform(1.0, 16.0), step + torch.log(-torch.expm1(-step))
        norm_w, conv_state, state = 1.0 + 0.1 * normal(DK), 0.5 * normal(conv_dim, 3), 0.05 * normal(HV, DK, DK)
        want, want_state = layer_in_64_bits(inp, conv_w, rec_a, dt_bias, norm_w, conv_state, state)
        for count in (tokens, 1):
            shape = K.GatedDeltaShape(count, hidden, HK, HV, DK, DK, 4, 1.0e-6)
            ws_bytes = K.qwen35_gated_delta_workspace_bytes(shape)
            ws, out = torch.zeros(ws_bytes // 4, device=dev()), torch.zeros(tokens, hidden, device=dev())
            cs, rs = conv_state.clone(), state.clone()
            for t in range(0, tokens, count):
                K.qwen35_gated_delta(inp[t:t + count], conv_w, rec_a, dt_bias, norm_w, out[t:t + count], cs, rs, ws,
                                     ws_bytes, shape, K.DTYPE_F32, K.DTYPE_F32, torch.cuda.current_stream())
            torch.cuda.synchronize()
            distances.append([((out - want).norm() / want.norm()).item(),
                              ((rs - want_state).norm() / want_state.norm()).item()])
    folded, single = np.mean(distances[0::2], axis=0), np.mean(distances[1::2], axis=0)
    assert (folded <= 0.97 * single).all(), (folded, single)


def test_layer_three_launches_share_device_state_without_a_sync():
    run = LayerRun(0xB2002200, 2, 4, 4, K.DTYPE_F32, K.DTYPE_F32, 6)
    results = [run.step(2, sync=False) for _ in range(3)]
    torch.cuda.synchronize()
    for out, want, _ in results[:-1]:
        m = compare(to_numpy_f32(out), want)
        assert m["max_abs"] <= 2.0e-3 and m["rel_l2"] <= 2.0e-4, m
    run.check(results[-1][0], results[-1][1])


def test_layer_conv_width_one_and_wide():
    for width in (1, 2, 6):
        run = LayerRun(0xB2002300 + width, 2, 4, width, K.DTYPE_F32, K.DTYPE_F32, 5)
        if width == 1:
            run.d_cs = torch.zeros(4, device=dev())
            run.cs = np.zeros((run.cs.shape[0], 0), dtype=np.float32)
        out, want, _ = run.step(5)
        m = compare(to_numpy_f32(out), want)
        assert m["max_abs"] <= 2.0e-3 and m["rel_l2"] <= 2.0e-4, (width, m)


def test_layer_saturation_edges_stay_finite():
    """Extreme gate inputs (cpp/tests/qwen35_cuda_delta_test.cu:568-603): A from -12 to -0.001, dt_bias -25..5,
    b = +-30, z = +-18.  Everything must stay finite and match the oracle."""
    hk, hv, width, tokens = 2, 4, 4, 4
    run = LayerRun(0xB2002400, hk, hv, width, K.DTYPE_F32, K.DTYPE_F32, tokens)
    hidden = hv * DK
    conv_dim = 2 * hk * DK + hidden
    run.rec_a = np.array([-12.0, -1.0, -0.05, -0.001], dtype=np.float32)
    run.dt_bias = np.array([-25.0, -3.0, 0.5, 5.0], dtype=np.float32)
    run.d_rec_a, run.d_dt = act_tensor(run.rec_a, K.DTYPE_F32), act_tensor(run.dt_bias, K.DTYPE_F32)
    run.inp[:, conv_dim:conv_dim + hv] = np.array([30.0, -30.0, 30.0, -30.0], dtype=np.float32)
    run.inp[:, conv_dim + 2 * hv::2] = 18.0
    run.inp[:, conv_dim + 2 * hv + 1::2] = -18.0
    out, want, _ = run.step(tokens)
    assert np.isfinite(to_numpy_f32(out)).all() and np.isfinite(to_numpy_f32(run.d_rs)).all()
    run.check(out, want)


def test_batched_decode_step_64_sequences_at_full_size():
    """The serving configuration's gated-delta half at its full size: one recurrent step on each of 64 sequences'
    FP32 [32][128][128] states in one launch (the kernel that splits the (sequence, head) units evenly over the SMs);
    every sequence's output and new state against the oracle."""
    batch, seed = 64, 0xB2001600
    q, k, v, beta, g = core_operands(seed, batch)  # one token per sequence
    gen = torch.Generator(device=dev()).manual_seed(seed)
    states = [0.05 * torch.randn(HV, DK, DK, device=dev(), generator=gen) for _ in range(batch)]
    states0 = [to_numpy_f32(s) for s in states]
    ptrs = torch.tensor([s.data_ptr() for s in states], device=dev(), dtype=torch.int64)
    out = torch.zeros(batch, HV, DK, device=dev())
    K.batched_gdn_decode(bf16_tensor(q), bf16_tensor(k), bf16_tensor(v), torch.from_numpy(beta).to(dev()),
                         torch.from_numpy(g).to(dev()), ptrs, out, batch, HK, HV, torch.cuda.current_stream())
    torch.cuda.synchronize()
    got = to_numpy_f32(out)
    for i in range(batch):
        want_out, want_state = ob.gdn_core(q[i:i + 1], k[i:i + 1], v[i:i + 1], beta[i:i + 1], np.exp(g[i:i + 1]),
                                           states0[i])
        assert compare(got[i], want_out[0])["rel_l2"] <= 1.0e-4, i
        assert compare(to_numpy_f32(states[i]), want_state)["rel_l2"] <= 1.0e-5, i


@pytest.mark.parametrize("batch", [8, 9, 37, 300])
def test_batched_decode_step_streaming_kernel(batch):
    """The batches the streaming kernel takes (8 sequences and up): unit counts that do not divide by the SM count,
    one or two units a CTA, and more units per CTA (300 x 32 over 148) than state pointers it keeps in shared memory.
    At 300 sequences every seventh one is checked against the oracle."""
    seed = 0xB2001700 + batch
    q, k, v, beta, g = core_operands(seed, batch)
    gen = torch.Generator(device=dev()).manual_seed(seed)
    states = [0.05 * torch.randn(HV, DK, DK, device=dev(), generator=gen) for _ in range(batch)]
    checked = range(batch) if batch <= 64 else range(0, batch, 7)
    states0 = {i: to_numpy_f32(states[i]) for i in checked}
    ptrs = torch.tensor([s.data_ptr() for s in states], device=dev(), dtype=torch.int64)
    out = torch.zeros(batch, HV, DK, device=dev())
    stream = torch.cuda.current_stream()
    K.batched_gdn_decode(bf16_tensor(q), bf16_tensor(k), bf16_tensor(v), torch.from_numpy(beta).to(dev()),
                         torch.from_numpy(g).to(dev()), ptrs, out, batch, HK, HV, stream)
    torch.cuda.synchronize()
    assert K.device_status(stream) == 0
    got = to_numpy_f32(out)
    for i in checked:
        want_out, want_state = ob.gdn_core(q[i:i + 1], k[i:i + 1], v[i:i + 1], beta[i:i + 1], np.exp(g[i:i + 1]),
                                           states0[i])
        assert compare(got[i], want_out[0])["rel_l2"] <= 1.0e-4, i
        assert compare(to_numpy_f32(states[i]), want_state)["rel_l2"] <= 1.0e-5, i


def test_batched_decode_step_reports_a_state_pointer_off_its_boundary():
    """The state pointers live in device memory, so the host cannot check them.  The streaming kernel looks at each
    one before it copies from it: a pointer off a 16-byte boundary is not read (the copy would fault); the kernel sets
    RIB200_DEVICE_POINTER_MISALIGNED instead, and the context carries on with the next, well-formed call."""
    batch, seed = 16, 0xB2001800
    q, k, v, beta, g = core_operands(seed, batch)
    gen = torch.Generator(device=dev()).manual_seed(seed)
    pool = 0.05 * torch.randn(batch, HV * DK * DK + 4, device=dev(), generator=gen)
    addresses = [pool[i].data_ptr() for i in range(batch)]
    bad = list(addresses)
    bad[5] += 4
    out = torch.zeros(batch, HV, DK, device=dev())
    stream = torch.cuda.current_stream()
    operands = (bf16_tensor(q), bf16_tensor(k), bf16_tensor(v), torch.from_numpy(beta).to(dev()),
                torch.from_numpy(g).to(dev()))
    assert K.device_status(stream) == 0
    K.batched_gdn_decode(*operands, torch.tensor(bad, device=dev(), dtype=torch.int64), out, batch, HK, HV, stream)
    torch.cuda.synchronize()
    assert K.device_status(stream) == K.DEVICE_POINTER_MISALIGNED
    assert K.device_status(stream) == 0  # reading cleared it
    fresh = 0.05 * torch.randn(batch, HV * DK * DK + 4, device=dev(), generator=gen)
    before = to_numpy_f32(fresh[3, :HV * DK * DK]).reshape(HV, DK, DK)
    K.batched_gdn_decode(*operands, torch.tensor([fresh[i].data_ptr() for i in range(batch)], device=dev(),
                                                 dtype=torch.int64), out, batch, HK, HV, stream)
    torch.cuda.synchronize()
    assert K.device_status(stream) == 0
    want_out, want_state = ob.gdn_core(q[3:4], k[3:4], v[3:4], beta[3:4], np.exp(g[3:4]), before)
    assert compare(to_numpy_f32(out)[3], want_out[0])["rel_l2"] <= 1.0e-4
    assert compare(to_numpy_f32(fresh[3, :HV * DK * DK]).reshape(HV, DK, DK), want_state)["rel_l2"] <= 1.0e-5
