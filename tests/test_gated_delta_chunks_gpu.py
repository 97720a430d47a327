"""The chunk kernels of the gated delta rule away from ordinary magnitudes, and the forms that only long calls take.

Their operands are FP16 with scales (powers of two) that have to hold every magnitude the FP32 tensors can bring.  A
result is compared per (chunk, head, column) with the token-sequential oracle: columns of V and of the state never meet
in a product, so none may lose to another.  Tolerance: a result passes five operands rounded to eleven significant bits
(K, T or W, U's V, the state, Delta), each 2^-11 relative at most: 5 x 2^-11 = 2.5e-3 of the column's 2-norm in the chunk."""
import numpy as np
import pytest
import torch

from oracle import bindings as ob
from raftinfer_b200 import kernels as K
from raftinfer_b200 import synth

from gpu_util import act_tensor, compare, dev, to_numpy_f32
from test_gated_delta_gpu import DK, HK, HV, LayerRun, core_operands

pytestmark = pytest.mark.gpu
COLUMN_TOLERANCE = 5 * 2.0 ** -11
CHUNK = 64


def column_errors(got, want, axis):
    """2-norm of the difference over 2-norm of the result, along `axis`; exact zeros have to be zeros."""
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    difference, size = np.sqrt(((got - want) ** 2).sum(axis)), np.sqrt((want ** 2).sum(axis))
    assert (difference[size == 0] == 0).all()
    return difference / np.where(size == 0, 1.0, size)


def run_core(q, k, v, beta, g, state0, dtype):
    tokens, hk, hv = q.shape[0], q.shape[1], v.shape[1]
    state = torch.from_numpy(state0.copy()).to(dev())
    out = torch.zeros(tokens, hv, DK, device=dev())
    nbytes = K.gdn_core_workspace_bytes(tokens, hk, hv, DK, DK)
    workspace = torch.zeros(nbytes // 4, device=dev())
    stream = torch.cuda.current_stream()
    K.gdn_core(act_tensor(q, dtype), act_tensor(k, dtype), act_tensor(v, dtype), torch.from_numpy(beta).to(dev()),
               torch.from_numpy(g).to(dev()), state, out, workspace, nbytes, tokens, hk, hv, DK, DK, dtype, stream)
    torch.cuda.synchronize()
    assert K.device_status(stream) == 0
    with np.errstate(all="ignore"):
        want_out, want_state = ob.gdn_core(q, k, v, beta, np.exp(g), state0)
    return to_numpy_f32(out), to_numpy_f32(state), want_out, want_state


def check_columns(got_out, got_state, want_out, want_state, columns=slice(None), fades=False):
    for first in range(0, got_out.shape[0], CHUNK):
        rows = slice(first, first + CHUNK)
        errors = column_errors(got_out[rows][..., columns], want_out[rows][..., columns], 0)
        assert errors.max() <= (8 if fades else 1) * COLUMN_TOLERANCE, (first, errors.max())
    errors = column_errors(got_state[..., columns], want_state[..., columns], 1)
    assert errors.max() <= COLUMN_TOLERANCE, errors.max()


def spread(v, state0, factors):
    """Columns of V and of the state times factors of their own."""
    factors = np.resize(np.asarray(factors, np.float32), DK)
    return synth.round_bf16(v * factors), state0 * factors


COLUMN_CASES = {
    "as they are": lambda v, s: (v, s),
    "ten decades": lambda v, s: spread(v, s, 10.0 ** -np.arange(10)),
    "every other one huge": lambda v, s: spread(v, s, [1.0, 1.0e10]),
    "all small": lambda v, s: spread(v, s, [1.0e-5]),
    "all large": lambda v, s: spread(v, s, [1.0e6]),
    "thousands": lambda v, s: spread(v, s, [1.0e3]),
    "large state": lambda v, s: (v, s * np.float32(1.0e4)),
    "small state, one column large": lambda v, s: (v, s * np.resize(np.float32([1.0e6] + 31 * [1.0]), DK)),
    "chunks up and down": lambda v, s: (synth.round_bf16(v * np.float32([1.0, 1.0e4, 1.0, 1.0e-4])[
        np.arange(len(v)) // CHUNK][:, None, None]), s),
    "a chunk of zeros": lambda v, s: (v * (np.arange(len(v)) // CHUNK != 1)[:, None, None].astype(np.float32), 0 * s),
    "zeros in front": lambda v, s: (v * (np.arange(len(v)) // CHUNK != 0)[:, None, None].astype(np.float32), 0 * s),
    "empty columns": lambda v, s: spread(v, s, [0.0, 1.0, 1.0]),
}
# What these chunks give is little of what they start with: a column whose first tokens read little of the large state has
# that state's rounding in its whole norm.  A factor of 8 (three bits) over the bound of the others.
FADES = ("large state", "chunks up and down", "a chunk of zeros")


@pytest.mark.parametrize("name", COLUMN_CASES)
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F32])
def test_columns_of_any_magnitude(name, dtype):
    tokens, hk, hv, seed = 230, 2, 4, 0xB2006000
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv, quantise=dtype == K.DTYPE_BF16)
    v, state0 = COLUMN_CASES[name](v, (0.05 * synth.normal(seed, 5, (hv, DK, DK))).astype(np.float32))
    check_columns(*run_core(q, k, v.astype(np.float32), beta, g, state0.astype(np.float32), dtype), fades=name in FADES)


@pytest.mark.parametrize("where,what", [("value", np.inf), ("value", np.nan), ("state", np.inf), ("state", np.nan)])
def test_what_is_not_finite_stays_in_its_column(where, what):
    tokens, hk, hv, seed = 200, 1, 2, 0xB2006100
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    state0 = (0.05 * synth.normal(seed, 5, (hv, DK, DK))).astype(np.float32)
    if where == "value":
        v[70, 1, 37] = what
    else:
        state0[1, 3, 37] = what
    got_out, got_state, want_out, want_state = run_core(q, k, v, beta, g, state0, K.DTYPE_BF16)
    others = [c for c in range(DK) if c != 37]
    check_columns(got_out, got_state, want_out, want_state, others)
    check_columns(got_out[:, :1], got_state[:1], want_out[:, :1], want_state[:1])
    assert not np.isfinite(got_state[1, :, 37]).any()
    if where == "value":  # the chunk in front of the infinity does not know of it
        assert column_errors(got_out[:CHUNK, 1, 37], want_out[:CHUNK, 1, 37], 0) <= COLUMN_TOLERANCE


@pytest.mark.parametrize("rise", [0.002, 0.08, 0.2])
def test_decays_above_one(rise):
    """The recurrence grows where a log decay is positive: up to e^(64 x 0.2) = 4e5 inside a chunk here."""
    tokens, hk, hv, seed = 64 if rise > 0.1 else 200, 2, 4, 0xB2006200
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    g = np.where(synth.normal(seed, 9, g.shape) > -1.0, rise, g * np.float32(0.02)).astype(np.float32)
    state0 = (0.05 * synth.normal(seed, 5, (hv, DK, DK))).astype(np.float32)
    check_columns(*run_core(q, k, v, beta, g, state0, K.DTYPE_BF16))


def test_decays_beyond_the_chunk_kernels_range_are_reported():
    tokens, hk, hv, seed = 130, 1, 2, 0xB2006280
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    g[70:] = 0.3  # e^(0.3 x 58) = 2^25 in the second chunk
    stream = torch.cuda.current_stream()
    nbytes = K.gdn_core_workspace_bytes(tokens, hk, hv, DK, DK)
    workspace, out = torch.zeros(nbytes // 4, device=dev()), torch.zeros(tokens, hv, DK, device=dev())
    state = torch.zeros(hv, DK, DK, device=dev())
    operands = [act_tensor(x, K.DTYPE_F32) for x in (q, k, v, beta, g)]
    assert K.device_status(stream) == 0
    K.gdn_core(*operands, state, out, workspace, nbytes, tokens, hk, hv, DK, DK, K.DTYPE_F32, stream)
    assert K.device_status(stream) == K.DEVICE_DECAY_OUT_OF_RANGE
    assert K.device_status(stream) == 0  # reading cleared it


@pytest.mark.parametrize("norm", [1.0e-4, 1.0, 100.0])
def test_queries_of_any_norm(norm):
    """q usually carries 1 / sqrt(128); the output is linear in it."""
    tokens, hk, hv, seed = 150, 2, 4, 0xB2006290
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    state0 = (0.05 * synth.normal(seed, 5, (hv, DK, DK))).astype(np.float32)
    q = synth.round_bf16(q * np.float32(norm * DK ** 0.5))
    check_columns(*run_core(q, k, v, beta, g, state0, K.DTYPE_BF16))


@pytest.mark.parametrize("beta_scale,decay_scale", [(1.0e-3, 0.01), (1.0e-5, 0.01), (1.0e-5, 0.0), (1.0, 0.0), (1.0, 8.0)])
def test_small_gates(beta_scale, decay_scale):
    """Tokens that hardly write (T diag(beta) is all there is), no decay at all, and decay of e^-6 a token."""
    tokens, hk, hv, seed = 200, 2, 4, 0xB2006300
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    beta, g = (beta * np.float32(beta_scale)).astype(np.float32), (g * np.float32(decay_scale)).astype(np.float32)
    check_columns(*run_core(q, k, v, beta, g, np.zeros((hv, DK, DK), np.float32), K.DTYPE_BF16))


def test_keys_that_repeat():
    """Equal keys with beta near 1 and no decay: A is full of elements near 1, and the state is overwritten with every token,
    so that a result is the difference of operands of its own size: one more rounding of either."""
    tokens, hk, hv, seed = 200, 2, 4, 0xB2006400
    q, k, v, beta, g = core_operands(seed, tokens, hk, hv)
    k[1:] = k[:1]
    beta, g = np.full_like(beta, 0.98), np.full_like(g, -1.0e-3)
    got_out, got_state, want_out, want_state = run_core(q, k, v, beta, g, np.zeros((hv, DK, DK), np.float32), K.DTYPE_BF16)
    assert compare(got_out, want_out)["rel_l2"] <= COLUMN_TOLERANCE + 2 * 2.0 ** -11
    assert compare(got_state, want_state)["rel_l2"] <= COLUMN_TOLERANCE + 2 * 2.0 ** -11


# ---- layer calls -----------------------------------------------------------------------------------------------------
def in_half(run, dtype):
    """Operands of a LayerRun that FP16 holds exactly on both sides."""
    if dtype == K.DTYPE_F16:
        run.inp = run.inp.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("hk,hv,tokens", [(HK, HV, 1900), (2, 6, 10400)])
@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F16])
def test_long_layer_calls(hk, hv, tokens, dtype):
    """16-bit calls of 1776 CTAs and more take the image kernel with eight dims a lane, here with a ragged tail and a
    history; with six value heads the packed rows lie off the 16-byte boundary.  One more token follows on the states."""
    run = LayerRun(0xB2006500 + hv, hk, hv, 4, dtype, K.DTYPE_F32, tokens + 1)
    in_half(run, dtype)
    for count in (tokens, 1):
        out, want, _ = run.step(count)
        # the output is rounded to 16 bits: 2^-8 or 2^-11 of the value at most, beside what the products leave
        got, rounding = to_numpy_f32(out).reshape(want.shape), 2.0 ** (-8 if dtype == K.DTYPE_BF16 else -11)
        assert np.isfinite(got).all() and (np.abs(got - want) <= rounding * np.abs(want) + 3.0e-2).all()
        assert compare(got, want)["rel_l2"] <= 1.0e-2
        assert compare(to_numpy_f32(run.d_cs).reshape(-1), run.cs.reshape(-1))["max_abs"] == 0.0
        assert compare(to_numpy_f32(run.d_rs).reshape(-1), run.rs.reshape(-1))["rel_l2"] <= 1.0e-3
    assert K.device_status(torch.cuda.current_stream()) == 0


@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F16])
def test_a_long_layer_call_equals_the_same_tokens_in_pieces(dtype):
    """Pieces of whole chunks take the image kernel with four dims a lane, the whole call the one with eight; outputs,
    recurrent states and histories are bit-identical."""
    def run(pieces):
        layer = LayerRun(0xB2006600, HK, HV, 4, dtype, K.DTYPE_F32, sum(pieces))
        in_half(layer, dtype)
        outs, done, hidden = [], 0, HV * DK
        for count in pieces:
            shape = K.GatedDeltaShape(count, hidden, HK, HV, DK, DK, 4, 1.0e-6)
            nbytes = K.qwen35_gated_delta_workspace_bytes(shape)
            workspace = torch.zeros(nbytes // 4, device=dev())
            out = torch.zeros(count, hidden, device=dev(), dtype=torch.float16 if dtype == K.DTYPE_F16 else torch.bfloat16)
            K.qwen35_gated_delta(act_tensor(layer.inp[done:done + count], dtype), layer.d_conv_w, layer.d_rec_a, layer.d_dt,
                                 layer.d_norm, out, layer.d_cs, layer.d_rs, workspace, nbytes, shape, dtype, K.DTYPE_F32,
                                 torch.cuda.current_stream())
            torch.cuda.synchronize()
            outs.append(out)
            done += count
        return torch.cat(outs), layer.d_rs, layer.d_cs

    for whole, parts in zip(run([1900]), run([960, 64, 876])):
        assert torch.equal(whole, parts)


def test_saturated_gates_in_chunks():
    """The gates of test_layer_saturation_edges_stay_finite over three chunks: A from -12 to -0.001, dt_bias -25..5,
    b = +-30, z = +-18."""
    hk, hv, tokens = 2, 4, 170
    run = LayerRun(0xB2006700, hk, hv, 4, K.DTYPE_F32, K.DTYPE_F32, tokens)
    conv_dim = 2 * hk * DK + hv * DK
    run.rec_a = np.array([-12.0, -1.0, -0.05, -0.001], dtype=np.float32)
    run.dt_bias = np.array([-25.0, -3.0, 0.5, 5.0], dtype=np.float32)
    run.d_rec_a, run.d_dt = act_tensor(run.rec_a, K.DTYPE_F32), act_tensor(run.dt_bias, K.DTYPE_F32)
    run.inp[:, conv_dim:conv_dim + hv] = np.array([30.0, -30.0, 30.0, -30.0], dtype=np.float32)
    run.inp[:, conv_dim + 2 * hv::2] = 18.0
    run.inp[:, conv_dim + 2 * hv + 1::2] = -18.0
    out, want, _ = run.step(tokens)
    m = compare(to_numpy_f32(out), want)
    assert m["nonfinite"] == 0 and m["rel_l2"] <= COLUMN_TOLERANCE, m
    m = compare(to_numpy_f32(run.d_rs).reshape(-1), run.rs.reshape(-1))
    assert m["nonfinite"] == 0 and m["rel_l2"] <= COLUMN_TOLERANCE, m


@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F16, K.DTYPE_F32])
def test_layer_with_columns_of_any_magnitude(dtype):
    """Value channels whose convolution weights are ten decades apart, so that every column has factors of its own, in the
    form of the chain that norms and gates the outputs; another call follows on the states."""
    hk, hv, calls = 2, 4, (200, 70)
    run = LayerRun(0xB2006900, hk, hv, 4, dtype, K.DTYPE_F32, sum(calls))
    if dtype == K.DTYPE_F16:
        run.inp = run.inp.astype(np.float16).astype(np.float32)
    factors = np.resize((10.0 ** -np.arange(10)).astype(np.float32), DK)
    run.conv_w[2 * hk * DK:] *= np.tile(factors, hv)[:, None]
    run.rs *= factors
    run.d_conv_w, run.d_rs = act_tensor(run.conv_w, K.DTYPE_F32), torch.from_numpy(run.rs.copy()).to(dev())
    for count in calls:
        out, want, _ = run.step(count)
        got = to_numpy_f32(out).reshape(want.shape)
        assert compare(got, want)["nonfinite"] == 0 and compare(got, want)["rel_l2"] <= 1.0e-2
        errors = column_errors(to_numpy_f32(run.d_rs).reshape(hv, DK, DK), run.rs.reshape(hv, DK, DK), 1)
        assert errors.max() <= COLUMN_TOLERANCE, errors.max()
    assert K.device_status(torch.cuda.current_stream()) == 0


def test_layer_whose_coefficients_are_positive():
    """recurrent_a > 0 lets the state grow, by e^10 over the call here."""
    hk, hv, tokens = 2, 4, 170
    run = LayerRun(0xB2006800, hk, hv, 4, K.DTYPE_F32, K.DTYPE_F32, tokens)
    run.rec_a = np.float32([0.05, 0.08, 0.02, -0.5])
    run.d_rec_a = act_tensor(run.rec_a, K.DTYPE_F32)
    out, want, _ = run.step(tokens)
    run.check(out, want, chunked=True)
