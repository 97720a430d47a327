"""The workloads that the speed of this library is measured on.

Every case is a piece of what a program on top of the library has it do for the hybrid model it serves (16 query and
4 KV heads of 256 dims; 16 key and 32 value heads of 128 dims; convolution width 4), through the public entry points:

  attn_decode   one generated token's pass through the full-attention layers of one sequence: per layer the step in
                front of attention, then split-k decode on the layer's own KV cache, the position read on the device.
                The launches of a token are captured once and replayed, as the reference's executor runs decode.
  gdn_decode    the same token's pass through the gated-delta layers: one single-token layer call per layer, captured
                and replayed.
  serving       one decode step of one layer pair for a batch of sequences with ragged contexts: batched attention
                (contiguous caches, or pages of 256 tokens) and the batched gated-delta recurrence.
  attn_prompt   a prompt through one full-attention layer: per chunk of tokens the step in front of attention, then
                causal prefill, which appends to the KV cache; earlier chunks are the past of later ones.
  gdn_prompt    a prompt through one gated-delta layer, states carried from chunk to chunk.

`projections` says how the attention layers are driven: "fused" is the single prologue launch that hands BF16 to
attention; "executor" is the reference executor's own sequence (query/gate split, two norm + RoPE calls, attention) on
FP32 tensors.  `chunking` says how a prompt is fed: "whole" is one call; "executor" cuts it into calls of 512, 128,
17, 4, 2 and 1 tokens, as the executor does.
"""
from __future__ import annotations

import math

import torch

from raftinfer_b200 import kernels as K

HQ, HKV, D = 16, 4, 256            # full attention
HK, HV, DK, WIDTH = 16, 32, 128, 4  # gated delta
HIDDEN = HV * DK
CONV_DIM = 2 * HK * DK + HIDDEN
STRIDE = CONV_DIM + 2 * HV + HIDDEN  # packed row: q | k | v | b | a | z
ROTARY, ROPE_BASE, EPSILON = 64, 1.0e7, 1.0e-6
EXECUTOR_CHUNKS = (512, 128, 17, 4, 2, 1)
ATTENTION_LAYERS, DELTA_LAYERS = 8, 24
POLICY = K.Qwen35AttentionLaunchPolicy(K.ONLINE_TILED, K.KV_BF16, K.HEAD_MAJOR)

TORCH_DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
LIB_DTYPE = {"f32": K.DTYPE_F32, "bf16": K.DTYPE_BF16, "f16": K.DTYPE_F16}

_stream = None


def stream():
    """The stream of this program; the library does not take the default one."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def listed():
    return [
        # generation early in a chat, driven as the reference's executor drives it: launches and latency
        {"name": "attn_decode_777_f32", "kind": "attn_decode", "context": 777, "capacity": 4096,
         "layers": ATTENTION_LAYERS, "projections": "executor"},
        # generation behind a long document, the configuration of the headline benchmark (context 32768)
        {"name": "attn_decode_32k", "kind": "attn_decode", "context": 32768, "capacity": 32768,
         "layers": ATTENTION_LAYERS, "projections": "fused"},
        # the longest context of the benchmark, two of the layers
        {"name": "attn_decode_128k", "kind": "attn_decode", "context": 131000, "capacity": 131072,
         "layers": 2, "projections": "fused"},
        # the gated-delta layers of every generated token
        {"name": "gdn_decode_token", "kind": "gdn_decode", "layers": DELTA_LAYERS, "dtype": "bf16"},
        # a busy server: 64 sequences of 1 K to 32 K tokens
        {"name": "serving_64", "kind": "serving", "batch": 64, "shortest": 1024, "longest": 32768, "paged": False},
        # a quiet server with a paged cache: nine sequences, some of them just begun
        {"name": "serving_9_paged", "kind": "serving", "batch": 9, "shortest": 100, "longest": 6000, "paged": True},
        # a long prompt in one call
        {"name": "attn_prompt_4096", "kind": "attn_prompt", "tokens": 4096, "past": 0, "projections": "fused",
         "chunking": "whole"},
        # the same kind of prompt as the drop-in user meets it: FP32 tensors, calls of 512 tokens and a ragged rest
        {"name": "attn_prompt_2709_executor", "kind": "attn_prompt", "tokens": 2709, "past": 0,
         "projections": "executor", "chunking": "executor"},
        # the next turn of a chat: a short question behind a longer past
        {"name": "attn_prompt_201_past_1500", "kind": "attn_prompt", "tokens": 201, "past": 1500,
         "projections": "fused", "chunking": "whole"},
        # the gated-delta layer on a long prompt in one call ...
        {"name": "gdn_prompt_4096", "kind": "gdn_prompt", "tokens": 4096, "dtype": "bf16", "chunking": "whole"},
        # ... on a prompt in the executor's calls, FP32 ...
        {"name": "gdn_prompt_1173_executor", "kind": "gdn_prompt", "tokens": 1173, "dtype": "f32",
         "chunking": "executor"},
        # ... and on a short one
        {"name": "gdn_prompt_149", "kind": "gdn_prompt", "tokens": 149, "dtype": "bf16", "chunking": "whole"},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["attn_decode", "gdn_decode", "serving", "attn_prompt", "attn_prompt", "gdn_prompt",
                       "gdn_prompt", "gdn_prompt"])
    if kind == "attn_decode":
        context = _log_uniform(rng, 16, 120000)
        capacity = rng.choice([context, -(-context // 256) * 256, max(4096, -(-context // 1024) * 1024)])
        layers = max(1, min(ATTENTION_LAYERS, 250000 // context))
        return {"kind": kind, "context": context, "capacity": capacity, "layers": layers,
                "projections": rng.choice(["fused", "executor"])}
    if kind == "gdn_decode":
        return {"kind": kind, "layers": rng.randint(2, DELTA_LAYERS), "dtype": rng.choice(["bf16", "f32", "f16"])}
    if kind == "serving":
        longest = _log_uniform(rng, 200, 32768)
        return {"kind": kind, "batch": _log_uniform(rng, 1, 56), "shortest": _log_uniform(rng, 16, longest),
                "longest": longest, "paged": rng.random() < 0.5}
    if kind == "attn_prompt":
        tokens = _log_uniform(rng, 2, 3500)
        past = rng.choice([0, _log_uniform(rng, 1, 4000)])
        projections = rng.choice(["fused", "executor"])
        return {"kind": kind, "tokens": tokens, "past": past, "projections": projections,
                "chunking": rng.choice(["whole", "executor"])}
    return {"kind": kind, "tokens": _log_uniform(rng, 2, 4000), "dtype": rng.choice(["bf16", "bf16", "f32", "f16"]),
            "chunking": rng.choice(["whole", "whole", "executor"])}


def pieces(tokens, chunking):
    """The calls a prompt is fed in."""
    if chunking == "whole":
        return [tokens]
    out = []
    for size in EXECUTOR_CHUNKS:
        while tokens >= size:
            out.append(size)
            tokens -= size
    return out


def lengths_of(case):
    """Contexts of a serving batch, the new token included: spread evenly over the range, in a shuffled order."""
    n = case["batch"]
    low, high = case["shortest"], case["longest"]
    values = [low + (high - low) * (2 * i + 1) // (2 * n) for i in range(n)]
    order = sorted(range(n), key=lambda i: (i * 37) % 101)
    return [values[i] for i in order]


class Inputs:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.device = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.device).manual_seed(seed)

    def normal(self, *shape, dtype=torch.float32, scale=1.0):
        out = torch.empty(*shape, device=self.device, dtype=dtype).normal_(generator=self.gen)
        return out if scale == 1.0 else out.mul_(scale)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.empty(*shape, device=self.device).uniform_(low, high, generator=self.gen)

    def zeros(self, *shape, dtype=torch.float32):
        return torch.zeros(*shape, device=self.device, dtype=dtype)

    def unit(self, *shape):
        x = self.normal(*shape)
        return x / x.norm(dim=-1, keepdim=True)


# ---- full attention ---------------------------------------------------------------------------------------------
class AttentionLayer:
    """One full-attention layer's projections of `tokens` tokens, its KV cache holding `past` rows, and the buffers
    between its calls."""

    def __init__(self, inputs, tokens, past, capacity, projections):
        self.fused = projections == "fused"
        dtype = torch.bfloat16 if self.fused else torch.float32
        self.tokens, self.past, self.capacity = tokens, past, capacity
        self.query_gate = inputs.normal(tokens, HQ, 2 * D)
        self.key_in = inputs.normal(tokens, HKV, D)
        self.value_in = inputs.normal(tokens, HKV, D)
        self.query_norm = inputs.normal(D, scale=0.1).add_(1.0)
        self.key_norm = inputs.normal(D, scale=0.1).add_(1.0)
        self.cache = inputs.normal(2, HKV, capacity, D, dtype=torch.bfloat16)
        self.cache[:, :, past:] = 0.0
        self.cache_bytes = self.cache.numel() * 2
        self.query = inputs.zeros(tokens, HQ, D, dtype=dtype)
        self.gate = inputs.zeros(tokens, HQ, D, dtype=dtype)
        self.key = inputs.zeros(tokens, HKV, D, dtype=dtype)
        self.value = inputs.zeros(tokens, HKV, D, dtype=dtype) if self.fused else self.value_in
        self.query_raw = None if self.fused else inputs.zeros(tokens, HQ, D)
        self.output = inputs.zeros(tokens, HQ, D, dtype=dtype)
        self.dtype = K.DTYPE_BF16 if self.fused else K.DTYPE_F32

    def project(self, first, count, device_position=None):
        """From the projections of tokens [first, first + count) to what attention takes."""
        rows = slice(first, first + count)
        position = 0 if device_position is not None else self.past + first
        if self.fused:
            shape = K.Qwen35AttentionShape(count, HQ, HKV, D, self.capacity, self.past + first)
            K.attention_prologue(self.query_gate[rows], self.key_in[rows], self.value_in[rows], self.query_norm,
                                 self.key_norm, self.query[rows], self.gate[rows], self.key[rows], self.value[rows],
                                 shape, ROTARY, ROPE_BASE, EPSILON, K.DTYPE_F32, K.DTYPE_F32, K.DTYPE_BF16, stream(),
                                 device_position)
            return
        K.qwen35_split_full_query_gate(self.query_gate[rows], self.query_raw[rows], self.gate[rows], count, HQ, D,
                                       K.DTYPE_F32, stream())
        for source, weight, out, heads in ((self.query_raw, self.query_norm, self.query, HQ),
                                           (self.key_in, self.key_norm, self.key, HKV)):
            K.qwen35_qk_norm_rope(source[rows], weight, out[rows],
                                  K.QkNormRopeShape(count, heads, D, ROTARY, position, ROPE_BASE), EPSILON,
                                  K.DTYPE_F32, K.DTYPE_F32, stream(), device_position)

    def prefill(self, first, count):
        rows = slice(first, first + count)
        shape = K.Qwen35AttentionShape(count, HQ, HKV, D, self.capacity, self.past + first)
        K.qwen35_causal_attention(self.query[rows], self.key[rows], self.value[rows], self.gate[rows],
                                  self.output[rows], self.cache, self.cache_bytes, None, 0, shape, self.dtype, POLICY,
                                  stream())


class AttentionPrompt:
    def __init__(self, case, seed):
        tokens, past = case["tokens"], case["past"]
        capacity = -(-(past + tokens) // 256) * 256
        self.layer = AttentionLayer(Inputs(seed), tokens, past, capacity, case["projections"])
        self.pieces = pieces(tokens, case["chunking"])

    def run(self):
        first = 0
        for count in self.pieces:
            self.layer.project(first, count)
            self.layer.prefill(first, count)
            first += count
        return {"output": self.layer.output, "cache": self.layer.cache}


class AttentionDecode:
    def __init__(self, case, seed):
        inputs = Inputs(seed)
        context, capacity = case["context"], case["capacity"]
        self.layers = [AttentionLayer(inputs, 1, context - 1, capacity, case["projections"])
                       for _ in range(case["layers"])]
        self.shape = K.Qwen35AttentionShape(1, HQ, HKV, D, capacity, context - 1)
        self.plan = K.qwen35_online_decode_plan(self.shape, K.AUTO_SELECT, context)
        layout = K.qwen35_online_decode_workspace_layout(self.shape, self.plan.resolved_mode)
        self.workspace, self.workspace_bytes = inputs.zeros(layout.bytes // 4), layout.bytes
        self.position = torch.tensor([context - 1], device=inputs.device, dtype=torch.int32)
        self.graph = capture(self.token)

    def token(self):
        for layer in self.layers:
            layer.project(0, 1, self.position)
            K.qwen35_online_attention_decode(layer.query, layer.key, layer.value, layer.gate, layer.output,
                                             layer.cache, layer.cache_bytes, self.workspace, self.workspace_bytes,
                                             self.shape, layer.dtype, K.KV_BF16, K.HEAD_MAJOR, self.plan,
                                             self.position, stream())

    def run(self):
        replay(self.graph)
        return {"output": [layer.output for layer in self.layers], "cache": [layer.cache for layer in self.layers]}


# ---- gated delta ------------------------------------------------------------------------------------------------
class DeltaLayer:
    """One gated-delta layer: weights, carried states, packed input of `tokens` tokens.  The decay parameters are
    spread as such layers are trained: coefficients of 1 to 16, time steps of 0.001 to 0.1 per token.  `conv_state`,
    `state` and `output` are the layer's rows of what the program holds for all of them."""

    def __init__(self, inputs, tokens, dtype, conv_state, state, output):
        self.dtype = LIB_DTYPE[dtype]
        self.packed = inputs.normal(tokens, STRIDE, dtype=TORCH_DTYPE[dtype])
        self.conv_weight = inputs.normal(CONV_DIM, WIDTH, scale=0.3)
        self.recurrent_a = -inputs.uniform(HV, low=1.0, high=16.0)
        step = torch.exp(inputs.uniform(HV, low=math.log(1.0e-3), high=math.log(1.0e-1)))
        self.dt_bias = step + torch.log(-torch.expm1(-step))  # the inverse of softplus
        self.norm_weight = inputs.normal(DK, scale=0.1).add_(1.0)
        self.conv_state, self.state, self.output = conv_state, state, output

    def call(self, first, count, workspace, workspace_bytes, policy):
        rows = slice(first, first + count)
        shape = K.GatedDeltaShape(count, HIDDEN, HK, HV, DK, DK, WIDTH, EPSILON)
        K.qwen35_gated_delta(self.packed[rows], self.conv_weight, self.recurrent_a, self.dt_bias, self.norm_weight,
                             self.output[rows], self.conv_state, self.state, workspace, workspace_bytes, shape,
                             self.dtype, K.DTYPE_F32, stream(), policy)


def delta_layers(inputs, layers, tokens, dtype):
    """`layers` gated-delta layers and the tensors that hold their states and outputs: (layers, tensors)."""
    held = {"conv_state": inputs.normal(layers, CONV_DIM, WIDTH - 1, scale=0.5),
            "state": inputs.normal(layers, HV, DK, DK, scale=0.05),
            "output": inputs.zeros(layers, tokens, HIDDEN, dtype=TORCH_DTYPE[dtype])}
    return [DeltaLayer(inputs, tokens, dtype, **{k: v[i] for k, v in held.items()}) for i in range(layers)], held


def delta_workspace(inputs, tokens):
    shape = K.GatedDeltaShape(tokens, HIDDEN, HK, HV, DK, DK, WIDTH, EPSILON)
    nbytes = K.qwen35_gated_delta_workspace_bytes(shape)
    return torch.empty(-(-nbytes // 4), device=inputs.device), nbytes, K.qwen35_gated_delta_select_policy(shape, tokens)


class DeltaPrompt:
    def __init__(self, case, seed):
        inputs = Inputs(seed)
        self.pieces = pieces(case["tokens"], case["chunking"])
        (self.layer,), self.held = delta_layers(inputs, 1, case["tokens"], case["dtype"])
        self.workspace = delta_workspace(inputs, max(self.pieces))

    def run(self):
        first = 0
        for count in self.pieces:
            self.layer.call(first, count, *self.workspace)
            first += count
        return self.held


class DeltaDecode:
    def __init__(self, case, seed):
        inputs = Inputs(seed)
        self.layers, self.held = delta_layers(inputs, case["layers"], 1, case["dtype"])
        self.workspace = delta_workspace(inputs, 1)
        self.graph = capture(self.token)

    def token(self):
        for layer in self.layers:
            layer.call(0, 1, *self.workspace)

    def run(self):
        replay(self.graph)
        return self.held


# ---- serving ----------------------------------------------------------------------------------------------------
class Serving:
    def __init__(self, case, seed):
        inputs = Inputs(seed)
        lengths = lengths_of(case)
        batch, dev = case["batch"], inputs.device
        self.batch, self.paged = batch, case["paged"]
        capacities = [-(-n // 256) * 256 for n in lengths]
        self.largest = max(capacities)
        self.positions = torch.tensor([n - 1 for n in lengths], device=dev, dtype=torch.int32)
        # the KV rows of all sequences: back to back, or in pages handed out in no particular order
        blocks = [c // K.PAGE_TOKENS for c in capacities]
        self.pages = sum(blocks)
        self.pool = inputs.normal(self.pages, 2 * HKV * K.PAGE_TOKENS * D, dtype=torch.bfloat16)
        if self.paged:
            shuffled = torch.randperm(self.pages, generator=torch.Generator().manual_seed(seed)).tolist()
            rows, handed = [], 0
            for n in blocks:
                rows.append(shuffled[handed:handed + n] + [0] * (max(blocks) - n))
                handed += n
            self.tables, self.table_width = torch.tensor(rows, device=dev, dtype=torch.int32), max(blocks)
        else:
            firsts = [sum(blocks[:i]) for i in range(batch)]
            self.cache_pointers = torch.tensor([self.pool[b].data_ptr() for b in firsts], device=dev,
                                               dtype=torch.int64)
            self.capacities = torch.tensor(capacities, device=dev, dtype=torch.int32)
        self.workspace_bytes = K.batched_decode_workspace_bytes(batch, self.largest)
        self.workspace = torch.empty(-(-self.workspace_bytes // 4), device=dev)
        bf16 = torch.bfloat16
        self.query, self.gate = inputs.normal(batch, HQ, D, dtype=bf16), inputs.normal(batch, HQ, D, dtype=bf16)
        self.key, self.value = inputs.normal(batch, HKV, D, dtype=bf16), inputs.normal(batch, HKV, D, dtype=bf16)
        self.output = inputs.zeros(batch, HQ, D, dtype=bf16)
        self.states = inputs.normal(batch, HV, DK, DK, scale=0.05)
        self.state_pointers = torch.tensor([s.data_ptr() for s in self.states], device=dev, dtype=torch.int64)
        self.delta_q = (inputs.unit(batch, HK, DK) / DK ** 0.5).to(bf16)
        self.delta_k = inputs.unit(batch, HK, DK).to(bf16)
        self.delta_v = inputs.normal(batch, HV, DK, dtype=bf16)
        self.beta = torch.sigmoid(inputs.normal(batch, HV))
        self.log_decay = -inputs.uniform(batch, HV, low=0.001, high=1.0)
        self.delta_output = inputs.zeros(batch, HV, DK)

    def run(self):
        if self.paged:
            K.paged_decode_attention(self.query, self.key, self.value, self.gate, self.output, self.pool, self.pages,
                                     self.tables, self.table_width, self.positions, self.batch, self.workspace,
                                     self.workspace_bytes, stream())
        else:
            K.batched_decode_attention(self.query, self.key, self.value, self.gate, self.output, self.cache_pointers,
                                       self.capacities, self.positions, self.batch, self.largest, self.workspace,
                                       self.workspace_bytes, stream())
        K.batched_gdn_decode(self.delta_q, self.delta_k, self.delta_v, self.beta, self.log_decay, self.state_pointers,
                             self.delta_output, self.batch, HK, HV, stream())
        return {"output": self.output, "delta_output": self.delta_output, "states": self.states, "cache": self.pool}


def capture(token):
    """The launches of `token` as a graph: run once as they are (the first call of a process sets the kernels up),
    then recorded."""
    torch.cuda.synchronize()
    token()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream()):
        token()
    return graph


def replay(graph):
    with torch.cuda.stream(stream()):
        graph.replay()


KINDS = {"attn_prompt": AttentionPrompt, "attn_decode": AttentionDecode, "gdn_prompt": DeltaPrompt,
         "gdn_decode": DeltaDecode, "serving": Serving}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ------------------------------------------------------------------------------
def _attention_tokens_bytes(tokens, projections):
    """Projections read, outputs written, new cache rows written."""
    return tokens * ((2 * HQ + 2 * HKV) * D * 4 + HQ * D * (2 if projections == "fused" else 4) + 2 * HKV * D * 2)


def _delta_work(tokens, dtype, calls):
    element = 4 if dtype == "f32" else 2
    weights = CONV_DIM * WIDTH * 4 + 2 * HV * 4 + DK * 4
    states = 2 * (HV * DK * DK + CONV_DIM * (WIDTH - 1)) * 4
    return {"bytes": tokens * (STRIDE + HIDDEN) * element + calls * (weights + states),
            "flops": tokens * HV * 6 * DK * DK}


def work(case):
    kind = case["kind"]
    if kind == "attn_prompt":
        tokens, past = case["tokens"], case["past"]
        return {"bytes": _attention_tokens_bytes(tokens, case["projections"]) + past * 2 * HKV * D * 2,
                "flops": 4 * HQ * D * (tokens * past + tokens * (tokens + 1) // 2)}
    if kind == "attn_decode":
        context, layers = case["context"], case["layers"]
        return {"bytes": layers * (_attention_tokens_bytes(1, case["projections"]) + (context - 1) * 2 * HKV * D * 2),
                "flops": layers * 4 * HQ * D * context}
    if kind == "gdn_prompt":
        return _delta_work(case["tokens"], case["dtype"], 1)
    if kind == "gdn_decode":
        one = _delta_work(1, case["dtype"], 1)
        return {key: case["layers"] * value for key, value in one.items()}
    batch, tokens = case["batch"], sum(lengths_of(case))
    attention = tokens * 2 * HKV * D * 2 + batch * (3 * HQ + 2 * HKV) * D * 2
    delta = batch * (2 * HV * DK * DK * 4 + (2 * HK + HV) * DK * 2 + HV * 8 + HV * DK * 4)
    return {"bytes": attention + delta, "flops": tokens * 4 * HQ * D + batch * HV * 6 * DK * DK}


def tolerance(case):
    """About four times the distance from the same pass computed in 64 bits (2-norm; largest single value)."""
    kind = case["kind"]
    if kind == "attn_decode":  # BF16 queries, keys and outputs; FP32 tensors against a BF16 cache
        return {"rel": 1.0e-2, "max": 4.0e-2} if case["projections"] == "fused" else {"rel": 3.0e-4, "max": 6.0e-3}
    if kind == "serving":
        return {"rel": 7.0e-3, "max": 1.6e-2}
    if kind == "attn_prompt":  # the probabilities are BF16 in both forms
        return {"rel": 1.4e-2, "max": 0.45}
    recurrent = kind == "gdn_decode" or max(pieces(case["tokens"], case["chunking"])) < 64
    if case["dtype"] == "bf16":
        return {"rel": 7.0e-3, "max": 2.0e-2 if recurrent else 0.1}
    if recurrent:  # FP32 throughout: what is left is the rounding of the output
        return {"rel": 1.0e-5, "max": 1.0e-4} if case["dtype"] == "f32" else {"rel": 1.0e-3, "max": 4.0e-3}
    return {"rel": 2.0e-3, "max": 0.12}  # products of chunks with 10-bit mantissas
