// The steps of qwen35_gated_delta on either side of the recurrence, for key_dim = value_dim = 128:
//   prologue  depthwise causal convolution + SiLU over the q|k|v channels, L2 normalisation of every q
//             and k head (q also scaled by 1/sqrt(128)), beta = sigmoid(b), log decay = A * softplus(a + dt)
//             (cpp/kernels/qwen35_delta.cu:236-276,375-411,522-529; CPU cpp/reference/qwen35.cpp:417-469);
//   state     shift of the convolution history [channel][W-1] (cpp/kernels/qwen35_delta.cu:267-275);
//   epilogue  per-head RMSNorm(128) * weight * SiLU(z) (cpp/kernels/qwen35_delta.cu:579-621).
// Unlike the reference's convolution kernel, which walks the tokens serially per channel, every
// (token, head vector) pair is independent: a tap is read from the token stream or, for the first W-1
// tokens, from the carried history.  These kernels are the general path: conv_width 4 on aligned tensors takes the
// warp-per-vector ones (16-byte accesses), other widths and odd alignments the one-CTA-per-vector ones.  Calls of up to
// 63 tokens with conv_width 4 and at most two value heads per key head are one launch (below), longer ones of that
// width the chunk kernels (gdn_image.cu, gdn_chunk.cu).

#include "common.hpp"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace rib200 {
namespace {

constexpr int kDim = 128;
constexpr float kQkEpsilon = 1.0e-6F;

__device__ __forceinline__ float load_any(const void *base, std::size_t index, int32_t dtype) {
  if (dtype == RIB200_DTYPE_F32) {
    return static_cast<const float *>(base)[index];
  }
  if (dtype == RIB200_DTYPE_F16) {
    return __half2float(static_cast<const __half *>(base)[index]);
  }
  return __bfloat162float(static_cast<const __nv_bfloat16 *>(base)[index]);
}

__device__ __forceinline__ void store_any(void *base, std::size_t index, int32_t dtype, float value) {
  if (dtype == RIB200_DTYPE_F32) {
    static_cast<float *>(base)[index] = value;
  } else if (dtype == RIB200_DTYPE_F16) {
    static_cast<__half *>(base)[index] = __float2half_rn(value);
  } else {
    static_cast<__nv_bfloat16 *>(base)[index] = __float2bfloat16_rn(value);
  }
}

__device__ __forceinline__ float silu(float x) { return x / (1.0F + expf(-x)); }

__device__ __forceinline__ float softplus(float x) {
  if (x > 20.0F) {
    return x;
  }
  if (x < -20.0F) {
    return expf(x);
  }
  return log1pf(expf(x));
}

// sum over the 128 threads of the block, returned to all of them
__device__ __forceinline__ float block_sum_128(float value, float *scratch) {
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    value += __shfl_xor_sync(0xFFFFFFFFU, value, offset);
  }
  if ((threadIdx.x & 31) == 0) {
    scratch[threadIdx.x >> 5] = value;
  }
  __syncthreads();
  return (scratch[0] + scratch[1]) + (scratch[2] + scratch[3]);
}

struct LayerParams {
  const void *input;
  const void *conv_weight, *recurrent_a, *dt_bias, *output_norm_weight;
  void *output;
  float *convolution_state;
  float *recurrent_state; // one-launch forms only (1 to 63 tokens)
  float *convolved;
  float *beta;
  float *log_decay;
  const float *raw;
  std::uint32_t tokens, key_heads, value_heads, conv_width;
  std::uint32_t conv_dim, token_stride;
  float epsilon;
  int32_t dtype, weight_dtype;
};

// grid (2*Hk + Hv head vectors, tokens), 128 threads = the 128 channels of the vector
__global__ void __launch_bounds__(kDim) gdn_prologue_kernel(const LayerParams p) {
  __shared__ float scratch[4];
  grid_dependency_wait();
  grid_dependents_may_launch();
  const std::uint32_t vec = blockIdx.x;
  const std::uint32_t tok = blockIdx.y;
  const std::uint32_t channel = vec * kDim + threadIdx.x;
  const std::uint32_t history = p.conv_width - 1;
  const std::size_t weight_base = static_cast<std::size_t>(channel) * p.conv_width;
  float sum = load_any(p.input, static_cast<std::size_t>(tok) * p.token_stride + channel, p.dtype) *
              load_any(p.conv_weight, weight_base + history, p.weight_dtype);
  for (std::uint32_t h = 0; h < history; ++h) {
    const std::uint32_t source = tok + h; // position in [history | tokens]
    const float previous =
        source < history
            ? p.convolution_state[static_cast<std::size_t>(channel) * history + source]
            : load_any(p.input, static_cast<std::size_t>(source - history) * p.token_stride + channel, p.dtype);
    sum += previous * load_any(p.conv_weight, weight_base + h, p.weight_dtype);
  }
  float value = silu(sum);
  if (vec < 2 * p.key_heads) {
    const float squares = block_sum_128(value * value, scratch);
    value *= rsqrtf(squares + kQkEpsilon);
    if (vec < p.key_heads) {
      value *= rsqrtf(static_cast<float>(kDim));
    }
  } else if (threadIdx.x == 0) {
    const std::uint32_t head = vec - 2 * p.key_heads;
    const std::size_t gates = static_cast<std::size_t>(tok) * p.token_stride + p.conv_dim;
    const float b = load_any(p.input, gates + head, p.dtype);
    const float a = load_any(p.input, gates + p.value_heads + head, p.dtype);
    p.beta[static_cast<std::size_t>(tok) * p.value_heads + head] = 1.0F / (1.0F + expf(-b));
    p.log_decay[static_cast<std::size_t>(tok) * p.value_heads + head] =
        load_any(p.recurrent_a, head, p.weight_dtype) * softplus(a + load_any(p.dt_bias, head, p.weight_dtype));
  }
  p.convolved[static_cast<std::size_t>(tok) * p.conv_dim + channel] = value;
}

// ---- fast forms for conv_width == 4 (the model's width) ---------------------------------------------
// A warp owns one head vector (128 channels, four per lane) over four consecutive tokens: the seven input rows
// it needs are fetched once, 8 or 16 bytes per lane and row, whole 256/512-byte segments per warp, and slide
// through registers; the sum of squares of a q or k vector is five shuffles.  Dtype is a template parameter.
template <int Dtype> struct Io;
template <> struct Io<RIB200_DTYPE_F32> {
  static __device__ __forceinline__ float4 load4(const void *base, std::size_t index) {
    return *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + index);
  }
  static __device__ __forceinline__ void store4(void *base, std::size_t index, float4 v) {
    *reinterpret_cast<float4 *>(static_cast<float *>(base) + index) = v;
  }
};
template <> struct Io<RIB200_DTYPE_BF16> {
  static __device__ __forceinline__ float4 load4(const void *base, std::size_t index) {
    const uint2 raw = *reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(base) + index);
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xFFFF0000U),
                       __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xFFFF0000U));
  }
  static __device__ __forceinline__ void store4(void *base, std::size_t index, float4 v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y);
    const __nv_bfloat162 hi = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(base) + index) =
        make_uint2(*reinterpret_cast<const std::uint32_t *>(&lo), *reinterpret_cast<const std::uint32_t *>(&hi));
  }
};
template <> struct Io<RIB200_DTYPE_F16> {
  static __device__ __forceinline__ float4 load4(const void *base, std::size_t index) {
    const uint2 raw = *reinterpret_cast<const uint2 *>(static_cast<const __half *>(base) + index);
    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  static __device__ __forceinline__ void store4(void *base, std::size_t index, float4 v) {
    const __half2 lo = __floats2half2_rn(v.x, v.y);
    const __half2 hi = __floats2half2_rn(v.z, v.w);
    *reinterpret_cast<uint2 *>(static_cast<__half *>(base) + index) =
        make_uint2(*reinterpret_cast<const std::uint32_t *>(&lo), *reinterpret_cast<const std::uint32_t *>(&hi));
  }
};

// SiLU on the special-function unit (ex2 + rcp instead of a full-precision exponential and division): the vector
// kernels are bound by instruction issue otherwise.  Relative error about 1e-6.
__device__ __forceinline__ float silu_fast(float x) {
  float e;
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(e) : "f"(x * -1.4426950408889634F));
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(1.0F + e));
  return x * r;
}

constexpr int kTokensPerWarp = 4;  // tokens of one step of a warp
constexpr int kStepsPerWarp = 4;   // steps a warp walks: its window of input rows slides, nothing is read twice
constexpr int kFastWidth = 4;

// grid (ceil(tokens / 16), ceil((2 Hk + Hv + 1) / 8)), 256 threads: warp w of the CTA takes head vector
// 8 blockIdx.y + w over 16 consecutive tokens, four at a time; the rows of the next four are in flight while the
// current four are convolved, and the last three rows of a step are the history of the next.  The vector after the
// last one stands for the gates (lane = value head, any head count).
template <int Dtype> __global__ void __launch_bounds__(256, 3) gdn_prologue_w4_kernel(const LayerParams p) {
  grid_dependency_wait();
  grid_dependents_may_launch(); // the kernels behind this one set themselves up early and wait for it to end
  const int lane = threadIdx.x & 31;
  const std::uint32_t vec = blockIdx.y * 8 + (threadIdx.x >> 5);
  const std::uint32_t vectors = 2 * p.key_heads + p.value_heads;
  const std::uint32_t first = blockIdx.x * (kTokensPerWarp * kStepsPerWarp);
  if (vec > vectors) {
    return;
  }
  if (vec == vectors) {
    for (std::uint32_t head = lane; head < p.value_heads; head += 32) {
      const float a_coeff = load_any(p.recurrent_a, head, p.weight_dtype);
      const float dt = load_any(p.dt_bias, head, p.weight_dtype);
      for (std::uint32_t tok = first; tok < min(p.tokens, first + kTokensPerWarp * kStepsPerWarp); ++tok) {
        const std::size_t gates = static_cast<std::size_t>(tok) * p.token_stride + p.conv_dim;
        const float b = load_any(p.input, gates + head, p.dtype);
        const float a = load_any(p.input, gates + p.value_heads + head, p.dtype);
        p.beta[static_cast<std::size_t>(tok) * p.value_heads + head] = 1.0F / (1.0F + expf(-b));
        p.log_decay[static_cast<std::size_t>(tok) * p.value_heads + head] = a_coeff * softplus(a + dt);
      }
    }
    return;
  }
  const std::uint32_t channel = vec * kDim + 4 * lane;
  // taps of this lane's four channels: weight[channel][4], oldest first
  float w[4][kFastWidth];
  if (p.weight_dtype == RIB200_DTYPE_F32) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 taps = *reinterpret_cast<const float4 *>(static_cast<const float *>(p.conv_weight) +
                                                            static_cast<std::size_t>(channel + c) * kFastWidth);
      w[c][0] = taps.x;
      w[c][1] = taps.y;
      w[c][2] = taps.z;
      w[c][3] = taps.w;
    }
  } else {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
      for (int h = 0; h < kFastWidth; ++h) {
        w[c][h] = load_any(p.conv_weight, static_cast<std::size_t>(channel + c) * kFastWidth + h, p.weight_dtype);
      }
    }
  }
  auto load_row = [&](long long tok) {
    if (tok >= 0 && tok < static_cast<long long>(p.tokens)) {
      return Io<Dtype>::load4(p.input, static_cast<std::size_t>(tok) * p.token_stride + channel);
    }
    return make_float4(0.0F, 0.0F, 0.0F, 0.0F);
  };
  // window: x[0..2] the three rows before the step, x[3..6] the step's own rows
  float4 x[kTokensPerWarp + kFastWidth - 1];
#pragma unroll
  for (int r = 0; r < kTokensPerWarp + kFastWidth - 1; ++r) {
    x[r] = load_row(static_cast<long long>(first) + r - (kFastWidth - 1));
  }
  if (first == 0) {
    // history [channel][3]: element h is the token 3 - h steps before this call's first one
    const float *hist = p.convolution_state + static_cast<std::size_t>(channel) * (kFastWidth - 1);
#pragma unroll
    for (int h = 0; h < kFastWidth - 1; ++h) {
      x[h] = make_float4(hist[h], hist[(kFastWidth - 1) + h], hist[2 * (kFastWidth - 1) + h],
                         hist[3 * (kFastWidth - 1) + h]);
    }
  }
  const bool is_qk = vec < 2 * p.key_heads;
  const float q_scale = vec < p.key_heads ? rsqrtf(static_cast<float>(kDim)) : 1.0F;
#pragma unroll
  for (int step = 0; step < kStepsPerWarp; ++step) {
    const std::uint32_t tok0 = first + step * kTokensPerWarp;
    if (tok0 >= p.tokens) {
      break;
    }
    float4 next[kTokensPerWarp];
    if (step + 1 < kStepsPerWarp) {
#pragma unroll
      for (int r = 0; r < kTokensPerWarp; ++r) {
        next[r] = load_row(static_cast<long long>(tok0) + kTokensPerWarp + r);
      }
    }
#pragma unroll
    for (int i = 0; i < kTokensPerWarp; ++i) {
      const std::uint32_t tok = tok0 + i;
      float4 sum = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
      // the reference adds the current token's tap first, then the history taps oldest first
      sum.x = x[i + 3].x * w[0][3];
      sum.y = x[i + 3].y * w[1][3];
      sum.z = x[i + 3].z * w[2][3];
      sum.w = x[i + 3].w * w[3][3];
#pragma unroll
      for (int h = 0; h < kFastWidth - 1; ++h) {
        sum.x += x[i + h].x * w[0][h];
        sum.y += x[i + h].y * w[1][h];
        sum.z += x[i + h].z * w[2][h];
        sum.w += x[i + h].w * w[3][h];
      }
      float4 value = make_float4(silu_fast(sum.x), silu_fast(sum.y), silu_fast(sum.z), silu_fast(sum.w));
      if (is_qk) {
        float squares = (value.x * value.x + value.y * value.y) + (value.z * value.z + value.w * value.w);
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
          squares += __shfl_xor_sync(0xFFFFFFFFU, squares, offset);
        }
        const float scale = rsqrtf(squares + kQkEpsilon) * q_scale;
        value.x *= scale;
        value.y *= scale;
        value.z *= scale;
        value.w *= scale;
      }
      if (tok < p.tokens) {
        *reinterpret_cast<float4 *>(p.convolved + static_cast<std::size_t>(tok) * p.conv_dim + channel) = value;
      }
    }
    if (step + 1 < kStepsPerWarp) {
#pragma unroll
      for (int h = 0; h < kFastWidth - 1; ++h) {
        x[h] = x[kTokensPerWarp + h];
      }
#pragma unroll
      for (int r = 0; r < kTokensPerWarp; ++r) {
        x[kFastWidth - 1 + r] = next[r];
      }
    }
  }
}

// grid (ceil(tokens * value_heads / 8)), 256 threads: a warp per (token, value head), four channels per lane
template <int Dtype> __global__ void __launch_bounds__(256) gdn_epilogue_warp_kernel(const LayerParams p) {
  grid_dependency_wait(); // launched with programmatic serialisation behind the recurrence, whose output it reads
  const int lane = threadIdx.x & 31;
  const std::size_t item = static_cast<std::size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  if (item >= static_cast<std::size_t>(p.tokens) * p.value_heads) {
    return;
  }
  const std::size_t tok = item / p.value_heads;
  const std::uint32_t head = static_cast<std::uint32_t>(item % p.value_heads);
  const std::size_t index = item * kDim + 4 * lane; // [token][head][128]
  const float4 value = *reinterpret_cast<const float4 *>(p.raw + index);
  const float4 z = Io<Dtype>::load4(p.input, tok * p.token_stride + p.conv_dim + 2 * p.value_heads + head * kDim +
                                                 4 * lane);
  float squares = (value.x * value.x + value.y * value.y) + (value.z * value.z + value.w * value.w);
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    squares += __shfl_xor_sync(0xFFFFFFFFU, squares, offset);
  }
  const float scale = rsqrtf(squares / static_cast<float>(kDim) + p.epsilon);
  float4 out;
  out.x = value.x * scale * load_any(p.output_norm_weight, 4 * lane, p.weight_dtype) * silu_fast(z.x);
  out.y = value.y * scale * load_any(p.output_norm_weight, 4 * lane + 1, p.weight_dtype) * silu_fast(z.y);
  out.z = value.z * scale * load_any(p.output_norm_weight, 4 * lane + 2, p.weight_dtype) * silu_fast(z.z);
  out.w = value.w * scale * load_any(p.output_norm_weight, 4 * lane + 3, p.weight_dtype) * silu_fast(z.w);
  Io<Dtype>::store4(p.output, index, out);
}

// Whether the vector forms apply: every row segment a lane touches must start on the boundary of its access.
bool vector_forms_apply(const LayerParams &p) {
  const std::size_t element = p.dtype == RIB200_DTYPE_F32 ? 4 : 2;
  const std::size_t access = 4 * element;
  if (p.weight_dtype == RIB200_DTYPE_F32 && reinterpret_cast<std::uintptr_t>(p.conv_weight) % 16 != 0) {
    return false; // the four taps of a channel are fetched as one 16-byte word
  }
  return reinterpret_cast<std::uintptr_t>(p.input) % access == 0 &&
         reinterpret_cast<std::uintptr_t>(p.output) % access == 0 && (p.token_stride * element) % access == 0 &&
         ((p.conv_dim + 2 * p.value_heads) * element) % access == 0;
}

// one thread per channel: new history[h] = element tokens + h of [old history | token stream]
__global__ void gdn_conv_state_kernel(const LayerParams p) {
  grid_dependents_may_launch();
  const std::uint32_t channel = blockIdx.x * blockDim.x + threadIdx.x;
  const std::uint32_t history = p.conv_width - 1;
  if (channel >= p.conv_dim || history == 0) {
    return;
  }
  float next[8];
  for (std::uint32_t h = 0; h < history; ++h) {
    const std::size_t source = static_cast<std::size_t>(p.tokens) + h;
    next[h] = source < history
                  ? p.convolution_state[static_cast<std::size_t>(channel) * history + source]
                  : load_any(p.input, (source - history) * p.token_stride + channel, p.dtype);
  }
  // launched with programmatic serialisation behind the prologue, which reads the old history: write after it ended
  grid_dependency_wait();
  for (std::uint32_t h = 0; h < history; ++h) {
    p.convolution_state[static_cast<std::size_t>(channel) * history + h] = next[h];
  }
}

// grid (value_heads, tokens), 128 threads
__global__ void __launch_bounds__(kDim) gdn_epilogue_kernel(const LayerParams p) {
  grid_dependency_wait();
  __shared__ float scratch[4];
  const std::uint32_t head = blockIdx.x;
  const std::uint32_t tok = blockIdx.y;
  const std::size_t hidden = static_cast<std::size_t>(p.value_heads) * kDim;
  const std::size_t index = static_cast<std::size_t>(tok) * hidden + head * kDim + threadIdx.x;
  const float value = p.raw[index];
  const float squares = block_sum_128(value * value, scratch);
  const float scale = rsqrtf(squares / static_cast<float>(kDim) + p.epsilon);
  const float z = load_any(p.input,
                           static_cast<std::size_t>(tok) * p.token_stride + p.conv_dim + 2 * p.value_heads +
                               head * kDim + threadIdx.x,
                           p.dtype);
  const float normalised = value * scale * load_any(p.output_norm_weight, threadIdx.x, p.weight_dtype);
  store_any(p.output, index, p.dtype, normalised * silu(z));
}

// ---- one token in one launch ---------------------------------------------------------------------------
// A decode step of the layer is latency: 4 MiB of state traffic (0.6 us of HBM) and 25 KB of input.  The four launches
// of the general path (prologue, history, recurrence, epilogue) cost 12.0 us a layer in a captured chain of 24 layers,
// most of it hand-over between grids; this form costs 3.6 us (4.2 MB of state in and out: 1.2 TB/s), 2.2
// to 2.6 of kernel and the rest hand-over; 4.4 us without the L2 hints in front of the wait.
//
// A cluster serves one key head: four CTAs (32 state columns each) per value head that shares it, one or two value
// heads.  Everything that has to meet across CTAs meets inside that cluster: the convolution history of the q and k
// channels is read by all of its CTAs and rewritten by one, and the output norm needs the squares of all four column
// slices; one cluster barrier covers both (the history is only written behind it).  Three value heads and more to a
// key head would need more than the portable eight CTAs and take the general path, as other convolution widths do.
// 128 CTAs of 16 KiB of state each at the model's head counts: a thread's 64 bytes are one round of loads.
template <int Dtype> struct Scalar;
template <> struct Scalar<RIB200_DTYPE_F32> {
  using Type = float;
  static __device__ __forceinline__ float widen(float x) { return x; }
  static __device__ __forceinline__ float narrow(float x) { return x; }
};
template <> struct Scalar<RIB200_DTYPE_F16> {
  using Type = __half;
  static __device__ __forceinline__ float widen(__half x) { return __half2float(x); }
  static __device__ __forceinline__ __half narrow(float x) { return __float2half_rn(x); }
};
template <> struct Scalar<RIB200_DTYPE_BF16> {
  using Type = __nv_bfloat16;
  static __device__ __forceinline__ float widen(__nv_bfloat16 x) { return __bfloat162float(x); }
  static __device__ __forceinline__ __nv_bfloat16 narrow(float x) { return __float2bfloat16_rn(x); }
};

constexpr int kStepThreads = 256;
constexpr int kStepSlices = 4;
constexpr int kStepColumns = kDim / kStepSlices;
constexpr std::uint32_t kStepMaxRatio = 2; // value heads per key head a portable cluster holds

// While the kernels in front still run, a single-launch call asks for what it will read: its state rows, and a line per
// eight channels of taps, history and input.  Hints, no reads: what those kernels write is current in L2 either way.
__device__ __forceinline__ void hint_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }
template <int Dtype, int WeightDtype>
__device__ __forceinline__ void hint_operands(const LayerParams &p, std::uint32_t key_head, std::uint32_t head,
                                              std::uint32_t slice) {
  const auto *input = static_cast<const typename Scalar<Dtype>::Type *>(p.input);
  const auto *taps = static_cast<const typename Scalar<WeightDtype>::Type *>(p.conv_weight);
  const std::uint32_t tid = threadIdx.x;
  auto channel_hints = [&](std::uint32_t channel) {
    hint_l2(taps + static_cast<std::size_t>(channel) * kFastWidth);
    hint_l2(p.convolution_state + static_cast<std::size_t>(channel) * (kFastWidth - 1));
    hint_l2(input + channel);
  };
  if (tid < kDim) {
    hint_l2(p.recurrent_state + static_cast<std::size_t>(head) * kDim * kDim + slice * kStepColumns +
            static_cast<std::size_t>(tid) * kDim);
  } else if (tid < kDim + 32) { // q, then k channels of the key head
    const std::uint32_t piece = tid - kDim;
    channel_hints((piece < 16 ? 0 : p.key_heads * kDim) + key_head * kDim + (piece & 15U) * 8);
  } else if (tid < kDim + 32 + 4) {
    const std::uint32_t column = head * kDim + slice * kStepColumns + (tid - kDim - 32) * 8;
    channel_hints(2 * p.key_heads * kDim + column);
    hint_l2(input + p.conv_dim + 2 * p.value_heads + column);
  } else if (tid == kDim + 64) {
    hint_l2(input + p.conv_dim + head);
    hint_l2(input + p.conv_dim + p.value_heads + head);
    hint_l2(static_cast<const typename Scalar<WeightDtype>::Type *>(p.recurrent_a) + head);
    hint_l2(static_cast<const typename Scalar<WeightDtype>::Type *>(p.dt_bias) + head);
    hint_l2(static_cast<const typename Scalar<WeightDtype>::Type *>(p.output_norm_weight) + slice * kStepColumns);
  }
}

template <int Dtype, int WeightDtype>
__global__ void __launch_bounds__(kStepThreads) gdn_layer_step_kernel(const LayerParams p) {
  using Act = Scalar<Dtype>;
  using Weight = Scalar<WeightDtype>;
  __shared__ float s_q[kDim];
  __shared__ float s_k[kDim];
  __shared__ float s_squares[8];
  __shared__ float s_gates[2]; // beta, decay
  __shared__ __align__(16) float s_a[8][kStepColumns];
  __shared__ __align__(16) float s_b[8][kStepColumns];
  __shared__ float s_dot[8];
  __shared__ __align__(16) float s_delta[kStepColumns];
  __shared__ float s_norm[kStepSlices]; // written by the CTAs of the value head, this one included
  std::uint32_t rank;
  std::uint32_t cluster_size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(cluster_size));
  const std::uint32_t key_head = blockIdx.x / cluster_size;
  const std::uint32_t head = key_head + (rank / kStepSlices) * p.key_heads;
  const std::uint32_t slice = rank % kStepSlices;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  float *state = p.recurrent_state + static_cast<std::size_t>(head) * kDim * kDim + slice * kStepColumns;
  hint_operands<Dtype, WeightDtype>(p, key_head, head, slice);
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); // every CTA of the cluster has started
  grid_dependency_wait();
  grid_dependents_may_launch();

  // ---- every load of the step in one round ----
  const int row0 = 16 * warp + (lane >> 3);
  const int col = 4 * (lane & 7);
  float4 s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    s[i] = *reinterpret_cast<const float4 *>(state + static_cast<std::size_t>(row0 + 4 * i) * kDim + col);
  }
  const auto *input = static_cast<const typename Act::Type *>(p.input);
  const auto *conv_weight = static_cast<const typename Weight::Type *>(p.conv_weight);
  constexpr int kHistory = kFastWidth - 1;
  struct Channel {
    typename Act::Type x;
    typename Weight::Type w[kFastWidth];
    float history[kHistory];
  };
  auto load_channel = [&](std::uint32_t channel, Channel &c) {
    c.x = input[channel];
#pragma unroll
    for (int h = 0; h < kFastWidth; ++h) {
      c.w[h] = conv_weight[static_cast<std::size_t>(channel) * kFastWidth + h];
    }
#pragma unroll
    for (int h = 0; h < kHistory; ++h) {
      c.history[h] = p.convolution_state[static_cast<std::size_t>(channel) * kHistory + h];
    }
  };
  auto convolve = [&](const Channel &c) { // the current token's tap first, then the history, oldest first
    float sum = Act::widen(c.x) * Weight::widen(c.w[kHistory]);
#pragma unroll
    for (int h = 0; h < kHistory; ++h) {
      sum += c.history[h] * Weight::widen(c.w[h]);
    }
    return silu(sum);
  };
  auto shift_history = [&](std::uint32_t channel, const Channel &c) {
    float *history = p.convolution_state + static_cast<std::size_t>(channel) * kHistory;
    history[0] = c.history[1];
    history[1] = c.history[2];
    history[2] = Act::widen(c.x);
  };
  // threads 0..127: the q channels of the key head, 128..255: its k channels; warp 0 also the slice's v channels
  const std::uint32_t qk_channel = (tid < kDim ? 0 : p.key_heads * kDim) + key_head * kDim + (tid & (kDim - 1));
  const std::uint32_t v_channel = 2 * p.key_heads * kDim + head * kDim + slice * kStepColumns + lane;
  Channel qk;
  Channel v;
  typename Act::Type z{};
  typename Act::Type b{};
  typename Act::Type a{};
  typename Weight::Type coefficient{};
  typename Weight::Type dt{};
  typename Weight::Type norm_weight{};
  load_channel(qk_channel, qk);
  if (warp == 0) {
    load_channel(v_channel, v);
    z = input[p.conv_dim + 2 * p.value_heads + head * kDim + slice * kStepColumns + lane];
    norm_weight = static_cast<const typename Weight::Type *>(p.output_norm_weight)[slice * kStepColumns + lane];
    b = input[p.conv_dim + head];
    a = input[p.conv_dim + p.value_heads + head];
    coefficient = static_cast<const typename Weight::Type *>(p.recurrent_a)[head];
    dt = static_cast<const typename Weight::Type *>(p.dt_bias)[head];
  }

  // ---- q, k: convolution, SiLU, sum of squares ----
  const float qk_value = convolve(qk);
  float squares = qk_value * qk_value;
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) {
    squares += __shfl_xor_sync(0xFFFFFFFFU, squares, offset);
  }
  (tid < kDim ? s_q : s_k)[tid & (kDim - 1)] = qk_value;
  float v_value = 0.0F;
  float z_gate = 0.0F;
  if (warp == 0) {
    v_value = convolve(v);
    z_gate = Weight::widen(norm_weight) * silu(Act::widen(z));
    if (lane == 0) {
      s_gates[0] = 1.0F / (1.0F + expf(-Act::widen(b)));
      s_gates[1] = expf(Weight::widen(coefficient) * softplus(Act::widen(a) + Weight::widen(dt)));
    }
  }
  if (lane == 0) {
    s_squares[warp] = squares;
  }
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
  __syncthreads();
  const float q_scale = rsqrtf((s_squares[0] + s_squares[1]) + (s_squares[2] + s_squares[3]) + kQkEpsilon) *
                        rsqrtf(static_cast<float>(kDim));
  const float k_scale = rsqrtf((s_squares[4] + s_squares[5]) + (s_squares[6] + s_squares[7]) + kQkEpsilon);
  const float beta = s_gates[0];
  const float decay = s_gates[1];

  // ---- S^T k and S^T q of the slice, k . q ----
  float k_row[4];
  float sums[9] = {};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float k = s_k[row0 + 4 * i] * k_scale;
    const float q = s_q[row0 + 4 * i] * q_scale;
    k_row[i] = k;
    sums[0] += s[i].x * k;
    sums[1] += s[i].y * k;
    sums[2] += s[i].z * k;
    sums[3] += s[i].w * k;
    sums[4] += s[i].x * q;
    sums[5] += s[i].y * q;
    sums[6] += s[i].z * q;
    sums[7] += s[i].w * q;
    sums[8] += k * q;
  }
#pragma unroll
  for (int offset = 16; offset >= 8; offset >>= 1) { // the four row groups of the warp
#pragma unroll
    for (int c = 0; c < 9; ++c) {
      sums[c] += __shfl_xor_sync(0xFFFFFFFFU, sums[c], offset);
    }
  }
  if (lane < 8) {
    *reinterpret_cast<float4 *>(&s_a[warp][col]) = make_float4(sums[0], sums[1], sums[2], sums[3]);
    *reinterpret_cast<float4 *>(&s_b[warp][col]) = make_float4(sums[4], sums[5], sums[6], sums[7]);
    if (lane == 0) {
      s_dot[warp] = sums[8];
    }
  }
  __syncthreads();
  float read = 0.0F; // the slice's output vector before the norm: one column per lane of warp 0
  if (warp == 0) {
    float a_sum = 0.0F;
    float b_sum = 0.0F;
    float dot = 0.0F;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      a_sum += s_a[w][lane];
      b_sum += s_b[w][lane];
      dot += s_dot[w];
    }
    const float delta = (v_value - decay * a_sum) * beta;
    s_delta[lane] = delta;
    read = decay * b_sum + delta * dot;
  }
  __syncthreads();
  if (warp == 0) {
    float norm = read * read;
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      norm += __shfl_xor_sync(0xFFFFFFFFU, norm, offset);
    }
    if (lane < kStepSlices) { // to the four CTAs of this value head
      std::uint32_t remote;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                   : "=r"(remote)
                   : "r"(static_cast<std::uint32_t>(__cvta_generic_to_shared(&s_norm[slice]))),
                     "r"(rank - slice + lane));
      asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(remote), "f"(norm) : "memory");
    }
    __syncwarp();
  }
  // The barrier orders the partial norms and marks the end of everybody's reads of the history.
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  const float4 delta = *reinterpret_cast<const float4 *>(&s_delta[col]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    *reinterpret_cast<float4 *>(state + static_cast<std::size_t>(row0 + 4 * i) * kDim + col) =
        make_float4(decay * s[i].x + k_row[i] * delta.x, decay * s[i].y + k_row[i] * delta.y,
                    decay * s[i].z + k_row[i] * delta.z, decay * s[i].w + k_row[i] * delta.w);
  }
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  if (rank == 0) {
    shift_history(qk_channel, qk);
  }
  if (warp == 0) {
    shift_history(v_channel, v);
    const float norm = (s_norm[0] + s_norm[1]) + (s_norm[2] + s_norm[3]);
    const float scale = rsqrtf(norm / static_cast<float>(kDim) + p.epsilon);
    static_cast<typename Act::Type *>(p.output)[head * kDim + slice * kStepColumns + lane] =
        Act::narrow(read * scale * z_gate);
  }
}

// ---- 2 .. 63 tokens in one launch --------------------------------------------------------------------------
// The calls that end a prompt (the executor cuts a rest into 17, 4 and 2 tokens) are latency as well: the general path
// took 53 us for 17 tokens and 25 us for 4 (prologue, history, recurrence, epilogue; launch list), this form 17.5 and 8.9
// (replayed calls, as the figures below).
// Same split as the one-token form - a cluster per key head, a CTA per 32 state columns - and the same arithmetic in
// FP32; the tokens go through in tiles of 32: convolution and norms of a tile with a warp per token, then the recurrence
// with the state in registers, then the output norm, for which the slices of a head exchange their sums once per tile.
// In the recurrence a warp owns four columns and a lane four rows of them, so that a token needs no barrier: nine
// shuffles bring the eight sums (S^T k, S^T q) to eight groups of lanes, four more hand the corrections back.
constexpr std::uint32_t kShortTile = 32;
// Longer calls run in chunks, which is faster (64 tokens 17.3 us, 63 here 45.6) but has products of ten-bit mantissas;
// calls of fewer tokens are FP32 throughout, as they always were.
constexpr std::uint32_t kShortMaxTokens = 63;
constexpr std::uint32_t kShortRounds = kShortTile / 8; // tokens per warp
constexpr std::uint32_t kShortGroup = 4;               // tokens convolved together

template <int Dtype, int WeightDtype>
__global__ void __launch_bounds__(kStepThreads) gdn_layer_short_kernel(const LayerParams p) {
  using Act = Scalar<Dtype>;
  using Weight = Scalar<WeightDtype>;
  using ActType = typename Act::Type;
  using WeightType = typename Weight::Type;
  constexpr int kHistory = kFastWidth - 1;
  __shared__ __align__(16) float s_qk[2][kShortTile][kDim];
  __shared__ float s_v[kShortTile][kStepColumns];
  __shared__ float s_out[kShortTile][kStepColumns];
  __shared__ float s_kq[kShortTile];
  __shared__ float s_beta[kShortTile];
  __shared__ float s_decay[kShortTile];
  __shared__ float s_norm[2][kStepSlices][kShortTile]; // by parity of the tile
  std::uint32_t rank;
  std::uint32_t cluster_size;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(cluster_size));
  const std::uint32_t key_head = blockIdx.x / cluster_size;
  const std::uint32_t head = key_head + (rank / kStepSlices) * p.key_heads;
  const std::uint32_t slice = rank % kStepSlices;
  const std::uint32_t tid = threadIdx.x;
  const std::uint32_t warp = tid >> 5;
  const std::uint32_t lane = tid & 31;
  float *state = p.recurrent_state + static_cast<std::size_t>(head) * kDim * kDim + slice * kStepColumns;
  hint_operands<Dtype, WeightDtype>(p, key_head, head, slice);
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); // every CTA of the cluster has started
  grid_dependency_wait();
  grid_dependents_may_launch();

  const auto *input = static_cast<const ActType *>(p.input);
  const auto *conv_weight = static_cast<const WeightType *>(p.conv_weight);
  // state: lane = rows 4 lane .. + 3, warp = columns 4 warp .. + 3 of the slice
  float4 s[4];
#pragma unroll
  for (std::uint32_t i = 0; i < 4; ++i) {
    s[i] = *reinterpret_cast<const float4 *>(state + static_cast<std::size_t>(4 * lane + i) * kDim + 4 * warp);
  }
  // threads 0..127 convolve the q channels of the key head, 128..255 its k channels; a lane a v channel of the slice
  const std::uint32_t qk_channel = (tid < kDim ? 0 : p.key_heads * kDim) + key_head * kDim + (tid & (kDim - 1));
  const std::uint32_t v_channel = 2 * p.key_heads * kDim + head * kDim + slice * kStepColumns + lane;
  const std::uint32_t z_channel = p.conv_dim + 2 * p.value_heads + head * kDim + slice * kStepColumns + lane;
  float qk_weight[kFastWidth];
  float v_weight[kFastWidth];
  float qk_history[kHistory]; // the three tokens in front of the call
  float v_history[kHistory];
#pragma unroll
  for (int h = 0; h < kFastWidth; ++h) {
    qk_weight[h] = Weight::widen(conv_weight[static_cast<std::size_t>(qk_channel) * kFastWidth + h]);
    v_weight[h] = Weight::widen(conv_weight[static_cast<std::size_t>(v_channel) * kFastWidth + h]);
  }
#pragma unroll
  for (int h = 0; h < kHistory; ++h) {
    qk_history[h] = p.convolution_state[static_cast<std::size_t>(qk_channel) * kHistory + h];
    v_history[h] = p.convolution_state[static_cast<std::size_t>(v_channel) * kHistory + h];
  }
  const float norm_weight =
      Weight::widen(static_cast<const WeightType *>(p.output_norm_weight)[slice * kStepColumns + lane]);
  const float coefficient = Weight::widen(static_cast<const WeightType *>(p.recurrent_a)[head]);
  const float dt = Weight::widen(static_cast<const WeightType *>(p.dt_bias)[head]);
  // a channel's input at a token of this call, or of the history in front of it
  auto row = [&](std::uint32_t channel, const float (&history)[kHistory], int tok) {
    return tok >= 0 ? Act::widen(input[static_cast<std::size_t>(tok) * p.token_stride + channel])
                    : (tok == -1 ? history[2] : (tok == -2 ? history[1] : history[0]));
  };
  const std::uint32_t last = p.tokens - 1;

  for (std::uint32_t first = 0, tile = 0; first < p.tokens; first += kShortTile, ++tile) {
    const std::uint32_t n = min(kShortTile, p.tokens - first);
    // ---- convolution and SiLU: q and k a channel per thread, v and the gates a token per warp.  Whole groups of
    // tokens without a branch, so that their long dependent chains overlap; rows past the last token are computed from
    // it and not used. ----
    {
      ActType x[kShortTile];
#pragma unroll
      for (std::uint32_t group = 0; group < kShortTile; group += kShortGroup) {
        if (group < n) {
#pragma unroll
          for (std::uint32_t t = group; t < group + kShortGroup; ++t) {
            x[t] = input[static_cast<std::size_t>(min(first + t, last)) * p.token_stride + qk_channel];
          }
        }
      }
      float before[kHistory];
#pragma unroll
      for (int h = 0; h < kHistory; ++h) {
        before[h] = row(qk_channel, qk_history, static_cast<int>(first) - kHistory + h);
      }
#pragma unroll
      for (std::uint32_t r = 0; r < kShortRounds; ++r) {
        if (8 * r < n) {
          const std::uint32_t t = warp + 8 * r;
          const int tok = static_cast<int>(min(first + t, last));
          // the current token's tap first, then the history, oldest first
          float sum = row(v_channel, v_history, tok) * v_weight[kHistory];
#pragma unroll
          for (int h = 0; h < kHistory; ++h) {
            sum += row(v_channel, v_history, tok - kHistory + h) * v_weight[h];
          }
          s_v[t][lane] = silu(sum);
        }
      }
      if (lane < kShortRounds && warp + 8 * lane < n) {
        const std::uint32_t t = warp + 8 * lane;
        const std::size_t gates = static_cast<std::size_t>(first + t) * p.token_stride + p.conv_dim + head;
        s_beta[t] = 1.0F / (1.0F + expf(-Act::widen(input[gates])));
        s_decay[t] = expf(coefficient * softplus(Act::widen(input[gates + p.value_heads]) + dt));
      }
#pragma unroll
      for (std::uint32_t group = 0; group < kShortTile; group += kShortGroup) {
        if (group < n) {
          float value[kShortGroup];
#pragma unroll
          for (std::uint32_t t = 0; t < kShortGroup; ++t) {
            const float now = Act::widen(x[group + t]);
            float sum = now * qk_weight[kHistory];
#pragma unroll
            for (int h = 0; h < kHistory; ++h) {
              sum += before[h] * qk_weight[h];
            }
            before[0] = before[1];
            before[1] = before[2];
            before[2] = now;
            value[t] = silu(sum);
          }
#pragma unroll
          for (std::uint32_t t = 0; t < kShortGroup; ++t) {
            s_qk[tid >> 7][group + t][tid & (kDim - 1)] = value[t];
          }
        }
      }
    }
    __syncthreads();
    // ---- norms of q and k, k . q ----
    for (std::uint32_t t = warp; t < n; t += 8) {
      float4 q = *reinterpret_cast<const float4 *>(&s_qk[0][t][4 * lane]);
      float4 k = *reinterpret_cast<const float4 *>(&s_qk[1][t][4 * lane]);
      float qq = (q.x * q.x + q.y * q.y) + (q.z * q.z + q.w * q.w);
      float kk = (k.x * k.x + k.y * k.y) + (k.z * k.z + k.w * k.w);
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) {
        qq += __shfl_xor_sync(0xFFFFFFFFU, qq, offset);
        kk += __shfl_xor_sync(0xFFFFFFFFU, kk, offset);
      }
      const float q_scale = rsqrtf(qq + kQkEpsilon) * rsqrtf(static_cast<float>(kDim));
      const float k_scale = rsqrtf(kk + kQkEpsilon);
      q = make_float4(q.x * q_scale, q.y * q_scale, q.z * q_scale, q.w * q_scale);
      k = make_float4(k.x * k_scale, k.y * k_scale, k.z * k_scale, k.w * k_scale);
      float kq = (k.x * q.x + k.y * q.y) + (k.z * q.z + k.w * q.w);
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) {
        kq += __shfl_xor_sync(0xFFFFFFFFU, kq, offset);
      }
      *reinterpret_cast<float4 *>(&s_qk[0][t][4 * lane]) = q;
      *reinterpret_cast<float4 *>(&s_qk[1][t][4 * lane]) = k;
      if (lane == 0) {
        s_kq[t] = kq;
      }
    }
    __syncthreads();
    // ---- the recurrence ----
    // after the three exchanges lane l holds the sum of column 2 (l / 8 % 2) + (l / 4) % 2, of S^T k below lane 16 and
    // of S^T q from there on
    const std::uint32_t my_column = ((lane >> 3) & 1U) * 2 + ((lane >> 2) & 1U);
    float4 next_k = *reinterpret_cast<const float4 *>(&s_qk[1][0][4 * lane]);
    float4 next_q = *reinterpret_cast<const float4 *>(&s_qk[0][0][4 * lane]);
    for (std::uint32_t t = 0; t < n; ++t) {
      const float k[4] = {next_k.x, next_k.y, next_k.z, next_k.w};
      const float q[4] = {next_q.x, next_q.y, next_q.z, next_q.w};
      const float decay = s_decay[t];
      const float beta = s_beta[t];
      const float v_value = s_v[t][4 * warp + my_column];
      const float kq = s_kq[t];
      const std::uint32_t following = min(t + 1, kShortTile - 1);
      next_k = *reinterpret_cast<const float4 *>(&s_qk[1][following][4 * lane]);
      next_q = *reinterpret_cast<const float4 *>(&s_qk[0][following][4 * lane]);
      float a[4] = {};
      float b[4] = {};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[0] += s[i].x * k[i];
        a[1] += s[i].y * k[i];
        a[2] += s[i].z * k[i];
        a[3] += s[i].w * k[i];
        b[0] += s[i].x * q[i];
        b[1] += s[i].y * q[i];
        b[2] += s[i].z * q[i];
        b[3] += s[i].w * q[i];
      }
      const bool upper = (lane & 16U) != 0;
      float four[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        four[c] = (upper ? b[c] : a[c]) + __shfl_xor_sync(0xFFFFFFFFU, upper ? a[c] : b[c], 16);
      }
      const bool high_pair = (lane & 8U) != 0;
      float two[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        two[c] = (high_pair ? four[2 + c] : four[c]) +
                 __shfl_xor_sync(0xFFFFFFFFU, high_pair ? four[c] : four[2 + c], 8);
      }
      const bool odd = (lane & 4U) != 0;
      float sum = (odd ? two[1] : two[0]) + __shfl_xor_sync(0xFFFFFFFFU, odd ? two[0] : two[1], 4);
      sum += __shfl_xor_sync(0xFFFFFFFFU, sum, 2);
      sum += __shfl_xor_sync(0xFFFFFFFFU, sum, 1);
      const float delta = (v_value - decay * sum) * beta; // below lane 16
      float correction[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        correction[c] = __shfl_sync(0xFFFFFFFFU, delta, 4 * c);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s[i].x = decay * s[i].x + k[i] * correction[0];
        s[i].y = decay * s[i].y + k[i] * correction[1];
        s[i].z = decay * s[i].z + k[i] * correction[2];
        s[i].w = decay * s[i].w + k[i] * correction[3];
      }
      const float low = odd ? correction[1] : correction[0];
      const float high = odd ? correction[3] : correction[2];
      if (upper && (lane & 3U) == 0) {
        s_out[t][4 * warp + my_column] = decay * sum + (high_pair ? high : low) * kq;
      }
    }
    __syncthreads();
    // ---- output norm over the four slices, gate ----
    float z_gate[kShortRounds];
    float read[kShortRounds];
#pragma unroll
    for (std::uint32_t r = 0; r < kShortRounds; ++r) {
      const std::uint32_t t = warp + 8 * r;
      if (t < n) {
        z_gate[r] = norm_weight * silu(Act::widen(input[static_cast<std::size_t>(first + t) * p.token_stride + z_channel]));
        read[r] = s_out[t][lane];
      }
    }
    if (tile == 0) { // the barrier that says that every CTA of the cluster has started
      asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
    }
#pragma unroll
    for (std::uint32_t r = 0; r < kShortRounds; ++r) {
      const std::uint32_t t = warp + 8 * r;
      if (t < n) {
        float norm = read[r] * read[r];
#pragma unroll
        for (int offset = 16; offset > 0; offset >>= 1) {
          norm += __shfl_xor_sync(0xFFFFFFFFU, norm, offset);
        }
        if (lane < kStepSlices) { // to the four CTAs of this value head
          std::uint32_t remote;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                       : "=r"(remote)
                       : "r"(static_cast<std::uint32_t>(__cvta_generic_to_shared(&s_norm[tile & 1U][slice][t]))),
                         "r"(rank - slice + lane));
          asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(remote), "f"(norm) : "memory");
        }
      }
    }
    __syncwarp();
    // Orders the partial norms; that of the first tile also marks the end of everybody's reads of the old history.
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
#pragma unroll
    for (std::uint32_t r = 0; r < kShortRounds; ++r) {
      const std::uint32_t t = warp + 8 * r;
      if (t < n) {
        const float (&norms)[kStepSlices][kShortTile] = s_norm[tile & 1U];
        const float norm = (norms[0][t] + norms[1][t]) + (norms[2][t] + norms[3][t]);
        const float scale = rsqrtf(norm / static_cast<float>(kDim) + p.epsilon);
        static_cast<ActType *>(p.output)[(static_cast<std::size_t>(first + t) * p.value_heads + head) * kDim +
                                         slice * kStepColumns + lane] = Act::narrow(read[r] * scale * z_gate[r]);
      }
    }
  }
#pragma unroll
  for (std::uint32_t i = 0; i < 4; ++i) {
    *reinterpret_cast<float4 *>(state + static_cast<std::size_t>(4 * lane + i) * kDim + 4 * warp) = s[i];
  }
  // the last three tokens of [old history | call] are the next call's history
  if (rank == 0) {
#pragma unroll
    for (int h = 0; h < kHistory; ++h) {
      p.convolution_state[static_cast<std::size_t>(qk_channel) * kHistory + h] =
          row(qk_channel, qk_history, static_cast<int>(p.tokens) - kHistory + h);
    }
  }
  if (warp == 0) {
#pragma unroll
    for (int h = 0; h < kHistory; ++h) {
      p.convolution_state[static_cast<std::size_t>(v_channel) * kHistory + h] =
          row(v_channel, v_history, static_cast<int>(p.tokens) - kHistory + h);
    }
  }
}

LayerParams make_params(const GdnLayerArgs &a) {
  LayerParams p{};
  p.input = a.input;
  p.conv_weight = a.conv_weight;
  p.recurrent_a = a.recurrent_a;
  p.dt_bias = a.dt_bias;
  p.output_norm_weight = a.output_norm_weight;
  p.output = a.output;
  p.convolution_state = a.convolution_state;
  p.recurrent_state = a.recurrent_state;
  p.convolved = a.convolved;
  p.beta = a.beta;
  p.log_decay = a.log_decay;
  p.raw = a.raw;
  p.tokens = a.tokens;
  p.key_heads = a.key_heads;
  p.value_heads = a.value_heads;
  p.conv_width = a.conv_width;
  p.conv_dim = (2 * a.key_heads + a.value_heads) * kDim;
  p.token_stride = p.conv_dim + 2 * a.value_heads + a.value_heads * kDim;
  p.epsilon = a.epsilon;
  p.dtype = a.dtype;
  p.weight_dtype = a.weight_dtype;
  return p;
}

template <int Dtype, int WeightDtype> void launch_step(const LayerParams &p, cudaStream_t stream) {
  const std::uint32_t cluster = kStepSlices * (p.value_heads / p.key_heads);
  auto *kernel = p.tokens == 1 ? gdn_layer_step_kernel<Dtype, WeightDtype> : gdn_layer_short_kernel<Dtype, WeightDtype>;
  launch_programmatic_cluster(kernel, dim3(cluster * p.key_heads), dim3(kStepThreads), cluster, 0, stream,
                              "gated-delta step launch", p);
}

} // namespace

bool gdn_layer_step_applies(const GdnLayerArgs &a) {
  return a.tokens <= kShortMaxTokens && a.conv_width == kFastWidth && a.value_heads / a.key_heads <= kStepMaxRatio;
}

void launch_gdn_layer_step(const GdnLayerArgs &a, cudaStream_t stream) {
  const LayerParams p = make_params(a);
  constexpr int kF32 = RIB200_DTYPE_F32;
  constexpr int kF16 = RIB200_DTYPE_F16;
  constexpr int kBf16 = RIB200_DTYPE_BF16;
  if (a.dtype == kF32) {
    if (a.weight_dtype == kF32) {
      launch_step<kF32, kF32>(p, stream);
    } else if (a.weight_dtype == kF16) {
      launch_step<kF32, kF16>(p, stream);
    } else {
      launch_step<kF32, kBf16>(p, stream);
    }
  } else if (a.dtype == kF16) {
    if (a.weight_dtype == kF32) {
      launch_step<kF16, kF32>(p, stream);
    } else {
      launch_step<kF16, kF16>(p, stream);
    }
  } else if (a.weight_dtype == kF32) {
    launch_step<kBf16, kF32>(p, stream);
  } else {
    launch_step<kBf16, kBf16>(p, stream);
  }
}

void launch_gdn_prologue(const GdnLayerArgs &a, cudaStream_t stream) {
  const LayerParams p = make_params(a);
  const char *what = "gated-delta prologue launch";
  // a call of a few tokens is latency, not bandwidth: the one-CTA-per-vector kernel spreads it wider
  if (a.conv_width == kFastWidth && a.tokens >= 2 * kTokensPerWarp && vector_forms_apply(p)) {
    constexpr std::uint32_t kTokensPerCta = kTokensPerWarp * kStepsPerWarp;
    const dim3 grid((a.tokens + kTokensPerCta - 1) / kTokensPerCta, (2 * a.key_heads + a.value_heads + 1 + 7) / 8);
    if (a.dtype == RIB200_DTYPE_F32) {
      launch_programmatic(gdn_prologue_w4_kernel<RIB200_DTYPE_F32>, grid, dim3(256), 0, stream, what, p);
    } else if (a.dtype == RIB200_DTYPE_F16) {
      launch_programmatic(gdn_prologue_w4_kernel<RIB200_DTYPE_F16>, grid, dim3(256), 0, stream, what, p);
    } else {
      launch_programmatic(gdn_prologue_w4_kernel<RIB200_DTYPE_BF16>, grid, dim3(256), 0, stream, what, p);
    }
  } else {
    launch_programmatic(gdn_prologue_kernel, dim3(2 * a.key_heads + a.value_heads, a.tokens), dim3(kDim), 0, stream, what,
                        p);
  }
  if (a.conv_width > 1) {
    launch_programmatic(gdn_conv_state_kernel, dim3((p.conv_dim + 255) / 256), dim3(256), 0, stream,
                        "gated-delta convolution-state launch", p);
  }
}

void launch_gdn_epilogue(const GdnLayerArgs &a, cudaStream_t stream) {
  const LayerParams p = make_params(a);
  if (vector_forms_apply(p)) {
    const std::size_t items = static_cast<std::size_t>(a.tokens) * a.value_heads;
    const unsigned int grid = static_cast<unsigned int>((items + 7) / 8);
    const char *what = "gated-delta epilogue launch";
    if (a.dtype == RIB200_DTYPE_F32) {
      launch_programmatic(gdn_epilogue_warp_kernel<RIB200_DTYPE_F32>, dim3(grid), dim3(256), 0, stream, what, p);
    } else if (a.dtype == RIB200_DTYPE_F16) {
      launch_programmatic(gdn_epilogue_warp_kernel<RIB200_DTYPE_F16>, dim3(grid), dim3(256), 0, stream, what, p);
    } else {
      launch_programmatic(gdn_epilogue_warp_kernel<RIB200_DTYPE_BF16>, dim3(grid), dim3(256), 0, stream, what, p);
    }
    return;
  }
  launch_programmatic(gdn_epilogue_kernel, dim3(a.value_heads, a.tokens), dim3(kDim), 0, stream,
                      "gated-delta epilogue launch", p);
}

} // namespace rib200
