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

#include <mutex>

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

// x / d for d >= 1 or infinite: the unit's reciprocal and one step of Newton's iteration on the quotient, q + (x - d q) r, in
// place of a division, whose slow path keeps the compiler from overlapping the chains of neighbouring tokens.  The
// remainder is not a number exactly where x or d is infinite or not a number; x r is the quotient then.  The unit makes the
// subnormal reciprocals of d above 2^126 zero, so it gets a quarter of d; r keeps 22 bits and more there.
__device__ __forceinline__ float quotient(float x, float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(0.25F * d));
  r *= 0.25F;
  const float q = x * r;
  const float remainder = fmaf(-d, q, x);
  return remainder == remainder ? fmaf(remainder, r, q) : q;
}
__device__ __forceinline__ float sigmoid(float x) { return quotient(1.0F, 1.0F + expf(-x)); }
__device__ __forceinline__ float silu(float x) { return quotient(x, 1.0F + expf(-x)); }

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
  unsigned int *status; // one-launch forms only
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
    p.beta[static_cast<std::size_t>(tok) * p.value_heads + head] = sigmoid(b);
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
        p.beta[static_cast<std::size_t>(tok) * p.value_heads + head] = sigmoid(b);
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
// most of it hand-over between grids; this form costs 3.2 us (4.2 MB of state in and out: 1.3 TB/s), about
// 2 of kernel and the rest hand-over; 3.6 us with a cluster barrier in place of the counted exchange of sums, and 4.4 us
// without the L2 hints in front of the wait.
//
// A cluster serves one key head: four CTAs (32 state columns each) per value head that shares it, one or two value
// heads.  Everything that has to meet across CTAs meets inside that cluster: the convolution history of the q and k
// channels is read by all of its CTAs and rewritten by one, and the output norm needs the squares of all four column
// slices; the exchange of those sums covers both (the history is only written behind it).  Three value heads and more to a
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

// The slices of a head exchange their sums of squares with stores that count on an mbarrier of the CTA they go to.  A cluster
// barrier in their place costs a call 0.3 to 0.6 us more: its release waits for whatever the thread has in flight.  Who has
// the sums of all slices also knows that their CTAs have read the old history.
constexpr long long kWaitLimitCycles = 1LL << 28;
__device__ __forceinline__ std::uint32_t smem_address(const void *p) {
  return static_cast<std::uint32_t>(__cvta_generic_to_shared(p));
}
// by one thread, in front of the barrier that says that every CTA of the cluster has started
__device__ __forceinline__ void expect_sums(std::uint64_t *bar, std::uint32_t bytes) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_address(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_address(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void send_sum(const float *slot, std::uint64_t *bar, std::uint32_t to_rank, float value) {
  std::uint32_t remote_slot;
  std::uint32_t remote_bar;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote_slot) : "r"(smem_address(slot)), "r"(to_rank));
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(remote_bar) : "r"(smem_address(bar)), "r"(to_rank));
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n" ::"r"(remote_slot),
               "r"(__float_as_uint(value)), "r"(remote_bar)
               : "memory");
}
// by every warp behind its last store to a peer; it releases nothing and so waits for nothing
__device__ __forceinline__ void all_sent() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
}
// bounded: when it runs out the status word says so, the call runs to its end and the answer is false
__device__ __forceinline__ bool wait_for_sums(std::uint64_t *bar, unsigned int *status) {
  const long long started = clock64();
  std::uint32_t done = 0;
  while (done == 0) {
    asm volatile("{\n"
                 ".reg .pred p;\n"
                 "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
                 "selp.u32 %0, 1, 0, p;\n"
                 "}\n"
                 : "=r"(done)
                 : "r"(smem_address(bar))
                 : "memory");
    if (done == 0 && clock64() - started > kWaitLimitCycles) {
      atomicOr(status, static_cast<unsigned int>(RIB200_DEVICE_WAIT_TIMED_OUT));
      return false;
    }
  }
  return true;
}
// At the end.  To a CTA that has its sums nobody sends any more, so it may leave (a wait of all for all costs a one-token call
// 0.06 of its 3.2 us); where the wait ran out, not before all have sent and that is here.
__device__ __forceinline__ void leave_cluster(std::uint64_t *bar, bool complete, unsigned int *status) {
  if (!complete) {
    asm volatile("barrier.cluster.wait;\n" ::: "memory");
    wait_for_sums(bar, status);
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
  // written by the CTAs of the value head, this one included; in the first CTA also by those of the other value head, to
  // say that they have read the history of q and k
  __shared__ float s_norm[kStepMaxRatio * kStepSlices];
  __shared__ __align__(8) std::uint64_t s_norm_bar;
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
  if (tid == 0) {
    expect_sums(&s_norm_bar, (rank == 0 ? cluster_size : kStepSlices) * 4);
  }
  __syncwarp();
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
      s_gates[0] = sigmoid(Act::widen(b));
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
      send_sum(&s_norm[slice], &s_norm_bar, rank - slice + lane, norm);
    } else if (lane == kStepSlices && rank >= kStepSlices) {
      send_sum(&s_norm[rank], &s_norm_bar, 0, 0.0F);
    }
  }
  all_sent();
  const float4 delta = *reinterpret_cast<const float4 *>(&s_delta[col]);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    *reinterpret_cast<float4 *>(state + static_cast<std::size_t>(row0 + 4 * i) * kDim + col) =
        make_float4(decay * s[i].x + k_row[i] * delta.x, decay * s[i].y + k_row[i] * delta.y,
                    decay * s[i].z + k_row[i] * delta.z, decay * s[i].w + k_row[i] * delta.w);
  }
  const bool complete = (rank != 0 && warp != 0) || wait_for_sums(&s_norm_bar, p.status);
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
  leave_cluster(&s_norm_bar, complete, p.status);
}

// ---- 2 .. 63 tokens in one launch --------------------------------------------------------------------------
// The calls that end a prompt (the executor cuts a rest into 17, 4 and 2 tokens) are latency as well.
// A cluster of four CTAs per key head, a CTA per 32 state columns of all its value heads, so that the q and k channels are
// convolved once for both heads and every cluster has SMs of its own: of the one-token form's clusters of eight, 15 fit on
// the GPU with a CTA per SM, and the CTAs of the sixteenth share.  FP32 throughout.  The whole call goes through in one pass:
//   loads         rows of 128 q or k channels, or of 32 v channels, a warp at a time into shared memory;
//   convolution   in place, a channel per thread of warps 0-7 (q, k) and 8-9 (v), while warps 10-11 make the gates;
//   norms         a warp per group of four tokens: the normalised vectors, and the products k_t . k_j and q_t . k_j of the
//                 group, of which warps 8-11 make the coefficients of all groups;
//   recurrence    a group at a time.  With G_t the product of the group's decays up to t and S0 the state in front of it,
//                   u_t = v_t - G_t S0^T k_t
//                   o_t = G_t S0^T q_t + sum over j <= t of R_tj u_j
//                   S   = G_3 S0 + sum over t of k_t (sum over j <= t of W_tj u_j)^T
//                   D = (I + L)^-1 diag(beta),  L_tj = beta_t (G_t / G_j) (k_t . k_j), j < t
//                   W_tj = (G_3 / G_t) D_tj,  R_tj = sum over i, j <= i <= t, of (G_t / G_i) (q_t . k_i) D_ij
//                 (the ratios are products of decays, nothing is divided; the coefficients are made in 64 bits and rounded
//                 once, and G_3 S0 is rounded with its sum and not before), so that eight reductions over the rows and a
//                 hand-back of corrections are paid once in four tokens.  A lane owns eight rows of four columns, a warp
//                 eight columns; 32 sums over 16 lanes are 30 exchanges and leave token t, column c with lane 4 t + c.
//                 A head with a decay above 1 (a positive coefficient) goes token by token: a product of its decays may be
//                 infinite where each decay is finite and what it multiplies is zero or small.
//   output norm   the slices of a head exchange their sums of squares.
// 24 layers' calls replayed, a call, BF16 and FP32: 2 tokens 6.2 and 6.4 us, 4 6.4 and 6.5, 17 11.2 and 11.3, 32 15.2 and 15.3,
// 63 27.1 and 26.4; a token at a time, a warp per four columns in clusters of eight: 7.8, 8.7, 17.2, 25.5 and 26.6, 48.4 and
// 49.2.  At 63 tokens its 64 SMs issue in 56 % of the cycles; a warp's 5.1 cycles between instructions are 1.2 at barriers,
// 0.8 for want of an issue slot, 0.7 waiting for memory.  A wait in front of the loop over groups in place of the one inside
// its first turn gains 0.8 us at 63 tokens and costs 0.25 at 2 to 4, which every prompt ends with.  FP32, distance from 64 bits
// at 63 tokens: output 1.68e-7, state 2.03e-7; a token at a time 1.72e-7 and 2.10e-7.
//
// The line to the chunks is one of accuracy: 64 tokens take 18.3 us (FP32 19.3) in chunks and would take 27.1 (26.5) here, but
// products of chunks have ten-bit mantissas, which leave the state 4.5e-4 from 64 bits.
constexpr std::uint32_t kShortMaxTokens = 63;
constexpr std::uint32_t kShortRows = 64;
constexpr std::uint32_t kShortGroup = 4;
constexpr int kShortThreads = 384;
constexpr std::uint32_t kShortWarps = kShortThreads / 32;
constexpr std::uint32_t kShortLoads = 6;  // q and k rows a warp has in flight
constexpr std::uint32_t kShortRounds = (kStepMaxRatio * kShortRows + 4 * kShortWarps - 1) / (4 * kShortWarps);

struct ShortShared {
  float qk[2][kShortRows][kDim];                  // inputs, then their convolutions, then normalised
  float v[kStepMaxRatio][kShortRows][kStepColumns]; // inputs, then their convolutions, then the outputs
  float2 gain[kStepMaxRatio][kShortRows];         // G_t, G_3
  float4 write[kStepMaxRatio][kShortRows];        // W_tj for j = t, t ^ 1, t ^ 2, t ^ 3
  float4 read[kStepMaxRatio][kShortRows];         // R_tj likewise
  float dots[kShortRows / kShortGroup][16];
  float beta[kStepMaxRatio][kShortRows];
  float decay[kStepMaxRatio][kShortRows];
  bool grows[kStepMaxRatio];                      // a decay is above 1
  float norm[kStepSlices][kStepMaxRatio * kShortRows];
  std::uint64_t norm_bar;
};

// Sums of N values over N neighbouring lanes: lane l of them gets the total of value l.
template <int N> __device__ __forceinline__ float fold(float (&v)[N]) {
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1) {
    const bool upper = (threadIdx.x & half) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float give = upper ? v[i] : v[i + half];
      const float keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xFFFFFFFFU, give, half);
    }
  }
  return v[0];
}
// four neighbouring elements; Wide: they start on the boundary of one access
template <int Dtype, bool Wide>
__device__ __forceinline__ float4 load_quad(const typename Scalar<Dtype>::Type *at) {
  if constexpr (Wide) {
    return Io<Dtype>::load4(at, 0);
  } else {
    using Act = Scalar<Dtype>;
    return make_float4(Act::widen(at[0]), Act::widen(at[1]), Act::widen(at[2]), Act::widen(at[3]));
  }
}

template <int Dtype, int WeightDtype, bool Wide>
__global__ void __launch_bounds__(kShortThreads, 1) gdn_layer_short_kernel(const LayerParams p) {
  using Act = Scalar<Dtype>;
  using Weight = Scalar<WeightDtype>;
  using ActType = typename Act::Type;
  using WeightType = typename Weight::Type;
  constexpr std::uint32_t kHistory = kFastWidth - 1;
  extern __shared__ __align__(16) unsigned char short_smem[];
  ShortShared &sh = *reinterpret_cast<ShortShared *>(short_smem);
  std::uint32_t slice;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(slice));
  const std::uint32_t key_head = blockIdx.x / kStepSlices;
  const std::uint32_t ratio = p.value_heads / p.key_heads;
  const std::uint32_t n = p.tokens;
  const std::uint32_t tid = threadIdx.x;
  const std::uint32_t warp = tid >> 5;
  const std::uint32_t lane = tid & 31;
  const auto *input = static_cast<const ActType *>(p.input);
  const auto *conv_weight = static_cast<const WeightType *>(p.conv_weight);
  auto head_of = [&](std::uint32_t index) { return key_head + (index < ratio ? index : 0U) * p.key_heads; };
  const std::uint32_t q_channel = key_head * kDim;
  const std::uint32_t k_channel = (p.key_heads + key_head) * kDim;
  auto v_channel = [&](std::uint32_t index) { return 2 * p.key_heads * kDim + head_of(index) * kDim + slice * kStepColumns; };
  auto z_column = [&](std::uint32_t index) {
    return p.conv_dim + 2 * p.value_heads + head_of(index) * kDim + slice * kStepColumns;
  };
  // the channel a thread of warps 0-9 convolves
  const bool convolves = warp < 8 || (warp < 10 && warp - 8 < ratio);
  const std::uint32_t channel = warp < 8 ? (warp < 4 ? q_channel : k_channel) + (tid & (kDim - 1)) : v_channel(warp & 1U) + lane;
  // recurrence: warps 0-3 have the first value head, 4-7 the second one if there is one; a lane's rows are
  // 4 row_lane + 64 i .. + 3 and its columns `column` .. + 3 of the slice
  const std::uint32_t h = (warp >> 2) & 1U;
  const bool recurs = warp < 8 && h < ratio;
  const std::uint32_t row_lane = lane & 15U;
  const std::uint32_t column = 8 * (warp & 3U) + 4 * (lane >> 4);
  float *state = p.recurrent_state + static_cast<std::size_t>(head_of(h)) * kDim * kDim + slice * kStepColumns;
  auto state_row = [&](std::uint32_t i) {
    return state + static_cast<std::size_t>(4 * row_lane + 64 * (i >> 2) + (i & 3U)) * kDim + column;
  };

  // While the kernels in front still run, this one asks for what it will read first (hints, no reads: what those kernels
  // write is current in L2 either way).
  if (recurs) {
    hint_l2(state + static_cast<std::size_t>(tid & (kDim - 1)) * kDim);
  }
  if (convolves && lane % 8 == 0) {
    hint_l2(conv_weight + static_cast<std::size_t>(channel) * kFastWidth);
    hint_l2(p.convolution_state + static_cast<std::size_t>(channel) * kHistory);
  }
  if (warp < n && lane < 16) {
    const ActType *row = input + static_cast<std::size_t>(warp) * p.token_stride;
    const std::uint32_t index = (lane >> 2) & 1U;
    const std::uint32_t what = lane & 3U;
    hint_l2(row + (lane < 4    ? q_channel + 32 * what
                   : lane < 8  ? k_channel + 32 * what
                   : what == 0 ? v_channel(index)
                   : what == 1 ? p.conv_dim + head_of(index)
                   : what == 2 ? p.conv_dim + p.value_heads + head_of(index)
                               : z_column(index)));
  }
  const std::uint32_t shift = ratio - 1;
  const std::uint32_t rows = n << shift; // of v, z and the output: (token, value head)
  if (tid == 0) {
    expect_sums(&sh.norm_bar, rows * kStepSlices * 4);
  }
  __syncwarp();
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); // every CTA of the cluster has started
  grid_dependency_wait();
  grid_dependents_may_launch();

  // ---- loads ----
  float4 raw[kShortLoads];
  auto load_rows = [&](std::uint32_t from) { // row r of the call's 2 n: q or k (bit 0) of token r / 2
#pragma unroll
    for (std::uint32_t i = 0; i < kShortLoads; ++i) {
      const std::uint32_t row = from + warp + kShortWarps * i;
      if (row < 2 * n) {
        raw[i] = load_quad<Dtype, Wide>(input + static_cast<std::size_t>(row >> 1) * p.token_stride +
                                        ((row & 1U) == 0 ? q_channel : k_channel) + 4 * lane);
      }
    }
  };
  auto store_rows = [&](std::uint32_t from) {
#pragma unroll
    for (std::uint32_t i = 0; i < kShortLoads; ++i) {
      const std::uint32_t row = from + warp + kShortWarps * i;
      if (row < 2 * n) {
        *reinterpret_cast<float4 *>(&sh.qk[row & 1U][row >> 1][4 * lane]) = raw[i];
      }
    }
  };
  load_rows(0);
  // v and z: eight lanes a row
  const std::uint32_t quad = 4 * (lane & 7U);
  float4 v_raw[kShortRounds];
  float4 z[kShortRounds];
#pragma unroll
  for (std::uint32_t r = 0; r < kShortRounds; ++r) {
    const std::uint32_t row = 4 * (warp + kShortWarps * r) + (lane >> 3);
    if (row < rows) {
      const ActType *at = input + static_cast<std::size_t>(row >> shift) * p.token_stride + quad;
      v_raw[r] = load_quad<Dtype, Wide>(at + v_channel(row & shift));
      z[r] = load_quad<Dtype, Wide>(at + z_column(row & shift));
    }
  }
  float taps[kFastWidth];
  float window[kHistory + kShortGroup]; // the three tokens in front of the call, then of the group
  if (convolves) {
    const float4 four = load_quad<WeightDtype, Wide && WeightDtype == RIB200_DTYPE_F32>(
        conv_weight + static_cast<std::size_t>(channel) * kFastWidth);
    taps[0] = four.x;
    taps[1] = four.y;
    taps[2] = four.z;
    taps[3] = four.w;
#pragma unroll
    for (std::uint32_t i = 0; i < kHistory; ++i) {
      window[i] = p.convolution_state[static_cast<std::size_t>(channel) * kHistory + i];
    }
  }
  float4 s[8];
  if (recurs) {
#pragma unroll
    for (std::uint32_t i = 0; i < 8; ++i) {
      s[i] = *reinterpret_cast<const float4 *>(state_row(i));
    }
  }
  store_rows(0);
  for (std::uint32_t from = kShortWarps * kShortLoads; from < 2 * n; from += kShortWarps * kShortLoads) {
    load_rows(from);
    store_rows(from);
  }
#pragma unroll
  for (std::uint32_t r = 0; r < kShortRounds; ++r) {
    const std::uint32_t row = 4 * (warp + kShortWarps * r) + (lane >> 3);
    if (row < rows) {
      *reinterpret_cast<float4 *>(&sh.v[row & shift][row >> shift][quad]) = v_raw[r];
    }
  }
  __syncthreads();

  // ---- convolution and SiLU, whole groups of four tokens, rows past the last one included (they are not used); gates ----
  float next_history[kHistory] = {}; // the last three tokens of [old history | call]
  if (convolves) {
    float *at = warp < 8 ? &sh.qk[warp >> 2][0][tid & (kDim - 1)] : &sh.v[warp & 1U][0][lane];
    const std::uint32_t pitch = warp < 8 ? kDim : kStepColumns;
#pragma unroll
    for (std::uint32_t i = 0; i < kHistory; ++i) {
      const std::uint32_t source = n + i; // position in [history | call], at least 2
      next_history[i] = source >= kHistory ? at[(source - kHistory) * pitch] : window[2];
    }
#pragma unroll 1
    for (std::uint32_t group = 0; group < n; group += kShortGroup) {
      float value[kShortGroup];
#pragma unroll
      for (std::uint32_t t = 0; t < kShortGroup; ++t) {
        window[kHistory + t] = at[t * pitch];
        // the current token's tap first, then the history, oldest first
        float sum = window[kHistory + t] * taps[kHistory];
#pragma unroll
        for (std::uint32_t i = 0; i < kHistory; ++i) {
          sum += window[t + i] * taps[i];
        }
        value[t] = silu(sum);
      }
#pragma unroll
      for (std::uint32_t t = 0; t < kShortGroup; ++t) {
        at[t * pitch] = value[t];
      }
#pragma unroll
      for (std::uint32_t i = 0; i < kHistory; ++i) {
        window[i] = window[kShortGroup + i];
      }
      at += kShortGroup * pitch;
    }
  } else if (warp - 10 < ratio) {
    const std::uint32_t index = warp - 10;
    const float coefficient = Weight::widen(static_cast<const WeightType *>(p.recurrent_a)[head_of(index)]);
    const float dt = Weight::widen(static_cast<const WeightType *>(p.dt_bias)[head_of(index)]);
    bool grows = false;
    for (std::uint32_t t = lane; t < n; t += 32) {
      const ActType *gates = input + static_cast<std::size_t>(t) * p.token_stride + p.conv_dim + head_of(index);
      const float b = Act::widen(gates[0]);
      const float a = Act::widen(gates[p.value_heads]);
      const float decay = expf(coefficient * softplus(a + dt));
      sh.beta[index][t] = sigmoid(b);
      sh.decay[index][t] = decay;
      grows = grows || !(decay <= 1.0F);
    }
    grows = __any_sync(0xFFFFFFFFU, grows);
    if (lane == 0) {
      sh.grows[index] = grows;
    }
  }
  __syncthreads();

  // ---- norms and products of a group of tokens per warp; tokens past the last one become zeros ----
#pragma unroll 1
  for (std::uint32_t group = warp; kShortGroup * group < n; group += kShortWarps) {
    const std::uint32_t t0 = kShortGroup * group;
    float4 q[kShortGroup];
    float4 k[kShortGroup];
    auto dot = [](const float4 &x, const float4 &y) { return (x.x * y.x + x.y * y.y) + (x.z * y.z + x.w * y.w); };
    float squares[2 * kShortGroup];
#pragma unroll
    for (std::uint32_t t = 0; t < kShortGroup; ++t) {
      q[t] = *reinterpret_cast<const float4 *>(&sh.qk[0][t0 + t][4 * lane]);
      k[t] = *reinterpret_cast<const float4 *>(&sh.qk[1][t0 + t][4 * lane]);
      squares[t] = dot(q[t], q[t]);
      squares[kShortGroup + t] = dot(k[t], k[t]);
    }
    float sum = fold(squares);
    sum += __shfl_xor_sync(0xFFFFFFFFU, sum, 8);
    sum += __shfl_xor_sync(0xFFFFFFFFU, sum, 16);
    const float scale = rsqrtf(sum + kQkEpsilon) * ((lane & kShortGroup) == 0 ? rsqrtf(static_cast<float>(kDim)) : 1.0F);
#pragma unroll
    for (std::uint32_t t = 0; t < kShortGroup; ++t) {
      const float q_scale = __shfl_sync(0xFFFFFFFFU, scale, t);
      const float k_scale = __shfl_sync(0xFFFFFFFFU, scale, kShortGroup + t);
      const bool live = t0 + t < n;
      q[t] = live ? make_float4(q[t].x * q_scale, q[t].y * q_scale, q[t].z * q_scale, q[t].w * q_scale)
                  : make_float4(0.0F, 0.0F, 0.0F, 0.0F);
      k[t] = live ? make_float4(k[t].x * k_scale, k[t].y * k_scale, k[t].z * k_scale, k[t].w * k_scale)
                  : make_float4(0.0F, 0.0F, 0.0F, 0.0F);
      *reinterpret_cast<float4 *>(&sh.qk[0][t0 + t][4 * lane]) = q[t];
      *reinterpret_cast<float4 *>(&sh.qk[1][t0 + t][4 * lane]) = k[t];
    }
    // k_t . k_j at 4 t + j for j < t, q_t . k_j at 4 j + t for j <= t: below, and on and above the diagonal of one square
    float dots[16];
#pragma unroll
    for (std::uint32_t t = 0; t < kShortGroup; ++t) {
#pragma unroll
      for (std::uint32_t j = 0; j <= t; ++j) {
        if (j < t) {
          dots[4 * t + j] = dot(k[t], k[j]);
        }
        dots[4 * j + t] = dot(q[t], k[j]);
      }
    }
    float total = fold(dots);
    total += __shfl_xor_sync(0xFFFFFFFFU, total, 16);
    if (lane < 16) {
      sh.dots[group][lane] = total;
    }
  }
  __syncthreads();

  // ---- coefficients, while the warps of the recurrence form the sums of their first group: a thread per group, value head
  // and token j of the group makes what u_j puts into the tokens from j on ----
  static_assert(kShortThreads - 256 == kShortRows * kStepMaxRatio, "a thread per value head and token");
  auto coefficients_made = [] { asm volatile("bar.sync 1, %0;\n" ::"n"(kShortThreads) : "memory"); };
  if (warp >= 8) {
    const std::uint32_t group = (tid - 256) / (kStepMaxRatio * kShortGroup);
    const std::uint32_t head = (tid / kShortGroup) % kStepMaxRatio;
    const std::uint32_t j = tid % kShortGroup;
    const std::uint32_t t0 = kShortGroup * group;
    if (t0 < n && head < ratio) {
      const float *d = sh.dots[group];
      double beta[kShortGroup];
      double decay[kShortGroup];
      double gain = 1.0; // up to token j
      double all = 1.0;
#pragma unroll
      for (std::uint32_t t = 0; t < kShortGroup; ++t) {
        const bool live = t0 + t < n;
        beta[t] = live ? sh.beta[head][t0 + t] : 0.0F;
        decay[t] = live ? sh.decay[head][t0 + t] : 1.0F;
        all *= decay[t];
        gain = t == j ? all : gain;
      }
      double product[kShortGroup][kShortGroup]; // [t][i]: the decays of the tokens after i up to t
#pragma unroll
      for (std::uint32_t i = 0; i < kShortGroup; ++i) {
        product[i][i] = 1.0;
#pragma unroll
        for (std::uint32_t t = i + 1; t < kShortGroup; ++t) {
          product[t][i] = product[t - 1][i] * decay[t];
        }
      }
      double column[kShortGroup]; // column j of (I + L)^-1 diag(beta)
#pragma unroll
      for (std::uint32_t t = 0; t < kShortGroup; ++t) {
        double sum = 0.0;
        double out = 0.0;
#pragma unroll
        for (std::uint32_t i = 0; i < t; ++i) {
          sum += product[t][i] * d[4 * t + i] * column[i];
          out += product[t][i] * d[4 * i + t] * column[i];
        }
        column[t] = t == j ? beta[t] : -beta[t] * sum;
        // the entry of token t at t ^ j; those in front of j are not used
        reinterpret_cast<float *>(&sh.write[head][t0 + t])[t ^ j] = static_cast<float>(product[kShortGroup - 1][t] * column[t]);
        reinterpret_cast<float *>(&sh.read[head][t0 + t])[t ^ j] = static_cast<float>(out + d[5 * t] * column[t]);
      }
      sh.gain[head][t0 + j] = make_float2(static_cast<float>(gain), static_cast<float>(all));
    }
    coefficients_made();
  } else if (!recurs) {
    coefficients_made();
  }

  // ---- the recurrence ----
  auto fetch = [&](const float *vector, float (&x)[8]) {
    const float4 low = *reinterpret_cast<const float4 *>(vector + 4 * row_lane);
    const float4 high = *reinterpret_cast<const float4 *>(vector + 4 * row_lane + 64);
    x[0] = low.x;
    x[1] = low.y;
    x[2] = low.z;
    x[3] = low.w;
    x[4] = high.x;
    x[5] = high.y;
    x[6] = high.z;
    x[7] = high.w;
  };
  auto products = [&](const float (&x)[8], float *to) { // two chains of four a column
    float4 low = make_float4(s[0].x * x[0], s[0].y * x[0], s[0].z * x[0], s[0].w * x[0]);
    float4 high = make_float4(s[4].x * x[4], s[4].y * x[4], s[4].z * x[4], s[4].w * x[4]);
#pragma unroll
    for (int i = 1; i < 4; ++i) {
      low.x = fmaf(s[i].x, x[i], low.x);
      low.y = fmaf(s[i].y, x[i], low.y);
      low.z = fmaf(s[i].z, x[i], low.z);
      low.w = fmaf(s[i].w, x[i], low.w);
      high.x = fmaf(s[4 + i].x, x[4 + i], high.x);
      high.y = fmaf(s[4 + i].y, x[4 + i], high.y);
      high.z = fmaf(s[4 + i].z, x[4 + i], high.z);
      high.w = fmaf(s[4 + i].w, x[4 + i], high.w);
    }
    to[0] = low.x + high.x;
    to[1] = low.y + high.y;
    to[2] = low.z + high.z;
    to[3] = low.w + high.w;
  };
  if (recurs && sh.grows[h]) { // token by token
    coefficients_made();
#pragma unroll 1
    for (std::uint32_t token = 0; token < n; ++token) {
      float key[8];
      float query[8];
      float sums[8]; // S^T k and S^T q of the lane's columns
      fetch(sh.qk[1][token], key);
      fetch(sh.qk[0][token], query);
      products(key, sums);
      products(query, sums + 4);
#pragma unroll
      for (int offset = 8; offset > 0; offset >>= 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          sums[i] += __shfl_xor_sync(0xFFFFFFFFU, sums[i], offset);
        }
      }
      const float beta = sh.beta[h][token];
      const float decay = sh.decay[h][token];
      const float dot = sh.dots[token / kShortGroup][5 * (token % kShortGroup)]; // q . k
      float4 &row = *reinterpret_cast<float4 *>(&sh.v[h][token][column]);
      const float4 delta = make_float4((row.x - decay * sums[0]) * beta, (row.y - decay * sums[1]) * beta,
                                       (row.z - decay * sums[2]) * beta, (row.w - decay * sums[3]) * beta);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        s[r] = make_float4(decay * s[r].x + key[r] * delta.x, decay * s[r].y + key[r] * delta.y,
                           decay * s[r].z + key[r] * delta.z, decay * s[r].w + key[r] * delta.w);
      }
      __syncwarp(); // all lanes of the columns have read the values
      if (row_lane == 0) {
        row = make_float4(decay * sums[4] + delta.x * dot, decay * sums[5] + delta.y * dot,
                          decay * sums[6] + delta.z * dot, decay * sums[7] + delta.w * dot);
      }
    }
  } else if (recurs) {
    const std::uint32_t t = row_lane >> 2;
    const bool second = (t & 1U) != 0; // has t ^ 1 in front of it
    const bool upper = (t & 2U) != 0;  // has t ^ 2 and t ^ 3 in front of it
#pragma unroll 1
    for (std::uint32_t group = 0; group < n; group += kShortGroup) {
      float k[kShortGroup][8];
      float a_sums[16];
      float b_sums[16];
#pragma unroll
      for (std::uint32_t i = 0; i < kShortGroup; ++i) {
        fetch(sh.qk[1][group + i], k[i]);
        products(k[i], a_sums + 4 * i);
      }
#pragma unroll
      for (std::uint32_t i = 0; i < kShortGroup; ++i) {
        float q[8];
        fetch(sh.qk[0][group + i], q);
        products(q, b_sums + 4 * i);
      }
      const float a = fold(a_sums);
      const float b = fold(b_sums);
      if (group == 0) {
        coefficients_made();
      }
      const float2 gain = sh.gain[h][group + t];
      float &slot = sh.v[h][group + t][column + (row_lane & 3U)];
      const float u = group + t < n ? fmaf(-gain.x, a, slot) : 0.0F;
      const float u1 = __shfl_xor_sync(0xFFFFFFFFU, u, 4);
      const float u2 = __shfl_xor_sync(0xFFFFFFFFU, u, 8);
      const float u3 = __shfl_xor_sync(0xFFFFFFFFU, u, 12);
      auto combine = [&](const float4 &entries) {
        float sum = upper ? fmaf(entries.z, u2, entries.w * u3) : 0.0F;
        sum = second ? fmaf(entries.y, u1, sum) : sum;
        return fmaf(entries.x, u, sum);
      };
      const float correction = combine(sh.write[h][group + t]);
      auto corrections = [&](int i) { // of token i for the lane's four columns
        const int from = static_cast<int>(lane & 16U) + 4 * i;
        return make_float4(__shfl_sync(0xFFFFFFFFU, correction, from), __shfl_sync(0xFFFFFFFFU, correction, from + 1),
                           __shfl_sync(0xFFFFFFFFU, correction, from + 2), __shfl_sync(0xFFFFFFFFU, correction, from + 3));
      };
      auto two = [](float k0, float c0, float k1, float c1, float sum) { return fmaf(k1, c1, fmaf(k0, c0, sum)); };
      {
        const float4 c0 = corrections(0);
        const float4 c1 = corrections(1);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          s[r] = make_float4(fmaf(gain.y, s[r].x, two(k[0][r], c0.x, k[1][r], c1.x, 0.0F)),
                             fmaf(gain.y, s[r].y, two(k[0][r], c0.y, k[1][r], c1.y, 0.0F)),
                             fmaf(gain.y, s[r].z, two(k[0][r], c0.z, k[1][r], c1.z, 0.0F)),
                             fmaf(gain.y, s[r].w, two(k[0][r], c0.w, k[1][r], c1.w, 0.0F)));
        }
      }
      {
        const float4 c2 = corrections(2);
        const float4 c3 = corrections(3);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          s[r] = make_float4(two(k[2][r], c2.x, k[3][r], c3.x, s[r].x), two(k[2][r], c2.y, k[3][r], c3.y, s[r].y),
                             two(k[2][r], c2.z, k[3][r], c3.z, s[r].z), two(k[2][r], c2.w, k[3][r], c3.w, s[r].w));
        }
      }
      slot = fmaf(gain.x, b, combine(sh.read[h][group + t]));
    }
  }
  __syncthreads();

  // ---- output norm over the four slices, gate ----
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory"); // every CTA of the cluster has started
  const float4 norm_weight = load_quad<WeightDtype, false>(static_cast<const WeightType *>(p.output_norm_weight) +
                                                           slice * kStepColumns + quad);
  float4 out[kShortRounds];
#pragma unroll
  for (std::uint32_t r = 0; r < kShortRounds; ++r) {
    if (4 * (warp + kShortWarps * r) >= rows) {
      continue;
    }
    const std::uint32_t row = min(4 * (warp + kShortWarps * r) + (lane >> 3), rows - 1);
    out[r] = *reinterpret_cast<const float4 *>(&sh.v[row & shift][row >> shift][quad]);
    float squares = (out[r].x * out[r].x + out[r].y * out[r].y) + (out[r].z * out[r].z + out[r].w * out[r].w);
#pragma unroll
    for (int offset = 4; offset > 0; offset >>= 1) {
      squares += __shfl_xor_sync(0xFFFFFFFFU, squares, offset);
    }
    if ((lane & 7U) < kStepSlices && 4 * (warp + kShortWarps * r) + (lane >> 3) < rows) { // to the four CTAs
      send_sum(&sh.norm[slice][row], &sh.norm_bar, lane & 7U, squares);
    }
  }
  all_sent();
#pragma unroll
  for (std::uint32_t r = 0; r < kShortRounds; ++r) {
    if (4 * (warp + kShortWarps * r) >= rows) {
      continue;
    }
    z[r] = make_float4(norm_weight.x * silu(z[r].x), norm_weight.y * silu(z[r].y), norm_weight.z * silu(z[r].z),
                       norm_weight.w * silu(z[r].w));
  }
  const bool complete = wait_for_sums(&sh.norm_bar, p.status);
#pragma unroll
  for (std::uint32_t r = 0; r < kShortRounds; ++r) {
    const std::uint32_t row = 4 * (warp + kShortWarps * r) + (lane >> 3);
    if (row < rows) {
      const float norm = (sh.norm[0][row] + sh.norm[1][row]) + (sh.norm[2][row] + sh.norm[3][row]);
      const float scale = rsqrtf(norm / static_cast<float>(kDim) + p.epsilon);
      const float4 x = make_float4(out[r].x * scale * z[r].x, out[r].y * scale * z[r].y, out[r].z * scale * z[r].z,
                                   out[r].w * scale * z[r].w);
      auto *to = static_cast<ActType *>(p.output) +
                 (static_cast<std::size_t>(row >> shift) * p.value_heads + head_of(row & shift)) * kDim +
                 slice * kStepColumns + quad;
      if constexpr (Wide) {
        Io<Dtype>::store4(to, 0, x);
      } else {
        to[0] = Act::narrow(x.x);
        to[1] = Act::narrow(x.y);
        to[2] = Act::narrow(x.z);
        to[3] = Act::narrow(x.w);
      }
    }
  }
  if (recurs) {
#pragma unroll
    for (std::uint32_t i = 0; i < 8; ++i) {
      *reinterpret_cast<float4 *>(state_row(i)) = s[i];
    }
  }
  if (convolves && (slice == 0 || warp >= 8)) {
#pragma unroll
    for (std::uint32_t i = 0; i < kHistory; ++i) {
      p.convolution_state[static_cast<std::size_t>(channel) * kHistory + i] = next_history[i];
    }
  }
  leave_cluster(&sh.norm_bar, complete, p.status);
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
  p.status = device_status_word();
  return p;
}

template <int Dtype, int WeightDtype, bool Wide> void launch_short(const LayerParams &p, cudaStream_t stream) {
  static std::once_flag flags[64];
  int device = 0;
  cuda_ok(cudaGetDevice(&device), "cudaGetDevice");
  require(device >= 0 && device < 64, "device ordinal out of range", RIB200_STATUS_INTERNAL);
  auto *kernel = gdn_layer_short_kernel<Dtype, WeightDtype, Wide>;
  std::call_once(flags[device], [&] {
    cuda_ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(ShortShared)),
            "gated-delta short call shared-memory opt-in");
  });
  launch_programmatic_cluster(kernel, dim3(kStepSlices * p.key_heads), dim3(kShortThreads), kStepSlices, sizeof(ShortShared),
                              stream, "gated-delta short call launch", p);
}

template <int Dtype, int WeightDtype> void launch_step(const LayerParams &p, cudaStream_t stream) {
  if (p.tokens == 1) {
    const std::uint32_t cluster = kStepSlices * (p.value_heads / p.key_heads);
    launch_programmatic_cluster(gdn_layer_step_kernel<Dtype, WeightDtype>, dim3(cluster * p.key_heads), dim3(kStepThreads),
                                cluster, 0, stream, "gated-delta step launch", p);
  } else if (vector_forms_apply(p)) {
    launch_short<Dtype, WeightDtype, true>(p, stream);
  } else {
    launch_short<Dtype, WeightDtype, false>(p, stream);
  }
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
