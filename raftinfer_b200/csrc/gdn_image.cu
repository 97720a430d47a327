// First kernel of the chunked gated-delta prefill: turns the operands of the recurrence into the FP16 images and gate
// arrays that the chunk kernels read (layout in gdn_chunk.hpp).  Two sources:
//   layer  the packed rows of qwen35_gated_delta: depthwise causal convolution (width 4) + SiLU over the q|k|v channels,
//          L2 normalisation of q and k (q also times 1/sqrt(128)), beta = sigmoid(b), log decay = A softplus(a + dt)
//          (cpp/kernels/qwen35_delta.cu:236-276,375-411,522-529; CPU cpp/reference/qwen35.cpp:417-469);
//   core   operands that are already convolved and normalised (rib200_gdn_core, and layer calls of other widths).
//
// FP16 keeps the 10 mantissa bits that the chunk kernels' products had in TF32, in half the bytes.  The range is no
// concern for q and k, which are normalised; V is brought under 2^14 by a power of two per (chunk, head), so that an
// element keeps its 10 bits down to 2^-27 of the largest one, and the factor is divided out of U in FP32.
//
// HBM-bound: 67 MB of BF16 rows read and 67 MB of images written at 4096 tokens (the FP32 q|k|v this replaces were
// 134 MB).  One CTA per (chunk, head vector), a warp per four tokens, a lane per four channels: the seven rows a warp
// convolves are fetched at once, whole 256- or 512-byte segments, and every image row leaves as full 128-byte lines.
// Rows a neighbouring warp fetches too come from L1; eight tokens a warp (256 threads) fetch less but leave 16 warps an
// SM instead of 32, too few to cover the latency of HBM.

#include "common.hpp"
#include "gdn_chunk.hpp"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace rib200 {
namespace {

constexpr int kImageThreads = 512;
constexpr int kTokensPerWarp = kGdnChunk / (kImageThreads / 32);
constexpr int kWidth = 4;
constexpr int kGateHeads = 32; // value heads per gate CTA
constexpr float kQkEpsilon = 1.0e-6F;

struct ImageParams {
  // layer: packed rows, convolution
  const void *input;
  const void *conv_weight, *recurrent_a, *dt_bias;
  const float *history; // [channel][3]
  std::uint32_t conv_dim, token_stride;
  int32_t weight_dtype;
  // core: operands and gates as they are
  const void *q, *k, *v;
  std::size_t q_stride, k_stride, v_stride;
  const float *beta, *log_decay; // [token][value head]
  GdnChunkScratch scratch;
  std::uint32_t tokens, chunks, key_heads, value_heads;
};

__device__ __forceinline__ float load_weight(const void *base, std::size_t index, int32_t dtype) {
  if (dtype == RIB200_DTYPE_F32) {
    return static_cast<const float *>(base)[index];
  }
  if (dtype == RIB200_DTYPE_F16) {
    return __half2float(static_cast<const __half *>(base)[index]);
  }
  return __bfloat162float(static_cast<const __nv_bfloat16 *>(base)[index]);
}

// Four consecutive elements as they lie in memory, and as FP32.
template <int Dtype> struct Quad;
template <> struct Quad<RIB200_DTYPE_F32> {
  float4 raw;
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
    raw = *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + index);
  }
  __device__ __forceinline__ void clear() { raw = make_float4(0.0F, 0.0F, 0.0F, 0.0F); }
  __device__ __forceinline__ float4 value() const { return raw; }
  static __device__ __forceinline__ float one(const void *base, std::size_t index) {
    return static_cast<const float *>(base)[index];
  }
};
template <> struct Quad<RIB200_DTYPE_BF16> {
  uint2 raw;
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
    raw = *reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(base) + index);
  }
  __device__ __forceinline__ void clear() { raw = make_uint2(0U, 0U); }
  __device__ __forceinline__ float4 value() const {
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xFFFF0000U),
                       __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xFFFF0000U));
  }
  static __device__ __forceinline__ float one(const void *base, std::size_t index) {
    return __bfloat162float(static_cast<const __nv_bfloat16 *>(base)[index]);
  }
};
template <> struct Quad<RIB200_DTYPE_F16> {
  uint2 raw;
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
    raw = *reinterpret_cast<const uint2 *>(static_cast<const __half *>(base) + index);
  }
  __device__ __forceinline__ void clear() { raw = make_uint2(0U, 0U); }
  __device__ __forceinline__ float4 value() const {
    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&raw.x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  static __device__ __forceinline__ float one(const void *base, std::size_t index) {
    return __half2float(static_cast<const __half *>(base)[index]);
  }
};

__device__ __forceinline__ float softplus(float x) {
  if (x > 20.0F) {
    return x;
  }
  if (x < -20.0F) {
    return expf(x);
  }
  return log1pf(expf(x));
}
// SiLU on the special-function unit (ex2 + rcp); relative error about 1e-6
__device__ __forceinline__ float silu_fast(float x) {
  float e;
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(e) : "f"(x * -1.4426950408889634F));
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(1.0F + e));
  return x * r;
}
__device__ __forceinline__ std::uint32_t pack_half(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const std::uint32_t *>(&v);
}
__device__ __forceinline__ unsigned char *record_of(const ImageParams &p, std::uint32_t chunk, std::uint32_t head) {
  return p.scratch.records + (static_cast<std::size_t>(chunk) * p.value_heads + head) * kGdnRecBytes;
}

// Gates of 32 value heads over one chunk: the running sum of the log decays and beta, zero past the last token.
template <int Dtype, bool Layer>
__device__ __forceinline__ void gate_arrays(const ImageParams &p, std::uint32_t chunk, std::uint32_t head0) {
  __shared__ float s_decay[kGdnChunk][kGateHeads + 1];
  __shared__ float s_beta[kGdnChunk][kGateHeads + 1];
  const std::uint32_t warp = threadIdx.x >> 5;
  const std::uint32_t lane = threadIdx.x & 31;
  const std::uint32_t head = head0 + lane;
  if (head < p.value_heads) {
    float coefficient = 0.0F;
    float dt = 0.0F;
    if constexpr (Layer) {
      coefficient = load_weight(p.recurrent_a, head, p.weight_dtype);
      dt = load_weight(p.dt_bias, head, p.weight_dtype);
    }
#pragma unroll
    for (int r = 0; r < kTokensPerWarp; ++r) {
      const std::uint32_t row = warp * kTokensPerWarp + r;
      const std::uint32_t tok = chunk * kGdnChunk + row;
      float decay = 0.0F;
      float beta = 0.0F;
      if (tok < p.tokens) {
        if constexpr (Layer) {
          const std::size_t at = static_cast<std::size_t>(tok) * p.token_stride + p.conv_dim;
          const float b = Quad<Dtype>::one(p.input, at + head);
          const float a = Quad<Dtype>::one(p.input, at + p.value_heads + head);
          beta = 1.0F / (1.0F + expf(-b));
          decay = coefficient * softplus(a + dt);
        } else {
          const std::size_t at = static_cast<std::size_t>(tok) * p.value_heads + head;
          beta = p.beta[at];
          decay = p.log_decay[at];
        }
      }
      s_decay[row][lane] = decay;
      s_beta[row][lane] = beta;
    }
  }
  __syncthreads();
  for (std::uint32_t h = warp; h < kGateHeads && head0 + h < p.value_heads; h += kImageThreads / 32) {
    float a = s_decay[lane][h];
    float b = s_decay[lane + 32][h];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float ua = __shfl_up_sync(0xFFFFFFFFU, a, d);
      const float ub = __shfl_up_sync(0xFFFFFFFFU, b, d);
      if (lane >= d) {
        a += ua;
        b += ub;
      }
    }
    b += __shfl_sync(0xFFFFFFFFU, a, 31);
    float *gates = reinterpret_cast<float *>(record_of(p, chunk, head0 + h) + kGdnRecGates);
    gates[kGdnGateG + lane] = a;
    gates[kGdnGateG + 32 + lane] = b;
    gates[kGdnGateBeta + lane] = s_beta[lane][h];
    gates[kGdnGateBeta + 32 + lane] = s_beta[lane + 32][h];
  }
}

// grid (chunks x (2 Hk + Hv head vectors + gate CTAs)), the chunk slowest: the CTAs of a chunk read the same rows
template <int Dtype, bool Layer> __global__ void __launch_bounds__(kImageThreads, 2) gdn_image_kernel(const ImageParams p) {
  grid_dependents_may_launch(); // the chunk kernels set themselves up early and wait for this grid to end
  grid_dependency_wait();
  const std::uint32_t vectors = 2 * p.key_heads + p.value_heads;
  const std::uint32_t per_chunk = vectors + (p.value_heads + kGateHeads - 1) / kGateHeads;
  const std::uint32_t chunk = blockIdx.x / per_chunk;
  const std::uint32_t vec = blockIdx.x - chunk * per_chunk;
  if (vec >= vectors) {
    gate_arrays<Dtype, Layer>(p, chunk, (vec - vectors) * kGateHeads);
    return;
  }
  const std::uint32_t warp = threadIdx.x >> 5;
  const std::uint32_t lane = threadIdx.x & 31;
  const std::uint32_t row0 = warp * kTokensPerWarp;
  const std::uint32_t tok0 = chunk * kGdnChunk + row0;
  const bool is_q = vec < p.key_heads;
  const bool is_v = vec >= 2 * p.key_heads;
  const std::uint32_t head = is_q ? vec : (is_v ? vec - 2 * p.key_heads : vec - p.key_heads);

  float4 out[kTokensPerWarp];
  if constexpr (Layer) {
    const std::uint32_t channel = vec * kGdnDim + 4 * lane;
    // rows tok0 - 3 .. tok0 + 7
    Quad<Dtype> x[kTokensPerWarp + kWidth - 1];
#pragma unroll
    for (int r = 0; r < kTokensPerWarp + kWidth - 1; ++r) {
      const long long tok = static_cast<long long>(tok0) + r - (kWidth - 1);
      if (tok >= 0 && tok < static_cast<long long>(p.tokens)) {
        x[r].load(p.input, static_cast<std::size_t>(tok) * p.token_stride + channel);
      } else {
        x[r].clear();
      }
    }
    float w[4][kWidth]; // taps of the lane's four channels, oldest first
    if (p.weight_dtype == RIB200_DTYPE_F32) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float4 taps = *reinterpret_cast<const float4 *>(static_cast<const float *>(p.conv_weight) +
                                                              static_cast<std::size_t>(channel + c) * kWidth);
        w[c][0] = taps.x;
        w[c][1] = taps.y;
        w[c][2] = taps.z;
        w[c][3] = taps.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int h = 0; h < kWidth; ++h) {
          w[c][h] = load_weight(p.conv_weight, static_cast<std::size_t>(channel + c) * kWidth + h, p.weight_dtype);
        }
      }
    }
    float4 before[kWidth - 1]; // the three rows in front of the warp's own
#pragma unroll
    for (int h = 0; h < kWidth - 1; ++h) {
      before[h] = x[h].value();
    }
    if (tok0 == 0) { // history [channel][3]: element h is the token 3 - h steps before this call's first one
      const float *hist = p.history + static_cast<std::size_t>(channel) * (kWidth - 1);
#pragma unroll
      for (int h = 0; h < kWidth - 1; ++h) {
        before[h] = make_float4(hist[h], hist[(kWidth - 1) + h], hist[2 * (kWidth - 1) + h], hist[3 * (kWidth - 1) + h]);
      }
    }
#pragma unroll
    for (int i = 0; i < kTokensPerWarp; ++i) {
      const float4 now = x[i + kWidth - 1].value();
      // the reference adds the current token's tap first, then the history taps oldest first
      float4 sum = make_float4(now.x * w[0][3], now.y * w[1][3], now.z * w[2][3], now.w * w[3][3]);
#pragma unroll
      for (int h = 0; h < kWidth - 1; ++h) {
        sum.x += before[h].x * w[0][h];
        sum.y += before[h].y * w[1][h];
        sum.z += before[h].z * w[2][h];
        sum.w += before[h].w * w[3][h];
      }
      before[0] = before[1];
      before[1] = before[2];
      before[2] = now;
      out[i] = make_float4(silu_fast(sum.x), silu_fast(sum.y), silu_fast(sum.z), silu_fast(sum.w));
      if (tok0 + i >= p.tokens) { // rows past the last token are inert
        out[i] = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
      }
    }
    if (!is_v) {
      const float q_scale = is_q ? rsqrtf(static_cast<float>(kGdnDim)) : 1.0F;
      float squares[kTokensPerWarp];
#pragma unroll
      for (int i = 0; i < kTokensPerWarp; ++i) {
        squares[i] = (out[i].x * out[i].x + out[i].y * out[i].y) + (out[i].z * out[i].z + out[i].w * out[i].w);
      }
#pragma unroll
      for (int offset = 16; offset > 0; offset >>= 1) {
#pragma unroll
        for (int i = 0; i < kTokensPerWarp; ++i) {
          squares[i] += __shfl_xor_sync(0xFFFFFFFFU, squares[i], offset);
        }
      }
#pragma unroll
      for (int i = 0; i < kTokensPerWarp; ++i) {
        const float scale = rsqrtf(squares[i] + kQkEpsilon) * q_scale;
        out[i] = make_float4(out[i].x * scale, out[i].y * scale, out[i].z * scale, out[i].w * scale);
      }
    }
  } else {
    const void *source = is_q ? p.q : (is_v ? p.v : p.k);
    const std::size_t stride = is_q ? p.q_stride : (is_v ? p.v_stride : p.k_stride);
    Quad<Dtype> x[kTokensPerWarp];
#pragma unroll
    for (int i = 0; i < kTokensPerWarp; ++i) {
      if (tok0 + i < p.tokens) {
        x[i].load(source, static_cast<std::size_t>(tok0 + i) * stride + head * kGdnDim + 4 * lane);
      } else {
        x[i].clear();
      }
    }
#pragma unroll
    for (int i = 0; i < kTokensPerWarp; ++i) {
      out[i] = x[i].value();
    }
  }

  unsigned char *image;
  std::uint32_t block;
  float scale = 1.0F;
  if (is_v) {
    __shared__ float s_max[kImageThreads / 32];
    float largest = 0.0F;
#pragma unroll
    for (int i = 0; i < kTokensPerWarp; ++i) {
      largest = fmaxf(largest, fmaxf(fmaxf(fabsf(out[i].x), fabsf(out[i].y)), fmaxf(fabsf(out[i].z), fabsf(out[i].w))));
    }
#pragma unroll
    for (int offset = 16; offset > 0; offset >>= 1) {
      largest = fmaxf(largest, __shfl_xor_sync(0xFFFFFFFFU, largest, offset));
    }
    if (lane == 0) {
      s_max[warp] = largest;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kImageThreads / 32; ++w) {
      largest = fmaxf(largest, s_max[w]);
    }
    // exponent e with largest in [2^e, 2^(e+1)); the scale is 2^(13 - e), kept away from the ends of the FP32 range
    const int biased = static_cast<int>(__float_as_uint(largest) >> 23);
    const int exponent = min(max(127 + 13 + 127 - biased, 27), 227);
    scale = __uint_as_float(static_cast<std::uint32_t>(exponent) << 23);
    if (threadIdx.x == 0) {
      float *gates = reinterpret_cast<float *>(record_of(p, chunk, head) + kGdnRecGates);
      gates[kGdnGateInvScale] = __uint_as_float(static_cast<std::uint32_t>(254 - exponent) << 23);
      gates[kGdnGateMax] = largest;
    }
    image = p.scratch.v + (static_cast<std::size_t>(chunk) * p.value_heads + head) * kGdnVBytes;
    block = kGdnBlock;
  } else {
    image = p.scratch.kq + (static_cast<std::size_t>(chunk) * p.key_heads + head) * kGdnKqBytes +
            (is_q ? kGdnBlock : 0U); // the Q rows follow the K rows of a block
    block = kGdnKqBlock;
  }
  // lane: dims 4 lane .. 4 lane + 3, half of the 16-byte piece (lane % 16) / 2 of block lane / 16
  unsigned char *at = image + (lane >> 4) * block + (lane & 1U) * 8U;
#pragma unroll
  for (int i = 0; i < kTokensPerWarp; ++i) {
    const std::uint32_t row = row0 + i;
    const std::uint32_t piece = ((lane & 15U) >> 1) ^ (row & 7U);
    *reinterpret_cast<uint2 *>(at + row * kGdnRowBytes + (piece << 4)) =
        make_uint2(pack_half(out[i].x * scale, out[i].y * scale), pack_half(out[i].z * scale, out[i].w * scale));
  }
}

template <int Dtype, bool Layer> void launch(const ImageParams &p, cudaStream_t stream) {
  const std::uint32_t gate_ctas = (p.value_heads + kGateHeads - 1) / kGateHeads;
  const std::size_t ctas = static_cast<std::size_t>(2 * p.key_heads + p.value_heads + gate_ctas) * p.chunks;
  require(ctas <= 0x7FFFFFFFU, "gated-delta prefill: too many tokens for one launch");
  launch_programmatic(gdn_image_kernel<Dtype, Layer>, dim3(static_cast<unsigned int>(ctas)), dim3(kImageThreads), 0,
                      stream, "gated-delta image launch", p);
}

void fill_sizes(ImageParams &p, void *workspace, std::uint32_t tokens, std::uint32_t key_heads,
                std::uint32_t value_heads) {
  p.tokens = tokens;
  p.chunks = (tokens + kGdnChunk - 1) / kGdnChunk;
  p.key_heads = key_heads;
  p.value_heads = value_heads;
  p.scratch = gdn_chunk_scratch(workspace, p.chunks, key_heads, value_heads);
}

} // namespace

void launch_gdn_layer_images(const GdnLayerArgs &a, void *workspace, cudaStream_t stream) {
  ImageParams p{};
  p.input = a.input;
  p.conv_weight = a.conv_weight;
  p.recurrent_a = a.recurrent_a;
  p.dt_bias = a.dt_bias;
  p.history = a.convolution_state;
  p.conv_dim = (2 * a.key_heads + a.value_heads) * kGdnDim;
  p.token_stride = p.conv_dim + 2 * a.value_heads + a.value_heads * kGdnDim;
  p.weight_dtype = a.weight_dtype;
  fill_sizes(p, workspace, a.tokens, a.key_heads, a.value_heads);
  if (a.dtype == RIB200_DTYPE_F32) {
    launch<RIB200_DTYPE_F32, true>(p, stream);
  } else if (a.dtype == RIB200_DTYPE_F16) {
    launch<RIB200_DTYPE_F16, true>(p, stream);
  } else {
    launch<RIB200_DTYPE_BF16, true>(p, stream);
  }
}

void launch_gdn_core_images(const GdnCoreArgs &a, void *workspace, cudaStream_t stream) {
  ImageParams p{};
  p.q = a.q;
  p.k = a.k;
  p.v = a.v;
  p.q_stride = a.q_stride;
  p.k_stride = a.k_stride;
  p.v_stride = a.v_stride;
  p.beta = a.beta;
  p.log_decay = a.log_decay;
  fill_sizes(p, workspace, a.tokens, a.key_heads, a.value_heads);
  if (a.qkv_f32) {
    launch<RIB200_DTYPE_F32, false>(p, stream);
  } else {
    launch<RIB200_DTYPE_BF16, false>(p, stream);
  }
}

} // namespace rib200
