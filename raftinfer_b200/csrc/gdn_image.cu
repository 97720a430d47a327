// First kernel of the chunked gated-delta prefill: turns the operands of the recurrence into the FP16 images and gate
// arrays that the chunk kernels read (layout in gdn_chunk.hpp).  Two sources:
//   layer  the packed rows of qwen35_gated_delta: depthwise causal convolution (width 4) + SiLU over the q|k|v channels,
//          L2 normalisation of q and k (q also times 1/sqrt(128)), beta = sigmoid(b), log decay = A softplus(a + dt)
//          (cpp/kernels/qwen35_delta.cu:236-276,375-411,522-529; CPU cpp/reference/qwen35.cpp:417-469);
//   core   operands that are already convolved and normalised (rib200_gdn_core, and layer calls of other widths).
//
// FP16 keeps the 10 mantissa bits of TF32 in half the bytes, but not its range.  q and k are normalised and stored times
// 2^7, so that an element keeps its 10 bits down to 2^-21.  V is brought under 2^14 by a power of two per (chunk, head,
// column), divided out of U in FP32: an element keeps its 10 bits down to 2^-27 of the largest one of its column in the
// chunk, and no column - one of large values, an infinity - takes precision from another.  (With one factor per (chunk,
// head) a column 2^-27 of the largest was lost, and an infinity wiped out the other 127.)
//
// 67 MB of BF16 rows read and 67 MB of images written at 4096 tokens (the FP32 q|k|v this replaces were 134 MB) in 47 us:
// DRAM 23 %, issue slots 53 %, L1 32 %, 22 warps an SM (80 registers), whose longest waits are for their rows and for an
// issue slot; neither bytes nor instructions alone bound it.  One CTA per (chunk, head vector); the lanes that share a row
// take four consecutive tokens, whose seven rows are fetched at once, and every image row leaves as full 128-byte lines.
// Rows that neighbouring lanes fetch too come from L1.

#include "common.hpp"
#include "gdn_chunk.hpp"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace rib200 {
namespace {

constexpr int kTokensPerRun = 4; // consecutive tokens of the lanes that share a row
constexpr int kRuns = kGdnChunk / kTokensPerRun;
// a lane has `Count` dims of a row; threads of a CTA and CTAs an SM should hold
template <int Count> struct Layout {
  static constexpr int kLanes = kGdnDim / Count;
  static constexpr int kThreads = kRuns * kLanes;
  static constexpr int kCtas = Count == 4 ? 2 : 3;
};
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
  std::uint32_t wide; // rows of 16-bit elements start on 16-byte boundaries
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

// `Count` consecutive elements of a row, four or (16-bit types) eight, as they lie in memory, and as FP32.  `wide`: rows
// start on 16-byte boundaries (else eight elements come in two pieces).
template <int Dtype, int Count> struct Piece;
template <> struct Piece<RIB200_DTYPE_F32, 4> {
  float4 raw;
  __device__ __forceinline__ void load(const void *base, std::size_t index, bool) {
    raw = *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + index);
  }
  __device__ __forceinline__ void clear() { raw = make_float4(0.0F, 0.0F, 0.0F, 0.0F); }
  __device__ __forceinline__ void value(float (&x)[4]) const {
    x[0] = raw.x;
    x[1] = raw.y;
    x[2] = raw.z;
    x[3] = raw.w;
  }
};
template <int Dtype, int Count> struct Piece {
  static_assert(Dtype == RIB200_DTYPE_BF16 || Dtype == RIB200_DTYPE_F16, "16-bit elements");
  std::uint32_t raw[Count / 2];
  __device__ __forceinline__ void load(const void *base, std::size_t index, bool wide) {
    const std::uint16_t *src = static_cast<const std::uint16_t *>(base) + index;
    if constexpr (Count == 8) {
      if (wide) {
        const uint4 v = *reinterpret_cast<const uint4 *>(src);
        raw[0] = v.x;
        raw[1] = v.y;
        raw[2] = v.z;
        raw[3] = v.w;
        return;
      }
    }
#pragma unroll
    for (int h = 0; h < Count / 4; ++h) {
      const uint2 v = *reinterpret_cast<const uint2 *>(src + 4 * h);
      raw[2 * h] = v.x;
      raw[2 * h + 1] = v.y;
    }
  }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < Count / 2; ++i) {
      raw[i] = 0U;
    }
  }
  __device__ __forceinline__ void value(float (&x)[Count]) const {
#pragma unroll
    for (int i = 0; i < Count / 2; ++i) {
      if constexpr (Dtype == RIB200_DTYPE_BF16) {
        x[2 * i] = __uint_as_float(raw[i] << 16);
        x[2 * i + 1] = __uint_as_float(raw[i] & 0xFFFF0000U);
      } else {
        const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(&raw[i]));
        x[2 * i] = v.x;
        x[2 * i + 1] = v.y;
      }
    }
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

// Gates of 32 value heads over one chunk: the running sum of the log decays and beta, zero past the last token; for the
// chain's bounds the largest product of consecutive decays, which exceeds 1 only where log decays are positive, and sum
// and maximum of beta.
template <int Dtype, int Count, bool Layer>
__device__ __forceinline__ void gate_arrays(const ImageParams &p, std::uint32_t chunk, std::uint32_t head0) {
  __shared__ float s_decay[kGdnChunk][kGateHeads + 1];
  __shared__ float s_beta[kGdnChunk][kGateHeads + 1];
  constexpr int kWarps = Layout<Count>::kThreads / 32;
  constexpr int kTokensPerWarp = kGdnChunk / kWarps;
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
          const float b = load_weight(p.input, at + head, Dtype);
          const float a = load_weight(p.input, at + p.value_heads + head, Dtype);
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
  for (std::uint32_t h = warp; h < kGateHeads && head0 + h < p.value_heads; h += kWarps) {
    float a = s_decay[lane][h];
    float b = s_decay[lane + 32][h];
    const bool grows = __any_sync(0xFFFFFFFFU, a > 0.0F || b > 0.0F);
    // magnitudes, NaN left out: a token that is NaN must not take the scales of the tokens in front of it along
    const float beta_a = fmaxf(fabsf(s_beta[lane][h]), 0.0F);
    const float beta_b = fmaxf(fabsf(s_beta[lane + 32][h]), 0.0F);
    float beta_sum = beta_a + beta_b;
    const float beta_max = __uint_as_float(__reduce_max_sync(0xFFFFFFFFU, __float_as_uint(fmaxf(beta_a, beta_b))));
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const float ua = __shfl_up_sync(0xFFFFFFFFU, a, d);
      const float ub = __shfl_up_sync(0xFFFFFFFFU, b, d);
      beta_sum += __shfl_xor_sync(0xFFFFFFFFU, beta_sum, d);
      if (lane >= d) {
        a += ua;
        b += ub;
      }
    }
    b += __shfl_sync(0xFFFFFFFFU, a, 31);
    float growth = 1.0F;
    if (grows) { // largest G_i - G_j over j <= i, the start of the chunk (0) among the j; NaN drops out
      float low_a = fminf(a, 0.0F);
      float low_b = b;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        low_a = fminf(low_a, __shfl_up_sync(0xFFFFFFFFU, low_a, d)); // a lane without a neighbour gets its own value
        low_b = fminf(low_b, __shfl_up_sync(0xFFFFFFFFU, low_b, d));
      }
      low_b = fminf(low_b, __shfl_sync(0xFFFFFFFFU, low_a, 31));
      const float rise = fmaxf(fmaxf(a - low_a, b - low_b), 0.0F);
      const float most = __uint_as_float(__reduce_max_sync(0xFFFFFFFFU, __float_as_uint(rise)));
      growth = fminf(expf(most), 0x1p100F);
    }
    float *gates = reinterpret_cast<float *>(record_of(p, chunk, head0 + h) + kGdnRecGates);
    gates[kGdnGateG + lane] = a;
    gates[kGdnGateG + 32 + lane] = b;
    gates[kGdnGateBeta + lane] = s_beta[lane][h];
    gates[kGdnGateBeta + 32 + lane] = s_beta[lane + 32][h];
    if (lane == 0) {
      gates[kGdnGateGrowth] = growth;
      gates[kGdnGateBetaSum] = beta_sum;
      gates[kGdnGateBetaMax] = beta_max;
    }
  }
}

// grid (chunks x (2 Hk + Hv head vectors + gate CTAs)), the chunk slowest: the CTAs of a chunk read the same rows
template <int Dtype, int Count, bool Layer>
__global__ void __launch_bounds__(Layout<Count>::kThreads, Layout<Count>::kCtas) gdn_image_kernel(const ImageParams p) {
  grid_dependents_may_launch(); // the chunk kernels set themselves up early and wait for this grid to end
  grid_dependency_wait();
  const std::uint32_t vectors = 2 * p.key_heads + p.value_heads;
  const std::uint32_t per_chunk = vectors + (p.value_heads + kGateHeads - 1) / kGateHeads;
  const std::uint32_t chunk = blockIdx.x / per_chunk;
  const std::uint32_t vec = blockIdx.x - chunk * per_chunk;
  if (vec >= vectors) {
    gate_arrays<Dtype, Count, Layer>(p, chunk, (vec - vectors) * kGateHeads);
    return;
  }
  constexpr std::uint32_t kLanes = Layout<Count>::kLanes;
  const std::uint32_t sub = threadIdx.x % kLanes; // a lane has dims Count sub .. Count sub + Count - 1
  const std::uint32_t row0 = threadIdx.x / kLanes * kTokensPerRun;
  const std::uint32_t tok0 = chunk * kGdnChunk + row0;
  const bool is_q = vec < p.key_heads;
  const bool is_v = vec >= 2 * p.key_heads;
  const std::uint32_t head = is_q ? vec : (is_v ? vec - 2 * p.key_heads : vec - p.key_heads);
  const bool wide = p.wide != 0;
  const bool whole = (chunk + 1) * kGdnChunk <= p.tokens; // no row of the chunk is past the last token
  __shared__ std::uint32_t s_largest[Count][kLanes]; // by column: bits of the largest |v| of the chunk
  if (threadIdx.x < kGdnDim) {
    s_largest[threadIdx.x / kLanes][threadIdx.x % kLanes] = 0U;
  }

  float out[kTokensPerRun][Count];
  if constexpr (Layer) {
    const std::uint32_t channel = vec * kGdnDim + Count * sub;
    // rows tok0 - 3 .. tok0 + 3
    Piece<Dtype, Count> x[kTokensPerRun + kWidth - 1];
    if (whole && chunk > 0) {
      const std::size_t first = static_cast<std::size_t>(tok0 - (kWidth - 1)) * p.token_stride + channel;
#pragma unroll
      for (int r = 0; r < kTokensPerRun + kWidth - 1; ++r) {
        x[r].load(p.input, first + static_cast<std::size_t>(r) * p.token_stride, wide);
      }
    } else {
#pragma unroll
      for (int r = 0; r < kTokensPerRun + kWidth - 1; ++r) {
        const int tok = static_cast<int>(tok0) + r - (kWidth - 1);
        if (tok >= 0 && tok < static_cast<int>(p.tokens)) {
          x[r].load(p.input, static_cast<std::size_t>(tok) * p.token_stride + channel, wide);
        } else {
          x[r].clear();
        }
      }
    }
    // Taps through shared memory, by tap: a lane's channels are 64 or 128 bytes apart in memory, and fetched from there
    // the weights took several times the L1 wavefronts of the rows.  Pieces of four channels, even ones first.
    __shared__ __align__(16) float s_taps[kWidth][kGdnDim];
    if (threadIdx.x < kGdnDim) {
      const std::uint32_t c = threadIdx.x;
      const std::size_t at = (static_cast<std::size_t>(vec) * kGdnDim + c) * kWidth;
      const std::uint32_t place = Count == 8 ? ((c >> 2) & 1U) * (kGdnDim / 2) + (c >> 3) * 4 + (c & 3U) : c;
      if (p.weight_dtype == RIB200_DTYPE_F32) {
        const float4 taps = *reinterpret_cast<const float4 *>(static_cast<const float *>(p.conv_weight) + at);
        s_taps[0][place] = taps.x;
        s_taps[1][place] = taps.y;
        s_taps[2][place] = taps.z;
        s_taps[3][place] = taps.w;
      } else {
#pragma unroll
        for (int h = 0; h < kWidth; ++h) {
          s_taps[h][place] = load_weight(p.conv_weight, at + h, p.weight_dtype);
        }
      }
    }
    __syncthreads();
    float w[Count][kWidth]; // taps of the lane's channels, oldest first
#pragma unroll
    for (int h = 0; h < kWidth; ++h) {
#pragma unroll
      for (int q = 0; q < Count / 4; ++q) {
        const float4 taps = *reinterpret_cast<const float4 *>(&s_taps[h][q * (kGdnDim / 2) + 4 * sub]);
        w[4 * q][h] = taps.x;
        w[4 * q + 1][h] = taps.y;
        w[4 * q + 2][h] = taps.z;
        w[4 * q + 3][h] = taps.w;
      }
    }
    float before[kWidth - 1][Count]; // the three rows in front of the run
#pragma unroll
    for (int h = 0; h < kWidth - 1; ++h) {
      x[h].value(before[h]);
    }
    if (tok0 == 0) { // history [channel][3]: element h is the token 3 - h steps before this call's first one
      const float *hist = p.history + static_cast<std::size_t>(channel) * (kWidth - 1);
#pragma unroll
      for (int h = 0; h < kWidth - 1; ++h) {
#pragma unroll
        for (int c = 0; c < Count; ++c) {
          before[h][c] = hist[c * (kWidth - 1) + h];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < kTokensPerRun; ++i) {
      float now[Count];
      x[i + kWidth - 1].value(now);
#pragma unroll
      for (int c = 0; c < Count; ++c) {
        // the reference adds the current token's tap first, then the history taps oldest first
        float sum = now[c] * w[c][3];
#pragma unroll
        for (int h = 0; h < kWidth - 1; ++h) {
          sum += before[h][c] * w[c][h];
        }
        before[0][c] = before[1][c];
        before[1][c] = before[2][c];
        before[2][c] = now[c];
        out[i][c] = silu_fast(sum);
      }
    }
    if (!whole) { // rows past the last token are inert
#pragma unroll
      for (int i = 0; i < kTokensPerRun; ++i) {
#pragma unroll
        for (int c = 0; c < Count; ++c) {
          out[i][c] = tok0 + i < p.tokens ? out[i][c] : 0.0F;
        }
      }
    }
    if (!is_v) {
      const float q_scale = is_q ? rsqrtf(static_cast<float>(kGdnDim)) : 1.0F;
      float squares[kTokensPerRun];
#pragma unroll
      for (int i = 0; i < kTokensPerRun; ++i) {
        squares[i] = 0.0F;
#pragma unroll
        for (int c = 0; c < Count; c += 4) {
          squares[i] += (out[i][c] * out[i][c] + out[i][c + 1] * out[i][c + 1]) +
                        (out[i][c + 2] * out[i][c + 2] + out[i][c + 3] * out[i][c + 3]);
        }
      }
      // the same order of additions for either layout, so that a row's image does not depend on the length of the call:
      // four dims a lane first join the neighbour that completes eight
      auto join = [&](int offset) {
#pragma unroll
        for (int i = 0; i < kTokensPerRun; ++i) {
          squares[i] += __shfl_xor_sync(0xFFFFFFFFU, squares[i], offset);
        }
      };
      if constexpr (Count == 4) {
        join(1);
      }
#pragma unroll
      for (int offset = static_cast<int>(kLanes) / 2; offset > (Count == 4 ? 1 : 0); offset >>= 1) {
        join(offset);
      }
#pragma unroll
      for (int i = 0; i < kTokensPerRun; ++i) {
        const float scale = rsqrtf(squares[i] + kQkEpsilon) * q_scale;
#pragma unroll
        for (int c = 0; c < Count; ++c) {
          out[i][c] *= scale;
        }
      }
    }
  } else {
    const void *source = is_q ? p.q : (is_v ? p.v : p.k);
    const std::size_t stride = is_q ? p.q_stride : (is_v ? p.v_stride : p.k_stride);
    Piece<Dtype, Count> x[kTokensPerRun];
#pragma unroll
    for (int i = 0; i < kTokensPerRun; ++i) {
      if (tok0 + i < p.tokens) {
        x[i].load(source, static_cast<std::size_t>(tok0 + i) * stride + head * kGdnDim + Count * sub, wide);
      } else {
        x[i].clear();
      }
    }
#pragma unroll
    for (int i = 0; i < kTokensPerRun; ++i) {
      x[i].value(out[i]);
    }
  }

  unsigned char *image;
  std::uint32_t block;
  float scale[Count];
  if (is_v) {
    if constexpr (!Layer) {
      __syncthreads(); // s_largest is set up (a layer call has had its barrier for the taps)
    }
    std::uint32_t largest[Count];
#pragma unroll
    for (int c = 0; c < Count; ++c) {
      largest[c] = 0U;
#pragma unroll
      for (int i = 0; i < kTokensPerRun; ++i) {
        largest[c] = max(largest[c], __float_as_uint(fabsf(out[i][c])));
      }
    }
#pragma unroll
    for (int c = 0; c < Count; ++c) {
      atomicMax(&s_largest[c][sub], largest[c]);
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < Count; ++c) {
      scale[c] = gdn_power(gdn_scale_exponent(__uint_as_float(s_largest[c][sub])));
    }
    if (threadIdx.x < kGdnDim) {
      float *gates = reinterpret_cast<float *>(record_of(p, chunk, head) + kGdnRecGates);
      gates[kGdnGateMax + threadIdx.x] = __uint_as_float(s_largest[threadIdx.x % Count][threadIdx.x / Count]);
    }
    image = p.scratch.v + (static_cast<std::size_t>(chunk) * p.value_heads + head) * kGdnVBytes;
    block = kGdnBlock;
  } else {
#pragma unroll
    for (int c = 0; c < Count; ++c) {
      scale[c] = kGdnUnit;
    }
    image = p.scratch.kq + (static_cast<std::size_t>(chunk) * p.key_heads + head) * kGdnKqBytes +
            (is_q ? kGdnBlock : 0U); // the Q rows follow the K rows of a block
    block = kGdnKqBlock;
  }
  // a lane's dims are a 16-byte piece of a row of the image (8 FP16), or half of one
  const std::uint32_t dim = Count * sub;
  unsigned char *at = image + (dim >> 6) * block + (dim & 7U) * 2U;
#pragma unroll
  for (int i = 0; i < kTokensPerRun; ++i) {
    const std::uint32_t row = row0 + i;
    unsigned char *to = at + row * kGdnRowBytes + ((((dim & 63U) >> 3) ^ (row & 7U)) << 4);
    std::uint32_t h[Count / 2];
#pragma unroll
    for (int c = 0; c < Count / 2; ++c) {
      h[c] = pack_half(out[i][2 * c] * scale[2 * c], out[i][2 * c + 1] * scale[2 * c + 1]);
    }
    if constexpr (Count == 8) {
      *reinterpret_cast<uint4 *>(to) = make_uint4(h[0], h[1], h[2], h[3]);
    } else {
      *reinterpret_cast<uint2 *>(to) = make_uint2(h[0], h[1]);
    }
  }
}

template <int Dtype, int Count, bool Layer> void launch(const ImageParams &p, std::size_t ctas, cudaStream_t stream) {
  launch_programmatic(gdn_image_kernel<Dtype, Count, Layer>, dim3(static_cast<unsigned int>(ctas)),
                      dim3(Layout<Count>::kThreads), 0, stream, "gated-delta image launch", p);
}

// Eight dims a lane is fewer instructions, four is more warps a CTA.  4096 tokens BF16 (4160 CTAs) 193.9 us for the
// layer call with four and 186.8 with eight; 149 tokens (195 CTAs) 22.1 and 22.9: eight from four waves on.  FP32 has
// four always (eight would hold 32 bytes a row in registers: 1173 tokens in the executor's calls 127.3 and 134.9 us).
template <int Dtype, bool Layer> void launch(const ImageParams &p, cudaStream_t stream) {
  const std::uint32_t gate_ctas = (p.value_heads + kGateHeads - 1) / kGateHeads;
  const std::size_t ctas = static_cast<std::size_t>(2 * p.key_heads + p.value_heads + gate_ctas) * p.chunks;
  require(ctas <= 0x7FFFFFFFU, "gated-delta prefill: too many tokens for one launch");
  if constexpr (Dtype != RIB200_DTYPE_F32) {
    if (ctas >= 4 * 3 * 148) {
      launch<Dtype, 8, Layer>(p, ctas, stream);
      return;
    }
  }
  launch<Dtype, 4, Layer>(p, ctas, stream);
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
  p.wide = p.token_stride % 8 == 0 && reinterpret_cast<std::uintptr_t>(a.input) % 16 == 0 ? 1U : 0U;
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
  p.wide = 1; // whole heads behind 16-byte aligned pointers
  fill_sizes(p, workspace, a.tokens, a.key_heads, a.value_heads);
  if (a.qkv_f32) {
    launch<RIB200_DTYPE_F32, false>(p, stream);
  } else {
    launch<RIB200_DTYPE_BF16, false>(p, stream);
  }
}

} // namespace rib200
