// Scratch layout shared by the kernels of the chunked gated-delta prefill (gdn_image.cu, gdn_chunk.cu).
//
// Chunks of 64 tokens, heads of 128 dims.  Every operand the tensor cores read lies in global memory as the image it
// has in shared memory: FP16, [block of 64 dims][row][128 bytes], the 16-byte piece index of a row XORed with row % 8
// (the 128-byte swizzle).  With 16-bit elements one such image serves both ways round: as a K-major operand (rows are
// M or N, dims are K) and as an MN-major one (dims are M or N, rows are K), so K, Q and V exist once.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace rib200 {

constexpr int kGdnDim = 128;
constexpr int kGdnChunk = 64;
constexpr int kGdnSlice = 32; // state columns per CTA of the chain kernel
constexpr int kGdnSlices = kGdnDim / kGdnSlice;

constexpr std::uint32_t kGdnRowBytes = 128;
// (chunk, key head): [2 blocks][128 rows: K, then Q][128 bytes]
constexpr std::uint32_t kGdnKqBlock = 2 * kGdnChunk * kGdnRowBytes;
constexpr std::uint32_t kGdnKqBytes = 2 * kGdnKqBlock;
// (chunk, value head): V, every column times a power of two of its own, [2 blocks][64 rows][128 bytes]
constexpr std::uint32_t kGdnBlock = kGdnChunk * kGdnRowBytes;
constexpr std::uint32_t kGdnVBytes = 2 * kGdnBlock;
// (chunk, value head) record: W as an image of 64 rows, P (64 tokens x 64 tokens) as one block of such rows, the gates,
// then U as four FP32 column slices [64 rows][32], the 16-byte piece index of a row XORed with row % 8.
constexpr std::uint32_t kGdnRecW = 0;
constexpr std::uint32_t kGdnRecP = kGdnRecW + 2 * kGdnBlock;
constexpr std::uint32_t kGdnRecGates = kGdnRecP + kGdnBlock;
// gates: running log decay G [64], beta [64], largest |v| of every column [128], the largest product of consecutive
// decays (1 where no decay exceeds 1), sum and maximum of beta, one unused
constexpr std::uint32_t kGdnGateG = 0;
constexpr std::uint32_t kGdnGateBeta = 64;
constexpr std::uint32_t kGdnGateMax = 128;
constexpr std::uint32_t kGdnGateGrowth = 256;
constexpr std::uint32_t kGdnGateBetaSum = 257;
constexpr std::uint32_t kGdnGateBetaMax = 258;
constexpr std::uint32_t kGdnGateBytes = 260 * 4;
constexpr std::uint32_t kGdnGateArea = 1152;
constexpr std::uint32_t kGdnSliceU = kGdnChunk * kGdnSlice * 4;
constexpr std::uint32_t kGdnRecU = kGdnRecGates + kGdnGateArea;
constexpr std::uint32_t kGdnRecBytes = kGdnRecU + kGdnSlices * kGdnSliceU;
static_assert(kGdnRecGates % 16 == 0 && kGdnGateBytes % 16 == 0 && kGdnGateBytes <= kGdnGateArea && kGdnRecU % 128 == 0 &&
                  kGdnRecBytes % 128 == 0,
              "bulk copies start and end on 16-byte boundaries");

// Units of the FP16 operands, powers of two that keep all ten mantissa bits of what is far below one: K and Q are stored
// times 2^7, T diag(beta) times 2^7 u, W times 2^14 u and P times 2^8 u, where u = 2^-floor(log2(growth)) is 1 unless some
// decay exceeds 1.  |k| <= 1 and 0 <= beta <= 1 make |T|, |W| <= growth and |P| <= growth |q|; P's unit is the smaller one
// because q need not be scaled.  Growth of more than 2^20 leaves the early rows of a chunk too few bits: that is reported.
constexpr float kGdnUnit = 128.0F;
constexpr int kGdnUnitW = 14;
constexpr int kGdnUnitP = 8;
constexpr float kGdnMostGrowth = 0x1p20F;

// exponent field of the power of two that brings `bound` into [2^13, 2^14), kept away from the ends of the range
__device__ __forceinline__ std::uint32_t gdn_scale_exponent(float bound) {
  const int biased = static_cast<int>((__float_as_uint(bound) >> 23) & 255U);
  return static_cast<std::uint32_t>(min(max(127 + 13 + 127 - biased, 27), 227));
}
__device__ __forceinline__ float gdn_power(std::uint32_t exponent) { return __uint_as_float(exponent << 23); }

struct GdnChunkScratch {
  unsigned char *kq;      // [chunk][key head] of kGdnKqBytes
  unsigned char *v;       // [chunk][value head] of kGdnVBytes
  unsigned char *records; // [chunk][value head] of kGdnRecBytes
};

inline GdnChunkScratch gdn_chunk_scratch(void *workspace, std::size_t chunks, std::size_t key_heads,
                                         std::size_t value_heads) {
  auto *base = static_cast<unsigned char *>(workspace);
  GdnChunkScratch s{};
  s.kq = base;
  s.v = s.kq + chunks * key_heads * kGdnKqBytes;
  s.records = s.v + chunks * value_heads * kGdnVBytes;
  return s;
}

} // namespace rib200
