// Chunk-64 WY-form prefill of the gated delta rule for key_dim = value_dim = 128.  The reference has only the
// token-sequential recurrence (cpp/kernels/qwen35_delta.cu:482-576, cpp/reference/qwen35.cpp:459-518); this is the
// same recurrence regrouped so that the dense work runs on the tensor cores.
//
// Per value head (key head = head % key_heads), for a chunk of C = 64 tokens entering with state S0 [128][128],
// with G_i the running sum of the log decays inside the chunk (decay applied before the read, as the reference):
//   A_ij  = beta_i exp(G_i - G_j) (k_i . k_j)   for j < i            T = (I + A)^-1
//   W     = T diag(beta exp(G)) K                U = T diag(beta) V
//   Delta = U - W S0
//   O     = diag(exp(G)) Q S0 + P Delta,         P_ij = exp(G_i - G_j) (q_i . k_j) for j <= i
//   S_C   = exp(G_C) S0 + K^T diag(exp(G_C - G)) Delta
// |k| <= 1, |q| <= 1 and 0 <= beta <= 1 are assumed.  Decays usually are at most 1; where log decays are positive, the
// largest product of consecutive ones in a chunk (`growth`) enters the scales below.  A ragged last chunk is padded with
// inert rows (beta = 0, log decay = 0, k = q = v = 0), which leave the state untouched.
//
// Three kernels: gdn_image.cu leaves K, Q and V as FP16 operand images and the gates as arrays; `prepare`, parallel over
// (chunk, value head), makes W, U and P of them; `chain` walks the chunks of one (value head, 32-column slice of the
// state) in order and writes the outputs - in a layer call after the output norm and gate.
//
// Products run on tcgen05 with FP16 operands and FP32 accumulators: the 10-bit mantissa of TF32, half its bytes, and
// - unlike 32-bit elements - one image serves as K-major and as MN-major operand, so K, Q and V are never transposed
// and K is never copied with its decays (the decay goes to the rows of Delta).  TF32 has FP32's range and FP16 has not, so
// every operand is scaled by powers of two that are divided out in FP32: K, Q, T, W and P, whose elements are at most 1
// (times growth), by the fixed units of gdn_chunk.hpp; V, Delta and the state, which may have any magnitude, by a factor
// per (chunk, head, column) from bounds that are known before they are formed.  The columns of V, Delta and the state
// never meet in a product, so a column loses nothing to the size of another; within a column an element keeps its ten
// bits down to 2^-27 of the chunk's bound.  FP32 copies of state and U are kept.
//
// Dense flops per launch: chunks * value_heads * [2 C^2 (3 dk + 2 dv) + 6 C dk dv].

#include "common.hpp"
#include "gdn_chunk.hpp"

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

namespace rib200 {
namespace {

constexpr int kDim = kGdnDim;
constexpr int kChunk = kGdnChunk;
constexpr int kSlice = kGdnSlice;
constexpr long long kWaitLimitCycles = 1LL << 28;

struct ChunkParams {
  GdnChunkScratch scratch;
  float *state;
  unsigned int *status;
  std::uint32_t tokens, chunks, key_heads, value_heads;
  float *out; // [token][value head][128], without the output norm
  // layer calls: output norm and gate, new convolution history
  const void *input; // packed rows
  std::size_t z_column;
  const void *norm_weight;
  void *output; // [token][value head][128]
  float *history; // [channel][3]
  std::uint32_t conv_dim, token_stride;
  int32_t dtype, weight_dtype;
  float epsilon;
};

// Optional timeline probe (compile with -DRIB200_TRACE): clock64() of the first CTA, row = chunk (or item), 16 slots.
#ifdef RIB200_TRACE
__device__ long long g_gdn_trace[256 * 16];
#define RIB200_GDN_STAMP(row, slot)                                                    \
  do {                                                                                 \
    if (blockIdx.x == 0 && blockIdx.y == 0 && (row) < 128) {                           \
      g_gdn_trace[(row) * 16 + (slot)] = clock64();                                    \
    }                                                                                  \
  } while (0)
#else
#define RIB200_GDN_STAMP(row, slot) \
  do {                              \
  } while (0)
#endif

__device__ __forceinline__ float load_any(const void *base, std::size_t index, int32_t dtype) {
  if (dtype == RIB200_DTYPE_F32) {
    return static_cast<const float *>(base)[index];
  }
  if (dtype == RIB200_DTYPE_F16) {
    return __half2float(static_cast<const __half *>(base)[index]);
  }
  return __bfloat162float(static_cast<const __nv_bfloat16 *>(base)[index]);
}
// e^x through the base-2 unit; results below the normal range are flushed to zero, which is what every use here
// (decay factors <= 1 and their products with bounded numbers) wants.
__device__ __forceinline__ float exp_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x * 1.4426950408889634F));
  return y;
}
__device__ __forceinline__ float silu_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(1.0F + exp_fast(-x)));
  return x * r;
}
__device__ __forceinline__ std::uint32_t pack_half(float lo, float hi) {
  const __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const std::uint32_t *>(&v);
}
// x = hi + lo with both parts FP16: hi * hi + hi * lo + lo * hi of two such numbers carries 22 bits of their product
__device__ __forceinline__ void split_half(float x, float y, std::uint32_t &hi, std::uint32_t &lo) {
  hi = pack_half(x, y);
  const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hi));
  lo = pack_half(x - h.x, y - h.y);
}

__device__ __forceinline__ std::uint32_t smem_address(const void *p) {
  return static_cast<std::uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbarrier_init(std::uint32_t bar, std::uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarrier_expect_tx(std::uint32_t bar, std::uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbarrier_arrive(std::uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbarrier_try_wait(std::uint32_t bar, std::uint32_t parity) {
  std::uint32_t done;
  asm volatile("{\n"
               ".reg .pred p;\n"
               "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
               "selp.u32 %0, 1, 0, p;\n"
               "}\n"
               : "=r"(done)
               : "r"(bar), "r"(parity)
               : "memory");
  return done != 0;
}
// Bounded wait: once a wait of this CTA has run out nobody in it waits any more.
__device__ __forceinline__ void bounded_wait(std::uint32_t bar, std::uint32_t parity, volatile std::uint32_t *abort_flag,
                                             unsigned int *status) {
  if (*abort_flag != 0 || mbarrier_try_wait(bar, parity)) {
    return;
  }
  const long long started = clock64();
  while (!mbarrier_try_wait(bar, parity)) {
    if (*abort_flag != 0) {
      return;
    }
    if (clock64() - started > kWaitLimitCycles) {
      *abort_flag = 1;
      atomicOr(status, static_cast<unsigned int>(RIB200_DEVICE_WAIT_TIMED_OUT));
      return;
    }
  }
}
__device__ __forceinline__ void bulk_copy_g2s(std::uint32_t dst, const void *src, std::uint32_t bytes,
                                              std::uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// bulk copy shared -> global, completion tracked by the issuing thread's bulk groups
__device__ __forceinline__ void bulk_copy_s2g(void *dst, std::uint32_t src, std::uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *src, std::uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ bool elect_one() {
  std::uint32_t chosen;
  asm volatile("{\n"
               ".reg .pred p;\n"
               "elect.sync _|p, 0xFFFFFFFF;\n"
               "selp.u32 %0, 1, 0, p;\n"
               "}\n"
               : "=r"(chosen));
  return chosen != 0;
}
// Shared-memory matrix descriptor (version 1).  K-major operands with the 128-byte swizzle: 8-row groups `sbo` bytes
// apart, `lbo` unused.  MN-major: one row per k index, groups of eight k indices `sbo` apart, blocks of a swizzle
// row's width (64 elements at 128 bytes, 32 at 64 bytes) `lbo` apart along M or N.
enum : std::uint32_t { kSwizzle128 = 2, kSwizzle64 = 4 };
__device__ __forceinline__ std::uint64_t smem_desc(std::uint32_t addr, std::uint32_t lbo, std::uint32_t sbo,
                                                   std::uint32_t swizzle = kSwizzle128) {
  std::uint64_t d = 0;
  d |= static_cast<std::uint64_t>((addr & 0x3FFFFU) >> 4);
  d |= static_cast<std::uint64_t>((lbo >> 4) & 0x3FFFU) << 16;
  d |= static_cast<std::uint64_t>((sbo >> 4) & 0x3FFFU) << 32;
  d |= static_cast<std::uint64_t>(1) << 46; // version
  d |= static_cast<std::uint64_t>(swizzle) << 61;
  return d;
}
__device__ __forceinline__ constexpr std::uint64_t desc_bytes(std::uint32_t bytes) { return bytes >> 4; }
// Instruction descriptor: FP16 x FP16 -> FP32, M 128; bit 15 / 16 mark an MN-major A / B operand.
__host__ __device__ constexpr std::uint32_t idesc_f16(std::uint32_t n, bool a_mn_major, bool b_mn_major) {
  return (1U << 4) | (a_mn_major ? 1U << 15 : 0U) | (b_mn_major ? 1U << 16 : 0U) | ((n >> 3) << 17) |
         (static_cast<std::uint32_t>(128 >> 4) << 24);
}
__device__ __forceinline__ void umma_f16(std::uint32_t d_tmem, std::uint64_t a_desc, std::uint64_t b_desc,
                                         std::uint32_t idesc, std::uint32_t accumulate) {
  asm volatile("{\n"
               ".reg .pred p;\n"
               "setp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
               "}\n" ::"r"(d_tmem),
               "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void umma_commit(std::uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(std::uint32_t taddr, float (&v)[32]) {
  std::uint32_t r[32];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                 "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                 "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                 "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    v[i] = __uint_as_float(r[i]);
  }
}
__device__ __forceinline__ void sts128(std::uint32_t addr, std::uint32_t a, std::uint32_t b, std::uint32_t c,
                                       std::uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ float lds32(std::uint32_t addr) {
  float value;
  asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(value) : "r"(addr));
  return value;
}
__device__ __forceinline__ float4 lds128(std::uint32_t addr) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

// ---- warp-level tiles of the inversion --------------------------------------------------------------------
__device__ __forceinline__ void ldmatrix_x4(std::uint32_t addr, std::uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(std::uint32_t addr, std::uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void stmatrix_x4_trans(std::uint32_t addr, const std::uint32_t (&r)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};\n" ::"r"(addr), "r"(r[0]),
               "r"(r[1]), "r"(r[2]), "r"(r[3])
               : "memory");
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const std::uint32_t (&a)[4], std::uint32_t b0, std::uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
               "{%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- prepare: per (chunk, value head), persistent CTAs, two per SM ----------------------------------------
// 256 threads.  Per item:
//   inputs   the [K; Q] image of the (chunk, key head), the V image and the gates, by bulk copies
//   G        = [K; Q] K^T            M 128, N 64, K 128   -> rows 0..63 K K^T, rows 64..127 Q K^T
//   rows 0..63: A = beta_i decay_ij (K K^T)_ij below the diagonal -> shared memory;  rows 64..127: P -> record
//            (a warp reads 32 rows x 32 columns of tensor memory; decay_ij = exp(G_i - G_j) is one exponential per
//            element in the two squares on the diagonal, in the one below it the product of a row and a column factor
//            taken against the running sum at the end of the block of 16 columns, both <= 1)
//   T        = (I + A)^-1: the four diagonal 16 x 16 blocks by back substitution in FP32 (a row per thread), then the
//            blocks below them by doubling, -M22^-1 M21 M11^-1, on warp-level tensor tiles with operands split in two
//            FP16 parts; A and T are held times 2^14 u there, so that the parts of an element carry 22 bits down to
//            2^-17 and an absolute 2^-39 below.  The tiles work on the transposed products, (T11^T A21^T) T22^T: the
//            first product's accumulators are then the second one's A operand, so no intermediate leaves the registers.
//   [W; *]   = [T diag(beta gamma); T diag(beta)] K      M 128, N 128, K 64   (rows 0..63 are W)
//   [*; U]   = [T diag(beta gamma); T diag(beta)] V      M 128, N 128, K 64   (rows 64..127 are U)
//   W (FP16) and U (FP32) leave through bulk copies from shared memory that is idle by then (the T image, V, A and T):
//            straight from the registers every store of a warp would touch 32 lines.
// A CTA's items are neighbours, so that the second value head of a key head finds the [K; Q] image in place (32 of an item's
// 50 KB of inputs), and no input waits for all of the item before to leave: the gates come during its inversion, the next
// image behind its two products, only V behind the stores.
// Each phase ends in a barrier and most of them occupy few warps, so a CTA alone leaves the SM mostly idle; two share it.
constexpr int kPrepThreads = 256;
constexpr std::uint32_t kAPitch = 112;                         // A: rows 16..63, columns 0..47 (what the tiles read)
constexpr std::uint32_t kALow = 48 * kAPitch;                  // low parts behind the high parts
constexpr std::uint32_t kTPitch = 80;                          // T: 64 rows, the 32 columns of the row's diagonal square
constexpr std::uint32_t kTLow = kChunk * kTPitch;
constexpr std::uint32_t kDiagPitch = 20;                       // floats per column of a diagonal block of A
constexpr std::uint32_t kDiagBlock = 16 * kDiagPitch + 16;     // floats per block: the two a warp reads miss each other's banks
constexpr std::uint32_t kPsKq = 0;
constexpr std::uint32_t kPsV = kPsKq + kGdnKqBytes;            //   later: slices 0 and 1 of U
// [T diag(beta gamma); T diag(beta)], 128 rows of 128 bytes; later: W
constexpr std::uint32_t kPsTstack = kPsV + kGdnVBytes;
constexpr std::uint32_t kPsPstage = kPsTstack + 128 * kGdnRowBytes;
constexpr std::uint32_t kPsA = kPsPstage + kGdnBlock;          //   later: slices 2 and 3 of U, over A and T
constexpr std::uint32_t kPsT = kPsA + 2 * kALow;
constexpr std::uint32_t kPsDiag = kPsT + 2 * kTLow;
constexpr std::uint32_t kPsGates = kPsDiag + 4 * kDiagBlock * 4;
// G log2(e), beta gamma and beta (both over the unit of K), column factors: 4 x 64 floats; what undoes U's scales: 128
constexpr std::uint32_t kPsFactors = kPsGates + kGdnGateBytes;
constexpr std::uint32_t kPsBars = kPsFactors + (4 * kChunk + kDim) * 4;
constexpr std::uint32_t kPsTmemSlot = kPsBars + 48;
constexpr std::uint32_t kPsAbort = kPsTmemSlot + 4;
constexpr std::uint32_t kPrepSmemBytes = kPsAbort + 4 + 1024;  // + room to align the base to 1 KiB
static_assert(kPsGates % 16 == 0 && kPsFactors % 16 == 0 && kPsBars % 8 == 0 && kPsA % 1024 == 0 && kPsT % 16 == 0 &&
                  kPsDiag - kPsA >= 2 * kGdnSliceU && kGdnVBytes == 2 * kGdnSliceU && 2 * kGdnBlock == 128 * kGdnRowBytes,
              "alignment, staging fits");
static_assert(2 * (kPrepSmemBytes + 1024) <= 233472, "two CTAs per SM");
constexpr std::uint32_t kPrepTmemColumns = 256; // W at 0, U at 128; G at 0 before them

// exponent field of u, the power of two that takes a chunk's growth into [1, 2)
__device__ __forceinline__ std::uint32_t growth_unit(float growth) { return 254U - (__float_as_uint(growth) >> 23); }
__device__ __forceinline__ std::uint32_t tstack_offset(std::uint32_t row, std::uint32_t col) {
  return row * kGdnRowBytes + (((col >> 3) ^ (row & 7U)) << 4) + ((col & 7U) << 1);
}
// 2^x, results below the normal range flushed to zero
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}

// acc[nt] += A B over one k block of 16: A as split fragments, B from a row-major matrix whose row index is N; `at` is
// the address of (first row, first column), the low parts lie `low` bytes behind the high parts.
template <int NT>
__device__ __forceinline__ void tile_step(float (&acc)[NT][4], const std::uint32_t (&a_hi)[4],
                                          const std::uint32_t (&a_lo)[4], std::uint32_t at, std::uint32_t pitch,
                                          std::uint32_t low) {
  const std::uint32_t lane = threadIdx.x & 31;
  at += (((lane >> 4) << 3) + (lane & 7U)) * pitch + ((lane >> 3) & 1U) * 16;
#pragma unroll
  for (int pair = 0; pair < NT / 2; ++pair) {
    std::uint32_t hi[4];
    std::uint32_t lo[4];
    ldmatrix_x4(at + pair * 16 * pitch, hi);
    ldmatrix_x4(at + pair * 16 * pitch + low, lo);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      mma_f16(acc[2 * pair + h], a_lo, hi[2 * h], hi[2 * h + 1]);
      mma_f16(acc[2 * pair + h], a_hi, lo[2 * h], lo[2 * h + 1]);
      mma_f16(acc[2 * pair + h], a_hi, hi[2 * h], hi[2 * h + 1]);
    }
  }
}
// A operand fragments of the transpose of the 16 x 16 block of T at `at`
__device__ __forceinline__ void transposed_fragments(std::uint32_t at, std::uint32_t (&hi)[4], std::uint32_t (&lo)[4]) {
  const std::uint32_t lane = threadIdx.x & 31;
  at += (((lane >> 4) << 3) + (lane & 7U)) * kTPitch + ((lane >> 3) & 1U) * 16;
  ldmatrix_x4_trans(at, hi);
  ldmatrix_x4_trans(at + kTLow, lo);
}
// the accumulators of two neighbouring column tiles, times a factor, and as the A fragments of a k block
__device__ __forceinline__ void rescale(float (&c0)[4], float (&c1)[4], float factor) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    c0[e] *= factor;
    c1[e] *= factor;
  }
}
__device__ __forceinline__ void accumulator_fragments(const float (&c0)[4], const float (&c1)[4], std::uint32_t (&hi)[4],
                                                      std::uint32_t (&lo)[4]) {
  split_half(c0[0], c0[1], hi[0], lo[0]);
  split_half(c0[2], c0[3], hi[1], lo[1]);
  split_half(c1[0], c1[1], hi[2], lo[2]);
  split_half(c1[2], c1[3], hi[3], lo[3]);
}

__global__ void __launch_bounds__(kPrepThreads, 2) gdn_chunk_prepare_kernel(const ChunkParams p) {
  extern __shared__ unsigned char prep_smem_raw[];
  const std::uint32_t base = (smem_address(prep_smem_raw) + 1023U) & ~1023U;
  unsigned char *smem = prep_smem_raw + (base - smem_address(prep_smem_raw));
  const float *gates = reinterpret_cast<const float *>(smem + kPsGates);
  const float *s_beta = gates + kGdnGateBeta;
  float *s_g2 = reinterpret_cast<float *>(smem + kPsFactors); // G log2(e)
  float *s_bg = s_g2 + kChunk;                                // beta exp(G) / kGdnUnit
  float *s_bu = s_bg + kChunk;                                // beta / kGdnUnit
  float *s_cf = s_bu + kChunk;                                // exp(G at the end of the token's block of 16 - G)
  float *s_undo = s_cf + kChunk;                              // by column: undoes the scales of the product that is U
  const std::uint32_t bar_kq = base + kPsBars; // the [K; Q] image has landed ...
  const std::uint32_t bar_gates = bar_kq + 8;  // ... the gates ...
  const std::uint32_t bar_v = bar_kq + 16;     // ... V
  const std::uint32_t bar_g = bar_kq + 24;
  const std::uint32_t bar_wu = bar_kq + 32;
  const std::uint32_t bar_left = bar_kq + 40; // what the item before has staged has been read
  volatile std::uint32_t *tmem_slot = reinterpret_cast<volatile std::uint32_t *>(smem + kPsTmemSlot);
  volatile std::uint32_t *abort_flag = reinterpret_cast<volatile std::uint32_t *>(smem + kPsAbort);
  const std::uint32_t tid = threadIdx.x;
  const std::uint32_t warp = tid >> 5;
  const std::uint32_t lane = tid & 31;
  // Items in the order (chunk, key head, value head of the key head), an equal share of them for every CTA: where two value
  // heads share a key head, the [K; Q] image of every second item is the one in hand.
  const std::uint32_t items = p.chunks * p.value_heads;
  const std::uint32_t ratio = p.value_heads / p.key_heads;
  auto share = [&](std::uint32_t cta) {
    return static_cast<std::uint32_t>(static_cast<std::uint64_t>(items) * cta / gridDim.x);
  };
  const bool one_each = items == gridDim.x; // short calls, in which 64-bit divisions would show
  const std::uint32_t first_item = one_each ? blockIdx.x : share(blockIdx.x);
  const std::uint32_t last_item = one_each ? blockIdx.x + 1 : share(blockIdx.x + 1);
  auto record_index = [&](std::uint32_t item) { // of V and the record: (chunk, value head)
    const std::uint32_t kq = item / ratio;
    const std::uint32_t chunk = kq / p.key_heads;
    return chunk * p.value_heads + (kq - chunk * p.key_heads) + (item - kq * ratio) * p.key_heads;
  };
  std::uint32_t record = record_index(first_item); // of the item in hand; the divisions are over before the wait below
  const std::uint32_t first_kq = first_item / ratio;
  std::uint32_t kq_index = first_kq;
  asm volatile("" : "+r"(record), "+r"(kq_index));

  if (tid == 0) {
    mbarrier_init(bar_kq, 1);
    mbarrier_init(bar_gates, 1);
    mbarrier_init(bar_v, 1);
    mbarrier_init(bar_g, 1);
    mbarrier_init(bar_wu, 1);
    mbarrier_init(bar_left, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + kPsTmemSlot),
                 "r"(kPrepTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const std::uint32_t tmem = *tmem_slot;
  // Launched with programmatic stream serialisation: what is above overlaps the image kernel, whose results are read
  // only after this.
  grid_dependency_wait();
  // Only now may the chain kernel set itself up: what it reads before its own wait, the recurrent state, is final once
  // the kernels in front of this one have ended.
  grid_dependents_may_launch();
  auto wait = [&](std::uint32_t b, std::uint32_t parity) { bounded_wait(b, parity, abort_flag, p.status); };

  if (p.history != nullptr) {
    // the convolution history [channel][3] of the next call: the last three rows (a chunked call has 64 at least)
    for (std::uint32_t channel = blockIdx.x * kPrepThreads + tid; channel < p.conv_dim; channel += gridDim.x * kPrepThreads) {
#pragma unroll
      for (std::uint32_t h = 0; h < 3; ++h) {
        p.history[static_cast<std::size_t>(channel) * 3 + h] =
            load_any(p.input, static_cast<std::size_t>(p.tokens - 3 + h) * p.token_stride + channel, p.dtype);
      }
    }
  }

  // One lane issues every copy (bulk groups belong to the issuing thread).  An input is asked for as soon as the item in hand
  // is done with its area: the gates behind A and P, the image behind the two products, V, whose area U leaves from, last.
  const bool copier = tid == kPrepThreads - 32;
  auto issue_kq = [&](std::uint32_t index) {
    mbarrier_expect_tx(bar_kq, kGdnKqBytes);
    bulk_copy_g2s(base + kPsKq, p.scratch.kq + static_cast<std::size_t>(index) * kGdnKqBytes, kGdnKqBytes, bar_kq);
    if ((index + 1) * ratio < last_item) { // into L2 while this image is worked on
      prefetch_l2(p.scratch.kq + static_cast<std::size_t>(index + 1) * kGdnKqBytes, kGdnKqBytes);
    }
  };
  auto issue_gates = [&](std::uint32_t at) {
    fence_proxy_async(); // those of the item before have been read by ordinary loads
    mbarrier_expect_tx(bar_gates, kGdnGateBytes);
    bulk_copy_g2s(base + kPsGates, p.scratch.records + static_cast<std::size_t>(at) * kGdnRecBytes + kGdnRecGates,
                  kGdnGateBytes, bar_gates);
  };
  auto issue_v = [&](std::uint32_t at) {
    fence_proxy_async(); // U has been staged here by ordinary stores
    mbarrier_expect_tx(bar_v, kGdnVBytes);
    bulk_copy_g2s(base + kPsV, p.scratch.v + static_cast<std::size_t>(at) * kGdnVBytes, kGdnVBytes, bar_v);
  };
  if (copier && first_item < last_item) {
    issue_kq(kq_index);
    issue_gates(record);
    issue_v(record);
    if (first_item + 1 < last_item) {
      prefetch_l2(p.scratch.v + static_cast<std::size_t>(record_index(first_item + 1)) * kGdnVBytes, kGdnVBytes);
    }
  }

  const std::uint32_t quarter = warp & 3; // the 32 tensor-memory lanes this warp may read
  const std::uint32_t half = warp >> 2;
  const std::uint32_t lane_base = (quarter * 32U) << 16;
  const std::uint32_t i = (quarter & 1U) * 32 + lane; // token of the lane's row
  const std::uint32_t a_matrix = base + kPsA - 16 * kAPitch; // address of row 0 (rows below 16 do not exist)
  const std::uint32_t t_matrix = base + kPsT;
  auto t_at = [&](std::uint32_t row, std::uint32_t col) { return t_matrix + row * kTPitch + (col & 31U) * 2; };
  std::uint32_t iteration = 0;
  for (std::uint32_t item = first_item; item < last_item; ++item, ++iteration) {
    const std::uint32_t phase = iteration & 1U;
    unsigned char *rec = p.scratch.records + static_cast<std::size_t>(record) * kGdnRecBytes;
    const bool next_kq = item + 1 < last_item && item + 1 == (kq_index + 1) * ratio; // the next item has another image
    const std::uint32_t next_record = item + 1 < last_item ? record_index(item + 1) : 0U;
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 0);
    }
    if (warp == 0) {
      wait(bar_kq, (kq_index - first_kq) & 1U);
      tcgen05_fence_after();
      if (elect_one() && *abort_flag == 0) {
        const std::uint64_t kq = smem_desc(base + kPsKq, 16, 1024);
#pragma unroll
        for (std::uint32_t ks = 0; ks < 8; ++ks) {
          const std::uint64_t at = desc_bytes((ks >> 2) * kGdnKqBlock + (ks & 3U) * 32U);
          umma_f16(tmem, kq + at, kq + at, idesc_f16(kChunk, false, false), ks);
        }
        umma_commit(bar_g);
      }
      __syncwarp();
    }
    wait(bar_gates, phase);
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 1);
    }
    if (warp == 2 || warp == 3) {
      const std::uint32_t t = tid - 64;
      const float g = gates[kGdnGateG + t];
      s_g2[t] = g * 1.4426950408889634F;
      s_bg[t] = s_beta[t] * exp_fast(g) * (1.0F / kGdnUnit);
      s_bu[t] = s_beta[t] * (1.0F / kGdnUnit);
      s_cf[t] = exp_fast(gates[kGdnGateG + (t | 15U)] - g);
      const float undo_t = gdn_power(254 - growth_unit(gates[kGdnGateGrowth])) * (1.0F / kGdnUnit);
      s_undo[t] = gdn_power(254 - gdn_scale_exponent(gates[kGdnGateMax + t])) * undo_t;
      s_undo[t + kChunk] = gdn_power(254 - gdn_scale_exponent(gates[kGdnGateMax + kChunk + t])) * undo_t;
    }
    const std::uint32_t unit = growth_unit(gates[kGdnGateGrowth]); // u; A and T are held times 2^14 u, as G comes times 2^14
    const float hold = gdn_power(unit + 14);
    const float release = gdn_power(254 - 14 - unit);
    if (tid == 0 && gates[kGdnGateGrowth] > kGdnMostGrowth) {
      atomicOr(p.status, static_cast<unsigned int>(RIB200_DEVICE_DECAY_OUT_OF_RANGE));
    }
    __syncthreads();

    // ---- rows of G: A (below the diagonal, to shared memory) and P (to its staging area) ----
    if (iteration > 0) { // until then the staging areas hold P, W and U of the item before
      wait(bar_left, phase ^ 1U);
    }
    wait(bar_g, phase);
    tcgen05_fence_after();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 2);
    }
    {
      const bool is_p = quarter >= 2; // rows 64..127 hold Q K^T
      const std::uint32_t row_half = quarter & 1U;
      float x[32];
      if (half <= row_half) {
        tmem_ld32(tmem + lane_base + 32 * half, x);
        const float g2_i = s_g2[i];
        const float scale_i = is_p ? gdn_power(unit + kGdnUnitP - 14) : s_beta[i] * gdn_power(unit);
        if (half < row_half) {
#pragma unroll
          for (std::uint32_t part = 0; part < 2; ++part) {
            const float row_factor = scale_i * exp2_fast(g2_i - s_g2[16 * part + 15]);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 f = *reinterpret_cast<const float4 *>(s_cf + 16 * part + 4 * c);
              x[16 * part + 4 * c] *= row_factor * f.x;
              x[16 * part + 4 * c + 1] *= row_factor * f.y;
              x[16 * part + 4 * c + 2] *= row_factor * f.z;
              x[16 * part + 4 * c + 3] *= row_factor * f.w;
            }
          }
        } else {
          const std::uint32_t last = is_p ? lane : lane - 1U; // columns of the square up to and with this one count
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 g = *reinterpret_cast<const float4 *>(s_g2 + 32 * half + 4 * c);
            const float gj[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = 4 * c + e;
              const float decayed = x[j] * (scale_i * exp2_fast(g2_i - gj[e]));
              x[j] = static_cast<int>(last) >= j ? decayed : 0.0F;
            }
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          x[e] = 0.0F;
        }
      }
      if (is_p) {
#pragma unroll
        for (std::uint32_t c = 0; c < 4; ++c) {
          sts128(base + kPsPstage + i * kGdnRowBytes + (((4 * half + c) ^ (i & 7U)) << 4), pack_half(x[8 * c], x[8 * c + 1]),
                 pack_half(x[8 * c + 2], x[8 * c + 3]), pack_half(x[8 * c + 4], x[8 * c + 5]),
                 pack_half(x[8 * c + 6], x[8 * c + 7]));
        }
        fence_proxy_async();
      } else if (half <= row_half) {
        if (half == row_half) { // the row's part of its diagonal block, by columns
          float *diag = reinterpret_cast<float *>(smem + kPsDiag) + (i >> 4) * kDiagBlock + (i & 15U);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            diag[e * kDiagPitch] = (lane < 16 ? x[e] : x[16 + e]) * release;
          }
        }
#pragma unroll
        for (std::uint32_t part = 0; part < 2; ++part) {
          if (half < row_half || (part == 0 && lane >= 16)) {
            const std::uint32_t at = a_matrix + i * kAPitch + (32 * half + 16 * part) * 2;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              std::uint32_t hi[4];
              std::uint32_t lo[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                split_half(x[16 * part + 8 * c + 2 * e], x[16 * part + 8 * c + 2 * e + 1], hi[e], lo[e]);
              }
              sts128(at + 16 * c, hi[0], hi[1], hi[2], hi[3]);
              sts128(at + 16 * c + kALow, lo[0], lo[1], lo[2], lo[3]);
            }
          }
        }
      }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 3);
    }
    if (copier && *abort_flag == 0) {
      bulk_copy_s2g(rec + kGdnRecP, base + kPsPstage, kGdnBlock);
      asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      if (item + 1 < last_item) {
        issue_gates(next_record);
      }
    }

    // ---- T = (I + A)^-1: diagonal blocks, a row per thread: x_c = [c = row] - sum over k > c of x_k A_kc ----
    if (tid < kChunk) {
      const std::uint32_t b = tid >> 4;
      const std::uint32_t r = tid & 15U;
      const float *diag = reinterpret_cast<const float *>(smem + kPsDiag) + b * kDiagBlock;
      float t[16];
#pragma unroll
      for (int c = 15; c >= 0; --c) {
        float a[16];
#pragma unroll
        for (int q = (c + 1) / 4; q < 4; ++q) {
          const float4 v = *reinterpret_cast<const float4 *>(diag + c * kDiagPitch + 4 * q);
          a[4 * q] = v.x;
          a[4 * q + 1] = v.y;
          a[4 * q + 2] = v.z;
          a[4 * q + 3] = v.w;
        }
        float even = c == static_cast<int>(r) ? 1.0F : 0.0F;
        float odd = 0.0F;
#pragma unroll
        for (int k = 15; k > c; --k) {
          if (k % 2 == 0) {
            even -= a[k] * t[k];
          } else {
            odd -= a[k] * t[k];
          }
        }
        t[c] = even + odd;
      }
#pragma unroll
      for (std::uint32_t c = 0; c < 2; ++c) {
        std::uint32_t hi[4];
        std::uint32_t lo[4];
        std::uint32_t with_gamma[4];
        std::uint32_t without[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const std::uint32_t k = 8 * c + 2 * e;
          const float t0 = t[k] * hold;
          const float t1 = t[k + 1] * hold;
          split_half(t0, t1, hi[e], lo[e]);
          const float2 bg = *reinterpret_cast<const float2 *>(s_bg + 16 * b + k);
          const float2 bu = *reinterpret_cast<const float2 *>(s_bu + 16 * b + k);
          with_gamma[e] = pack_half(t0 * bg.x, t1 * bg.y);
          without[e] = pack_half(t0 * bu.x, t1 * bu.y);
        }
        sts128(t_at(tid, 16 * b + 8 * c), hi[0], hi[1], hi[2], hi[3]);
        sts128(t_at(tid, 16 * b + 8 * c) + kTLow, lo[0], lo[1], lo[2], lo[3]);
        sts128(base + kPsTstack + tstack_offset(tid, 16 * b + 8 * c), with_gamma[0], with_gamma[1], with_gamma[2],
               with_gamma[3]);
        sts128(base + kPsTstack + tstack_offset(kChunk + tid, 16 * b + 8 * c), without[0], without[1], without[2], without[3]);
      }
    } else { // the other warps: zeros above the diagonal blocks of the T image, where W of the item before was
      const std::uint32_t at = tid - kChunk; // of 16 rows each of 6, 4 and 2 pieces of eight columns
      const std::uint32_t b = at < 96 ? 0U : (at < 160 ? 1U : 2U);
      const std::uint32_t within = at - (b == 0 ? 0U : (b == 1 ? 96U : 160U));
      const std::uint32_t pieces = 6 - 2 * b;
      const std::uint32_t row = 16 * b + within / pieces;
      const std::uint32_t col = 8 * (2 * (b + 1) + within % pieces);
      sts128(base + kPsTstack + tstack_offset(row, col), 0U, 0U, 0U, 0U);
      sts128(base + kPsTstack + tstack_offset(kChunk + row, col), 0U, 0U, 0U, 0U);
    }
    __syncthreads();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 4);
    }
    // Two accumulator tiles (rows = columns m0 .. m0 + 15 of T, columns = rows r0 .. r0 + 15 of T) go, negated, into the
    // T image, scaled per column of T.
    auto store_scaled = [&](const float (&z0)[4], const float (&z1)[4], std::uint32_t r0, std::uint32_t m0) {
      const std::uint32_t lo_col = m0 + (lane >> 2);
      const std::uint32_t row = r0 + ((lane >> 4) << 3) + (lane & 7U);
      const std::uint32_t col = m0 + ((lane >> 3) & 1U) * 8;
      const float bg0 = -s_bg[lo_col];
      const float bg1 = -s_bg[lo_col + 8];
      const float be0 = -s_bu[lo_col];
      const float be1 = -s_bu[lo_col + 8];
      const std::uint32_t with_gamma[4] = {pack_half(z0[0] * bg0, z0[1] * bg0), pack_half(z0[2] * bg1, z0[3] * bg1),
                                           pack_half(z1[0] * bg0, z1[1] * bg0), pack_half(z1[2] * bg1, z1[3] * bg1)};
      const std::uint32_t without[4] = {pack_half(z0[0] * be0, z0[1] * be0), pack_half(z0[2] * be1, z0[3] * be1),
                                        pack_half(z1[0] * be0, z1[1] * be0), pack_half(z1[2] * be1, z1[3] * be1)};
      stmatrix_x4_trans(base + kPsTstack + tstack_offset(row, col), with_gamma);
      stmatrix_x4_trans(base + kPsTstack + tstack_offset(kChunk + row, col), without);
    };
    // ---- ... the 16 x 16 blocks beside them, T_10 = -T_11 (A_10 T_00) and T_32, a warp each ----
    if (warp < 2) {
      const std::uint32_t m0 = 32 * warp;
      const std::uint32_t r0 = m0 + 16;
      std::uint32_t hi[4];
      std::uint32_t lo[4];
      float y[2][4] = {};
      transposed_fragments(t_at(m0, m0), hi, lo);
      tile_step<2>(y, hi, lo, a_matrix + r0 * kAPitch + m0 * 2, kAPitch, kALow);
      rescale(y[0], y[1], release);
      accumulator_fragments(y[0], y[1], hi, lo);
      float z[2][4] = {};
      tile_step<2>(z, hi, lo, t_at(r0, r0), kTPitch, kTLow);
      rescale(z[0], z[1], release);
      store_scaled(z[0], z[1], r0, m0);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          z[t][e] = -z[t][e];
        }
      }
      accumulator_fragments(z[0], z[1], hi, lo);
      const std::uint32_t at = t_at(r0 + ((lane >> 4) << 3) + (lane & 7U), m0 + ((lane >> 3) & 1U) * 8);
      stmatrix_x4_trans(at, hi);
      stmatrix_x4_trans(at + kTLow, lo);
    }
    __syncthreads();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 5);
    }
    // ---- ... and the lower left 32 x 32 block: warp (m tile, row block); triangular factors are only walked over
    // their non-zero blocks ----
    if (warp < 4) {
      const std::uint32_t m0 = 16 * (warp & 1U);
      std::uint32_t hi[4];
      std::uint32_t lo[4];
      float y[4][4] = {};
      if (m0 == 0) {
        transposed_fragments(t_at(0, 0), hi, lo);
        tile_step<4>(y, hi, lo, a_matrix + 32 * kAPitch, kAPitch, kALow);
      }
      transposed_fragments(t_at(16, m0), hi, lo);
      tile_step<4>(y, hi, lo, a_matrix + 32 * kAPitch + 32, kAPitch, kALow);
      float z[2][4] = {};
      rescale(y[0], y[1], release);
      accumulator_fragments(y[0], y[1], hi, lo);
      if (warp < 2) { // rows 32..47
        tile_step<2>(z, hi, lo, t_at(32, 32), kTPitch, kTLow);
        rescale(z[0], z[1], release);
        store_scaled(z[0], z[1], 32, m0);
      } else { // rows 48..63
        tile_step<2>(z, hi, lo, t_at(48, 32), kTPitch, kTLow);
        rescale(y[2], y[3], release);
        accumulator_fragments(y[2], y[3], hi, lo);
        tile_step<2>(z, hi, lo, t_at(48, 48), kTPitch, kTLow);
        rescale(z[0], z[1], release);
        store_scaled(z[0], z[1], 48, m0);
      }
    }
    fence_proxy_async(); // the T image is read through the async proxy
    tcgen05_fence_before();
    __syncthreads();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 6);
    }

    // ---- the two products with T: B operands are K and V as stored, sixteen tokens = 2 KiB per step ----
    if (warp == 0) {
      wait(bar_v, phase);
      tcgen05_fence_after();
      if (elect_one() && *abort_flag == 0) {
        const std::uint64_t t_desc = smem_desc(base + kPsTstack, 16, 1024);
        const std::uint64_t k_desc = smem_desc(base + kPsKq, kGdnKqBlock, 1024);
        const std::uint64_t v_desc = smem_desc(base + kPsV, kGdnBlock, 1024);
#pragma unroll
        for (std::uint32_t ks = 0; ks < 4; ++ks) {
          umma_f16(tmem, t_desc + desc_bytes(ks * 32U), k_desc + desc_bytes(ks * 2048U), idesc_f16(kDim, false, true), ks);
        }
#pragma unroll
        for (std::uint32_t ks = 0; ks < 4; ++ks) {
          umma_f16(tmem + 128, t_desc + desc_bytes(ks * 32U), v_desc + desc_bytes(ks * 2048U), idesc_f16(kDim, false, true),
                   ks);
        }
        umma_commit(bar_wu);
      }
      __syncwarp();
    }
    wait(bar_wu, phase);
    tcgen05_fence_after();
    if (copier && next_kq && *abort_flag == 0) {
      issue_kq(kq_index + 1);
    }
    __syncwarp();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 7);
    }

    // ---- W (rows 0..63 of the first) and U (rows 64..127 of the second), 64 columns per warp, to their staging areas --
    if (quarter < 2) {
#pragma unroll
      for (std::uint32_t part = 0; part < 2; ++part) {
        float x[32];
        tmem_ld32(tmem + lane_base + 64 * half + 32 * part, x);
#pragma unroll
        for (std::uint32_t c = 0; c < 4; ++c) {
          sts128(base + kPsTstack + half * kGdnBlock + i * kGdnRowBytes + (((4 * part + c) ^ (i & 7U)) << 4),
                 pack_half(x[8 * c], x[8 * c + 1]), pack_half(x[8 * c + 2], x[8 * c + 3]),
                 pack_half(x[8 * c + 4], x[8 * c + 5]), pack_half(x[8 * c + 6], x[8 * c + 7]));
        }
      }
    } else {
      const std::uint32_t stage = base + (half == 0 ? kPsV : kPsA);
      const std::uint32_t undo_at = smem_address(s_undo);
#pragma unroll
      for (std::uint32_t part = 0; part < 2; ++part) {
        float4 undo[8]; // all of them first: a load behind a store of this loop would wait for it
#pragma unroll
        for (std::uint32_t c = 0; c < 8; ++c) {
          undo[c] = lds128(undo_at + (64 * half + 32 * part + 4 * c) * 4);
        }
        float x[32];
        tmem_ld32(tmem + lane_base + 128 + 64 * half + 32 * part, x);
#pragma unroll
        for (std::uint32_t c = 0; c < 8; ++c) {
          sts128(stage + part * kGdnSliceU + i * kGdnRowBytes + ((c ^ (i & 7U)) << 4),
                 __float_as_uint(x[4 * c] * undo[c].x), __float_as_uint(x[4 * c + 1] * undo[c].y),
                 __float_as_uint(x[4 * c + 2] * undo[c].z), __float_as_uint(x[4 * c + 3] * undo[c].w));
        }
      }
    }
    fence_proxy_async();
    tcgen05_fence_before();
    __syncthreads();
    if (tid == 0) {
      RIB200_GDN_STAMP(100 + iteration, 8);
    }
    if (copier && *abort_flag == 0) {
      bulk_copy_s2g(rec + kGdnRecW, base + kPsTstack, 2 * kGdnBlock);
      bulk_copy_s2g(rec + kGdnRecU, base + kPsV, 2 * kGdnSliceU);
      bulk_copy_s2g(rec + kGdnRecU + 2 * kGdnSliceU, base + kPsA, 2 * kGdnSliceU);
      asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
      mbarrier_arrive(bar_left);
      if (item + 1 < last_item) {
        issue_v(next_record);
        if (item + 2 < last_item) {
          prefetch_l2(p.scratch.v + static_cast<std::size_t>(record_index(item + 2)) * kGdnVBytes, kGdnVBytes);
        }
      }
    }
    __syncwarp();
    record = next_record;
    kq_index += next_kq ? 1U : 0U;
  }
  if (copier) {
    asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    if (*abort_flag != 0) { // inputs may be on their way for an item that nobody waits for
      for (const long long started = clock64(); clock64() - started < (1LL << 17);) {
      }
    }
  }
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 0) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kPrepTmemColumns) : "memory");
  }
}

// ---- chain: per (state slice, value head), chunks in order -------------------------------------------------
// 352 threads.  Warps 0-3 own the 128 lanes of tensor memory and the state (thread = row of every product), warps 4-5
// make the outputs of the even chunks and warps 8-9 those of the odd ones (a chunk's outputs cost a pair of warps about
// 3000 cycles, the chain itself 2100 a chunk: with one pair every first product waited for the outputs two chunks back;
// 4096 tokens 224.2 -> 197.4 us, a chunk 3100 -> 2500 cycles), warp 6 issues the products, lane 0 of warp 7 streams the operand images of each chunk into a
// three-stage ring, asking for them in L2 some chunks earlier (the records of a long call do not all stay there).  Per chunk:
//   X  = [Q; W] S0            M 128 (rows 0..63 Q S0, rows 64..127 W S0), N 32, K 128
//   warps 2-3: Delta = U - X[64..] -> diag(e) Delta and Delta as B operands
//   SD = K^T (diag(e) Delta)  M 128, N 32, K 64 (K as stored: MN-major A operand)
//   O2 = P Delta              M 128 (rows 64..127 are don't-care), N 32, K 64
//   warps 0-3: S = gamma_C S + SD (FP32 registers) -> B operand: the next chunk's first product waits for this
//   warps 4-5, 8-9: O = gamma_i (Q S0)_i + O2; in a layer call the four slices of a head are a cluster, exchange the sums of
//   squares of every token and write norm(O) * weight * SiLU(z)
// The chain X -> Delta -> SD -> S is latency: nothing but that chain runs in warps 0-3, everything they need from memory
// is in registers before they wait, and a row of a B operand (32 columns, 64 bytes) is four 16-byte stores because the
// operand is MN-major (64-byte swizzle).
// Scales, per column: with M the largest |S0| of the column, no |S| after the chunk exceeds
//   b_S = 11.5 exp(G_C) M + growth sum(beta) max|v|
// (the column of S0 has norm <= sqrt(128) M, a token adds at most beta |v|; 11.5 and not 11.32 because M is cut to BF16), and
// no |Delta| exceeds b_D = max(beta) (max|v| + growth (11.5 M + sum(beta) max|v|)).  Delta is scaled by the power of two
// that brings b_D to [2^13, 2^14).  The new state is scaled by 2 whenever 2^-4 <= b_S < 2^14 and like Delta, from b_S,
// elsewhere: its image is written before its own maximum is known, and a factor that is the same for all ordinary magnitudes
// keeps a prompt fed in pieces of whole chunks bit-identical to the same prompt in one call (a bound that follows every
// chunk rounds the few elements below FP16's normal range differently on either side of a cut).  Inside that window the
// image of the state is exact to 2^-26.
// Columns whose bounds lie within 2^10 of each other, as they nearly always do, share the factor of the largest, and
// everybody works with one number; else every column has its own, which costs up to 700 cycles a chunk (4096 tokens 216 us
// and not 194 if all chunks do so).  One factor per (chunk, slice) at all times left a column that is 1e-6 of the slice's
// largest with errors of 2e-3.  All of the scales together, columns of V, units and growth included, cost 3 to 5 % of a
// layer call (replayed calls of 64 tokens 16.8 -> 17.4 us, 512 tokens 30.9 -> 32.5, 4096 tokens 185.5 -> 193.8).
// Warp 10 makes the factors while the first product of the chunk runs, from column maxima that warps 0-3 leave as soon as
// the state is on its way; the gates it needs it reads from memory two chunks ahead.
// Every mbarrier wait is bounded; when one runs out the CTA records RIB200_DEVICE_WAIT_TIMED_OUT, stops waiting and
// copying, and runs to its end.
constexpr int kChainThreads = 352;
constexpr std::uint32_t kStages = 3;
constexpr std::uint32_t kPrefetchAhead = 3; // chunks between the L2 prefetch and the copy that uses it
constexpr std::uint32_t kStageQw = 0;                              // [2 blocks][rows 0..63 Q, 64..127 W][128 bytes]
constexpr std::uint32_t kStageK = kStageQw + 2 * kGdnKqBlock;      // [2 blocks][64 rows][128 bytes]
constexpr std::uint32_t kStageP = kStageK + 2 * kGdnBlock;         // 64 rows; the product's rows 64.. read on into U
constexpr std::uint32_t kStageU = kStageP + kGdnBlock;
constexpr std::uint32_t kStageGates = kStageU + kGdnSliceU;
constexpr std::uint32_t kStageBytes = (kStageGates + kChunk * 4 + 1023) / 1024 * 1024; // of the gates, G
constexpr std::uint32_t kOperandRow = kSlice * 2;                  // bytes of a B operand row
constexpr std::uint32_t kCsState = kStages * kStageBytes;               // S, 128 rows
constexpr std::uint32_t kCsEDelta = kCsState + kDim * kOperandRow; // diag(e) Delta, 64 rows
constexpr std::uint32_t kCsDelta = kCsEDelta + kChunk * kOperandRow;
// [chunk & 3][4 slices][64 tokens]: a peer sends the sums of chunk c + 4 only after this CTA's sums of c + 2, which
// leave after its threads have read those of c (even and odd chunks have warps of their own, two slots would not do)
constexpr std::uint32_t kCsNorm = kCsDelta + kChunk * kOperandRow;
constexpr std::uint32_t kNormSlots = 4;
constexpr std::uint32_t kCsWeight = kCsNorm + kNormSlots * kGdnSlices * kChunk * 4;
constexpr std::uint32_t kCsMax = kCsWeight + kSlice * 4;           // [4 warps][columns] largest |S0|
// [chunk & 3][factors below][columns].  Warp 10 makes those of a chunk at its head; by then the outputs of the chunk that
// had the slot before, which may lag, have read theirs: the first product of the chunk before this one waited for them.
constexpr std::uint32_t kCsScale = kCsMax + 4 * kSlice * 4;
enum : std::uint32_t {
  kScaleX = 0,                      // takes X to the scale of Delta
  kScaleDelta = 1 * kSlice * 4,     // scale of Delta
  kScaleSd = 2 * kSlice * 4,        // undoes the scale of SD
  kScaleOutX = 3 * kSlice * 4,      // undoes that of Q S0
  kScaleOutDelta = 4 * kSlice * 4,  // undoes that of P Delta
  kScaleState = 5 * kSlice * 4,     // scale of the new S
  kScaleEqual = 6 * kSlice * 4,     // not 0: the columns have the same factors
  kScaleBytes = 6 * kSlice * 4 + 16
};
constexpr std::uint32_t kScaleSlots = 4;
constexpr std::uint32_t kCsBars = kCsScale + kScaleSlots * kScaleBytes;
enum : std::uint32_t {
  kBarQwFull = 0,                      // [stages] bytes of Q and W
  kBarRestFull = kBarQwFull + kStages, // [stages] bytes of K, P, U and the gates
  kBarRead = kBarRestFull + kStages,   // [stages] the threads that read U and the gates have done so
  kBarUsed = kBarRead + kStages,       // [stages] the products that read the stage have completed
  kBarXDone = kBarUsed + kStages,      // [2] by parity of the chunk, as the outputs may lag the chain by more than a chunk
  kBarO2Done = kBarXDone + 2,          // [2]
  kBarOutRead = kBarO2Done + 2,        // [2] X (rows 0..63), O2 and the scales of a chunk have been read (64 threads)
  kBarNorm = kBarOutRead + 2,          // [chunk & 3] the four slices' sums of squares
  kBarEDelta = kBarNorm + kNormSlots,          // diag(e) Delta is in shared memory (64 writers)
  kBarDelta,                           // Delta is in shared memory (64 writers)
  kBarSdDone,
  kBarState,                           // S is in shared memory, X and SD have been read (128 threads)
  kBarCount
};
// a role's place in the ring
struct RingPlace {
  std::uint32_t stage = 0;
  std::uint32_t phase = 0; // parity of the barrier phase that belongs to this visit of the stage
  __device__ __forceinline__ void next() {
    if (++stage == kStages) {
      stage = 0;
      phase ^= 1U;
    }
  }
};
constexpr std::uint32_t kCsTmemSlot = kCsBars + kBarCount * 8;
constexpr std::uint32_t kCsAbort = kCsTmemSlot + 4;
constexpr std::uint32_t kChainSmemBytes = kCsAbort + 4 + 1024;
static_assert(kStageBytes % 1024 == 0 && kStageP % 1024 == 0 && kCsState % 1024 == 0 && kCsEDelta % 512 == 0 &&
                  kCsDelta % 512 == 0 && kCsBars % 8 == 0 && kCsWeight % 16 == 0,
              "operand images sit on the boundaries of their swizzle atoms");
static_assert(kStageP + 2 * kGdnBlock <= kStageBytes, "the don't-care rows of P lie inside the stage");
static_assert(kCsScale % 16 == 0 && kChainSmemBytes <= 232448, "aligned, fits an SM");
constexpr std::uint32_t kChainTmemColumns = 256; // X at 0 and 32, O2 at 64 and 96 (by parity), SD at 128

// byte offset of the 16-byte piece `piece` of row `row` of a B operand (64-byte rows, 64-byte swizzle)
__device__ __forceinline__ std::uint32_t operand_piece(std::uint32_t row, std::uint32_t piece) {
  return row * kOperandRow + ((piece ^ ((row >> 1) & 3U)) << 4);
}
__device__ __forceinline__ void store_operand_row(std::uint32_t operand, std::uint32_t row, const std::uint32_t (&h)[16]) {
#pragma unroll
  for (std::uint32_t c = 0; c < 4; ++c) {
    sts128(operand + operand_piece(row, c), h[4 * c], h[4 * c + 1], h[4 * c + 2], h[4 * c + 3]);
  }
}
// exponent field of the scale of a state bounded by `bound`
__device__ __forceinline__ std::uint32_t state_exponent_of(float bound) {
  return bound >= 0.0625F && bound < 16384.0F ? 128U : gdn_scale_exponent(bound);
}
// Lane = column: the bound to scale by, the largest one where the columns' bounds lie within 2^10 of each other (columns of
// zeros aside), else the column's own.
__device__ __forceinline__ float level(float bound, bool &equal) {
  const std::uint32_t bits = __float_as_uint(bound);
  const float high = __uint_as_float(__reduce_max_sync(0xFFFFFFFFU, bits));
  const float low = __uint_as_float(__reduce_min_sync(0xFFFFFFFFU, bits == 0U ? 0x7F7FFFFFU : bits));
  const bool same = low >= high * 0x1p-10F;
  equal = equal && same;
  return same ? high : bound;
}
// factors of the columns in shared memory: one for all, or an array
struct EqualFactors {
  float value;
  __device__ __forceinline__ explicit EqualFactors(std::uint32_t at) : value(lds32(at)) {}
  __device__ __forceinline__ float4 quad(int) const { return make_float4(value, value, value, value); }
};
struct ColumnFactors {
  std::uint32_t at;
  __device__ __forceinline__ explicit ColumnFactors(std::uint32_t at) : at(at) {}
  __device__ __forceinline__ float4 quad(int c) const { return lds128(at + 16 * c); }
};
template <class Factors> struct Kind {
  using Type = Factors;
};
// Largest magnitude of every column over the 32 rows of a warp, cut to BF16: lane c gets column c's.  Two columns ride in a
// word, and each exchange halves the words a lane still holds.
__device__ __forceinline__ float column_maximum(const float (&s)[kSlice]) {
  const std::uint32_t lane = threadIdx.x & 31;
  std::uint32_t held[kSlice / 2];
#pragma unroll
  for (int i = 0; i < kSlice / 2; ++i) {
    held[i] = __byte_perm(__float_as_uint(s[2 * i]), __float_as_uint(s[2 * i + 1]), 0x7632) & 0x7FFF7FFFU;
  }
#pragma unroll
  for (int words = kSlice / 4; words > 0; words >>= 1) { // lanes 2 `words` apart
    const bool upper = (lane & (2 * words)) != 0;
#pragma unroll
    for (int i = 0; i < words; ++i) {
      const std::uint32_t give = upper ? held[i] : held[i + words];
      const std::uint32_t keep = upper ? held[i + words] : held[i];
      held[i] = __vmaxs2(keep, __shfl_xor_sync(0xFFFFFFFFU, give, 2 * words));
    }
  }
  held[0] = __vmaxs2(held[0], __shfl_xor_sync(0xFFFFFFFFU, held[0], 1));
  return __uint_as_float((lane & 1U) != 0 ? held[0] & 0xFFFF0000U : held[0] << 16);
}

template <int Dtype> struct RowPart; // 32 elements of a row of activations
template <> struct RowPart<RIB200_DTYPE_F32> {
  float4 raw[8];
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      raw[c] = *reinterpret_cast<const float4 *>(static_cast<const float *>(base) + index + 4 * c);
    }
  }
  __device__ __forceinline__ float4 quad(int c) const { return raw[c]; }
  static __device__ __forceinline__ void store(void *base, std::size_t index, const float (&x)[32]) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      *reinterpret_cast<float4 *>(static_cast<float *>(base) + index + 4 * c) =
          make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
    }
  }
};
template <> struct RowPart<RIB200_DTYPE_BF16> {
  uint2 raw[8];
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      raw[c] = *reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(base) + index + 4 * c);
    }
  }
  __device__ __forceinline__ float4 quad(int c) const {
    return make_float4(__uint_as_float(raw[c].x << 16), __uint_as_float(raw[c].x & 0xFFFF0000U),
                       __uint_as_float(raw[c].y << 16), __uint_as_float(raw[c].y & 0xFFFF0000U));
  }
  static __device__ __forceinline__ void store(void *base, std::size_t index, const float (&x)[32]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      std::uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __nv_bfloat162 pair = __floats2bfloat162_rn(x[8 * c + 2 * e], x[8 * c + 2 * e + 1]);
        w[e] = *reinterpret_cast<const std::uint32_t *>(&pair);
      }
      *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(base) + index + 8 * c) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
};
template <> struct RowPart<RIB200_DTYPE_F16> {
  uint2 raw[8];
  __device__ __forceinline__ void load(const void *base, std::size_t index) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      raw[c] = *reinterpret_cast<const uint2 *>(static_cast<const __half *>(base) + index + 4 * c);
    }
  }
  __device__ __forceinline__ float4 quad(int c) const {
    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&raw[c].x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&raw[c].y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
  static __device__ __forceinline__ void store(void *base, std::size_t index, const float (&x)[32]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      *reinterpret_cast<uint4 *>(static_cast<__half *>(base) + index + 8 * c) =
          make_uint4(pack_half(x[8 * c], x[8 * c + 1]), pack_half(x[8 * c + 2], x[8 * c + 3]),
                     pack_half(x[8 * c + 4], x[8 * c + 5]), pack_half(x[8 * c + 6], x[8 * c + 7]));
    }
  }
};

constexpr int kCore = 0; // "dtype" of the form that writes the recurrence's FP32 output as it is

// grid (4 slices, value heads); a layer call's four slices form a cluster
template <int Dtype> __global__ void __launch_bounds__(kChainThreads, 1) gdn_chunk_chain_kernel(const ChunkParams p) {
  constexpr bool kLayer = Dtype != kCore;
  extern __shared__ unsigned char chain_smem_raw[];
  const std::uint32_t base = (smem_address(chain_smem_raw) + 1023U) & ~1023U;
  unsigned char *smem = chain_smem_raw + (base - smem_address(chain_smem_raw));
  const std::uint32_t bars = base + kCsBars;
  auto bar = [&](std::uint32_t index) { return bars + index * 8; };
  volatile std::uint32_t *tmem_slot = reinterpret_cast<volatile std::uint32_t *>(smem + kCsTmemSlot);
  volatile std::uint32_t *abort_flag = reinterpret_cast<volatile std::uint32_t *>(smem + kCsAbort);
  volatile float *s_max = reinterpret_cast<volatile float *>(smem + kCsMax);
  auto wait = [&](std::uint32_t b, std::uint32_t parity) { bounded_wait(b, parity, abort_flag, p.status); };

  grid_dependents_may_launch();
  const std::uint32_t slice = blockIdx.x;
  const std::uint32_t head = blockIdx.y;
  const std::uint32_t warp = threadIdx.x >> 5;
  const std::uint32_t lane = threadIdx.x & 31;
  float *state = p.state + static_cast<std::size_t>(head) * kDim * kDim + slice * kSlice;

  if (threadIdx.x == 0) {
    for (std::uint32_t i = 0; i < kBarCount; ++i) {
      std::uint32_t count = 1;
      if (i == kBarState) {
        count = 128;
      } else if (i >= kBarRead && i < kBarRead + kStages) {
        count = 128 + 64;
      } else if (i == kBarEDelta || i == kBarDelta || i == kBarOutRead || i == kBarOutRead + 1) {
        count = 64;
      }
      mbarrier_init(bar(i), count);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 6) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + kCsTmemSlot),
                 "r"(kChainTmemColumns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }

  // State slice: row `key` of S in this thread's registers.
  float s_reg[kSlice];
  const std::uint32_t key = threadIdx.x; // warps 0-3
  if (warp < 4) {
#pragma unroll
    for (int c = 0; c < kSlice; c += 4) {
      const float4 v = *reinterpret_cast<const float4 *>(state + static_cast<std::size_t>(key) * kDim + c);
      s_reg[c] = v.x;
      s_reg[c + 1] = v.y;
      s_reg[c + 2] = v.z;
      s_reg[c + 3] = v.w;
    }
    s_max[warp * kSlice + lane] = column_maximum(s_reg);
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const std::uint32_t tmem = *tmem_slot;
  if constexpr (kLayer) { // every barrier of the cluster is set up before a peer's sum can arrive
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  // Launched with programmatic stream serialisation behind the prepare kernel: barriers, tensor memory and the state
  // slice (which that kernel does not touch) are set up while its last CTAs finish; the records are read after this.
  grid_dependency_wait();

  auto scales_of = [&](std::uint32_t chunk) { return base + kCsScale + (chunk & (kScaleSlots - 1)) * kScaleBytes; };

  if (warp == 7) {
    // ---- producer ----
    if (lane == 0) {
      auto record = [&](std::uint32_t chunk) {
        return p.scratch.records + (static_cast<std::size_t>(chunk) * p.value_heads + head) * kGdnRecBytes;
      };
      auto key_image = [&](std::uint32_t chunk) {
        return p.scratch.kq + (static_cast<std::size_t>(chunk) * p.key_heads + head % p.key_heads) * kGdnKqBytes;
      };
      RingPlace at;
      std::uint32_t issued = 0;
      for (std::uint32_t chunk = 0; chunk < p.chunks; ++chunk, at.next()) {
        const unsigned char *rec = record(chunk);
        const unsigned char *kq = key_image(chunk);
        const std::uint32_t stage = base + at.stage * kStageBytes;
        if (chunk + kPrefetchAhead < p.chunks) { // its own U and a quarter of what the four slices share
          const unsigned char *ahead = record(chunk + kPrefetchAhead);
          prefetch_l2(ahead + kGdnRecU + slice * kGdnSliceU, kGdnSliceU);
          prefetch_l2(ahead + slice * (kGdnRecU / 4), kGdnRecU / 4);
          prefetch_l2(key_image(chunk + kPrefetchAhead) + slice * (kGdnKqBytes / 4), kGdnKqBytes / 4);
        }
        if (chunk >= kStages) {
          wait(bar(kBarUsed + at.stage), at.phase ^ 1U);
          wait(bar(kBarRead + at.stage), at.phase ^ 1U);
        }
        if (*abort_flag != 0) {
          break;
        }
        fence_proxy_async(); // U and the gates were read by ordinary loads
        const std::uint32_t full = bar(kBarQwFull + at.stage);
        mbarrier_expect_tx(full, 2 * kGdnKqBlock);
#pragma unroll
        for (std::uint32_t b = 0; b < 2; ++b) {
          bulk_copy_g2s(stage + kStageQw + b * kGdnKqBlock, kq + b * kGdnKqBlock + kGdnBlock, kGdnBlock, full);
          bulk_copy_g2s(stage + kStageQw + b * kGdnKqBlock + kGdnBlock, rec + kGdnRecW + b * kGdnBlock, kGdnBlock, full);
        }
        const std::uint32_t rest = bar(kBarRestFull + at.stage);
        mbarrier_expect_tx(rest, 2 * kGdnBlock + kGdnBlock + kGdnSliceU + kChunk * 4);
        bulk_copy_g2s(stage + kStageU, rec + kGdnRecU + slice * kGdnSliceU, kGdnSliceU, rest);
        bulk_copy_g2s(stage + kStageGates, rec + kGdnRecGates + kGdnGateG * 4, kChunk * 4, rest);
#pragma unroll
        for (std::uint32_t b = 0; b < 2; ++b) {
          bulk_copy_g2s(stage + kStageK + b * kGdnBlock, kq + b * kGdnKqBlock, kGdnBlock, rest);
        }
        bulk_copy_g2s(stage + kStageP, rec + kGdnRecP, kGdnBlock, rest);
        issued = chunk + 1;
      }
      if (*abort_flag != 0) { // let the copies already issued land before the CTA's shared memory goes away
        for (std::uint32_t chunk = issued > kStages ? issued - kStages : 0; chunk < issued; ++chunk) {
          const std::uint32_t s = chunk % kStages;
          const std::uint32_t parity = (chunk / kStages) & 1U;
          const long long started = clock64();
          while (!(mbarrier_try_wait(bar(kBarQwFull + s), parity) && mbarrier_try_wait(bar(kBarRestFull + s), parity)) &&
                 clock64() - started < kWaitLimitCycles) {
          }
        }
      }
    }
  } else if (warp == 6) {
    // ---- tensor-core issue: the whole warp walks the chunks, one elected lane issues ----
    const bool issuer = elect_one();
    constexpr std::uint32_t kIdesc = idesc_f16(kSlice, false, true);
    constexpr std::uint32_t kIdescK = idesc_f16(kSlice, true, true);
    const std::uint64_t s_desc = smem_desc(base + kCsState, 16, 8 * kOperandRow, kSwizzle64);
    const std::uint64_t ed_desc = smem_desc(base + kCsEDelta, 16, 8 * kOperandRow, kSwizzle64);
    const std::uint64_t d_desc = smem_desc(base + kCsDelta, 16, 8 * kOperandRow, kSwizzle64);
    RingPlace at;
    for (std::uint32_t chunk = 0; chunk < p.chunks; ++chunk, at.next()) {
      const std::uint32_t s = chunk & 1U;
      const std::uint32_t stage = base + at.stage * kStageBytes;
      wait(bar(kBarQwFull + at.stage), at.phase);
      if (issuer) {
        RIB200_GDN_STAMP(chunk, 7);
      }
      if (chunk >= 2) {
        wait(bar(kBarOutRead + s), ((chunk >> 1) - 1) & 1U);
      }
      if (issuer) {
        RIB200_GDN_STAMP(chunk, 8);
      }
      wait(bar(kBarState), chunk & 1U);
      tcgen05_fence_after();
      if (issuer) {
        RIB200_GDN_STAMP(chunk, 5);
      }
      if (issuer && *abort_flag == 0) {
        const std::uint64_t qw_desc = smem_desc(stage + kStageQw, 16, 1024);
#pragma unroll
        for (std::uint32_t ks = 0; ks < 8; ++ks) {
          umma_f16(tmem + 32 * s, qw_desc + desc_bytes((ks >> 2) * kGdnKqBlock + (ks & 3U) * 32U),
                   s_desc + desc_bytes(ks * 16 * kOperandRow), kIdesc, ks);
        }
        umma_commit(bar(kBarXDone + s));
      }
      __syncwarp();
      wait(bar(kBarRestFull + at.stage), at.phase);
      wait(bar(kBarEDelta), chunk & 1U);
      tcgen05_fence_after();
      if (issuer) {
        RIB200_GDN_STAMP(chunk, 6);
      }
      if (issuer && *abort_flag == 0) {
        const std::uint64_t k_desc = smem_desc(stage + kStageK, kGdnBlock, 1024);
#pragma unroll
        for (std::uint32_t ks = 0; ks < 4; ++ks) {
          umma_f16(tmem + 128, k_desc + desc_bytes(ks * 2048U), ed_desc + desc_bytes(ks * 16 * kOperandRow), kIdescK, ks);
        }
        umma_commit(bar(kBarSdDone));
      }
      __syncwarp();
      wait(bar(kBarDelta), chunk & 1U);
      tcgen05_fence_after();
      if (issuer && *abort_flag == 0) {
        const std::uint64_t p_desc = smem_desc(stage + kStageP, 16, 1024);
#pragma unroll
        for (std::uint32_t ks = 0; ks < 4; ++ks) {
          umma_f16(tmem + 64 + 32 * s, p_desc + desc_bytes(ks * 32U), d_desc + desc_bytes(ks * 16 * kOperandRow), kIdesc, ks);
        }
        umma_commit(bar(kBarO2Done + s));
        umma_commit(bar(kBarUsed + at.stage));
      }
      __syncwarp();
      if (*abort_flag != 0) {
        break;
      }
    }
  } else if (warp == 10) {
    // ---- the factors of the chunks, lane = column.  It waits for the maxima of the chain's warps (barrier 1), they for its
    // factors (barrier 3); the five warps walk all chunks whatever happens. ----
    struct Gates {
      float largest, growth, beta_sum, beta_max, g_end;
    };
    auto gates_of = [&](std::uint32_t chunk) {
      const float *gates = reinterpret_cast<const float *>(
          p.scratch.records + (static_cast<std::size_t>(chunk) * p.value_heads + head) * kGdnRecBytes + kGdnRecGates);
      return Gates{gates[kGdnGateMax + slice * kSlice + lane], gates[kGdnGateGrowth], gates[kGdnGateBetaSum],
                   gates[kGdnGateBetaMax], gates[kGdnGateG + kChunk - 1]};
    };
    auto state_bound = [](const Gates &g, float m) {
      return 11.5F * exp_fast(g.g_end) * m + g.growth * g.beta_sum * g.largest;
    };
    auto column_bound = [&] { // largest |S0| that the four warps have left
      const volatile float *maxima = s_max + lane;
      return fmaxf(fmaxf(maxima[0], maxima[kSlice]), fmaxf(maxima[2 * kSlice], maxima[3 * kSlice]));
    };
    auto factors_of = [&](std::uint32_t chunk) { return reinterpret_cast<float *>(smem + (scales_of(chunk) - base)) + lane; };
    Gates now = gates_of(0);                           // of this chunk ...
    Gates following = gates_of(min(1U, p.chunks - 1)); // ... and of the next
    std::uint32_t state_exponent;                      // of the scale of S0
    bool state_equal = true;
    {
      const float m = column_bound();
      state_exponent = state_exponent_of(level(fmaxf(state_bound(now, m), 1.01F * m), state_equal));
      factors_of(kScaleSlots - 1)[kScaleState / 4] = gdn_power(state_exponent);
      asm volatile("bar.arrive 3, 160;\n" ::: "memory");
    }
    for (std::uint32_t chunk = 0; chunk < p.chunks; ++chunk) {
      asm volatile("bar.sync 1, 160;\n" ::: "memory");
      const float m = column_bound();
      bool equal = state_equal;
      const std::uint32_t delta_exponent = gdn_scale_exponent(
          level(now.beta_max * (now.largest + now.growth * (11.5F * m + now.beta_sum * now.largest)), equal));
      const std::uint32_t unit = growth_unit(now.growth);
      // X times 2^(unit of W) / (scale of S0) into Delta's scale; out of FP32's range only where X is 0
      const int x_exponent = static_cast<int>(delta_exponent + 254) - static_cast<int>(state_exponent + unit + kGdnUnitW);
      float *to = factors_of(chunk);
      to[kScaleX / 4] = gdn_power(static_cast<std::uint32_t>(min(max(x_exponent, 1), 254)));
      to[kScaleDelta / 4] = gdn_power(delta_exponent);
      to[kScaleSd / 4] = gdn_power(254 - delta_exponent) * (1.0F / kGdnUnit);
      to[kScaleOutX / 4] = gdn_power(254 - state_exponent) * (1.0F / kGdnUnit);
      to[kScaleOutDelta / 4] = gdn_power(254 - delta_exponent) * gdn_power(254 - kGdnUnitP - unit);
      state_equal = true;
      state_exponent = state_exponent_of(level(state_bound(now, m), state_equal));
      to[kScaleState / 4] = gdn_power(state_exponent);
      if (lane == 0) {
        to[kScaleEqual / 4] = equal && state_equal ? 1.0F : 0.0F;
      }
      __syncwarp();
      asm volatile("bar.arrive 3, 160;\n" ::: "memory");
      now = following;
      following = gates_of(min(chunk + 2, p.chunks - 1));
    }
  } else if (warp < 4) {
    // ---- the chain: thread = lane of tensor memory ----
    const std::uint32_t lane_base = (warp * 32U) << 16;
    const bool has_w = warp >= 2;                  // rows 64..127 of X: W S0 of token threadIdx.x - 64
    const std::uint32_t token = threadIdx.x & 63U;
    std::uint32_t half_row[16];
    auto put_state = [&](const auto &scale) {
#pragma unroll
      for (int c = 0; c < kSlice / 4; ++c) {
        const float4 f = scale.quad(c);
        half_row[2 * c] = pack_half(s_reg[4 * c] * f.x, s_reg[4 * c + 1] * f.y);
        half_row[2 * c + 1] = pack_half(s_reg[4 * c + 2] * f.z, s_reg[4 * c + 3] * f.w);
      }
      store_operand_row(base + kCsState, key, half_row);
      fence_proxy_async();
      tcgen05_fence_before();
      mbarrier_arrive(bar(kBarState));
    };
    asm volatile("bar.sync 3, 160;\n" ::: "memory"); // the scale of the first S0
    put_state(ColumnFactors(scales_of(kScaleSlots - 1) + kScaleState));
    RingPlace at;
    for (std::uint32_t chunk = 0; chunk < p.chunks; ++chunk, at.next()) {
      const std::uint32_t s = chunk & 1U;
      const std::uint32_t stage = base + at.stage * kStageBytes;
      const std::uint32_t scales = scales_of(chunk);
      if (threadIdx.x == 64) {
        RIB200_GDN_STAMP(chunk, 0);
      }
      s_max[warp * kSlice + lane] = column_maximum(s_reg);
      asm volatile("bar.arrive 1, 160;\n" ::: "memory");
      wait(bar(kBarRestFull + at.stage), at.phase);
      const float g_end = lds32(stage + kStageGates + (kChunk - 1) * 4);
      const float gamma_c = exp_fast(g_end);
      float4 u[kSlice / 4]; // rows 64..127 alone
      float decay_to_end = 0.0F;
      if (has_w) {
        decay_to_end = exp_fast(g_end - lds32(stage + kStageGates + token * 4));
#pragma unroll
        for (std::uint32_t c = 0; c < kSlice / 4; ++c) {
          u[c] = lds128(stage + kStageU + token * kGdnRowBytes + ((c ^ (token & 7U)) << 4));
        }
      }
      mbarrier_arrive(bar(kBarRead + at.stage));
      __syncwarp(); // lanes may have left the wait above one by one
      asm volatile("bar.sync 3, 160;\n" ::: "memory");
      auto walk = [&](auto kind) {
        using Factors = typename decltype(kind)::Type;
        if (has_w) {
          const Factors x_scale(scales + kScaleX);
          {
            const Factors scale(scales + kScaleDelta);
#pragma unroll
            for (int c = 0; c < kSlice / 4; ++c) {
              const float4 f = scale.quad(c);
              u[c] = make_float4(u[c].x * f.x, u[c].y * f.y, u[c].z * f.z, u[c].w * f.w);
            }
          }
          wait(bar(kBarXDone + s), (chunk >> 1) & 1U);
          tcgen05_fence_after();
          if (threadIdx.x == 64) {
            RIB200_GDN_STAMP(chunk, 1);
          }
          float x[kSlice];
          tmem_ld32(tmem + lane_base + 32 * s, x);
#pragma unroll
          for (int c = 0; c < kSlice / 4; ++c) { // Delta at its scale
            const float4 f = x_scale.quad(c);
            x[4 * c] = u[c].x - x[4 * c] * f.x;
            x[4 * c + 1] = u[c].y - x[4 * c + 1] * f.y;
            x[4 * c + 2] = u[c].z - x[4 * c + 2] * f.z;
            x[4 * c + 3] = u[c].w - x[4 * c + 3] * f.w;
          }
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            half_row[c] = pack_half(x[2 * c] * decay_to_end, x[2 * c + 1] * decay_to_end);
          }
          store_operand_row(base + kCsEDelta, token, half_row);
          fence_proxy_async();
          tcgen05_fence_before();
          mbarrier_arrive(bar(kBarEDelta));
          if (threadIdx.x == 64) {
            RIB200_GDN_STAMP(chunk, 2);
          }
#pragma unroll
          for (int c = 0; c < 16; ++c) {
            half_row[c] = pack_half(x[2 * c], x[2 * c + 1]);
          }
          if (chunk >= 1) { // P Delta of the chunk before has read its operand
            wait(bar(kBarO2Done + (s ^ 1U)), ((chunk - 1) >> 1) & 1U);
          }
          store_operand_row(base + kCsDelta, token, half_row);
          fence_proxy_async();
          mbarrier_arrive(bar(kBarDelta));
        }
#pragma unroll
        for (int c = 0; c < kSlice; ++c) {
          s_reg[c] *= gamma_c;
        }
        const Factors undo(scales + kScaleSd);
        const Factors scale(scales + kScaleState);
        wait(bar(kBarSdDone), chunk & 1U);
        tcgen05_fence_after();
        if (threadIdx.x == 64) {
          RIB200_GDN_STAMP(chunk, 3);
        }
        float sd[kSlice];
        tmem_ld32(tmem + lane_base + 128, sd);
#pragma unroll
        for (int c = 0; c < kSlice / 4; ++c) {
          const float4 f = undo.quad(c);
          s_reg[4 * c] += sd[4 * c] * f.x;
          s_reg[4 * c + 1] += sd[4 * c + 1] * f.y;
          s_reg[4 * c + 2] += sd[4 * c + 2] * f.z;
          s_reg[4 * c + 3] += sd[4 * c + 3] * f.w;
        }
        put_state(scale);
      };
      if (lds32(scales + kScaleEqual) != 0.0F) {
        walk(Kind<EqualFactors>{});
      } else {
        walk(Kind<ColumnFactors>{});
      }
      if (threadIdx.x == 64) {
        RIB200_GDN_STAMP(chunk, 4);
      }
    }
#pragma unroll
    for (int c = 0; c < kSlice; c += 4) {
      *reinterpret_cast<float4 *>(state + static_cast<std::size_t>(key) * kDim + c) =
          make_float4(s_reg[c], s_reg[c + 1], s_reg[c + 2], s_reg[c + 3]);
    }
  } else {
    // ---- warps 4-5 and 8-9: the outputs of the even and of the odd chunks, thread = token of the chunk ----
    const std::uint32_t parity = warp >> 3;
    const std::uint32_t token = threadIdx.x & 63U;
    const std::uint32_t lane_base = ((warp & 3U) * 32U) << 16;
    const std::size_t column = static_cast<std::size_t>(head) * kDim + slice * kSlice;
    const std::size_t row_stride = static_cast<std::size_t>(p.value_heads) * kDim;
    std::uint32_t norm_target[kGdnSlices];
    std::uint32_t norm_bar[kGdnSlices];
    if constexpr (kLayer) {
      if (threadIdx.x < 128 + kSlice) {
        reinterpret_cast<float *>(smem + kCsWeight)[threadIdx.x - 128] =
            load_any(p.norm_weight, slice * kSlice + threadIdx.x - 128, p.weight_dtype);
      }
      asm volatile("bar.sync 2, 128;\n" ::: "memory");
#pragma unroll
      for (std::uint32_t r = 0; r < kGdnSlices; ++r) {
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                     : "=r"(norm_target[r])
                     : "r"(base + kCsNorm + (slice * kChunk + token) * 4), "r"(r));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(norm_bar[r]) : "r"(bar(kBarNorm)), "r"(r));
      }
    }
    RingPlace at;
    if (parity != 0) {
      at.next();
    }
    for (std::uint32_t chunk = parity; chunk < p.chunks; chunk += 2, at.next(), at.next()) {
      const std::uint32_t s = chunk & 1U;
      const std::uint32_t stage = base + at.stage * kStageBytes;
      [[maybe_unused]] const std::uint32_t norm_slot = chunk & (kNormSlots - 1);
      const std::uint32_t tok = chunk * kChunk + token;
      const bool live = tok < p.tokens;
      RowPart<kLayer ? Dtype : RIB200_DTYPE_F32> z{};
      if constexpr (kLayer) {
        if (live) {
          z.load(p.input, static_cast<std::size_t>(tok) * p.token_stride + p.z_column + column);
        }
        if (token == 0) {
          RIB200_GDN_STAMP(chunk, 9);
          mbarrier_expect_tx(bar(kBarNorm + norm_slot), kGdnSlices * kChunk * 4);
        }
      }
      wait(bar(kBarRestFull + at.stage), at.phase);
      const float gamma = exp_fast(lds32(stage + kStageGates + token * 4));
      mbarrier_arrive(bar(kBarRead + at.stage));
      wait(bar(kBarXDone + s), (chunk >> 1) & 1U);
      tcgen05_fence_after();
      if (token == 0) {
        RIB200_GDN_STAMP(chunk, 10);
      }
      float o[kSlice];
      tmem_ld32(tmem + lane_base + 32 * s, o);
      wait(bar(kBarO2Done + s), (chunk >> 1) & 1U);
      tcgen05_fence_after();
      {
        float o2[kSlice];
        tmem_ld32(tmem + lane_base + 64 + 32 * s, o2);
        const std::uint32_t scales = scales_of(chunk);
        if (lds32(scales + kScaleEqual) != 0.0F) {
          const float scale_x = gamma * lds32(scales + kScaleOutX);
          const float scale_o2 = lds32(scales + kScaleOutDelta);
#pragma unroll
          for (int c = 0; c < kSlice; ++c) {
            o[c] = o[c] * scale_x + o2[c] * scale_o2;
          }
        } else {
#pragma unroll
          for (std::uint32_t c = 0; c < kSlice / 4; ++c) {
            const float4 undo_x = lds128(scales + kScaleOutX + 16 * c);
            const float4 undo_delta = lds128(scales + kScaleOutDelta + 16 * c);
            o[4 * c] = o[4 * c] * (gamma * undo_x.x) + o2[4 * c] * undo_delta.x;
            o[4 * c + 1] = o[4 * c + 1] * (gamma * undo_x.y) + o2[4 * c + 1] * undo_delta.y;
            o[4 * c + 2] = o[4 * c + 2] * (gamma * undo_x.z) + o2[4 * c + 2] * undo_delta.z;
            o[4 * c + 3] = o[4 * c + 3] * (gamma * undo_x.w) + o2[4 * c + 3] * undo_delta.w;
          }
        }
        tcgen05_fence_before();
        mbarrier_arrive(bar(kBarOutRead + s));
      }
      if constexpr (kLayer) {
        float squares = 0.0F;
#pragma unroll
        for (int c = 0; c < kSlice; ++c) {
          squares += o[c] * o[c];
        }
#pragma unroll
        for (std::uint32_t r = 0; r < kGdnSlices; ++r) {
          asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n" ::"r"(
                           norm_target[r] + norm_slot * (kGdnSlices * kChunk * 4)),
                       "r"(__float_as_uint(squares)), "r"(norm_bar[r] + norm_slot * 8)
                       : "memory");
        }
        const std::uint32_t weights = base + kCsWeight;
#pragma unroll
        for (std::uint32_t c = 0; c < kSlice / 4; ++c) {
          const float4 w = lds128(weights + 16 * c);
          const float4 gate = z.quad(c);
          o[4 * c] *= w.x * silu_fast(gate.x);
          o[4 * c + 1] *= w.y * silu_fast(gate.y);
          o[4 * c + 2] *= w.z * silu_fast(gate.z);
          o[4 * c + 3] *= w.w * silu_fast(gate.w);
        }
        if (token == 0) {
          RIB200_GDN_STAMP(chunk, 11);
        }
        wait(bar(kBarNorm + norm_slot), (chunk >> 2) & 1U);
        if (token == 0) {
          RIB200_GDN_STAMP(chunk, 12);
        }
        const std::uint32_t norms = base + kCsNorm + norm_slot * (kGdnSlices * kChunk * 4) + token * 4;
        const float sum = (lds32(norms) + lds32(norms + kChunk * 4)) + (lds32(norms + 2 * kChunk * 4) + lds32(norms + 3 * kChunk * 4));
        const float scale = rsqrtf(sum / static_cast<float>(kDim) + p.epsilon);
#pragma unroll
        for (int c = 0; c < kSlice; ++c) {
          o[c] *= scale;
        }
        if (live) {
          RowPart<Dtype>::store(p.output, static_cast<std::size_t>(tok) * row_stride + column, o);
        }
      } else if (live) {
        RowPart<RIB200_DTYPE_F32>::store(p.out, static_cast<std::size_t>(tok) * row_stride + column, o);
      }
      if (*abort_flag != 0) {
        break;
      }
    }
  }

  // every role comes here; the products issued so far have completed or the CTA has given up waiting for them
  tcgen05_fence_before();
  __syncthreads();
  if (warp == 6) {
    // warps 0-5, 8 and 9 waited for the last commits, so nothing is still writing tensor memory
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kChainTmemColumns) : "memory");
  }
  if constexpr (kLayer) { // nobody leaves while a peer may still send it a sum
    if (*abort_flag != 0) {
      for (const long long started = clock64(); clock64() - started < (1LL << 17);) {
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
}

// SMs of the current device
int sm_count() {
  static int counts[64] = {};
  int device = 0;
  cuda_ok(cudaGetDevice(&device), "cudaGetDevice");
  require(device >= 0 && device < 64, "device ordinal out of range", RIB200_STATUS_INTERNAL);
  if (counts[device] == 0) {
    int count = 0;
    cuda_ok(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device), "SM count");
    counts[device] = count > 0 ? count : 1;
  }
  return counts[device];
}

void configure_once() {
  static std::once_flag flags[64];
  int device = 0;
  cuda_ok(cudaGetDevice(&device), "cudaGetDevice");
  require(device >= 0 && device < 64, "device ordinal out of range", RIB200_STATUS_INTERNAL);
  std::call_once(flags[device], [] {
    cuda_ok(cudaFuncSetAttribute(gdn_chunk_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPrepSmemBytes),
            "gated-delta prepare shared-memory opt-in");
    for (auto *kernel : {gdn_chunk_chain_kernel<kCore>, gdn_chunk_chain_kernel<RIB200_DTYPE_F32>,
                         gdn_chunk_chain_kernel<RIB200_DTYPE_F16>, gdn_chunk_chain_kernel<RIB200_DTYPE_BF16>}) {
      cuda_ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kChainSmemBytes),
              "gated-delta chain shared-memory opt-in");
    }
  });
}

// behind the image kernel: prepare, then the chain; `dtype` kCore writes p.out, anything else the layer's output
void launch_chunks(const ChunkParams &p, int dtype, cudaStream_t stream) {
  configure_once();
  const std::uint32_t items = p.chunks * p.value_heads;
  const std::uint32_t slots = 2U * static_cast<std::uint32_t>(sm_count());
  launch_programmatic(gdn_chunk_prepare_kernel, dim3(items < slots ? items : slots), dim3(kPrepThreads), kPrepSmemBytes,
                      stream, "gated-delta prepare launch", p);
  const dim3 grid(kGdnSlices, p.value_heads);
  const char *what = "gated-delta chain launch";
  auto layer = [&](auto kernel) {
    launch_programmatic_cluster(kernel, grid, dim3(kChainThreads), kGdnSlices, kChainSmemBytes, stream, what, p);
  };
  if (dtype == kCore) {
    launch_programmatic(gdn_chunk_chain_kernel<kCore>, grid, dim3(kChainThreads), kChainSmemBytes, stream, what, p);
  } else if (dtype == RIB200_DTYPE_F32) {
    layer(gdn_chunk_chain_kernel<RIB200_DTYPE_F32>);
  } else if (dtype == RIB200_DTYPE_F16) {
    layer(gdn_chunk_chain_kernel<RIB200_DTYPE_F16>);
  } else {
    layer(gdn_chunk_chain_kernel<RIB200_DTYPE_BF16>);
  }
}

ChunkParams base_params(void *workspace, float *state, std::uint32_t tokens, std::uint32_t key_heads,
                        std::uint32_t value_heads) {
  require(workspace != nullptr, "gated-delta chunked prefill needs its workspace");
  require(reinterpret_cast<std::uintptr_t>(workspace) % 16 == 0, "gated-delta chunk workspace is not 16-byte aligned");
  require(reinterpret_cast<std::uintptr_t>(state) % 16 == 0, "gated-delta chunked prefill: state must be 16-byte aligned");
  ChunkParams p{};
  p.tokens = tokens;
  p.chunks = (tokens + kChunk - 1) / kChunk;
  p.key_heads = key_heads;
  p.value_heads = value_heads;
  p.scratch = gdn_chunk_scratch(workspace, p.chunks, key_heads, value_heads);
  p.state = state;
  p.status = device_status_word();
  return p;
}

} // namespace

#ifdef RIB200_TRACE
extern "C" int rib200_debug_read_gdn_trace(long long *host, std::size_t count) {
  return static_cast<int>(cudaMemcpyFromSymbol(host, g_gdn_trace, count * sizeof(long long)));
}
#endif

std::size_t gdn_chunk_workspace_bytes(std::size_t tokens, std::size_t key_heads, std::size_t value_heads) {
  const char *what = "gated-delta chunk workspace overflows";
  const std::size_t chunks = ceil_div(tokens, kChunk, "gated-delta chunk count overflows");
  return mul(chunks,
             add(mul(key_heads, kGdnKqBytes, what), mul(value_heads, kGdnVBytes + kGdnRecBytes, what), what), what);
}

void launch_gdn_chunked(const GdnCoreArgs &a, void *workspace, cudaStream_t stream) {
  ChunkParams p = base_params(workspace, a.state, a.tokens, a.key_heads, a.value_heads);
  require(reinterpret_cast<std::uintptr_t>(a.out) % 16 == 0,
          "gated-delta chunked prefill: output must be 16-byte aligned");
  p.out = a.out;
  launch_gdn_core_images(a, workspace, stream);
  launch_chunks(p, kCore, stream);
}

bool gdn_layer_chunks_apply(const GdnLayerArgs &a) {
  // the rows are read four elements at a time and written sixteen bytes at a time
  const std::size_t element = a.dtype == RIB200_DTYPE_F32 ? 4 : 2;
  const std::size_t stride = static_cast<std::size_t>(2 * a.key_heads + 2 * a.value_heads) * kDim + 2 * a.value_heads;
  return a.conv_width == 4 && reinterpret_cast<std::uintptr_t>(a.input) % (4 * element) == 0 && stride % 4 == 0 &&
         reinterpret_cast<std::uintptr_t>(a.output) % 16 == 0 &&
         (a.weight_dtype != RIB200_DTYPE_F32 || reinterpret_cast<std::uintptr_t>(a.conv_weight) % 16 == 0);
}

void launch_gdn_layer_chunks(const GdnLayerArgs &a, void *workspace, cudaStream_t stream) {
  ChunkParams p = base_params(workspace, a.recurrent_state, a.tokens, a.key_heads, a.value_heads);
  p.input = a.input;
  p.norm_weight = a.output_norm_weight;
  p.output = a.output;
  p.history = a.convolution_state;
  p.conv_dim = (2 * a.key_heads + a.value_heads) * kDim;
  p.token_stride = p.conv_dim + 2 * a.value_heads + a.value_heads * kDim;
  p.z_column = p.conv_dim + 2 * a.value_heads;
  p.dtype = a.dtype;
  p.weight_dtype = a.weight_dtype;
  p.epsilon = a.epsilon;
  launch_gdn_layer_images(a, workspace, stream);
  launch_chunks(p, a.dtype, stream);
}

} // namespace rib200
