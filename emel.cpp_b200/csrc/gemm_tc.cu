// Q4_K x Q8_K matrix product for many columns (prompt processing) on the Blackwell tensor cores: tcgen05.mma kind::f16,
// weights as the A operand in TMEM, activations as the B operand in shared memory, f32 accumulators in TMEM that only
// ever hold exact integers.
//
// What is computed is exactly the reference's per-super-block value,
//   fma(d*dx, isum, -(dmin*dx)*msum),   isum = sum_j sc_j * dot_j(q, x),   msum = sum_j m_j * bsum_j
//   (src/emel/kernel/x86_64/actions.hpp:859-866)
// added in ascending block order, so the result equals the mat-vec kernels' (and the x86 AVX2 route's) bit for bit.
//   * A weight times its scale, q * sc <= 15 * 63 = 945, is exact in f16, so one operand carries both.
//   * f32 sums are exact below 2^24, which sum 945 * |x| over 256 can pass.  So the activations are centred: u = x - v with
//     v = the rounded mean of the super-block's 256 values, an integer within +-255 and exact in f16.  The positive
//     and the negative u of a super-block then sum to at most 16448 each, so any partial sum of q * sc * u stays
//     below 945 * 16448 < 2^24 in any order, and (float)isum = fma(v, T, D) with T = sum q * sc of the row: v * T + D is
//     the exact integer, rounded once.
//   * msum comes from one K = 16 instruction: the row's mins (each twice) times the 16 block sums, all exact.
// The expanded weights pass through neither the shared memory nor its port: a thread owns a weight row = a TMEM lane
// and writes the operand with tcgen05.st.  Expanding two weights is one mask and one half2 fma: a masked 4-bit quant
// under the exponent of 1024 is 1024 + q (1024 + 16 q), times sc (sc / 16) minus 1024 sc (64 sc) is q * sc without a
// rounding.  The order of a super-block's 256 weights along the MMA's K is free (the sums are exact), so it follows
// from the masks; a pre-pass lays the activations out alike.
//
// CTA = 128 weight rows (TMEM lanes) x TN columns (32, 64 or 128), one super-block of K per turn, 20 warps:
//   warps 0-7   producers: two warps per TMEM lane quarter, one for each half (128 weights) of a super-block; a thread
//               expands its row's half into TMEM, 64 weights at a time
//   warps 8-15  epilogue: two warps per TMEM lane quarter, half of the columns each, a thread a row: the row's constants stay
//               in registers, the float chain runs on packed f32x2 instructions
//   warps 16, 17 MMA issue, msum included, half of the columns each; TMEM allocation
//   warp  18    copies of the weights (TMA, 128 rows x 144 bytes) and of the activations, a quarter super-block each
//   warp  19    copies of block sums, column scales and table
// TMEM at TN = 128: two turns' accumulators (256 columns), msum of one turn (128, made and read in two parts, so that
// the next turn's first part is made while the epilogue works on the second), the operand of one super-block (128, handed
// over in quarters).  Narrower tiles keep two super-blocks of operand.
// Where it pays (TN = 128, many waves: plan_tiles) the mins' operand and {d, -dmin, T} of every row and super-block come from a
// table that a pre-pass over the weights makes once; else the producers work them out while they expand.
// Registers are split by setmaxnreg: 640 threads x 96 at launch = 256 x 80 + 256 x 136 + 128 x 48.
// Every mbarrier wait is bounded; on a timeout the CTA raises the status word, lets its copies land and frees its TMEM.
//
// What bounds it: instruction issue, 61 % of the slots with some eight cycles between two instructions of a warp.  Per
// 128 x 128 x 256: 6,700 warp instructions (1,536 packed float ones, 1,150 for the expansion), of 2,760 cycles the MMAs take
// 1,090.  Measured, B200, 14336 x 4096 by 2048 columns: pre-passes and product 352 us, product alone 333 (683 and 722
// TFLOP/s); the int8 kernel before it (two operands of scale pieces, sums of mins on mma.sync) 439.  Whole calls on planes,
// before and now: 14336 x 4096 by 32 columns 47.7 -> 30.5, by 128 48.4 -> 39.9, by 512 159 -> 118; 4096 x 14336 by 32 134 -> 78,
// by 333 136 -> 104, by 1900 517 -> 354; 1024 x 4096 by 333 47.6 -> 31.4.  What gave it: TMEM loads of whole lanes (32x32b, half
// a cycle a register against two of 16x256b: 16 % of the product without its arithmetic), roles in few instructions (the
// producers' loop not unrolled 374 -> 349), the table (233 -> 188 million instructions), the second MMA warp (a call, quantizer
// included, 385 -> 372; the figures above are from before it).  Without effect: tiles of 96 columns with
// msum double-buffered (400), 16 epilogue warps (355), copies or MMAs left out (the memories and the tensor core wait).
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace emelb {
namespace {

using namespace tc;

constexpr int BM = 128;
constexpr int kEpilogueWarp0 = 8, kEpilogueWarps = 8, kMmaWarp = 16, kLoaderWarp = 18;   // two MMA warps; the meta loader's warp
constexpr int kThreads = 20 * 32;

constexpr int kRawBytes = BM * Q4_K_BYTES;   // 128 rows of a super-block as they lie in memory; 144 bytes a row spread reads over the banks
constexpr int kMetaSlots = 3;
constexpr int kStageRow = 80;             // an epilogue warp's store: 16 columns of a row; a multiple of 16 that spreads rows over the banks
constexpr int kRowMeta = 32;              // per row: d, d, -dmin, -dmin, then T of either half, each twice
constexpr int kMinsBytes = BM * 32;       // A operand of the msum instruction: two 16-byte chunks of K
constexpr int kSumBytes = kColumnSumBytes, kPairBytes = kColumnPairBytes;

constexpr int kTableRow = 24;             // per row of the table: d, d, -dmin, -dmin, T, T
constexpr int kTableBytes = kMinsBytes + BM * kTableRow;   // of 128 rows x one super-block

template <int TN, bool kTable>
struct Cfg {
  static constexpr int kProducerRegs = 80, kEpilogueRegs = 136, kOtherRegs = 48;
  static_assert(8 * kProducerRegs + 8 * kEpilogueRegs + 4 * kOtherRegs <= 20 * 96, "register split");
  static constexpr int kTurns = TN == 32 ? 4 : 2;       // super-blocks of activations in shared memory
  static constexpr int kRawSlots = TN == 128 ? 2 : 4;   // and of weights
  static constexpr int kOperands = TN == 128 ? 1 : 2;   // super-blocks of operand in TMEM
  static constexpr int kParts = TN >= 64 ? 2 : 1;       // of the columns: each has its msum made and is read by itself
  static constexpr int kPart = TN / kParts;
  // TMEM columns: accumulators of two turns, msum of one, then the operand
  static constexpr uint32_t kTmemM = 2 * TN, kTmemA = TN == 128 ? 384 : 256;
  static constexpr int kQuarterBytes = TN / 8 * kAtomBytes;   // activations of a quarter super-block (64 K)
  // what a bulk-copied slot holds for a super-block: block sums, dx and v of the columns; with the table also mins and row meta
  static constexpr int kOffPairs = TN * kSumBytes, kOffTable = kOffPairs + TN / 2 * kPairBytes;
  static constexpr int kMetaBytes = kOffTable + (kTable ? kTableBytes : 0);
  static constexpr int kMinsSlots = kTable ? 0 : kOperands + 2, kRowMetaSlots = kTable ? 0 : kOperands + 2;
  // shared memory map
  static constexpr int kOffRaw = 4 * kTurns * kQuarterBytes;
  static constexpr int kOffMins = kOffRaw + kRawSlots * kRawBytes;
  static constexpr int kOffRowMeta = kOffMins + kMinsSlots * kMinsBytes;
  static constexpr int kOffMeta = kOffRowMeta + kRowMetaSlots * BM * kRowMeta;
  static constexpr int kOffStage = kOffMeta + kMetaSlots * kMetaBytes;
  static constexpr int kOffBars = kOffStage + kEpilogueWarps * 32 * kStageRow;
  static constexpr int kSmemBytes = kOffBars + 512 + 1024;   // barriers; slack for the base's alignment
  static_assert(kSmemBytes <= 227 * 1024, "shared memory");
};

// K-major, no swizzle, 8-row groups of 128 bytes; chunk_stride: between the two 16-byte K chunks
__device__ __forceinline__ uint64_t plain_desc(uint32_t saddr, uint32_t chunk_stride) {
  return (uint64_t)((saddr >> 4) & 0x3fffu) | (uint64_t)(chunk_stride >> 4) << 16 | (uint64_t)(128 >> 4) << 32 | (uint64_t)1 << 46;
}

struct GemmArgs {
  int M, K, N;
  const uint8_t* x;       // [K/64][npad/8] swizzle atoms of 8 columns
  const uint8_t* sums;    // [K/256][2 chunks][npad][16 bytes]
  const uint8_t* pairs;   // [K/256][npad/2]{dx, dx, v, v}
  const uint8_t* table;   // [ceil(M/128)][K/256]{mins, row meta}
  int npad;
  float* y;
  int64_t ldy;
  int* status;
};

// 16-byte pieces of the result's rows
__host__ __device__ __forceinline__ bool rows_aligned(const GemmArgs& p) {
  return ((p.ldy | (int64_t)(reinterpret_cast<uintptr_t>(p.y) >> 2)) & 3) == 0;
}

// pre-pass: the quantized activation planes of columns col0.. -> operand order.  K position 128 n + 16 w + 8 c + j of
// a super-block holds element 128 n + 64 c + 32 (j / 4) + 4 w + {0, 2, 1, 3}[j % 4], which is what the producers'
// masks leave side by side.  grid (K/256, npad/64), 256 threads; columns past N are zero.
constexpr int kPreCols = 64, kPreRow = QK_K + 4;   // 65 words: column-wise reads fall on all banks

__global__ void __launch_bounds__(256) operand_layout_kernel(ActPlanes act, int col0, int N, int npad, bool centre, uint8_t* x, uint8_t* sums, uint8_t* pairs) {
  __shared__ __align__(16) uint8_t t8[kPreCols * kPreRow];
  __shared__ int mean[kPreCols];
  const int kb = blockIdx.x, c0 = blockIdx.y * kPreCols;
  for (int q = threadIdx.x; q < kPreCols * 16; q += 256) {
    const int col = q >> 4, piece = q & 15;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (c0 + col < N) v = *reinterpret_cast<const uint4*>(act.qs + (int64_t)(col0 + c0 + col) * act.col_stride_qs + kb * QK_K + 16 * piece);
    uint32_t* o = reinterpret_cast<uint32_t*>(t8 + col * kPreRow + 16 * piece);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
  if (threadIdx.x < kPreCols) {
    const int col = threadIdx.x;
    __half h[16];
    float d = 0.0f;
    int total = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) h[i] = __float2half_rn(0.0f);
    if (c0 + col < N) {
      const int4* bs = reinterpret_cast<const int4*>(act.bsums + (int64_t)(col0 + c0 + col) * act.col_stride_bs + kb * 16);
      const int4 b0 = bs[0], b1 = bs[1];
      const int w[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int j = 0; j < 8; ++j) {   // |sum of 16| <= 2048: exact in f16
        const int s0 = (int)(short)(w[j] & 0xffff), s1 = w[j] >> 16;
        h[2 * j] = __int2half_rn(s0);
        h[2 * j + 1] = __int2half_rn(s1);
        total += s0 + s1;
      }
      d = act.d[(int64_t)(col0 + c0 + col) * act.col_stride_d + kb];
    }
    const int v = centre ? (total + 128) >> 8 : 0;
    mean[col] = v;
#pragma unroll
    for (int c = 0; c < 2; ++c)
      *reinterpret_cast<uint4*>(sums + (((size_t)kb * 2 + c) * npad + c0 + col) * 16) = *reinterpret_cast<const uint4*>(h + 8 * c);
    float* p = reinterpret_cast<float*>(pairs + ((size_t)kb * (npad >> 1) + ((c0 + col) >> 1)) * kPairBytes) + (col & 1);
    p[0] = d;
    p[2] = (float)v;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < kPreCols * 32; q += 256) {
    const int col = q & (kPreCols - 1), ch = q >> 6;               // chunk ch of 8 K positions
    const int n = ch >> 4, w = (ch >> 1) & 7, c = ch & 1;
    const uint8_t* s = t8 + col * kPreRow + 128 * n + 64 * c + 4 * w;
    const __half2 bias = __float2half2_rn(-1152.0f - (float)mean[col]);   // (x ^ 0x80) | 0x6400 is 1152 + x
    auto halves = [&](uint32_t word, uint32_t& even, uint32_t& odd) {     // four int8 -> f16 {0, 2}, {1, 3}
      const uint32_t u = word ^ 0x80808080u;
      even = h2_bits(__hadd2(bits_h2((u & 0x00ff00ffu) | 0x64006400u), bias));
      odd = h2_bits(__hadd2(bits_h2(((u >> 8) & 0x00ff00ffu) | 0x64006400u), bias));
    };
    uint4 o;
    halves(*reinterpret_cast<const uint32_t*>(s), o.x, o.y);
    halves(*reinterpret_cast<const uint32_t*>(s + 32), o.z, o.w);
    uint8_t* dst = x + ((size_t)(4 * kb + (ch >> 3)) * (npad >> 3) + ((c0 + col) >> 3)) * kAtomBytes + (col & 7) * 128 + (((ch ^ col) & 7) << 4);
    *reinterpret_cast<uint4*>(dst) = o;
  }
}

// pre-pass over the weights, for products of several column tiles: the mins as the msum instruction's A operand, and d, -dmin
// and T = sum q * sc of every row and super-block, which the producers would else work out anew for each column tile.
// grid (K/256, ceil(M/128)), 128 threads; rows past M repeat the last one
__global__ void __launch_bounds__(128) q4k_table_kernel(const uint8_t* W, int64_t row_bytes, int M, uint8_t* table) {
  __shared__ __align__(16) uint8_t blocks[BM * Q4_K_BYTES];
  const int kb = blockIdx.x, r0 = blockIdx.y * BM, t = threadIdx.x;
#pragma unroll
  for (int j = 0; j < 9; ++j) {
    const int g = t + BM * j, rr = g / 9, part = g - 9 * rr;
    *reinterpret_cast<uint4*>(blocks + 16 * g) =
        *reinterpret_cast<const uint4*>(W + (size_t)min(r0 + rr, M - 1) * row_bytes + (size_t)kb * Q4_K_BYTES + 16 * part);
  }
  __syncthreads();
  const uint4* blk = reinterpret_cast<const uint4*>(blocks + t * Q4_K_BYTES);
  const uint4 h = blk[0];
  const uint32_t sc[2] = {h.y & 0x3f3f3f3fu, (h.w & 0x0f0f0f0fu) | (((h.y >> 6) & 0x03030303u) << 4)};
  const uint32_t mn[2] = {h.z & 0x3f3f3f3fu, ((h.w >> 4) & 0x0f0f0f0fu) | (((h.z >> 6) & 0x03030303u) << 4)};
  int total = 0;
#pragma unroll
  for (int g = 0; g < 4; ++g) {          // sub-blocks 2g (low nibbles), 2g + 1
    int lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint4 v = blk[1 + 2 * g + i];
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        lo = __dp4a(w[k] & 0x0f0f0f0fu, 0x01010101u, (unsigned)lo);
        hi = __dp4a((w[k] >> 4) & 0x0f0f0f0fu, 0x01010101u, (unsigned)hi);
      }
    }
    const uint32_t s = sc[g >> 1] >> (16 * (g & 1));
    total += (int)(s & 0xffu) * lo + (int)((s >> 8) & 0xffu) * hi;
  }
  uint8_t* out = table + ((size_t)blockIdx.y * gridDim.x + kb) * kTableBytes;
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    __half2 m[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) m[f] = __half2half2(__ushort2half_rn((unsigned short)((mn[n] >> (8 * f)) & 0xffu)));
    *reinterpret_cast<uint4*>(out + n * (BM * 16) + t * 16) = *reinterpret_cast<const uint4*>(m);
  }
  const float d = h2f((uint16_t)(h.x & 0xffffu)), dm = -h2f((uint16_t)(h.x >> 16)), tt = (float)total;
  float2* row = reinterpret_cast<float2*>(out + kMinsBytes + t * kTableRow);
  row[0] = make_float2(d, d);
  row[1] = make_float2(dm, dm);
  row[2] = make_float2(tt, tt);
}

template <int TN, bool kTable>
__global__ void __launch_bounds__(kThreads, 1) gemm_q4k_tc_kernel(const GemmArgs p, const __grid_constant__ CUtensorMap wmap) {
  using C = Cfg<TN, kTable>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw = smem + C::kOffRaw;
  uint8_t* mins = smem + C::kOffMins;
  uint8_t* rowmeta = smem + C::kOffRowMeta;
  uint8_t* meta = smem + C::kOffMeta;
  // barriers, by their shared memory addresses
  const uint32_t bars = smem_u32(smem + C::kOffBars);
  const uint32_t h_full = bars;                       // [turns][4 quarters] producers and bulk copies -> MMA; the last quarter brings the meta slot
  const uint32_t h_free = h_full + 8 * 4 * C::kTurns; // MMA -> producers and loader
  const uint32_t r_full = h_free + 8 * 4 * C::kTurns; // [raw slots] TMA -> producers: the weights of a super-block
  const uint32_t r_free = r_full + 8 * C::kRawSlots;
  const uint32_t m_free = r_free + 8 * C::kRawSlots;  // [3] epilogue -> loader: the meta slot is read
  const uint32_t s_full = m_free + 8 * kMetaSlots;    // [parts] MMA -> epilogue: the part's accumulators and msum are complete
  const uint32_t s_free = s_full + 8 * 2;             // [parts] epilogue -> MMA: they are read
  const uint32_t drained = s_free + 8 * 2;            // [2] only after a wait that gave up
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::kOffBars + 8 * 60);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // from one lane: the compiler then keeps what follows from it in uniform registers (TMEM addresses, barriers, pointers)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::kRawSlots; ++s) { mbar_init(r_full + 8 * s, 1); mbar_init(r_free + 8 * s, 8); }
    for (int s = 0; s < 4 * C::kTurns; ++s) { mbar_init(h_full + 8 * s, (s & 3) == 3 ? 6 : 5); mbar_init(h_free + 8 * s, C::kParts); }
    for (int s = 0; s < kMetaSlots; ++s) mbar_init(m_free + 8 * s, kEpilogueWarps);
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + 8 * s, 1);
      mbar_init(s_free + 8 * s, kEpilogueWarps);
      mbar_init(drained + 8 * s, 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  const int mt = (p.M + BM - 1) / BM, nt = (p.N + TN - 1) / TN, ntiles = mt * nt, nkb = p.K / QK_K;
  const int my_tiles = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int turns = my_tiles * nkb;   // super-blocks this CTA walks

  if (warp < 8) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kProducerRegs));
    const int quarter = warp & 3, n = warp >> 2;   // TMEM lanes 32 * quarter .., half n of every super-block
    const uint32_t a_lane = tmem_base + C::kTmemA + ((uint32_t)(32 * quarter) << 16) + 64u * n;
    const uint32_t low = in_register(0x000f000fu), high = in_register(0x00f000f0u), k1024 = in_register(0x64006400u);
    int slot = 0, mslot = 0, rslot = 0;
    uint32_t rphase = 0;
    bool live = true;
    for (int it = 0; it < turns; ++it) {
      live = mbar_wait(r_full + 8 * slot, rphase, abort_flag);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      const int buf = it & 1, hb = 4 * (it & (C::kTurns - 1)) + 2 * n;
      const uint8_t* blk = raw + slot * kRawBytes + (32 * quarter + lane) * Q4_K_BYTES;
      const uint4 h = *reinterpret_cast<const uint4*>(blk);
      const uint32_t scw = n ? (h.w & 0x0f0f0f0fu) | (((h.y >> 6) & 0x03030303u) << 4) : h.y & 0x3f3f3f3fu;   // of sub-blocks 4n .. 4n+3
      const uint32_t mnw = n ? ((h.w >> 4) & 0x0f0f0f0fu) | (((h.z >> 6) & 0x03030303u) << 4) : h.z & 0x3f3f3f3fu;
      const __half2 bias = __float2half2_rn(-1024.0f);
      __half2 s[4], c[4];    // even sub-blocks {sc, -1024 sc}, odd ones {sc / 16, -64 sc}
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const __half2 sc = __hadd2(bits_h2(__byte_perm(scw, 0x64646464u, 0x4040 | (f * 0x0101))), bias);
        s[f] = f & 1 ? __hmul2(sc, __float2half2_rn(0.0625f)) : sc;
        c[f] = __hmul2(sc, __float2half2_rn(f & 1 ? -64.0f : -1024.0f));
      }
      uint32_t sum[4] = {0u, 0u, 0u, 0u};   // of the masked words: 16 exponents and the quants of either lane
      auto expand = [&](int w, uint32_t* o, const uint4& a, const uint4& b) {   // words w & 3 of a (sub-blocks 4n, 4n+1) and b (4n+2, 4n+3)
        const uint32_t av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t u = e ? bv[w] : av[w], u8 = u >> 8;
          const uint32_t l0 = mask_or(u, low, k1024), l1 = mask_or(u8, low, k1024), h0 = mask_or(u, high, k1024), h1 = mask_or(u8, high, k1024);
          if constexpr (!kTable) {
            sum[2 * e] += l0 + l1;
            sum[2 * e + 1] += h0 + h1;
          }
          o[4 * e + 0] = expand2(l0, s[2 * e], c[2 * e]);
          o[4 * e + 1] = expand2(l1, s[2 * e], c[2 * e]);
          o[4 * e + 2] = expand2(h0, s[2 * e + 1], c[2 * e + 1]);
          o[4 * e + 3] = expand2(h1, s[2 * e + 1], c[2 * e + 1]);
        }
      };
      // a quarter's columns are free once the MMAs of the turn that used them last are done.  Not unrolled: six roles'
      // instructions share the caches
      const int prev = it - C::kOperands;
#pragma unroll 1
      for (int e = 0; e < 2; ++e) {
        const uint8_t* quants = blk + 16 + 64 * n + 16 * e;
        const uint4 a = *reinterpret_cast<const uint4*>(quants), b = *reinterpret_cast<const uint4*>(quants + 32);
        if (e == 1) {                          // the slot is read
          __syncwarp();
          mbar_arrive_if(lane == 0, r_free + 8 * slot);
        }
        uint32_t o[32];
#pragma unroll
        for (int w = 0; w < 4; ++w) expand(w, o + 8 * w, a, b);
        live = prev < 0 || mbar_wait(h_free + 8 * (4 * (prev & (C::kTurns - 1)) + 2 * n + e), (uint32_t)(prev / C::kTurns) & 1u, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        fence_after();
        tmem_st32(a_lane + (C::kOperands == 2 ? 128u * buf : 0u) + 32u * e, o);
        if (!kTable && e == 1) {
          // row meta: the slot's last readers, the epilogue of the turn two before prev, were done before the MMAs of prev
          // could be issued, and so were the mins' last readers, that turn's msum instructions
          {
            float t = 0.0f;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              const uint32_t pair = sum[f] - 16u * 0x64006400u;
              const int q = (int)((pair & 0xffffu) + (pair >> 16));
              t += (float)(((int)(scw >> (8 * f)) & 0xff) * (f & 1 ? q >> 4 : q));
            }
            uint8_t* rm = rowmeta + (rslot * BM + 32 * quarter + lane) * kRowMeta;
            if (n == 0) {
              const float d = h2f((uint16_t)(h.x & 0xffffu)), dm = -h2f((uint16_t)(h.x >> 16));
              *reinterpret_cast<float4*>(rm) = make_float4(d, d, dm, dm);
            }
            *reinterpret_cast<float2*>(rm + 16 + 8 * n) = make_float2(t, t);
            uint4 mv;
            mv.x = h2_bits(__hadd2(bits_h2(__byte_perm(mnw, 0x64646464u, 0x4040)), bias));
            mv.y = h2_bits(__hadd2(bits_h2(__byte_perm(mnw, 0x64646464u, 0x4141)), bias));
            mv.z = h2_bits(__hadd2(bits_h2(__byte_perm(mnw, 0x64646464u, 0x4242)), bias));
            mv.w = h2_bits(__hadd2(bits_h2(__byte_perm(mnw, 0x64646464u, 0x4343)), bias));
            *reinterpret_cast<uint4*>(mins + mslot * kMinsBytes + n * (BM * 16) + (32 * quarter + lane) * 16) = mv;
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the mins -> visible to the tensor core's reads
        }
        tmem_wait_st();
        fence_before();
        __syncwarp();
        mbar_arrive_if(lane == 0, h_full + 8 * (hb + e));
      }
      if (!live) break;
      if (++slot == C::kRawSlots) { slot = 0; rphase ^= 1u; }
      if (++mslot >= C::kMinsSlots) mslot = 0;
      if (++rslot >= C::kRowMetaSlots) rslot = 0;
    }
  } else if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kOtherRegs));
    // One lane issues, but the whole warp walks the loops, so that descriptors and addresses are worked out in uniform
    // registers.  D = f32, A = B = f16, both K-major, M = 128 weight rows, N = columns
    constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(BM >> 4) << 24);
    const bool leader = elect_one();
    bool live = true;
    if (warp < kLoaderWarp) {
      // -------------------------------------------------------------- MMA issue: a warp for either part of the columns, so that
      // the one's waits pass while the other's instructions run.  A part's accumulators have two buffers, its msum one:
      // when the epilogue has read the part of turn it - 1, msum of turn it and the accumulators of turn it + 1 are made
      constexpr uint32_t kIdescN = kIdesc | ((uint32_t)(C::kPart >> 3) << 17);
      const int s = warp - kMmaWarp;
      const uint64_t x0 = operand_desc(smem_u32(smem), kAtomBytes) + (uint64_t)((C::kPart / 8 * s * kAtomBytes) >> 4);
      const uint64_t sums0 = plain_desc(smem_u32(meta), TN * 16) + (uint64_t)(C::kPart * s);
      const uint64_t mins0 = plain_desc(smem_u32(kTable ? meta + C::kOffTable : mins), BM * 16);
      const uint32_t d0 = tmem_base + (uint32_t)(C::kPart * s);
      auto accumulate = [&](int it) {
        const int buf = it & 1, h0 = 4 * (it & (C::kTurns - 1));
        bool ok = true;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          ok = ok && mbar_wait(h_full + 8 * (h0 + q), (uint32_t)(it / C::kTurns) & 1u, abort_flag);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          fence_after();
          const uint64_t x = x0 + (uint64_t)((h0 + q) * (C::kQuarterBytes >> 4));
          const uint32_t a_op = tmem_base + C::kTmemA + (C::kOperands == 2 ? 128u * buf : 0u) + 32u * q;
          if (leader) {
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_f16(d0 + (uint32_t)(TN * buf), a_op + 8u * j, x + (uint64_t)(2 * j), kIdescN, (q | j) ? 1u : 0u);
            mma_commit(h_free + 8 * (h0 + q));
          }
          __syncwarp();
        }
        return ok;
      };
      const int my_turns = s < C::kParts ? turns : 0;
      int ms = 0, mslot = 0;
#pragma unroll 1
      for (int it = -1; live && it < my_turns; ++it) {
        if (it >= 0) {
          live = mbar_wait(s_free + 8 * s, ((uint32_t)it & 1u) ^ 1u, abort_flag);
          live = __all_sync(0xffffffffu, live);
          if (!live) break;
          fence_after();
          if (leader) {
            mma_f16_ss(d0 + C::kTmemM, mins0 + (uint64_t)((kTable ? ms * C::kMetaBytes : mslot * kMinsBytes) >> 4), sums0 + (uint64_t)(ms * C::kMetaBytes >> 4), kIdescN);
            mma_commit(s_full + 8 * s);
          }
          __syncwarp();
          if (++ms == kMetaSlots) ms = 0;
          if (++mslot >= C::kMinsSlots) mslot = 0;
        }
        if (it + 1 < my_turns) live = accumulate(it + 1);
      }
      if (!live && leader) {
        // gave up: let the tensor core finish what was issued before the TMEM goes away (bounded)
        mma_commit(drained + 8 * s);
        for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(drained + 8 * s, 0u); ++spins) {}
      }
    } else if (warp == kLoaderWarp) {
      // -------------------------------------------------------------- activations, a quarter super-block a copy, and weights
      const size_t stride = (size_t)(p.npad >> 3) * kAtomBytes;
      int kb = 0, tile = blockIdx.x, it = 0;
      const uint8_t* src = p.x + (size_t)((tile % nt) * (TN / 8)) * kAtomBytes;
      int wkb = 0, wtile = blockIdx.x, wslot = 0, asked = 0;
      uint32_t wphase = 1u;
      auto weights = [&]() {                   // of the next turn not asked for yet
        if (asked >= turns) return true;
        bool ok = mbar_wait(r_free + 8 * wslot, wphase, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (ok && leader) {
          mbar_arrive_expect_tx(r_full + 8 * wslot, kRawBytes);
          tma_load_2d(raw + wslot * kRawBytes, &wmap, wkb * Q4_K_BYTES, wtile / nt * BM, r_full + 8 * wslot);
        }
        __syncwarp();
        ++asked;
        if (++wslot == C::kRawSlots) { wslot = 0; wphase ^= 1u; }
        if (++wkb == nkb) { wkb = 0; wtile += gridDim.x; }
        return ok;
      };
      for (int i = 0; i < C::kRawSlots - 1; ++i) live = live && weights();
#pragma unroll 1
      for (; live && it < turns; ++it) {
        live = weights();
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          const int hq = 4 * (it & (C::kTurns - 1)) + q;
          const uint32_t full = h_full + 8 * hq;
          live = live && mbar_wait(h_free + 8 * hq, ((uint32_t)(it / C::kTurns) & 1u) ^ 1u, abort_flag);
          live = __all_sync(0xffffffffu, live);
          if (!live) break;
          if (leader) {
            mbar_arrive_expect_tx(full, C::kQuarterBytes);
            bulk_g2s(smem + hq * C::kQuarterBytes, src, C::kQuarterBytes, full);
          }
          __syncwarp();
          src += stride;
        }
        if (++kb == nkb) {
          kb = 0;
          tile += gridDim.x;
          src = p.x + (size_t)((tile % nt) * (TN / 8)) * kAtomBytes;
        }
      }
      if (!live && leader) {
        // gave up: let the copies in flight land (bounded).  A quarter's barrier also counts producers, who may have gone:
        // the copies' landing shows in its phase only if all came, so this waits out its bound otherwise
        for (int i = max(0, it - C::kTurns); i <= it; ++i)
          for (int q = 0; q < 4; ++q)
            for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(h_full + 8 * (4 * (i & (C::kTurns - 1)) + q), (uint32_t)(i / C::kTurns) & 1u); ++spins) {}
        for (int i = max(0, asked - C::kRawSlots); i < asked; ++i)
          for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(r_full + 8 * (i % C::kRawSlots), (uint32_t)(i / C::kRawSlots) & 1u); ++spins) {}
      }
    } else {
      // -------------------------------------------------------------- block sums, scales and table of a super-block
      int kb = 0, tile = blockIdx.x, it = 0, ms = 0;
      uint32_t phase = 1u;
#pragma unroll 1
      for (; it < turns; ++it) {
        const int hq = 4 * (it & (C::kTurns - 1)) + 3;
        const uint32_t full = h_full + 8 * hq;
        live = mbar_wait(m_free + 8 * ms, phase, abort_flag);
        // the barrier's phase before this one is over once the accumulators of turn it - kTurns are complete
        live = live && mbar_wait(h_free + 8 * hq, ((uint32_t)(it / C::kTurns) & 1u) ^ 1u, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        if (leader) {
          const int tm = tile / nt, c0 = (tile - tm * nt) * TN;
          uint8_t* cm = meta + ms * C::kMetaBytes;
          mbar_arrive_expect_tx(full, C::kMetaBytes);
#pragma unroll
          for (int c = 0; c < 2; ++c) bulk_g2s(cm + c * TN * 16, p.sums + (((size_t)kb * 2 + c) * p.npad + c0) * 16, TN * 16, full);
          bulk_g2s(cm + C::kOffPairs, p.pairs + ((size_t)kb * (p.npad >> 1) + (c0 >> 1)) * kPairBytes, TN / 2 * kPairBytes, full);
          if (kTable) bulk_g2s(cm + C::kOffTable, p.table + ((size_t)tm * nkb + kb) * kTableBytes, kTableBytes, full);
        }
        __syncwarp();
        if (++ms == kMetaSlots) { ms = 0; phase ^= 1u; }
        if (++kb == nkb) { kb = 0; tile += gridDim.x; }
      }
      if (!live && leader) {
        for (int i = max(0, it - C::kTurns); i <= it; ++i)
          for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(h_full + 8 * (4 * (i & (C::kTurns - 1)) + 3), (uint32_t)(i / C::kTurns) & 1u); ++spins) {}
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- epilogue
    // TMEM lanes are weight rows, TMEM columns the product's columns.  The warp owns 32 rows (its lane quarter) and of every
    // column part one half, a thread one row: its d, -dmin and T stay in registers, the columns' dx and v come as
    // broadcasts.  (TMEM loads of whole lanes take half a cycle a register, those in the m16n8 fragment layout two.)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kEpilogueRegs));
    constexpr int kMine = C::kPart / 2, kLoads = kMine / 8;        // columns of a part; loads of eight
    static_assert(kLoads % 2 == 0, "rows leave 16 columns at a time");
    const int quarter = warp & 3, side = (warp - kEpilogueWarp0) >> 2;
    const uint32_t tb = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(kMine * side), lead = lane == 0;
    int ms = 0, rslot = 0, it = 0;
    bool live = true;
    for (int tile = blockIdx.x; live && tile < ntiles; tile += gridDim.x) {
      f2 acc[C::kParts][kLoads][4];       // [part][load][column pair]
#pragma unroll
      for (int i = 0; i < 4 * kLoads * C::kParts; ++i) acc[i / (4 * kLoads)][(i >> 2) % kLoads][i & 3] = 0ull;
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const uint8_t* cm = meta + ms * C::kMetaBytes + C::kOffPairs + kMine / 2 * side * kPairBytes;
        const uint8_t* rmeta = kTable ? meta + ms * C::kMetaBytes + C::kOffTable + kMinsBytes + (32 * quarter + lane) * kTableRow
                                      : rowmeta + (rslot * BM + 32 * quarter + lane) * kRowMeta;
        const uint32_t parity = (uint32_t)it & 1u;
        f2 dw, ndm, tq;          // d, -dmin, T of the row, each twice
#pragma unroll
        for (int s = 0; s < C::kParts; ++s) {
          const uint32_t td = tb + TN * parity + C::kPart * s, tm = tb + C::kTmemM + C::kPart * s;
          // after a wait that gave up the turn's arithmetic is nonsense, which nobody stores
          live = mbar_wait(s_full + 8 * s, parity, abort_flag) && live;
          __syncwarp();
          fence_after();
          uint32_t dv[2][8], sv[2][8];
          tmem_ld8(td, dv[0]);
          tmem_ld8(tm, sv[0]);
          if (s == 0) {
            if constexpr (kTable) {
              const f2* m = reinterpret_cast<const f2*>(rmeta);
              dw = m[0];
              ndm = m[1];
              tq = m[2];
            } else {
              const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(rmeta), tt = *reinterpret_cast<const ulonglong2*>(rmeta + 16);
              dw = m.x;
              ndm = m.y;
              tq = add2(tt.x, tt.y);
            }
          }
#pragma unroll
          for (int i = 0; i < kLoads; ++i) {
            tmem_wait_ld(dv[i & 1], sv[i & 1]);
            if (i + 1 == kLoads) {
              fence_before();
              __syncwarp();
              mbar_arrive_if(lead, s_free + 8 * s);
            } else {
              tmem_ld8(td + 8u * (i + 1), dv[(i + 1) & 1]);
              tmem_ld8(tm + 8u * (i + 1), sv[(i + 1) & 1]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const ulonglong2 cv = *reinterpret_cast<const ulonglong2*>(cm + (C::kPart / 2 * s + 4 * i + q) * kPairBytes);   // dx, dx, v, v
              const f2 isum = fma2(cv.y, tq, pack2u(dv[i & 1][2 * q], dv[i & 1][2 * q + 1]));
              const f2 off = mul2(mul2(cv.x, ndm), pack2u(sv[i & 1][2 * q], sv[i & 1][2 * q + 1]));
              acc[s][i][q] = add2(acc[s][i][q], fma2(mul2(cv.x, dw), isum, off));
            }
          }
        }
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        mbar_arrive_if(lead, m_free + 8 * ms);
        if (++ms == kMetaSlots) ms = 0;
        if (++rslot >= C::kRowMetaSlots) rslot = 0;
      }
      if (!live) break;
      // rows leave through shared memory, 16 columns at a time, four lanes a row: 64 bytes of a row side by side (16 bytes
      // of 32 rows an instruction took twice as long, and longer than the pairs of the fragment layout)
      const int tm = tile / nt, r0 = tm * BM + 32 * quarter, j = lane & 3;
      uint8_t* stage = smem + C::kOffStage + (warp - kEpilogueWarp0) * 32 * kStageRow;
      const bool aligned = rows_aligned(p);
#pragma unroll
      for (int s = 0; s < C::kParts; ++s)
#pragma unroll
        for (int i = 0; i < kLoads; i += 2) {
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 4; ++e)
            *reinterpret_cast<ulonglong2*>(stage + lane * kStageRow + 16 * e) = make_ulonglong2(acc[s][i + (e >> 1)][2 * (e & 1)], acc[s][i + (e >> 1)][2 * (e & 1) + 1]);
          __syncwarp();
          const int c = (tile - tm * nt) * TN + C::kPart * s + kMine * side + 8 * i + 4 * j;
          // Other strides: single floats, 16 of a row side by side (four floats a lane: 14336 x 1024 by 333 52, so 48 us).  Not with
          // the table, whose products are long: there the code in its way takes 0.6 % of 14336 x 4096 by 2048
          if (!kTable && !aligned) {
            const int cc = c - 4 * j + (lane & 15);
            if (cc < p.N)
#pragma unroll 1
              for (int row = lane >> 4; row < 32 && r0 + row < p.M; row += 2) p.y[(size_t)(r0 + row) * p.ldy + cc] = *reinterpret_cast<const float*>(stage + row * kStageRow + 4 * (lane & 15));
            continue;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int row = r0 + 8 * k + (lane >> 2);
            const float4 v = *reinterpret_cast<const float4*>(stage + (8 * k + (lane >> 2)) * kStageRow + 16 * j);
            if (row >= p.M) continue;
            float* yr = p.y + (size_t)row * p.ldy + c;
            if (aligned && c + 3 < p.N) {
              *reinterpret_cast<float4*>(yr) = v;
            } else {
              if (c < p.N) yr[0] = v.x;
              if (c + 1 < p.N) yr[1] = v.y;
              if (c + 2 < p.N) yr[2] = v.z;
              if (c + 3 < p.N) yr[3] = v.w;
            }
          }
        }
    }
  }

  fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, 1);
  if (warp == kMmaWarp) {
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

// the workspace's columns: whole tiles, whole pre-pass blocks
int padded_columns(int ncols) { return ncols <= 64 ? 64 : (ncols + 127) / 128 * 128; }

}  // namespace


size_t operand_layout_bytes(int K, int npad) { return (size_t)npad * (size_t)(K / QK_K) * (2 * QK_K + kSumBytes + kPairBytes / 2); }

OperandLayout operand_layout(uint8_t* workspace, int K, int npad) {
  const size_t columns = (size_t)(K / QK_K) * npad;
  OperandLayout o;
  o.x = workspace;
  o.sums = o.x + columns * (2 * QK_K);
  o.pairs = o.sums + columns * kSumBytes;
  return o;
}

cudaError_t launch_operand_layout(const ActPlanes& act, int col0, int ncols, int npad, int K, const OperandLayout& out, bool centre, cudaStream_t st) {
  operand_layout_kernel<<<dim3(K / QK_K, npad / kPreCols), 256, 0, st>>>(act, col0, ncols, npad, centre, out.x, out.sums, out.pairs);
  return cudaGetLastError();
}

bool planes_aligned(const ActPlanes& act) {
  return act.bsums != nullptr && (reinterpret_cast<uintptr_t>(act.qs) & 15) == 0 && act.col_stride_qs % 16 == 0 &&
         (reinterpret_cast<uintptr_t>(act.bsums) & 15) == 0 && act.col_stride_bs % 8 == 0;
}

size_t gemm_tc_workspace_bytes(int K, int ncols) { return operand_layout_bytes(K, padded_columns(ncols)); }

bool gemm_tc_supported(int type, int K, int ncols, const void* W, int64_t row_bytes, const ActPlanes& act) {
  return type == T_Q4_K && ncols >= kGemmTcMinCols && K % QK_K == 0 && (reinterpret_cast<uintptr_t>(W) & 15) == 0 && row_bytes % 16 == 0 &&
         row_bytes < (1 << 27) && planes_aligned(act);
}

namespace {

// the weights as bytes {rows, K/256 * 144}, boxes of 128 rows x one block
bool encode_rows(CUtensorMap* map, const GemvArgs& a) {
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  const cuuint64_t dims[2] = {(cuuint64_t)(a.K / QK_K) * Q4_K_BYTES, (cuuint64_t)a.M}, strides[1] = {(cuuint64_t)a.row_bytes};
  const cuuint32_t box[2] = {Q4_K_BYTES, BM}, estr[2] = {1, 1};
  return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(a.W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int TN, bool kTable>
cudaError_t launch_tiles(const GemmArgs& g, const CUtensorMap& wmap, int sm_count, cudaStream_t st) {
  constexpr int kSmem = Cfg<TN, kTable>::kSmemBytes;
  // per host thread (one context, one lane per thread): no shared mutable state between lanes
  static thread_local unsigned configured = 0;  // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_q4k_tc_kernel<TN, kTable>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  const int tiles = ((g.M + BM - 1) / BM) * ((g.N + TN - 1) / TN);
  gemm_q4k_tc_kernel<TN, kTable><<<tiles < sm_count ? tiles : sm_count, kThreads, kSmem, st>>>(g, wmap);
  return cudaGetLastError();
}

// Columns per tile, and whether a table of the rows is made first: what takes the least time by a model of hundredths of a us.  A
// wave of CTAs takes a start and a time per super-block; the table is a launch and a pass over the weights, and saves a part
// of every wave and super-block.  Fitted to 190 calls of 3000 to 32000 rows, K of 256 to 4096 and 32 to 1900 columns, of which it takes
// six 3 to 8 % longer than the best does.  us, tiles of 32, 64, 128 without and 128 with table: 14336 x 256 by 160 columns 24.3, 24.5, 26.5,
// 29.4; 6500 x 768 by 256 30.7, 27.9, 25.6, 29.7; 4096 x 1024 by 512 39.9, 31.7, 27.6, 31.8; 14336 x 2048 by 333 109, 78.9, 68.7, 70.7, by 1900 472, 280,
// 199, 191; 4096 x 14336, one wave, 78, 88 and (table) 97
struct Plan {
  int columns;
  bool table;
};
Plan plan_tiles(int M, int K, int ncols, int call_columns, int sm_count, bool table_fits, bool aligned) {
  const int64_t mt = (M + BM - 1) / BM, nkb = K / QK_K;
  auto waves = [&](int tn) { return (mt * ((ncols + tn - 1) / tn) + sm_count - 1) / sm_count; };
  const int64_t c32 = waves(32) * (45 + 119 * nkb), c64 = waves(64) * (90 + 132 * nkb);
  const int64_t saved = waves(128) * (18 + 12 * nkb) - 320 - mt * nkb * 26 / 100;
  // calls of 1024 column tiles and more make the table either way, in each of their turns: its launches are 2 % of them at most
  if (table_fits && call_columns > 1023 * 128 && ncols > 64) return Plan{128, true};
  // strides of no 16 bytes: the kernels without table store them better (14336 x 256 by 1901 83, with table 96)
  const bool table = table_fits && saved > 0 && (aligned || nkb > 4);
  const int64_t c128 = waves(128) * (190 + 162 * nkb) - (table ? saved : 0);
  if (ncols > 64 && c128 <= c64 && c128 <= c32) return Plan{128, table};
  return Plan{c64 <= c32 ? 64 : 32, false};
}

// columns of a turn: what the workspace holds, and a grid's y extent; ncols where one turn takes all
int turn_columns(const GemvArgs& a, int ncols) {
  const size_t groups = a.tc_ws_bytes / gemm_tc_workspace_bytes(a.K, 128);
  const int fit = (int)(groups < 32767 ? groups : 32767) * 128;
  return fit >= ncols || (ncols <= 64 && fit == 0) ? ncols : fit;   // a single group of 64 columns may fit where 128 do not
}

}  // namespace

bool gemm_q4k_tc_one_turn(const GemvArgs& a, int ncols) { return turn_columns(a, ncols) == ncols; }

// launches: the activation pre-pass (into the workspace), the pre-pass over the weights where it pays and its results fit beside
// the columns, and the product; the three again for columns whose operand the workspace does not hold beside the others'.  (A
// table never sends columns to another turn: what a turn holds follows from K and the columns alone, for every matrix of an
// input.)
cudaError_t launch_gemm_q4k_tc(const GemvArgs& a, int ncols, int sm_count, cudaStream_t st, int* launches) {
  GemmArgs g{};
  g.M = a.M;
  g.K = a.K;
  g.ldy = a.ldy;
  g.status = a.status;
  const int nkb = a.K / QK_K, mt = (a.M + BM - 1) / BM, fit = turn_columns(a, ncols);
  CUtensorMap wmap;
  if (!encode_rows(&wmap, a)) return cudaErrorNotSupported;
  for (int c = 0; c < ncols; c += fit) {
    g.N = ncols - c < fit ? ncols - c : fit;
    g.npad = padded_columns(g.N);
    g.y = a.y + a.col0 + c;
    const OperandLayout x = operand_layout(a.tc_ws, a.K, g.npad);
    const size_t used = operand_layout_bytes(a.K, g.npad);
    uint8_t* table = a.tc_ws + used;
    g.x = x.x;
    g.sums = x.sums;
    g.pairs = x.pairs;
    g.table = table;
    cudaError_t e = cudaSuccess;
    if (!a.tc_ws_reuse || fit < ncols) {  // else the workspace still holds these planes in operand order (same K, columns, col0)
      e = launch_operand_layout(a.act, a.col0 + c, g.N, g.npad, a.K, x, true, st);
      ++*launches;
      if (e != cudaSuccess) return e;
    }
    const Plan plan = plan_tiles(a.M, a.K, g.N, ncols, sm_count, used + (size_t)mt * nkb * kTableBytes <= a.tc_ws_bytes && mt <= 65535, rows_aligned(g));
    if (plan.table) {
      q4k_table_kernel<<<dim3(nkb, mt), BM, 0, st>>>(a.W, a.row_bytes, a.M, table);
      ++*launches;
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      e = launch_tiles<128, true>(g, wmap, sm_count, st);
    } else {
      e = plan.columns == 128 ? launch_tiles<128, false>(g, wmap, sm_count, st)
          : plan.columns == 64 ? launch_tiles<64, false>(g, wmap, sm_count, st) : launch_tiles<32, false>(g, wmap, sm_count, st);
    }
    ++*launches;
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace emelb
