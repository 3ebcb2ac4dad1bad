// Q6_K x Q8_K matrix product for many columns (prompt processing) on the Blackwell tensor cores: tcgen05.mma kind::f16,
// weights as the A operand in TMEM, activations as the B operand in shared memory, f32 accumulators in TMEM that only
// ever hold exact integers.
//
// What is computed is exactly the reference's per-super-block value (src/emel/kernel/x86_64/actions.hpp:1036-1077)
//   (dx*d) * (float)isum,  isum = sum_g sc_g * dot16_g(q - 32, x)
// added in ascending block order, so the result equals the mat-vec kernels' (and the x86 AVX2 route's) bit for bit.
// A weight times its scale is a small integer, and f16 operands with f32 sums are exact as long as every partial sum
// of a super-block stays below 2^24.  (q - 32) * sc needs 13 bits, f16 holds 11, so sc = 16 * hi + lo with
// |hi|, |lo| <= 8 and two operands of |.| <= 256 each: |sum| <= 256 * 128 * 256 = 2^23 in any order of addition, and
// (float)isum = fma(16, D_hi, D_lo), one rounding.
// The expanded weights pass through neither the shared memory nor its port: a thread owns a weight row = a TMEM lane
// and writes the operand with tcgen05.st.  Expanding two weights is one mask and one half2 fma: the masked 6-bit
// quants are f16 subnormals q * 2^-24, times piece * 2^10 plus -32 * piece * 2^-14 is (q - 32) * piece * 2^-14 without a
// rounding; the factor 2^14 returns in the fma that joins the pieces.  The order of a super-block's 256 weights along
// the MMA's K is free (the sums are exact), so it follows from the masks; a pre-pass lays the activations out alike.
//
// CTA = 128 weight rows (TMEM lanes) x TN columns (32 or 64), one super-block of K per turn, 20 warps:
//   warps 0-7   producers: two warps per TMEM lane quarter, one for each half (128 weights) of a super-block; what a
//               half needs of the GGUF blocks of the warp's 32 rows comes by cp.async two turns ahead (ring of three,
//               no barrier beyond the warp), a thread expands its row's half into TMEM
//   warps 8-15  epilogue: two warps per TMEM lane quarter, TN/2 columns each, accumulators read in the m16n8 fragment
//               layout, the float chain on packed f32x2 instructions
//   warp  16    one elected thread: MMA issue; TMEM allocation
//   warp  17    one thread: bulk copies of the activations (by half super-blocks) and of their scales
// TMEM: two turns' accumulators (lo and hi, TN columns each), operands lo and hi of one turn, handed over in halves.
// Registers are split by setmaxnreg: 640 threads x 96 at launch = 256 x 80 + 256 x 136 + 128 x 48.
// Every mbarrier wait is bounded; on a timeout the CTA raises the status word, lets its copies land and frees its TMEM.
//
// What bounds it: the producers, a chain of dependent steps of about 3,400 cycles a turn, of which the copies into the ring
// (256 cp.async of a row each a turn) are a large part: as many as twice, for 16 producer warps with a quarter each, made the
// turn 25 % longer, addresses that step from row to row instead of a product and a minimum per copy 8 % shorter; scales taken
// apart two in a half2 and odd bytes by a permutation 4 %.  The MMAs take 1040 (64 columns).  Measured, B200, us a
// call: 4096 x 11008 by 77 columns 66.3 -> 60.2 (a call by itself; one behind the other 105 -> 93), 14336 x
// 11008 by 200 414 -> 363, 11008 x 4096 by 77 82 -> 74, 14336 x 2816 by 16 35.5 -> 31.3.
// Dispatch: K and rows that the streaming kernels and gemm_q6k_mma.cu do not take (their copies need rows of a multiple
// of 16 bytes, K % 2048 == 0), up to the columns where gemm_q6k_wide.cu, which unpacks the blocks once for all column tiles,
// is the cheaper one (its line is there).  Rows that both take are faster there with few columns (4096 x 14336 by 32: 124 + 3
// against 99; by 8 127 against the mat-vec kernels' 60, by 5 127 against 49), so those kernels keep their sizes.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace emelb {
namespace {

using namespace tc;

constexpr int BM = 128;
constexpr int kEpilogueWarp0 = 8, kEpilogueWarps = 8, kMmaWarp = 16, kLoaderWarp = 17;
constexpr int kThreads = 20 * 32;
constexpr int kProducerRegs = 80, kEpilogueRegs = 136, kOtherRegs = 48;
static_assert(8 * 32 * kProducerRegs + 8 * 32 * kEpilogueRegs + 4 * 32 * kOtherRegs <= kThreads * 96, "register split");

// activations in the workspace, and in shared memory: half super-blocks of 128 K, 8-column groups of two swizzle atoms
constexpr int kGroupBytes = 2 * kAtomBytes;             // one 8-column group of a half
constexpr int kColPad = 64;                             // the workspace's columns come in groups: whole tiles, whole pre-pass blocks

constexpr int kMaxTN = 64, kHalves = 6;
// a row's half of a raw block: 17 words of ql, 9 of qh, 3 of scales, the word of d; an odd number: rows on all 32 banks
constexpr int kRawRow = 124, kRawSlots = 3, kRowMetaSlots = 4, kColMetaSlots = 3;
constexpr int kHalfBytes = kMaxTN / 8 * kGroupBytes;

// shared memory map
constexpr int kOffRaw = kHalves * kHalfBytes;
constexpr int kOffRowMeta = kOffRaw + kRawSlots * 2 * BM * kRawRow;      // [slot][row]: d
constexpr int kOffColMeta = kOffRowMeta + kRowMetaSlots * BM * 4;        // [slot][column]: dx
constexpr int kOffBars = kOffColMeta + kColMetaSlots * kMaxTN * 4;
constexpr int kSmemBytes = kOffBars + 256 + 1024;   // barriers; slack for the base's alignment

constexpr uint32_t kTmemA = 256;   // first operand column

struct GemmArgs {
  const uint8_t* W;
  int64_t row_bytes;
  int M, K, N, TN;
  const uint8_t* x;       // [K/128][npad/8] 8-column groups
  const float* dx;        // [K/256][npad]
  int npad;
  float* y;
  int64_t ldy;
  int* status;
};

// pre-pass: the quantized activation planes of columns col0.. -> operand order.  K position 128 n + 16 w + 8 c + j of
// a super-block holds element 128 n + 64 c + 32 (j / 4) + 4 w + {0, 2, 1, 3}[j % 4], which is what the producers'
// masks leave side by side.  grid (K/256, ceil(N/64)), 256 threads; columns past N are zero.
constexpr int kPreCols = kColPad, kPreRow = QK_K + 4;   // 65 words: column-wise reads fall on all banks

__global__ void __launch_bounds__(256) tile_activations_f16_kernel(ActPlanes act, int col0, int N, int npad, uint8_t* x, float* dx) {
  __shared__ __align__(16) uint8_t t8[kPreCols * kPreRow];
  const int kb = blockIdx.x, c0 = blockIdx.y * kPreCols;
  for (int q = threadIdx.x; q < kPreCols * 16; q += 256) {
    const int col = q >> 4, piece = q & 15;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (c0 + col < N) v = *reinterpret_cast<const uint4*>(act.qs + (int64_t)(col0 + c0 + col) * act.col_stride_qs + kb * QK_K + 16 * piece);
    uint32_t* o = reinterpret_cast<uint32_t*>(t8 + col * kPreRow + 16 * piece);
    o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
  __syncthreads();
  auto halves = [](uint32_t w, uint32_t& even, uint32_t& odd) {   // four int8 -> f16 {0, 2}, {1, 3}
    const uint32_t u = w ^ 0x80808080u;
    const __half2 bias = __float2half2_rn(-1152.0f);
    even = h2_bits(__hadd2(bits_h2((u & 0x00ff00ffu) | 0x64006400u), bias));
    odd = h2_bits(__hadd2(bits_h2(((u >> 8) & 0x00ff00ffu) | 0x64006400u), bias));
  };
  for (int q = threadIdx.x; q < kPreCols * 32; q += 256) {
    const int col = q & (kPreCols - 1), ch = q >> 6;               // chunk ch of 8 K positions
    const int n = ch >> 4, w = (ch >> 1) & 7, c = ch & 1;
    const uint8_t* s = t8 + col * kPreRow + 128 * n + 64 * c + 4 * w;
    uint4 o;
    halves(*reinterpret_cast<const uint32_t*>(s), o.x, o.y);
    halves(*reinterpret_cast<const uint32_t*>(s + 32), o.z, o.w);
    uint8_t* dst = x + ((size_t)(2 * kb + n) * (npad >> 3) + ((c0 + col) >> 3)) * kGroupBytes + ((ch >> 3) & 1) * kAtomBytes +
                   (col & 7) * 128 + (((ch ^ col) & 7) << 4);
    *reinterpret_cast<uint4*>(dst) = o;
  }
  if (threadIdx.x < kPreCols) {
    const int col = c0 + threadIdx.x;
    dx[(size_t)kb * npad + col] = col < N ? act.d[(int64_t)(col0 + col) * act.col_stride_d + kb] : 0.0f;
  }
}

__global__ void __launch_bounds__(kThreads, 1) gemm_q6k_tc_kernel(const GemmArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw = smem + kOffRaw;
  uint8_t* rowmeta = smem + kOffRowMeta;
  uint8_t* colmeta = smem + kOffColMeta;
  const uint32_t bars = smem_u32(smem + kOffBars);
  const uint32_t a_full = bars;                      // [2 halves] producers -> MMA
  const uint32_t a_free = a_full + 8 * 2;
  const uint32_t x_full = a_free + 8 * 2;            // [kHalves] bulk copies -> MMA
  const uint32_t x_free = x_full + 8 * kHalves;
  const uint32_t m_full = x_free + 8 * kHalves;      // [3] bulk copies -> epilogue: the columns' scales of a super-block
  const uint32_t m_free = m_full + 8 * kColMetaSlots;
  const uint32_t d_full = m_free + 8 * kColMetaSlots;   // [2] MMA -> epilogue: the accumulators hold a finished super-block
  const uint32_t d_free = d_full + 8 * 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBars + 8 * (8 + 2 * kHalves + 2 * kColMetaSlots));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int TN = p.TN;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) { mbar_init(a_full + 8 * s, 4); mbar_init(a_free + 8 * s, 1); }
    for (int s = 0; s < kHalves; ++s) { mbar_init(x_full + 8 * s, 1); mbar_init(x_free + 8 * s, 1); }
    for (int s = 0; s < kColMetaSlots; ++s) { mbar_init(m_full + 8 * s, 1); mbar_init(m_free + 8 * s, kEpilogueWarps); }
    for (int s = 0; s < 2; ++s) { mbar_init(d_full + 8 * s, 1); mbar_init(d_free + 8 * s, kEpilogueWarps); }
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
  const uint32_t tmem_base = *tmem_slot;

  const int mt = (p.M + BM - 1) / BM, nt = (p.N + TN - 1) / TN, ntiles = mt * nt, nkb = p.K / QK_K;
  const int my_tiles = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int turns = my_tiles * nkb;   // super-blocks this CTA walks

  if (warp < 8) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
    const int quarter = warp & 3, n = warp >> 2;   // TMEM lanes 32 * quarter .., half n of every super-block
    const uint32_t a_lane = tmem_base + kTmemA + ((uint32_t)(32 * quarter) << 16) + 64u * n;
    uint8_t* const raw0 = raw + (n * BM + 32 * quarter) * kRawRow;
    constexpr int kSlotBytes = 2 * BM * kRawRow;
    int itile = blockIdx.x, ikb = 0, islot = 0;    // the turn staged next
    auto issue_raw = [&](int it) {
      if (it < turns) {
        const int r0 = (itile / nt) * BM + 32 * quarter;
        uint8_t* dst = raw0 + islot * kSlotBytes;
        // blocks start at any even byte: a half needs up to 30 of the 53 aligned words that cover its block, one a lane
        const int word = lane < 17 ? 16 * n + lane : lane < 26 ? 32 + 8 * n + lane - 17 : lane < 29 ? 48 + 2 * n + lane - 26 : 52;
        if (lane < 30) {
          // two rows a step: rows may start at odd halves of a word, every other one in the same way.  Rows past M repeat the
          // last one or the one before; never stored
          const int last = p.M - 1 - r0;
          const uintptr_t first = reinterpret_cast<uintptr_t>(p.W) + (size_t)min(r0, p.M - 1) * p.row_bytes + (size_t)ikb * Q6_K_BYTES;
          uintptr_t s0 = (first & ~uintptr_t(3)) + 4 * word, s1 = ((first + (last > 0 ? p.row_bytes : 0)) & ~uintptr_t(3)) + 4 * word;
          const uint32_t d = smem_u32(dst) + 4 * lane;
#pragma unroll 4
          for (int rr = 0; rr < 32; rr += 2) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + rr * kRawRow), "l"(s0) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + (rr + 1) * kRawRow), "l"(s1) : "memory");
            if (rr + 3 <= last) {
              s0 += 2 * p.row_bytes;
              s1 += 2 * p.row_bytes;
            } else if (rr + 2 <= last) {
              s0 += 2 * p.row_bytes;
            }
          }
        }
        if (++ikb == nkb) { ikb = 0; itile += gridDim.x; }
        if (++islot == kRawSlots) islot = 0;
      }
      cp_async_commit();
    };
    issue_raw(0);
    issue_raw(1);
    int tile = blockIdx.x, kb = 0, slot = 0;
    bool live = true;
    for (int it = 0; it < turns; ++it) {
      issue_raw(it + 2);     // into the slot of turn it - 1
      cp_async_wait<2>();
      __syncwarp();
      const uint8_t* blk = raw0 + slot * kSlotBytes + lane * kRawRow;
      uint8_t* rm = rowmeta + ((it & (kRowMetaSlots - 1)) * BM + 32 * quarter + lane) * 4;
      const int row = min((tile / nt) * BM + 32 * quarter + lane, p.M - 1);
      const uint32_t sh = (uint32_t)((reinterpret_cast<uintptr_t>(p.W) + (size_t)row * p.row_bytes + (size_t)kb * Q6_K_BYTES) & 2) * 8;
      const uint32_t* bw = reinterpret_cast<const uint32_t*>(blk);
      auto word = [&](int i) { return __funnelshift_r(bw[i], bw[i + 1], sh); };   // i: 0 ql, 17 qh, 26 scales of the half
      const uint32_t sw[2] = {word(26), word(27)};   // the half's eight scales
      live = mbar_wait(a_free + 8 * n, (it & 1) ^ 1, abort_flag);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      fence_after();
      // the slot's last readers were done before the MMAs of turn it - 1 could be issued
      if (n == 0) *reinterpret_cast<uint32_t*>(rm) = sh ? bw[29] >> 16 : bw[29] & 0xffffu;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        // weights 16q .. 16q+15 of each 32: scale 2f + q of the half for form f, two forms in a half2.  sc + 136 = 16 (hi + 8) +
        // (lo + 8), with 1024 in front each part is an f16
        __half2 sl[2], cl[2], sh2[2], ch[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t u = (((sw[e] >> (8 * q)) & 0x00ff00ffu) ^ 0x00800080u) + 0x00080008u;
          const __half2 lo = __hsub2(bits_h2((u & 0x000f000fu) | 0x64006400u), __float2half2_rn(1032.0f));
          const __half2 hi = __hsub2(bits_h2(((u >> 4) & 0x001f001fu) | 0x64006400u), __float2half2_rn(1032.0f));
          sl[e] = __hmul2(lo, __float2half2_rn(1024.0f));
          cl[e] = __hmul2(lo, __float2half2_rn(-0.001953125f));   // -32 * 2^-14
          sh2[e] = __hmul2(hi, __float2half2_rn(1024.0f));
          ch[e] = __hmul2(hi, __float2half2_rn(-0.001953125f));
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t ol[8], oh[8];
          const int i = 4 * q + w;
          const uint32_t qa = word(i), qb = word(8 + i), qh = word(17 + i);
          const uint32_t v[4] = {(qa & 0x0f0f0f0fu) | ((qh << 4) & 0x30303030u), (qb & 0x0f0f0f0fu) | ((qh << 2) & 0x30303030u),
                                 ((qa >> 4) & 0x0f0f0f0fu) | (qh & 0x30303030u), ((qb >> 4) & 0x0f0f0f0fu) | ((qh >> 2) & 0x30303030u)};
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const uint32_t e = v[f] & 0x00ff00ffu, d = __byte_perm(v[f], 0, 0x4341);
            const __half2 l = f & 1 ? __high2half2(sl[f >> 1]) : __low2half2(sl[f >> 1]), lc = f & 1 ? __high2half2(cl[f >> 1]) : __low2half2(cl[f >> 1]);
            const __half2 h = f & 1 ? __high2half2(sh2[f >> 1]) : __low2half2(sh2[f >> 1]), hc = f & 1 ? __high2half2(ch[f >> 1]) : __low2half2(ch[f >> 1]);
            ol[2 * f] = expand2(e, l, lc);
            ol[2 * f + 1] = expand2(d, l, lc);
            oh[2 * f] = expand2(e, h, hc);
            oh[2 * f + 1] = expand2(d, h, hc);
          }
          tmem_st8(a_lane + 8u * i, ol);
          tmem_st8(a_lane + 128u + 8u * i, oh);
        }
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full + 8 * n);
      if (++slot == kRawSlots) slot = 0;
      if (++kb == nkb) { kb = 0; tile += gridDim.x; }
    }
    cp_async_wait<0>();
  } else if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    if (warp == kMmaWarp && elect_one()) {
      // -------------------------------------------------------------- MMA issue (one thread)
      // D = f32, A = B = f16, both K-major, M = 128 weight rows, N = TN columns
      const uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint64_t x0 = operand_desc(smem_u32(smem), kGroupBytes);
      bool live = true, issued = false;
      int last = 0, xs = 0, xphase = 0;
      for (int it = 0; live && it < turns; ++it) {
        const int buf = it & 1;
        const uint32_t d = tmem_base + (uint32_t)(2 * TN * buf);
        live = mbar_wait(d_free + 8 * buf, ((it >> 1) & 1) ^ 1, abort_flag);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (!live) break;
          live = mbar_wait(a_full + 8 * n, (uint32_t)it & 1u, abort_flag) && mbar_wait(x_full + 8 * xs, xphase, abort_flag);
          if (!live) break;
          fence_after();
          const uint64_t x = x0 + (uint64_t)(xs * (kHalfBytes >> 4));
          const uint32_t a_op = tmem_base + kTmemA + 64u * n;
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int j = 0; j < 8; ++j)
              mma_f16(d + (uint32_t)(r * TN), a_op + 128u * r + 8u * j, x + (uint64_t)(((j >> 2) * kAtomBytes + (j & 3) * 32) >> 4), idesc,
                      (n | j) ? 1u : 0u);
          mma_commit(a_free + 8 * n);
          mma_commit(x_free + 8 * xs);
          if (++xs == kHalves) { xs = 0; xphase ^= 1; }
          issued = true;
        }
        if (issued) {
          mma_commit(d_full + 8 * buf);
          last = it;
        }
      }
      if (!live && issued) {
        // gave up: let the tensor core finish what was issued before the TMEM goes away (bounded)
        for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(d_full + 8 * (last & 1), (uint32_t)(last >> 1) & 1u); ++spins) {}
      }
    } else if (warp == kLoaderWarp && lane == 0) {
      // -------------------------------------------------------------- activation loader (one thread)
      bool live = true;
      int xs = 0, xphase = 0, ms = 0, mphase = 0, sent_x = 0, sent_m = 0;
      const uint32_t xbytes = (uint32_t)(TN / 8) * kGroupBytes, dbytes = (uint32_t)TN * 4;
      int tile = blockIdx.x, kb = 0;
      for (int it = 0; live && it < turns; ++it) {
        const int c0 = (tile % nt) * TN;
        for (int n = 0; live && n < 2; ++n) {
          live = mbar_wait(x_free + 8 * xs, xphase ^ 1, abort_flag);
          if (!live) break;
          mbar_arrive_expect_tx(x_full + 8 * xs, xbytes);
          bulk_g2s(smem + xs * kHalfBytes, p.x + ((size_t)(2 * kb + n) * (p.npad >> 3) + (c0 >> 3)) * kGroupBytes, xbytes, x_full + 8 * xs);
          ++sent_x;
          if (++xs == kHalves) { xs = 0; xphase ^= 1; }
        }
        live = live && mbar_wait(m_free + 8 * ms, mphase ^ 1, abort_flag);
        if (live) {
          mbar_arrive_expect_tx(m_full + 8 * ms, dbytes);
          bulk_g2s(colmeta + ms * kMaxTN * 4, p.dx + (size_t)kb * p.npad + c0, dbytes, m_full + 8 * ms);
          ++sent_m;
          if (++ms == kColMetaSlots) { ms = 0; mphase ^= 1; }
        }
        if (++kb == nkb) { kb = 0; tile += gridDim.x; }
      }
      if (!live) {
        // gave up: let the copies in flight land (bounded)
        for (int i = max(0, sent_x - kHalves); i < sent_x; ++i)
          for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(x_full + 8 * (i % kHalves), (i / kHalves) & 1); ++spins) {}
        for (int i = max(0, sent_m - kColMetaSlots); i < sent_m; ++i)
          for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(m_full + 8 * (i % kColMetaSlots), (i / kColMetaSlots) & 1); ++spins) {}
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    // TMEM lanes are weight rows, TMEM columns the product's columns.  The warp owns 32 rows (its lane quarter) x TN/2
    // columns; thread (g = lane/4, t = lane%4) holds rows g and g+8, columns 2t and 2t+1 of every 16 x 8 block.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    const int quarter = warp & 3, col0 = ((warp - kEpilogueWarp0) >> 2) * (TN / 2), ncp = TN / 32;   // 16-column pieces
    constexpr int kPieces = kMaxTN / 32;
    const int g = lane >> 2, t = lane & 3;
    int ms = 0, mphase = 0, tile = blockIdx.x, kb = 0;
    f2 acc[kPieces][2][2][2];   // [piece][16-row half][8-column block][row g, g + 8]: columns 2t, 2t+1
    const f2 up14 = pack2(16384.0f, 16384.0f), up18 = pack2(262144.0f, 262144.0f);
    // added with fma(v, 1, acc), the 1 from a run-time value: ptxas contracts a packed multiply that only feeds a
    // packed add (seen with 12.9, in spite of .rn), and the reference rounds both
    const float one1 = p.K > 0 ? 1.0f : 2.0f;
    const f2 one = pack2(one1, one1);
    for (int it = 0; it < turns; ++it) {
      const int buf = it & 1;
      if (kb == 0) {
#pragma unroll
        for (int i = 0; i < 8 * kPieces; ++i) acc[i >> 3][(i >> 2) & 1][(i >> 1) & 1][i & 1] = 0ull;
      }
      bool live = mbar_wait(m_full + 8 * ms, mphase, abort_flag) && mbar_wait(d_full + 8 * buf, (uint32_t)(it >> 1) & 1u, abort_flag);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      fence_after();
      const float* dxs = reinterpret_cast<const float*>(colmeta) + ms * kMaxTN + col0 + 2 * t;
      const uint8_t* rmeta = rowmeta + ((it & (kRowMetaSlots - 1)) * BM + 32 * quarter + g) * 4;
      const uint32_t tbase = tmem_base + (uint32_t)(2 * TN * buf) + ((uint32_t)(32 * quarter) << 16) + (uint32_t)col0;
      f2 dw[4];                 // rows g, g + 8, g + 16, g + 24
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float d = h2f((uint16_t)*reinterpret_cast<const uint32_t*>(rmeta + 32 * r));
        dw[r] = pack2(d, d);
      }
#pragma unroll
      for (int cp = 0; cp < kPieces; ++cp) {
        if (cp >= ncp) break;
        uint32_t lo[2][8], hi[2][8];
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          tmem_ld_16x256b_x2(tbase + ((uint32_t)(16 * hh) << 16) + 16u * cp, lo[hh]);
          tmem_ld_16x256b_x2(tbase + ((uint32_t)(16 * hh) << 16) + (uint32_t)TN + 16u * cp, hi[hh]);
        }
        f2 dx[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 dxv = *reinterpret_cast<const float2*>(dxs + 16 * cp + 8 * q);
          dx[q] = pack2(dxv.x, dxv.y);
        }
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          if (hh == 0) tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 2; ++q) {
#pragma unroll
            for (int rr = 0; rr < 2; ++rr) {
              const f2 dl = pack2u(lo[hh][4 * q + 2 * rr], lo[hh][4 * q + 2 * rr + 1]);
              f2& a = acc[cp][hh][q][rr];
              const f2 d_all = mul2(dx[q], dw[2 * hh + rr]);
              const f2 isum = fma2(pack2u(hi[hh][4 * q + 2 * rr], hi[hh][4 * q + 2 * rr + 1]), up18, mul2(dl, up14));
              a = fma2(mul2(d_all, isum), one, a);
            }
          }
        }
      }
      fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(d_free + 8 * buf);
        mbar_arrive(m_free + 8 * ms);
      }
      if (++ms == kColMetaSlots) { ms = 0; mphase ^= 1; }
      if (++kb == nkb) {
        const int tm = tile / nt, c0 = (tile - tm * nt) * TN + col0 + 2 * t;
        const bool pairs = ((p.ldy | (int64_t)(reinterpret_cast<uintptr_t>(p.y) >> 2)) & 1) == 0;   // 8-byte stores
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int row = tm * BM + 32 * quarter + 8 * r + g;
          if (row >= p.M) continue;
          float* yr = p.y + (size_t)row * p.ldy + c0;
#pragma unroll
          for (int nb = 0; nb < 2 * kPieces; ++nb) {
            if (nb >= 2 * ncp) break;
            const float2 v = unpack2(acc[nb >> 1][r >> 1][nb & 1][r & 1]);
            const int c = c0 + 8 * nb;
            if (pairs && c + 1 < p.N) {
              *reinterpret_cast<float2*>(yr + 8 * nb) = v;
            } else {
              if (c < p.N) yr[8 * nb] = v.x;
              if (c + 1 < p.N) yr[8 * nb + 1] = v.y;
            }
          }
        }
        kb = 0;
        tile += gridDim.x;
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

int padded_columns(int ncols) { return (ncols + kColPad - 1) / kColPad * kColPad; }

// columns per tile: 64, or 32 where the 64-column tiles leave SMs idle (a turn of 32 columns takes as long as the
// producers need, about 0.7 of a 64-column one)
int tile_columns(int M, int ncols, int sm_count) {
  const int mt = (M + BM - 1) / BM;
  const int waves64 = (mt * ((ncols + 63) / 64) + sm_count - 1) / sm_count, waves32 = (mt * ((ncols + 31) / 32) + sm_count - 1) / sm_count;
  return 10 * waves64 <= 7 * waves32 ? 64 : 32;
}

}  // namespace

size_t gemm_q6k_tc_workspace_bytes(int K, int ncols) { return (size_t)padded_columns(ncols) * (size_t)(K / QK_K) * (2 * QK_K + 4); }

// Against gemv_odd_kernel (one pass over the weights per four columns, CTAs of eight rows): its time is that of the passes,
// this kernel's that of K (2.25 us a super-block however few rows and columns there are), so the line is in passes x
// rows.  us a call, calls one behind the other, there and here.  8192 row passes: 4096 x 11008 by 8 columns 92.5 / 107.5,
// 1024 x 11008 by 32 84.7 / 108.2, 4096 x 2816 by 8 37.7 / 38.9, 1024 x 2816 by 32 37.2 / 40.6.  12288: 4096 x 11008 by 12
// 142 / 108, 4096 x 2816 by 12 55.6 / 39.1.  Far from it: 256 x 11008 by 16 21.9 / 106.5, 14336 x 11008 by 5 262 / 108
constexpr int64_t kMinRowPasses = 9216;

bool gemm_q6k_tc_supported(int type, const GemvArgs& a, int ncols) {
  if (type != T_Q6_K || ncols < kGemmQ6kTcMinCols || a.K % QK_K != 0 || !a.tc_ws) return false;
  if (a.residual || a.W2 || a.W3 || a.pro_x || a.rope_cos || a.join_in || a.join_out) return false;
  if ((int64_t)((ncols + 3) / 4) * ((a.M + 7) / 8 * 8) < kMinRowPasses) return false;
  if (gemv_fast_path_ok(type, a.W, a.row_bytes, a.K)) return false;   // whatever the column count: see above
  return reinterpret_cast<uintptr_t>(a.W) % 2 == 0 && a.row_bytes % 2 == 0 && reinterpret_cast<uintptr_t>(a.act.qs) % 16 == 0 &&
         a.act.col_stride_qs % 16 == 0 && gemm_q6k_tc_workspace_bytes(a.K, kColPad) <= a.tc_ws_bytes;
}

// two launches: the activation pre-pass (into the tensor-core workspace) and the product; the two again for columns whose
// operand the workspace does not hold beside the others'
cudaError_t launch_gemm_q6k_tc(const GemvArgs& a, int ncols, int sm_count, cudaStream_t st, int* launches) {
  // per host thread (one context, one lane per thread): no shared mutable state between lanes
  static thread_local unsigned configured = 0;  // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_q6k_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  GemmArgs g{};
  g.W = a.W;
  g.row_bytes = a.row_bytes;
  g.M = a.M;
  g.K = a.K;
  g.x = a.tc_ws;
  g.ldy = a.ldy;
  g.status = a.status;
  const size_t groups = a.tc_ws_bytes / gemm_q6k_tc_workspace_bytes(a.K, kColPad);
  const int fit = (int)(groups < 65535 ? groups : 65535) * kColPad;   // at least one group: gemm_q6k_tc_supported
  for (int c = 0; c < ncols; c += fit) {
    g.N = ncols - c < fit ? ncols - c : fit;
    g.npad = padded_columns(g.N);
    g.TN = tile_columns(a.M, g.N, sm_count);
    g.y = a.y + a.col0 + c;
    float* dx = reinterpret_cast<float*>(a.tc_ws + (size_t)(a.K / QK_K) * g.npad * (2 * QK_K));
    g.dx = dx;
    tile_activations_f16_kernel<<<dim3(a.K / QK_K, (g.N + kPreCols - 1) / kPreCols), 256, 0, st>>>(a.act, a.col0 + c, g.N, g.npad, a.tc_ws, dx);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int tiles = ((a.M + BM - 1) / BM) * ((g.N + g.TN - 1) / g.TN);
    gemm_q6k_tc_kernel<<<tiles < sm_count ? tiles : sm_count, kThreads, kSmemBytes, st>>>(g);
    *launches += 2;
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace emelb
