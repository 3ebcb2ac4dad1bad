// Q6_K x Q8_K matrix product for prompts (many columns) on the Blackwell tensor cores: tcgen05.mma kind::f16, weights as two
// A operands in TMEM, activations as the B operand in shared memory, f32 accumulators in TMEM that only ever hold exact
// integers.
//
// What is computed is exactly the reference's per-super-block value (src/emel/kernel/x86_64/actions.hpp:1036-1077)
//   (dx*d) * (float)isum,  isum = sum_g sc_g * dot16_g(q - 32, x)
// added in ascending block order, so the result equals the mat-vec kernels' (and the x86 AVX2 route's) bit for bit.
// A weight times its scale needs 13 bits, f16 holds 11, so sc = 16 * hi + lo with |hi|, |lo| <= 8 and two operands
// (q - 32) * piece of |.| <= 256 each: |sum| <= 256 * 128 * 256 = 2^23 in any order of addition, and (float)isum =
// fma(16, D_hi, D_lo), one rounding.
// Every column tile would unpack the same 6-bit blocks anew, from 210-byte blocks at any even address.  So a pre-pass
// over the weights writes them once as bytes, in the order in which a thread (a weight row = a TMEM lane) expands them,
// with the scales' pieces as f16 and d as f32: 41 KB for 128 rows of a super-block, one plain copy a turn.
//
// CTA = 128 weight rows x 128 columns, one super-block of K per turn, 28 warps:
//   warps 0-15   producers: a thread expands 64 weights of its row into TMEM: per two weights one mask under the exponent
//                of 1024 and one half2 fma an operand, (1024 + q) * piece - 1056 * piece, exact
//   warps 16-23  epilogue: two warps per TMEM lane quarter, half of the columns each, a thread a row, packed f32x2
//   warps 24, 25 MMA issue, a part of 64 columns each; TMEM allocation
//   warp  26     copies of weights and of activations, a quarter super-block each
//   warp  27     copies of the columns' scales
// TMEM: accumulators lo and hi of two parts of 64 columns (256 columns), operands lo and hi of one super-block (256, handed
// over in quarters).  A part's accumulators have one buffer: the epilogue reads one part while the MMAs make the other.
// Registers are split by setmaxnreg: 896 threads x 72 at launch = 512 x 64 + 256 x 104 + 128 x 40.
// Every mbarrier wait is bounded; on a timeout the CTA raises the status word, lets its copies land and frees its TMEM.
//
// What bounds it: the chain through one operand buffer, MMAs of either part (2,050 cycles a turn, both) -> expansion -> MMAs, 3,370
// cycles a turn (14336 x 4096 by 512 columns: tensor pipe 61 %, issue slots 52 %).  Measured, B200, 14336 x 4096 by 1900 columns: 377 us a call on planes (layout 12, slabs 18, product 340:
// 656 TFLOP/s), mma.sync kernel 977; 4096 x 14336: 430, 972.  One warp for all MMAs took 541 (its waits stood in the way of
// its instructions), two with the loop over quarters rolled 428, four 384.  The slabs' loads all in flight: 33 -> 18 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace emelb {
namespace {

using namespace tc;

constexpr int BM = 128, TN = 128, kPart = 64;
constexpr int kProducerWarps = 16, kEpilogueWarp0 = 16, kEpilogueWarps = 8, kMmaWarp = 24, kLoaderWarp = 26, kMetaWarp = 27;   // two MMA warps
constexpr int kThreads = 28 * 32;
constexpr int kProducerRegs = 64, kEpilogueRegs = 104, kOtherRegs = 40;
static_assert(kProducerWarps * kProducerRegs + kEpilogueWarps * kEpilogueRegs + 4 * kOtherRegs <= 28 * 72, "register split");

// 128 rows of a super-block as the pre-pass writes them
constexpr int kChunk = BM * 16;                   // 16 bytes of every row
constexpr int kOffScales = 16 * kChunk;           // behind the quants, [half][word 0..7][row]: four bytes of each of the four 32-weight runs
constexpr int kOffD = kOffScales + 4 * kChunk;    // behind the scales, [quarter][row]: {lo, hi} as f16 of four 16-weight groups
constexpr int kSlab = kOffD + BM * 8;             // d as f32, twice
constexpr int kSlabs = 2, kMetaSlots = 3;
constexpr int kQuarterBytes = TN / 8 * kAtomBytes;   // activations of a quarter super-block (64 K)
constexpr int kMetaBytes = TN / 2 * kColumnPairBytes;
constexpr int kStageRow = 48;                     // an epilogue warp's store: 8 columns of a row; a multiple of 16 that spreads rows over the banks

// shared memory map
constexpr int kOffSlab = 8 * kQuarterBytes;
constexpr int kOffMeta = kOffSlab + kSlabs * kSlab;
constexpr int kOffStage = kOffMeta + kMetaSlots * kMetaBytes;
constexpr int kOffBars = kOffStage + kEpilogueWarps * 32 * kStageRow;
constexpr int kSmemBytes = kOffBars + 512 + 1024;   // barriers; slack for the base's alignment
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

constexpr uint32_t kTmemA = 256;   // operand lo; hi 128 columns on

struct GemmArgs {
  int M, K, N;
  const uint8_t* slabs;   // [ceil(M/128)][K/256]
  const uint8_t* x;       // [K/64][npad/8] swizzle atoms of 8 columns
  const uint8_t* pairs;   // [K/256][npad/2]{dx, dx, -, -}
  int npad;
  float* y;
  int64_t ldy;
  int* status;
};

// pre-pass over the weights, rows at any even address.  grid (K/256, ceil(M/128)), 256 threads; rows past M repeat the last one
constexpr int kPreWords = 55;    // 54 aligned words cover a block; an odd number: rows on all banks

__global__ void __launch_bounds__(256) q6k_slab_kernel(const uint8_t* W, int64_t row_bytes, int M, uint8_t* slabs) {
  __shared__ uint32_t blocks[BM * kPreWords];
  const int kb = blockIdx.x, r0 = blockIdx.y * BM, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t part[16][2];      // all requested at once: a row of 53 words is one or two loads of a warp
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int rr = 16 * warp + i;
    const uintptr_t src = (reinterpret_cast<uintptr_t>(W) + (size_t)min(r0 + rr, M - 1) * row_bytes + (size_t)kb * Q6_K_BYTES) & ~uintptr_t(3);
    const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
    part[i][0] = w[lane];
    part[i][1] = lane < 21 ? w[32 + lane] : 0u;   // the 53 words that hold 210 bytes from byte 0 or 2 on
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int rr = 16 * warp + i;
    blocks[rr * kPreWords + lane] = part[i][0];
    if (lane < 21) blocks[rr * kPreWords + 32 + lane] = part[i][1];
  }
  __syncthreads();
  const int row = threadIdx.x & (BM - 1), n = threadIdx.x >> 7;         // half n of a row
  const uint32_t sh = (uint32_t)((reinterpret_cast<uintptr_t>(W) + (size_t)min(r0 + row, M - 1) * row_bytes + (size_t)kb * Q6_K_BYTES) & 2) * 8;
  const uint32_t* b = blocks + row * kPreWords;
  auto word = [&](int i) { return sh ? __funnelshift_r(b[i], b[i + 1], 16) : b[i]; };
  uint8_t* out = slabs + ((size_t)blockIdx.y * gridDim.x + kb) * kSlab;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const uint32_t qa = word(16 * n + i), qb = word(16 * n + 8 + i), qh = word(32 + 8 * n + i);
    uint4 v;
    v.x = (qa & 0x0f0f0f0fu) | ((qh << 4) & 0x30303030u);
    v.y = (qb & 0x0f0f0f0fu) | ((qh << 2) & 0x30303030u);
    v.z = ((qa >> 4) & 0x0f0f0f0fu) | (qh & 0x30303030u);
    v.w = ((qb >> 4) & 0x0f0f0f0fu) | ((qh >> 2) & 0x30303030u);
    *reinterpret_cast<uint4*>(out + (8 * n + i) * kChunk + row * 16) = v;
  }
  const uint32_t sw[2] = {word(48 + 2 * n), word(49 + 2 * n)};          // the half's eight scales
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    __half2 s[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int at = 2 * f + q, sc = (int)(int8_t)(sw[at >> 2] >> (8 * (at & 3)));
      const int hi = (sc + 8) >> 4, lo = sc - 16 * hi;                  // both in -8 .. 8
      s[f] = __halves2half2(__int2half_rn(lo), __int2half_rn(hi));
    }
    *reinterpret_cast<uint4*>(out + kOffScales + (2 * n + q) * kChunk + row * 16) = *reinterpret_cast<const uint4*>(s);
  }
  if (n == 0) {
    const float d = h2f((uint16_t)((sh ? b[52] >> 16 : b[52]) & 0xffffu));
    *reinterpret_cast<float2*>(out + kOffD + row * 8) = make_float2(d, d);
  }
}

// kAligned: rows of results go in 16-byte pieces.  A kernel of its own, because the other form in its way costs it 2 %
template <bool kAligned>
__global__ void __launch_bounds__(kThreads, 1) gemm_q6k_wide_kernel(const GemmArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* slab = smem + kOffSlab;
  uint8_t* meta = smem + kOffMeta;
  // barriers, by their shared memory addresses
  const uint32_t h_full = smem_u32(smem + kOffBars);  // [2 turns][4 quarters] producers and copies -> MMA; the last quarter brings the meta slot
  const uint32_t h_free = h_full + 8 * 8;             // MMA -> producers and loader
  const uint32_t r_full = h_free + 8 * 8;             // [slabs] copies -> producers: the weights of a super-block
  const uint32_t r_free = r_full + 8 * kSlabs;        // epilogue (the last reader, of d) -> loader
  const uint32_t m_free = r_free + 8 * kSlabs;        // [3] epilogue -> loader: the meta slot is read
  const uint32_t s_full = m_free + 8 * kMetaSlots;    // [parts] MMA -> epilogue: the part's accumulators are complete
  const uint32_t s_free = s_full + 8 * 2;             // [parts] epilogue -> MMA: they are read
  const uint32_t drained = s_free + 8 * 2;            // [2] only after a wait that gave up
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBars + 8 * 60);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // from one lane: the compiler then keeps what follows from it in uniform registers (TMEM addresses, barriers, pointers)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 8; ++s) { mbar_init(h_full + 8 * s, (s & 3) == 3 ? 6 : 5); mbar_init(h_free + 8 * s, 2); }
    for (int s = 0; s < kSlabs; ++s) { mbar_init(r_full + 8 * s, 1); mbar_init(r_free + 8 * s, kProducerWarps + kEpilogueWarps); }
    for (int s = 0; s < kMetaSlots; ++s) mbar_init(m_free + 8 * s, kEpilogueWarps);
    for (int s = 0; s < 2; ++s) { mbar_init(s_full + 8 * s, 1); mbar_init(s_free + 8 * s, kEpilogueWarps); mbar_init(drained + 8 * s, 1); }
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

  if (warp < kProducerWarps) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
    const int quarter = warp & 3, q4 = warp >> 2;   // TMEM lanes 32 * quarter .., quarter q4 of every super-block
    const uint32_t a_lane = tmem_base + kTmemA + ((uint32_t)(32 * quarter) << 16) + 32u * q4, lead = lane == 0;
    const uint32_t mask = in_register(0x00ff00ffu), k1024 = in_register(0x64006400u);
    const uint8_t* mine = slab + (32 * quarter + lane) * 16 + 4 * q4 * kChunk;
    for (int it = 0; it < turns; ++it) {
      const int slot = it & 1, prev = it - 1;
      bool live = mbar_wait(r_full + 8 * slot, (uint32_t)(it >> 1) & 1u, abort_flag);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      const uint8_t* src = mine + slot * kSlab;
      const uint4 sc = *reinterpret_cast<const uint4*>(src + kOffScales - 3 * q4 * kChunk);
      const uint32_t sw[4] = {sc.x, sc.y, sc.z, sc.w};
      __half2 sl[4], cl[4], sh[4], ch[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        sl[f] = bits_h2(__byte_perm(sw[f], 0u, 0x1010));
        sh[f] = bits_h2(__byte_perm(sw[f], 0u, 0x3232));
        cl[f] = __hmul2(sl[f], __float2half2_rn(-1056.0f));
        ch[f] = __hmul2(sh[f], __float2half2_rn(-1056.0f));
      }
      uint4 v4[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) v4[w] = *reinterpret_cast<const uint4*>(src + w * kChunk);
      __syncwarp();
      mbar_arrive_if(lead, r_free + 8 * slot);
      // the quarter's columns are free once the MMAs of the turn before are done with them
      live = prev < 0 || mbar_wait(h_free + 8 * (4 * (prev & 1) + q4), (uint32_t)(prev >> 1) & 1u, abort_flag);
      live = __all_sync(0xffffffffu, live);
      if (!live) break;
      fence_after();
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint32_t v[4] = {v4[w].x, v4[w].y, v4[w].z, v4[w].w};
        uint32_t ol[8], oh[8];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const uint32_t e = mask_or(v[f], mask, k1024), d = mask_or(v[f] >> 8, mask, k1024);
          ol[2 * f] = expand2(e, sl[f], cl[f]);
          ol[2 * f + 1] = expand2(d, sl[f], cl[f]);
          oh[2 * f] = expand2(e, sh[f], ch[f]);
          oh[2 * f + 1] = expand2(d, sh[f], ch[f]);
        }
        tmem_st8(a_lane + 8u * w, ol);
        tmem_st8(a_lane + 128u + 8u * w, oh);
      }
      tmem_wait_st();
      fence_before();
      __syncwarp();
      mbar_arrive_if(lead, h_full + 8 * (4 * slot + q4));
    }
  } else if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    // One lane issues, but the whole warp walks the loops, so that descriptors and addresses are worked out in uniform
    // registers.  D = f32, A = B = f16, both K-major, M = 128 weight rows, N = a part's columns
    const bool leader = elect_one();
    bool live = true;
    if (warp < kLoaderWarp) {
      // -------------------------------------------------------------- MMA issue: a warp for either part, so that the one's waits
      // pass while the other's instructions run
      constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(BM >> 4) << 24) | ((uint32_t)(kPart >> 3) << 17);
      const uint64_t x0 = operand_desc(smem_u32(smem), kAtomBytes);
      const int s = warp - kMmaWarp;
      const uint32_t d = tmem_base + (uint32_t)(2 * kPart * s);
#pragma unroll 1
      for (int it = 0; live && it < turns; ++it) {
        const int buf = it & 1;
        live = mbar_wait(s_free + 8 * s, ((uint32_t)it & 1u) ^ 1u, abort_flag);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          live = live && mbar_wait(h_full + 8 * (4 * buf + q), (uint32_t)(it >> 1) & 1u, abort_flag);
          live = __all_sync(0xffffffffu, live);
          if (!live) break;
          fence_after();
          const uint64_t x = x0 + (uint64_t)(((4 * buf + q) * kQuarterBytes + s * (kPart / 8) * kAtomBytes) >> 4);
          const uint32_t a_op = tmem_base + kTmemA + 32u * q, more = q > 0;
          if (leader) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              mma_f16(d, a_op + 8u * j, x + (uint64_t)(2 * j), kIdesc, more | (j > 0));
              mma_f16(d + kPart, a_op + 128u + 8u * j, x + (uint64_t)(2 * j), kIdesc, more | (j > 0));
            }
            mma_commit(h_free + 8 * (4 * buf + q));
            if (q == 3) mma_commit(s_full + 8 * s);
          }
          __syncwarp();
        }
      }
      if (!live && leader) {
        // gave up: let the tensor core finish what was issued before the TMEM goes away (bounded)
        mma_commit(drained + 8 * s);
        for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(drained + 8 * s, 0u); ++spins) {}
      }
    } else if (warp == kLoaderWarp) {
      // -------------------------------------------------------------- weights, and activations a quarter super-block a copy
      const size_t stride = (size_t)(p.npad >> 3) * kAtomBytes;
      int kb = 0, tile = blockIdx.x, it = 0;
      const uint8_t* src = p.x + (size_t)((tile % nt) * (TN / 8)) * kAtomBytes;
      const uint8_t* weights = p.slabs + (size_t)(tile / nt) * nkb * kSlab;
#pragma unroll 1
      for (; live && it < turns; ++it) {
        const int buf = it & 1;
        const uint32_t phase = ((uint32_t)(it >> 1) & 1u) ^ 1u;
        live = mbar_wait(r_free + 8 * buf, phase, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        if (leader) {
          mbar_arrive_expect_tx(r_full + 8 * buf, kSlab);
          bulk_g2s(slab + buf * kSlab, weights, kSlab, r_full + 8 * buf);
        }
        __syncwarp();
        weights += kSlab;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          const uint32_t full = h_full + 8 * (4 * buf + q);
          live = live && mbar_wait(h_free + 8 * (4 * buf + q), phase, abort_flag);
          live = __all_sync(0xffffffffu, live);
          if (!live) break;
          if (leader) {
            mbar_arrive_expect_tx(full, kQuarterBytes);
            bulk_g2s(smem + (4 * buf + q) * kQuarterBytes, src, kQuarterBytes, full);
          }
          __syncwarp();
          src += stride;
        }
        if (++kb == nkb) {
          kb = 0;
          tile += gridDim.x;
          src = p.x + (size_t)((tile % nt) * (TN / 8)) * kAtomBytes;
          weights = p.slabs + (size_t)(tile / nt) * nkb * kSlab;
        }
      }
      if (!live && leader) {
        // gave up: let the copies in flight land (bounded).  A quarter's barrier also counts producers, who may have gone:
        // the copies' landing shows in its phase only if all came, so this waits out its bound otherwise
        for (int i = max(0, it - 2); i <= it; ++i) {
          for (int q = 0; q < 4; ++q)
            for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(h_full + 8 * (4 * (i & 1) + q), (uint32_t)(i >> 1) & 1u); ++spins) {}
          for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(r_full + 8 * (i & 1), (uint32_t)(i >> 1) & 1u); ++spins) {}
        }
      }
    } else if (warp == kMetaWarp) {
      // -------------------------------------------------------------- scales of the columns
      int kb = 0, tile = blockIdx.x, it = 0, ms = 0;
      uint32_t phase = 1u;
#pragma unroll 1
      for (; live && it < turns; ++it) {
        const uint32_t full = h_full + 8 * (4 * (it & 1) + 3);
        live = mbar_wait(m_free + 8 * ms, phase, abort_flag);
        // the barrier's phase before this one is over once the MMAs of turn it - 2 are done
        live = live && mbar_wait(h_free + 8 * (4 * (it & 1) + 3), ((uint32_t)(it >> 1) & 1u) ^ 1u, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        if (leader) {
          mbar_arrive_expect_tx(full, kMetaBytes);
          bulk_g2s(meta + ms * kMetaBytes, p.pairs + ((size_t)kb * (p.npad >> 1) + (tile % nt) * (TN / 2)) * kColumnPairBytes, kMetaBytes, full);
        }
        __syncwarp();
        if (++ms == kMetaSlots) { ms = 0; phase ^= 1u; }
        if (++kb == nkb) { kb = 0; tile += gridDim.x; }
      }
      if (!live && leader) {
        for (int i = max(0, it - 2); i <= it; ++i)
          for (int spins = 0; spins < (1 << 14) && !mbar_try_wait(h_full + 8 * (4 * (i & 1) + 3), (uint32_t)(i >> 1) & 1u); ++spins) {}
      }
    }
    __syncwarp();
  } else {
    // ---------------------------------------------------------------- epilogue
    // TMEM lanes are weight rows, TMEM columns the product's columns.  The warp owns 32 rows (its lane quarter) and of either
    // part one half, a thread one row.
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    constexpr int kMine = kPart / 2, kLoads = kMine / 8;           // columns of a part; loads of eight
    const int quarter = warp & 3, side = (warp - kEpilogueWarp0) >> 2;
    const uint32_t tb = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)(kMine * side), lead = lane == 0;
    // added with fma(v, 1, acc), the 1 from a run-time value: ptxas contracts a packed multiply that only feeds a
    // packed add (seen with 12.9, in spite of .rn), and the reference rounds both
    const float one1 = p.K > 0 ? 1.0f : 2.0f;
    const f2 one = pack2(one1, one1), k16 = pack2(16.0f, 16.0f);
    int ms = 0, it = 0;
    bool live = true;
    for (int tile = blockIdx.x; live && tile < ntiles; tile += gridDim.x) {
      f2 acc[2][kLoads][4];       // [part][load][column pair]
#pragma unroll
      for (int i = 0; i < 8 * kLoads; ++i) acc[i / (4 * kLoads)][(i >> 2) % kLoads][i & 3] = 0ull;
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb, ++it) {
        const uint8_t* cm = meta + ms * kMetaBytes + kMine / 2 * side * kColumnPairBytes;
        const int slot = it & 1;
        f2 dw = 0ull;
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const uint32_t td = tb + 2 * kPart * s;
          // after a wait that gave up the turn's arithmetic is nonsense, which nobody stores
          live = mbar_wait(s_full + 8 * s, (uint32_t)it & 1u, abort_flag) && live;
          __syncwarp();
          fence_after();
          if (s == 0) {
            dw = *reinterpret_cast<const f2*>(slab + slot * kSlab + kOffD + (32 * quarter + lane) * 8);
            __syncwarp();
            mbar_arrive_if(lead, r_free + 8 * slot);
          }
          uint32_t lo[2][8], hi[2][8];
          tmem_ld8(td, lo[0]);
          tmem_ld8(td + kPart, hi[0]);
#pragma unroll
          for (int i = 0; i < kLoads; ++i) {
            tmem_wait_ld(lo[i & 1], hi[i & 1]);
            if (i + 1 == kLoads) {
              fence_before();
              __syncwarp();
              mbar_arrive_if(lead, s_free + 8 * s);
            } else {
              tmem_ld8(td + 8u * (i + 1), lo[(i + 1) & 1]);
              tmem_ld8(td + kPart + 8u * (i + 1), hi[(i + 1) & 1]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const f2 dx = *reinterpret_cast<const f2*>(cm + (kPart / 2 * s + 4 * i + q) * kColumnPairBytes);
              const f2 isum = fma2(pack2u(hi[i & 1][2 * q], hi[i & 1][2 * q + 1]), k16, pack2u(lo[i & 1][2 * q], lo[i & 1][2 * q + 1]));
              acc[s][i][q] = fma2(mul2(mul2(dx, dw), isum), one, acc[s][i][q]);
            }
          }
        }
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        mbar_arrive_if(lead, m_free + 8 * ms);
        if (++ms == kMetaSlots) ms = 0;
      }
      if (!live) break;
      // rows leave through shared memory, 8 columns at a time, two lanes a row: 32 bytes of a row side by side
      const int tm = tile / nt, r0 = tm * BM + 32 * quarter, j = lane & 1;
      uint8_t* stage = smem + kOffStage + (warp - kEpilogueWarp0) * 32 * kStageRow;
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < kLoads; ++i) {
          __syncwarp();
#pragma unroll
          for (int e = 0; e < 2; ++e) *reinterpret_cast<ulonglong2*>(stage + lane * kStageRow + 16 * e) = make_ulonglong2(acc[s][i][2 * e], acc[s][i][2 * e + 1]);
          __syncwarp();
          const int c = (tile - tm * nt) * TN + kPart * s + kMine * side + 8 * i + 4 * j;
          if constexpr (!kAligned) {
            // other strides: single floats, 8 of a row side by side (four floats a lane: 4096 x 4096 by 1901 188, so 171 us)
            const int cc = c - 4 * j + (lane & 7);
            if (cc < p.N)
#pragma unroll 1
              for (int row = lane >> 3; row < 32 && r0 + row < p.M; row += 4) p.y[(size_t)(r0 + row) * p.ldy + cc] = *reinterpret_cast<const float*>(stage + row * kStageRow + 4 * (lane & 7));
          } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const int row = r0 + 16 * k + (lane >> 1);
              const float4 v = *reinterpret_cast<const float4*>(stage + (16 * k + (lane >> 1)) * kStageRow + 16 * j);
              if (row >= p.M) continue;
              float* yr = p.y + (size_t)row * p.ldy + c;
              if (c + 3 < p.N) {
                *reinterpret_cast<float4*>(yr) = v;
              } else {
                if (c < p.N) yr[0] = v.x;
                if (c + 1 < p.N) yr[1] = v.y;
                if (c + 2 < p.N) yr[2] = v.z;
              }
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

}  // namespace

// Against the kernels for fewer columns.  From one of their tiles an SM on, or for long rows, the cheaper one by a model in us: of
// this kernel a start, the pass over the weights and a time per wave and super-block; of gemm_q6k_mma.cu (K % 2048 == 0, aligned
// rows) its first wave of 64 x 64 tiles and what each further tile an SM adds, more where the last column tile is partial;
// of gemm_q6k_tc.cu (other rows) its waves of 128 x 64.  Fitted to 250 calls; us there and here: 2048 x 2048 by 512 columns 35.9 / 39.9,
// by 640 47.2 / 41.9, 5632 x 2048 by 192 36.3 / 43.0, by 256 46.1 / 43.0, 4096 x 4096 by 192 60.5 / 56.4, by 512 110 / 60, 14336 x 4096 by 1900 977 / 377,
// 4096 x 14336 by 128 136 / 140, by 1900 972 / 430; 6500 x 768 by 320 33.4 / 40.0, by 1024 58.5 / 48.1, 4096 x 2816 by 320 64.6 / 47.2, by 576 67.8 / 69.7,
// 4096 x 11008 by 200 109.5 / 116.7, by 320 202 / 121.
// Rows of a single super-block stay here from the first line on, though the other kernel is 2 to 8 us faster at that (6500 x 256 by
// 201 23.7 / 28.7, 14336 x 256 by 1024 50.2 / 50.2): tests hold sizes of theirs to this kernel
bool gemm_q6k_wide_supported(int type, const GemvArgs& a, int ncols, int sm_count) {
  if (type != T_Q6_K || a.M < BM || a.K % QK_K != 0 || !a.tc_ws) return false;
  const bool streamed = gemv_fast_path_ok(type, a.W, a.row_bytes, a.K);
  if (ncols < (streamed ? 96 : 192)) return false;
  const int64_t nkb = a.K / QK_K, column_tiles = (ncols + 63) / 64, tile_rows = streamed ? 64 : BM;
  const int64_t tiles = (a.M + tile_rows - 1) / tile_rows * column_tiles;
  if (nkb < 40 && tiles <= sm_count) return false;
  const auto waves = [&](int64_t n) { return (double)((n + sm_count - 1) / sm_count); };
  const double here = 22.5 + 3.6e-7 * a.M * a.K + waves((int64_t)((a.M + BM - 1) / BM) * ((ncols + TN - 1) / TN)) * (2.5 + 1.75 * nkb);
  double there;
  if (streamed) {
    const double w = waves(tiles);
    there = 11.5 + nkb * (2.2 + (w > 1 ? 1.3 * (w - 1) - 0.4 : 0.0) + (ncols % 64 ? 4.5 / column_tiles : 0.0));
  } else {
    there = 17.5 + waves(tiles) * (0.5 + 2.1 * nkb);
  }
  if (nkb > 1 && there <= here) return false;
  if (a.residual || a.W2 || a.W3 || a.pro_x || a.rope_cos || a.join_in || a.join_out) return false;
  return reinterpret_cast<uintptr_t>(a.W) % 2 == 0 && a.row_bytes % 2 == 0 && planes_aligned(a.act) &&
         operand_layout_bytes(a.K, TN) + (size_t)nkb * kSlab <= a.tc_ws_bytes;
}

template <bool kAligned>
static cudaError_t launch_product(const GemmArgs& g, int grid, cudaStream_t st) {
  // per host thread (one context, one lane per thread): no shared mutable state between lanes
  static thread_local unsigned configured = 0;  // one bit per device
  int dev = 0;
  cudaGetDevice(&dev);
  if (!(configured & (1u << (dev & 31)))) {
    const cudaError_t e = cudaFuncSetAttribute(gemm_q6k_wide_kernel<kAligned>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (e != cudaSuccess) return e;
    configured |= 1u << (dev & 31);
  }
  gemm_q6k_wide_kernel<kAligned><<<grid, kThreads, kSmemBytes, st>>>(g);
  return cudaGetLastError();
}

// launches: the activation pre-pass, then for as many rows as the workspace holds the pre-pass over the weights and the
// product; all again for columns whose operand it does not hold beside them
cudaError_t launch_gemm_q6k_wide(const GemvArgs& a, int ncols, int sm_count, cudaStream_t st, int* launches) {
  const int nkb = a.K / QK_K, mt = (a.M + BM - 1) / BM;
  const size_t group = operand_layout_bytes(a.K, TN), tile_row = (size_t)nkb * kSlab;
  // columns first: a slab is worth its making for many of them.  At least one tile row stays
  const size_t room = (a.tc_ws_bytes - tile_row) / group;
  const int fit = (int)(room < 32767 ? room : 32767) * TN;
  for (int c = 0; c < ncols; c += fit) {
    const int n = ncols - c < fit ? ncols - c : fit, npad = (n + TN - 1) / TN * TN;
    const OperandLayout x = operand_layout(a.tc_ws, a.K, npad);
    cudaError_t e = launch_operand_layout(a.act, a.col0 + c, n, npad, a.K, x, false, st);
    ++*launches;
    if (e != cudaSuccess) return e;
    const size_t rows = (a.tc_ws_bytes - operand_layout_bytes(a.K, npad)) / tile_row;
    const int step = (int)(rows < 65535 ? rows : 65535);
    for (int t = 0; t < mt; t += step) {
      GemmArgs g{};
      const int r0 = t * BM, tiles_m = mt - t < step ? mt - t : step;
      g.M = a.M - r0 < tiles_m * BM ? a.M - r0 : tiles_m * BM;
      g.K = a.K;
      g.N = n;
      uint8_t* slabs = a.tc_ws + operand_layout_bytes(a.K, npad);
      g.slabs = slabs;
      g.x = x.x;
      g.pairs = x.pairs;
      g.npad = npad;
      g.y = a.y + (size_t)r0 * a.ldy + a.col0 + c;
      g.ldy = a.ldy;
      g.status = a.status;
      q6k_slab_kernel<<<dim3(nkb, tiles_m), 256, 0, st>>>(a.W + (size_t)r0 * a.row_bytes, a.row_bytes, g.M, slabs);
      e = cudaGetLastError();
      if (e != cudaSuccess) return e;
      const int tiles = tiles_m * ((n + TN - 1) / TN);
      const int grid = tiles < sm_count ? tiles : sm_count;
      const bool aligned = ((g.ldy | (int64_t)(reinterpret_cast<uintptr_t>(g.y) >> 2)) & 3) == 0;
      e = aligned ? launch_product<true>(g, grid, st) : launch_product<false>(g, grid, st);
      *launches += 2;
      if (e != cudaSuccess) return e;
    }
  }
  return cudaSuccess;
}

}  // namespace emelb
