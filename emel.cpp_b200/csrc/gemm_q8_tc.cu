// Q8_0 / Q4_0 x Q8_0 matrix product for prompts (many columns) on the Blackwell tensor cores: tcgen05.mma kind::f16, weights
// as the A operand in TMEM, activations as the B operand in shared memory, f32 accumulators in TMEM that only ever hold exact
// integers.
//
// What is computed is exactly the reference's per-block value (src/emel/kernel/detail.hpp:3131-3153, 3252-3269)
//   (float)isum * (d_w * d_x),  isum = dot32(q, x)
// added in ascending block order, so the result equals the mat-vec kernels' bit for bit.  Quants and activations are f16
// integers of at most 128, a block's sum stays below 2^20: exact in f32 in any order of addition, and there as a float.
// Both formats scale every 32 weights on their own, so every two MMAs (K = 16 each) end an accumulator.  The scales are f16 on
// either side, so their product is exact in f32, and a third MMA makes it for all rows and columns of the tile: (d_w, 0 ...)
// times (d_x, 0 ...).  The CUDA cores read both accumulators and spend two packed operations per two products and block.
//
// CTA = 128 weight rows (TMEM lanes) x 64 columns, 28 warps; copies come by turns of 8 blocks of K:
//   warps 0-7    producers: four warps (a TMEM lane quarter each) for even pairs of blocks, four for odd ones; a thread expands
//                a row's two blocks into TMEM
//   warps 8-23   epilogue: four warps per TMEM lane quarter, 16 columns each, a thread a row, packed f32x2
//   warps 24-26  MMA issue, every third block each; TMEM allocation
//   warp  27     copies of weights (TMA, 128 rows x 272 or 144 bytes) and activations
// TMEM: accumulators of three blocks (sums and scale products, 384 columns), operands of two pairs of blocks (96).
// Registers are split by setmaxnreg: 896 threads x 72 at launch = 256 x 96 + 512 x 64 + 128 x 48.
// Every mbarrier wait is bounded; on a timeout the CTA raises the status word, lets its copies land and frees its TMEM.
//
// What bounds it: instruction issue, 77 % of the slots (1,270 warp instructions and 416 cycles a block of a tile, MMAs 96), behind
// it the round of an accumulator, MMAs -> epilogue -> MMAs, with three on their way.
// Measured, B200, us a call on planes, mma.sync kernel and here: Q8_0 5632 x 5632 by 1024 columns 296 -> 216, 2048 x 5632 by 333 79 -> 56;
// Q4_0 255 -> 215, 69 -> 56.  With the product of the scales on the CUDA cores (three packed operations, the columns' scales from
// shared memory, whose 16-byte loads took more than half of the time) 248 and 62.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"
#include "q8_tc_order.h"
#include "tc_common.cuh"

namespace emelb {
namespace {

using namespace tc;

constexpr int BM = 128, TN = 64, kBlocks = 8, kTurnK = kBlocks * QK32;
constexpr int kProducerWarps = 8, kEpilogueWarps = 16, kMmaWarp = 24, kMmaWarps = q8tc::kMmaWarps, kLoaderWarp = 27;
constexpr int kThreads = 28 * 32;
constexpr int kProducerRegs = 96, kEpilogueRegs = 64, kOtherRegs = 48;
static_assert(kProducerWarps * kProducerRegs + kEpilogueWarps * kEpilogueRegs + 4 * kOtherRegs <= 28 * 72, "register split");

template <int T>
constexpr int kRowBytes = kBlocks * (T == T_Q8_0 ? Q8_0_BYTES : Q4_0_BYTES);   // of a turn; an odd number of 16 bytes

constexpr int kRawSlots = 3, kXStages = 2;
constexpr int kChunkBytes = TN / 8 * kAtomBytes;         // 64 columns x 128 bytes: activations of 64 K, scales of four blocks
constexpr int kChunks = kTurnK / 64 + kBlocks / 4;       // of a turn
constexpr int kXBytes = kChunks * kChunkBytes;

// shared memory map
constexpr int kOffRaw = kXStages * kXBytes;
constexpr int kOffBars = kOffRaw + kRawSlots * BM * kRowBytes<T_Q8_0>;
constexpr int kSmemBytes = kOffBars + 512 + 1024;   // barriers; slack for the base's alignment
static_assert(kSmemBytes <= 227 * 1024, "shared memory");

constexpr uint32_t kTmemA = 384, kPairColumns = 48;   // operands of a pair: quants 2 x 16 columns, scales 2 x 8

struct GemmArgs {
  int M, K, N;
  const uint8_t* x;    // [K/256][6][npad/8] swizzle atoms of 8 columns
  int npad;
  float* y;
  int64_t ldy;
  int* status;
};

// pre-pass: the quantized activation planes of columns col0.. -> operand order; of every four elements {0, 2, 1, 3}, which is
// what the producers' byte permutations leave side by side.  A block's scale is the first of 16 f16, the others are zero.
// grid (K/256, npad/64), 256 threads; columns past N are zero
constexpr int kPreRow = kTurnK + 4;   // 65 words: column-wise reads fall on all banks

__global__ void __launch_bounds__(256) q8_layout_kernel(ActPlanes act, int col0, int N, int npad, uint8_t* x) {
  __shared__ __align__(16) uint8_t t8[TN * kPreRow];
  const int kb = blockIdx.x, c0 = blockIdx.y * TN;
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int q = threadIdx.x + 256 * i, col = q >> 4, piece = q & 15;
    v[i] = make_uint4(0, 0, 0, 0);
    if (c0 + col < N) v[i] = *reinterpret_cast<const uint4*>(act.qs + (int64_t)(col0 + c0 + col) * act.col_stride_qs + kb * kTurnK + 16 * piece);
  }
  auto piece_at = [&](int chunk, int col, int piece) {   // 16 bytes
    return reinterpret_cast<uint4*>(x + ((size_t)(kChunks * kb + chunk) * (npad >> 3) + ((c0 + col) >> 3)) * kAtomBytes + (col & 7) * 128 +
                                    (((piece ^ col) & 7) << 4));
  };
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int q = threadIdx.x + 256 * i, col = q >> 3, b = q & 7;
    const float d = c0 + col < N ? act.d[(int64_t)(col0 + c0 + col) * act.col_stride_d + kb * kBlocks + b] : 0.0f;
    *piece_at(4 + (b >> 2), col, 2 * (b & 3)) = make_uint4(__half_as_ushort(__float2half_rn(d)), 0, 0, 0);   // a plane's scale is an f16
    *piece_at(4 + (b >> 2), col, 2 * (b & 3) + 1) = make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int q = threadIdx.x + 256 * i, col = q >> 4, piece = q & 15;
    uint32_t* o = reinterpret_cast<uint32_t*>(t8 + col * kPreRow + 16 * piece);
    o[0] = v[i].x; o[1] = v[i].y; o[2] = v[i].z; o[3] = v[i].w;
  }
  __syncthreads();
  auto halves = [](uint32_t w, uint32_t& even, uint32_t& odd) {   // four int8 -> f16 {0, 2}, {1, 3}
    const uint32_t u = w ^ 0x80808080u;
    const __half2 bias = __float2half2_rn(-1152.0f);
    even = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4240)), bias));
    odd = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4341)), bias));
  };
  for (int q = threadIdx.x; q < TN * 32; q += 256) {
    const int col = q & (TN - 1), ch = q >> 6;               // chunk ch of 8 elements
    const uint32_t* s = reinterpret_cast<const uint32_t*>(t8 + col * kPreRow + 8 * ch);
    uint4 o;
    halves(s[0], o.x, o.y);
    halves(s[1], o.z, o.w);
    *piece_at(ch >> 3, col, ch) = o;
  }
}

template <int T>
__global__ void __launch_bounds__(kThreads, 1) gemm_q8_tc_kernel(const GemmArgs p, const __grid_constant__ CUtensorMap wmap) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* raw = smem + kOffRaw;
  const uint32_t bars = smem_u32(smem + kOffBars);
  const uint32_t r_full = bars;                       // [kRawSlots] TMA -> producers: the weights of a turn
  const uint32_t r_free = r_full + 8 * kRawSlots;
  const uint32_t a_full = r_free + 8 * kRawSlots;     // [pair & 1] producers -> MMA
  const uint32_t a_free = a_full + 8 * 2;
  const uint32_t x_full = a_free + 8 * 2;             // [kXStages] bulk copies -> MMA
  const uint32_t x_free = x_full + 8 * kXStages;
  const uint32_t d_full = x_free + 8 * kXStages;      // [kMmaWarps] MMA -> epilogue: accumulators of a block
  const uint32_t d_free = d_full + 8 * kMmaWarps;
  const uint32_t drained = d_free + 8 * kMmaWarps;    // [kMmaWarps] all that was issued is done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kOffBars + 8 * (4 + 2 * kRawSlots + 2 * kXStages + 3 * kMmaWarps));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // from one lane: the compiler then keeps what follows from it in uniform registers (TMEM addresses, barriers, pointers)
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRawSlots; ++s) { mbar_init(r_full + 8 * s, 1); mbar_init(r_free + 8 * s, kProducerWarps); }
    for (int s = 0; s < 2; ++s) { mbar_init(a_full + 8 * s, 4); mbar_init(a_free + 8 * s, 2); }   // a pair's blocks are two warps'
    for (int s = 0; s < kXStages; ++s) { mbar_init(x_full + 8 * s, 1); mbar_init(x_free + 8 * s, kMmaWarps); }
    for (int s = 0; s < kMmaWarps; ++s) { mbar_init(d_full + 8 * s, 1); mbar_init(d_free + 8 * s, kEpilogueWarps); mbar_init(drained + 8 * s, 1); }
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

  const int mt = (p.M + BM - 1) / BM, nt = (p.N + TN - 1) / TN, ntiles = mt * nt, nkb = p.K / kTurnK;
  const int my_tiles = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int turns = my_tiles * nkb;

  if (warp < kProducerWarps) {
    // ---------------------------------------------------------------- producers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
    const int quarter = warp & 3, odd = warp >> 2;
    const uint32_t a_lane = tmem_base + kTmemA + kPairColumns * odd + ((uint32_t)(32 * quarter) << 16), lead = lane == 0;
    constexpr int kPairWords = kRowBytes<T> / 16, kMid = kPairWords / 2;   // words of a pair of blocks; the second one's first
    int rs = 0, rphase = 0;
    bool live = true;
    for (int it = 0; it < turns; ++it) {
      const uint8_t* mine = raw + (rs * BM + 32 * quarter + lane) * kRowBytes<T>;
      live = mbar_wait(r_full + 8 * rs, rphase, abort_flag);
      live = __all_sync(0xffffffffu, live);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (!live) break;
        // pair 2 h + odd of the turn: 16-byte pieces as they come, the pair starts at word 0 .. 3 of one
        uint32_t w[4 * ((kPairWords + 6) / 4)];
        const int first = (2 * h + odd) * kPairWords;
#pragma unroll
        for (int i = 0; i < (kPairWords + 6) / 4; ++i) {
          const int at = min(first / 4 + i, kRowBytes<T> / 16 - 1);
          const uint4 v = *reinterpret_cast<const uint4*>(mine + 16 * at);
          w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
        }
        if (h == 1) {
          __syncwarp();
          mbar_arrive_if(lead, r_free + 8 * rs);
        }
        // to word 0: kPairWords is 1 mod 4, so pair j starts at word j of a piece
        if (odd) {
#pragma unroll
          for (int i = 0; i < kPairWords; ++i) w[i] = w[i + 2 * h + 1];
        } else if (h == 1) {
#pragma unroll
          for (int i = 0; i < kPairWords; ++i) w[i] = w[i + 2];
        }
        // the first block has its scale in the low half of word 0 and its quants across words, the second one in the high
        // half of the middle word and its quants in the words behind it
        uint32_t o[32], dw[2][8] = {{w[0] & 0xffffu}, {w[kMid] >> 16}};
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int i = 0; i < kMid; ++i) {
            const uint32_t q = e ? w[kMid + 1 + i] : __funnelshift_r(w[i], w[i + 1], 16);
            if constexpr (T == T_Q8_0) {
              const uint32_t u = q ^ 0x80808080u;
              const __half2 bias = __float2half2_rn(-1152.0f);
              o[16 * e + 2 * i] = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4240)), bias));
              o[16 * e + 2 * i + 1] = h2_bits(__hadd2(bits_h2(__byte_perm(u, 0x64646464u, 0x4341)), bias));
            } else {
              const __half2 bias = __float2half2_rn(-1032.0f);
#pragma unroll
              for (int s = 0; s < 4; ++s)   // low nibbles of bytes 0 and 2, high ones, bytes 1 and 3
                o[16 * e + 8 * (s & 1) + 2 * i + (s >> 1)] = h2_bits(__hadd2(bits_h2(((q >> (4 * s)) & 0x000f000fu) | 0x64006400u), bias));
            }
          }
        // the pair's columns are free once the MMAs of the pair before last are done with them (use 2 it + h)
        live = mbar_wait(a_free + 8 * odd, h ^ 1, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        fence_after();
        tmem_st32(a_lane, o);
        tmem_st8(a_lane + 32u, dw[0]);
        tmem_st8(a_lane + 40u, dw[1]);
        tmem_wait_st();
        fence_before();
        __syncwarp();
        mbar_arrive_if(lead, a_full + 8 * odd);
      }
      if (!live) break;
      if (++rs == kRawSlots) { rs = 0; rphase ^= 1; }
    }
  } else if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    if (warp < kLoaderWarp && elect_one()) {
      // -------------------------------------------------------------- MMA issue (one thread for every third block)
      // D = f32, A = B = f16, both K-major, M = 128 weight rows, N = 64 columns
      constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const int r = warp - kMmaWarp, blocks = kBlocks * turns;
      const uint64_t x0 = operand_desc(smem_u32(smem), kAtomBytes);
      const uint32_t d = tmem_base + 2 * TN * r;
      bool live = true;
      int xs = 0, xphase = 0, b = r;   // block b of the turn
      uint32_t fresh = 1;              // parity of d_free
      for (int g = r; g < blocks; g += kMmaWarps) {
        const uint32_t pair = (uint32_t)(g >> 1) & 1u;
        live = q8tc::wait_for_block(g, xs, xphase, fresh, [&](q8tc::Barrier what, int index, uint32_t parity) {
          return mbar_wait((what == q8tc::kXFull ? x_full : what == q8tc::kDFree ? d_free : a_full) + 8 * index, parity, abort_flag);
        });
        if (!live) break;
        fence_after();
        const uint64_t x = x0 + (uint64_t)((xs * kXBytes + (b >> 1) * kChunkBytes + (b & 1) * 64) >> 4);
        const uint64_t xd = x0 + (uint64_t)((xs * kXBytes + (4 + (b >> 2)) * kChunkBytes + (b & 3) * 32) >> 4);
        const uint32_t a_op = tmem_base + kTmemA + kPairColumns * pair + 16u * (b & 1);
        mma_f16(d + TN, tmem_base + kTmemA + kPairColumns * pair + 32u + 8u * (b & 1), xd, idesc, 0u);
        mma_f16(d, a_op, x, idesc, 0u);
        mma_f16(d, a_op + 8u, x + (32 >> 4), idesc, 1u);
        mma_commit(d_full + 8 * r);
        mma_commit(a_free + 8 * pair);
        fresh ^= 1u;
        b += kMmaWarps;
        if (b >= kBlocks) {
          mma_commit(x_free + 8 * xs);
          b -= kBlocks;
          if (++xs == kXStages) { xs = 0; xphase ^= 1; }
        }
      }
      if (!live) {
        // gave up: let the tensor core finish what was issued before the TMEM goes away (bounded)
        mma_commit(drained + 8 * r);
        for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(drained + 8 * r, 0); ++spins) {}
      }
    } else if (warp == kLoaderWarp && lane == 0) {
      // -------------------------------------------------------------- copies (one thread): activations of turn it, weights of
      // the turn after it
      bool live = true;
      int sent_r = 0, sent_x = 0, wtile = blockIdx.x, wkb = 0, tile = blockIdx.x, kb = 0;
      auto weights = [&]() {
        if (sent_r == turns) return;
        const int rs = sent_r % kRawSlots;
        live = mbar_wait(r_free + 8 * rs, ((sent_r / kRawSlots) & 1) ^ 1, abort_flag);
        if (!live) return;
        mbar_arrive_expect_tx(r_full + 8 * rs, BM * kRowBytes<T>);
        tma_load_2d(raw + rs * BM * kRowBytes<T>, &wmap, wkb * (kRowBytes<T> / 4), wtile / nt * BM, r_full + 8 * rs);
        ++sent_r;
        if (++wkb == nkb) { wkb = 0; wtile += gridDim.x; }
      };
      for (int s = 0; s + 1 < kRawSlots; ++s) weights();
      for (int it = 0; it < turns; ++it) {
        const int c0 = (tile % nt) * TN, xs = it % kXStages;
        live = mbar_wait(x_free + 8 * xs, ((it / kXStages) & 1) ^ 1, abort_flag);
        if (!live) break;
        mbar_arrive_expect_tx(x_full + 8 * xs, kXBytes);
        for (int c = 0; c < kChunks; ++c)
          bulk_g2s(smem + xs * kXBytes + c * kChunkBytes, p.x + ((size_t)(kChunks * kb + c) * (p.npad >> 3) + (c0 >> 3)) * kAtomBytes, kChunkBytes,
                   x_full + 8 * xs);
        ++sent_x;
        if (++kb == nkb) { kb = 0; tile += gridDim.x; }
        weights();
        if (!live) break;
      }
      if (!live) {
        // gave up: let the copies in flight land (bounded)
        auto land = [&](uint32_t bar, int sent, int slots) {
          for (int i = max(0, sent - slots); i < sent; ++i)
            for (int spins = 0; spins < (1 << 16) && !mbar_try_wait(bar + 8 * (i % slots), (i / slots) & 1); ++spins) {}
        };
        land(r_full, sent_r, kRawSlots);
        land(x_full, sent_x, kXStages);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
    const int quarter = warp & 3, col0 = 16 * ((warp - kProducerWarps) >> 2);
    const uint32_t lead = lane == 0, tbase = tmem_base + ((uint32_t)(32 * quarter) << 16) + (uint32_t)col0;
    // added with fma(v, 1, acc), the 1 from a run-time value: ptxas contracts a packed multiply that only feeds a
    // packed add (seen with 12.9, in spite of .rn), and the reference rounds both
    const float one1 = p.K > 0 ? 1.0f : 2.0f;
    const f2 one = pack2(one1, one1);
    f2 acc[8];
    int tile = blockIdx.x, kb = 0, slot = 0;
    uint32_t phase = 0;
    bool live = true;
    for (int it = 0; it < turns; ++it) {
      if (kb == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0ull;
      }
#pragma unroll 2
      for (int b = 0; b < kBlocks; ++b) {
        if (!mbar_try_wait(d_full + 8 * slot, phase)) live = mbar_wait(d_full + 8 * slot, phase, abort_flag);
        live = __all_sync(0xffffffffu, live);
        if (!live) break;
        fence_after();
        uint32_t v[2][8], d[2][8];
        const uint32_t at = tbase + (uint32_t)(2 * TN * slot);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          tmem_ld8(at + 8u * c, v[c]);
          tmem_ld8(at + TN + 8u * c, d[c]);
        }
        tmem_wait_ld(v[0], v[1]);
        tmem_wait_ld(d[0], d[1]);
        fence_before();
        __syncwarp();
        mbar_arrive_if(lead, d_free + 8 * slot);
        if (++slot == kMmaWarps) { slot = 0; phase ^= 1u; }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          acc[i] = fma2(mul2(pack2u(v[i >> 2][2 * i & 7], v[i >> 2][(2 * i & 7) + 1]), pack2u(d[i >> 2][2 * i & 7], d[i >> 2][(2 * i & 7) + 1])), one, acc[i]);
      }
      if (!live) break;
      if (++kb == nkb) {
        const int tm = tile / nt, c = (tile - tm * nt) * TN + col0, row = tm * BM + 32 * quarter + lane;
        if (row < p.M) {
          float* yr = p.y + (size_t)row * p.ldy + c;
          const bool quads = p.ldy % 4 == 0 && reinterpret_cast<uintptr_t>(p.y) % 16 == 0;   // 16-byte stores
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            const float2 a = unpack2(acc[i]), b = unpack2(acc[i + 1]);
            if (quads && c + 2 * i + 3 < p.N) {
              *reinterpret_cast<float4*>(yr + 2 * i) = make_float4(a.x, a.y, b.x, b.y);
            } else {
              if (c + 2 * i < p.N) yr[2 * i] = a.x;
              if (c + 2 * i + 1 < p.N) yr[2 * i + 1] = a.y;
              if (c + 2 * i + 2 < p.N) yr[2 * i + 2] = b.x;
              if (c + 2 * i + 3 < p.N) yr[2 * i + 3] = b.y;
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

int padded_columns(int ncols) { return (ncols + TN - 1) / TN * TN; }
size_t workspace_bytes(int K, int npad) { return (size_t)npad * (K / kTurnK) * kChunks * 128; }

// the weights as words {rows, K/256 * (68 or 36)}, boxes of 128 rows x a turn
bool encode_rows(CUtensorMap* map, int row_bytes, const GemvArgs& a) {
  static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }();
  const cuuint64_t dims[2] = {(cuuint64_t)(a.K / kTurnK) * (row_bytes / 4), (cuuint64_t)a.M}, strides[1] = {(cuuint64_t)a.row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)row_bytes / 4, BM}, estr[2] = {1, 1};
  return encode && encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<uint8_t*>(a.W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int T>
cudaError_t launch_product(const GemmArgs& g, const CUtensorMap& wmap, int sm_count, cudaStream_t st) {
  const cudaError_t e = cudaFuncSetAttribute(gemm_q8_tc_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
  if (e != cudaSuccess) return e;
  const int64_t tiles = (int64_t)((g.M + BM - 1) / BM) * ((g.N + TN - 1) / TN);
  gemm_q8_tc_kernel<T><<<(int)(tiles < sm_count ? tiles : sm_count), kThreads, kSmemBytes, st>>>(g, wmap);
  return cudaGetLastError();
}

}  // namespace

// Against gemm_q8_mma.cu: two launches and the start of a CTA cost 8 to 10 us more, a block of K less.  us a call, there and
// here: 2048 x 2048 by 333 columns 32 / 31, 5632 x 2048 by 64 23 / 26, by 333 54 / 52, by 1024 115 / 91; 2048 x 5632 by 333 79 / 56,
// 5632 x 5632 by 64 56 / 50.  Where 64 x 64 tiles leave half of the SMs idle that kernel takes narrow ones (2048 x 5632 by 64
// 29 / 50), so those stay there; and Q4_0, half the bytes, needs longer sums or more tiles (1024 x 4096 by 333 41.8 / 43.6, 4096 x
// 4096 by 128 37.6 / 38.9; 14336 x 4096 by 64 49.9 / 39.7, 2048 x 5632 by 333 68.5 / 55.7).  A thread stores a row's columns, which
// without 16-byte pieces takes a tenth more (5632 x 2048 by 1900 171, by 1901 211): for Q4_0 and short sums that is the
// advantage and more (2750 x 2048 by 1440 95.4 / 92.0, by 1441 97.4 / 104.4, 4096 x 3072 by 1441 168.8 / 166.7)
bool gemm_q8_tc_supported(int type, const GemvArgs& a, int ncols, int sm_count) {
  const int64_t columns = (ncols + TN - 1) / TN, tiles = (a.M + BM - 1) / BM * columns;
  if (2 * ((a.M + 63) / 64) * columns <= sm_count) return false;
  if (a.K < 4096 && (a.K < 2048 || tiles < 2 * sm_count)) return false;
  if (type == T_Q4_0 && a.K < 5120 && 3 * tiles < 2 * sm_count) return false;
  if (type == T_Q4_0 && a.K < 3072 && ((a.ldy | a.col0 | (int64_t)(reinterpret_cast<uintptr_t>(a.y) >> 2)) & 3) != 0) return false;
  if ((type != T_Q8_0 && type != T_Q4_0) || ncols < kGemmQ8TcMinCols || a.K % kTurnK != 0 || !a.tc_ws) return false;
  if (a.residual || a.W2 || a.W3 || a.pro_x || a.rope_cos || a.join_in || a.join_out) return false;
  return reinterpret_cast<uintptr_t>(a.W) % 16 == 0 && a.row_bytes % 16 == 0 && a.row_bytes < (1 << 27) && reinterpret_cast<uintptr_t>(a.act.qs) % 16 == 0 &&
         a.act.col_stride_qs % 16 == 0 && workspace_bytes(a.K, TN) <= a.tc_ws_bytes;
}

// two launches: the activation pre-pass (into the workspace) and the product; the two again for columns whose operand the
// workspace does not hold beside the others'
cudaError_t launch_gemm_q8_tc(int type, const GemvArgs& a, int ncols, int sm_count, cudaStream_t st, int* launches) {
  GemmArgs g{};
  g.M = a.M;
  g.K = a.K;
  g.x = a.tc_ws;
  g.ldy = a.ldy;
  g.status = a.status;
  CUtensorMap wmap;
  if (!encode_rows(&wmap, type == T_Q8_0 ? kRowBytes<T_Q8_0> : kRowBytes<T_Q4_0>, a)) return cudaErrorNotSupported;
  const size_t groups = a.tc_ws_bytes / workspace_bytes(a.K, TN);
  const int fit = (int)(groups < 65535 ? groups : 65535) * TN;
  for (int c = 0; c < ncols; c += fit) {
    g.N = ncols - c < fit ? ncols - c : fit;
    g.npad = padded_columns(g.N);
    g.y = a.y + a.col0 + c;
    q8_layout_kernel<<<dim3(a.K / kTurnK, g.npad / TN), 256, 0, st>>>(a.act, a.col0 + c, g.N, g.npad, a.tc_ws);
    ++*launches;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = type == T_Q8_0 ? launch_product<T_Q8_0>(g, wmap, sm_count, st) : launch_product<T_Q4_0>(g, wmap, sm_count, st);
    ++*launches;
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace emelb
