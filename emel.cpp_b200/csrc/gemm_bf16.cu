// y {rows, M} = act(x {rows, K} W {M, K}^T + bias) with bf16 operands on the Blackwell tensor cores: tcgen05.mma
// kind::f16, f32 accumulators in TMEM, operands brought by TMA in the 128-byte swizzled K-major layout.
//
// The weights are the M operand (TMEM lanes), BN rows of x the N operand, so few rows cost a narrow tile.  GLU tiles hold a
// gate tile and the up tile of the same outputs side by side in TMEM and store silu(gate) * up.
//
// A tile belongs to the two CTAs of a cluster on neighbouring SMs (cta_group::2): 256 features x BN rows, of which either CTA
// holds the weights and accumulators of 128 features, but half of the rows of x, which the tensor cores of both read.  Pairs
// stay for tile after tile, one CTA per SM: 10 warps, of which warp 8 issues the TMA copies, warp 9 of the first CTA the MMAs of
// the pair (its copies and those of the second CTA count on its barriers, its commits arrive at both), and warps 0-7 read the
// accumulators back (a TMEM lane quarter and half of the columns each) while the next tile's MMAs fill the other half of
// TMEM.
//
// What it replaced, a CTA and a tile of 128 features each, two CTAs per SM with 2 to 4 stages, waited on copies (a round trip
// is over a microsecond) and on last waves.  us, mean of 8 launches: 14336 x 2 x 4096, 2048 rows 438 -> 329 (1,460 TFLOP/s), 300
// rows 125 -> 84; 8192 x 2 x 2048, 2048 rows 144 -> 99; 4096 x 14336, 2048 rows 182 -> 162 (1,480), 300 rows 62 -> 50; 2048 x 8192,
// 200 rows 49 -> 27.  Bounds: large products the tensor cores, few rows the chain of a wait, the MMAs and a commit per stage
// (about 290 cycles beside the MMAs' own, whether addresses are constants of an unrolled loop or not, hence two slabs of K a
// stage where shared memory has room for enough of these).
//
// Short sums over few tiles run on single CTAs (gemm_bf16_one_kernel below), because a cluster's start costs 1 to 2 us more than a
// CTA's, and so do sizes that leave most pairs idle in a last turn, but not the SMs (one_cta).
// Every wait is bounded; when one runs out the CTA, or both, stop, let the copies and MMAs in flight end, raise the status word and free
// their TMEM.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "act.cuh"
#include "common.cuh"
#include "layered.h"

// true: the wait of `role` of CTA `rank` in front of its use (or tile) `use` is taken to have run out.  Nothing but a test, which
// compiles this file for itself, says so (tests/gemm_bf16_giveup_harness.cu)
#ifndef EMELB_GIVE_UP
#define EMELB_GIVE_UP(rank, role, use) false
#endif

namespace emelb {
namespace {

enum Role : int { kCopies, kMmas, kMmaTiles, kStores };
constexpr int kEpilogueWarps = 8, kTmaWarp = 8, kMmaWarp = 9, kThreads = 320;
constexpr int kBM = kGemmWeightBox, kBK = 64;
constexpr int kWeightTile = kBM * kBK * 2;
constexpr int kWaitSpins = 1 << 22;
constexpr uint32_t kSuspendHintNs = 10000;
constexpr unsigned long long kWaitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendHintNs)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  unsigned long long t0 = 0;
  for (int spins = 0; spins < kWaitSpins; ++spins) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((spins & 15) == 15) {
      if (*abort_flag) return false;
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitNs) break;
    }
  }
  *abort_flag = 1;
  return false;
}
// one thread of the warp, in a form that tells the compiler that a single one issues what follows (2048 prompt
// rows: 39.8 and 75.4 us a launch of 128- and 256-row tiles with a lane test, 38.7 and 73.8 with elect.sync)
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e != 0;
}

// K-major operand in 8-row x 128-byte swizzled atoms, 1024 bytes apart (descriptor version 1, swizzle mode 2)
__device__ __forceinline__ uint64_t operand_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fffu) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
               "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
               "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                 "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                 "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                 "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
               : "r"(taddr)
               : "memory");
}

struct GemmParams {
  int M, K, rows;          // M: outputs (half of the stored rows for GLU)
  const float* bias;
  int act, act_split;
  float* y;
  __nv_bfloat16* yb;
  int64_t ldy;
  int* status;
  float out_scale, softcap;
  int tail;                // first feature stored as f32 at tail_y
  float* tail_y;
  int64_t tail_ld;
};

constexpr int kTileLd = 40;   // elements from row to row where bf16 outputs turn

// one warp: 32 features x rows [c_begin, c_end) of accumulators -> y
template <int BN, bool GLU>
__device__ __forceinline__ void store_tile(const GemmParams p, uint32_t tmem, int f0, int t0, int quarter, int lane, __nv_bfloat16* tile, int c_begin, int c_end) {
  const int f = f0 + quarter * 32 + lane;
  const bool live = f < p.M;
  const float b0 = live && p.bias ? p.bias[f] : 0.0f, b1 = GLU && live && p.bias ? p.bias[p.M + f] : 0.0f;
  const uint32_t lane_base = tmem + ((uint32_t)(quarter * 32) << 16);
  const bool sigm = p.act == ACT_SILU_SIGMOID, gelu = p.act == ACT_GLU_GELU, cap = p.act == ACT_SOFTCAP, tail = f >= p.tail;
  // bf16 outputs turn in shared memory, 32 features x kCh rows of a warp at a time, and leave as 16-byte stores
  constexpr int kCh = BN < 64 ? 16 : 32;
  const int f_end = min(p.M, p.tail), fw = f0 + quarter * 32;
  for (int c = c_begin; c < c_end && t0 + c < p.rows; c += kCh) {
    uint32_t v[kCh], u[GLU ? kCh : 1];
    tmem_ld(lane_base + c, v);
    if constexpr (GLU) tmem_ld(lane_base + BN + c, u);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    float o[kCh];
#pragma unroll
    for (int j = 0; j < kCh; ++j) {
      o[j] = __uint_as_float(v[j]) + b0;
      if constexpr (GLU) {
        o[j] = (gelu ? gelu_tanhf_(o[j]) : siluf_(o[j])) * (__uint_as_float(u[j]) + b1);
      } else if (sigm) {
        const float sg = sigmoidf_(o[j]);
        o[j] = f < p.act_split ? o[j] * sg : sg;
      } else if (cap) {
        o[j] = softcapf_(o[j] * p.out_scale, p.softcap);
      }
    }
    if (live && (tail || !p.yb)) {
      float* y = tail ? p.tail_y + f - p.tail : p.y + f;
      const int64_t ld = tail ? p.tail_ld : p.ldy;
#pragma unroll
      for (int j = 0; j < kCh; ++j)
        if (t0 + c + j < p.rows) y[(int64_t)(t0 + c + j) * ld] = o[j];
    }
    if (!p.yb) continue;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kCh; ++j) tile[j * kTileLd + lane] = __float2bfloat16_rn(o[j]);
    __syncwarp();
#pragma unroll
    for (int i = lane; i < 4 * kCh; i += 32) {
      const int j = i / 4, q = 8 * (i % 4), n = f_end - fw - q;   // n features of this piece are stored
      if (t0 + c + j >= p.rows || n <= 0) continue;
      const __nv_bfloat16* src = tile + j * kTileLd + q;
      __nv_bfloat16* dst = p.yb + (int64_t)(t0 + c + j) * p.ldy + fw + q;
      if (n >= 8) {
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
      } else {
        // no loop: as one it cost every piece of a ragged tile (136 features, 64 rows: 5.7 us, so 4.6)
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (e < n) dst[e] = src[e];
      }
    }
  }
}

// BN rows; SL slabs of 64 elements of K a stage
template <int BN, bool GLU, int SL>
struct Tile {
  static constexpr int kRows = BN / 2;                // rows of x of either CTA
  static constexpr int kXTile = kRows * kBK * 2;
  static constexpr int kSlabBytes = (GLU ? 2 : 1) * kWeightTile + kXTile;
  static constexpr int kStageBytes = SL * kSlabBytes;
  static constexpr int kAccCols = (GLU ? 2 : 1) * BN, kTmemCols = 2 * kAccCols;
  static constexpr int kTurnBytes = kEpilogueWarps * 32 * kTileLd * 2;
  static constexpr int kRest = kTurnBytes + 1024 + 512;   // beside the stages; 1024 to align these
  static constexpr int kStages = std::min((226 * 1024 - kRest) / kStageBytes, 8);
  static constexpr int kSmem = kStages * kStageBytes + kRest;
  static_assert(kTmemCols <= 512 && kStages >= 2, "accumulators of two tiles");
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of the first CTA's copy of a shared memory object
__device__ __forceinline__ uint32_t in_first(const void* ptr) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(ptr)));
  return a;
}
// a word of the other CTA's shared memory, at the place that ptr has in this one's
__device__ __forceinline__ void store_at(const volatile int* ptr, uint32_t rank, int v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(const_cast<const int*>(ptr))), "r"(rank));
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// stands in for copies that nobody asked for
__device__ __forceinline__ void mbar_complete_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void prefetch_map(const TmaMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
// into this CTA's shared memory, counted on a barrier of the pair
__device__ __forceinline__ void tma_load(void* dst, const TmaMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                   smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(bar)
               : "memory");
}
// D = f32, A = B = bf16, both K-major, M = 256
template <int BN>
constexpr uint32_t kInstrDesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(2 * kBM >> 4) << 24);
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrives at both CTAs' barriers
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive_at(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}

// a wait of this CTA ran out: both are told
__device__ __noinline__ void give_up(volatile int* abort_flag, uint32_t rank) {
  *abort_flag = 1;
  store_at(abort_flag, rank ^ 1u, 1);
}

// After a wait that ran out, when no role of either CTA issues any more: MMAs and copies in flight end, bounded.  All threads
// of both CTAs call it.  (This and give_up are calls, and so out of the way: inlined they cost short products 0.3 to 1 us.)
__device__ __noinline__ void end_in_flight(uint32_t rank, bool mma_warp, bool copier, bool leader, int issued, uint64_t* full, int stages,
                                           uint32_t stage_bytes, uint64_t* drained, volatile int* second_issued) {
  if (mma_warp) {
    if (leader) mma_commit(drained);
    if ((threadIdx.x & 31) == 0)
      for (int spin = 0; spin < 1 << 16 && !mbar_try_wait(drained, 0); ++spin) {}
  }
  if (copier && rank == 1) store_at(second_issued, 0, issued);
  __syncwarp();
  cluster_sync();
  if (copier && rank == 0) {
    // The two may have stopped at different stages, at most `stages` apart (a stage comes free through MMAs that read both
    // CTAs' copies); where one did not ask for copies, the first CTA stands in for its share of the barrier
    const int other = *second_issued, both = min(issued, other), any = max(issued, other);
    for (int i = max(0, any - stages); i < any; ++i) {
      uint64_t* bar = full + i % stages;
      if (i >= both) {
        if (issued > other) mbar_complete_tx(bar, stage_bytes);
        else mbar_arrive_expect_tx(bar, stage_bytes);
      }
      for (int spin = 0; spin < 1 << 16 && !mbar_try_wait(bar, (i / stages) & 1); ++spin) {}
    }
  }
  __syncwarp();
  cluster_sync();
}

template <int BN, bool GLU, int SL>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    gemm_bf16_kernel(const __grid_constant__ TmaMap wmap, const __grid_constant__ TmaMap xmap, const GemmParams p) {
  using T = Tile<BN, GLU, SL>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __nv_bfloat16* turn = reinterpret_cast<__nv_bfloat16*>(smem + T::kStages * T::kStageBytes);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStageBytes + T::kTurnBytes);   // of the first CTA: copies of both have landed
  uint64_t* empty = full + T::kStages;       // of either: the MMAs are done with the stage
  uint64_t* acc_full = empty + T::kStages;   // of either: a tile's accumulators stand
  uint64_t* acc_empty = acc_full + 2;        // of the first CTA: both have read theirs
  uint64_t* drained = acc_empty + 2;         // of either, only after a wait that ran out: all MMAs are done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);   // set in both or in neither
  volatile int* second_issued = abort_flag + 1;                                // of the first, after a wait that ran out
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int slabs = (p.K + kBK - 1) / kBK, nk = (slabs + SL - 1) / SL;
  const int nt = (p.rows + BN - 1) / BN, tiles = nt * ((p.M + 2 * kBM - 1) / (2 * kBM));
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + b, 1);
      mbar_init(acc_empty + b, 2 * kEpilogueWarps);
    }
    mbar_init(drained, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  if (warp == kTmaWarp && lane == 0) {
    prefetch_map(&wmap);
    prefetch_map(&xmap);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();            // the barriers and accumulators of both CTAs stand
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const auto wait = [&](uint64_t* bar, uint32_t parity, Role role, int use) {
    if (!EMELB_GIVE_UP(rank, role, use) && mbar_wait(bar, parity, abort_flag)) return true;
    give_up(abort_flag, rank);
    return false;
  };
  int issued = 0;         // stages that this CTA asked copies for (the copying thread)
  bool leader = false;    // the thread that issues the pair's MMAs

  if (warp == kTmaWarp) {
    if (lane == 0) {
      int s = 0, lap = 0;
      bool ok = true;
      for (int tile = first; ok && tile < tiles; tile += step) {
        const int t0 = tile % nt * BN + (int)rank * T::kRows, f0 = (tile / nt * 2 + (int)rank) * kBM;
        for (int i = 0; i < nk; ++i) {
          if ((lap > 0 || EMELB_GIVE_UP(rank, kCopies, s)) && !(ok = wait(empty + s, (lap - 1) & 1, kCopies, lap * T::kStages + s))) break;
          uint8_t* st = smem + s * T::kStageBytes;
          const uint32_t bar = in_first(full + s);
          if (rank == 0) mbar_arrive_expect_tx(full + s, 2 * T::kStageBytes);
#pragma unroll
          for (int l = 0; l < SL; ++l) {
            const int k = (i * SL + l) * kBK;
            uint8_t* at = st + l * T::kSlabBytes;
            tma_load(at, &wmap, k, f0, bar);
            if (GLU) tma_load(at + kWeightTile, &wmap, k, p.M + f0, bar);
            tma_load(at + (GLU ? 2 : 1) * kWeightTile, &xmap, k, t0, bar);
          }
          if (++s == T::kStages) s = 0, ++lap;
        }
      }
      issued = lap * T::kStages + s;
      // every commit to this CTA's barriers has arrived before it leaves
      for (int e = 0; ok && e < T::kStages; ++e) {
        const int uses = lap + (e < s);
        if (uses > 0) ok = wait(empty + e, (uses - 1) & 1, kCopies, issued + e);
      }
    }
  } else if (warp == kMmaWarp) {
    leader = rank == 0 && elect_one();
    if (leader) {
      int s = 0, use = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first, n = 0; tile < tiles; tile += step, ++n) {
        const int b = n & 1;
        if (n >= 2 && !wait(acc_empty + b, ((n >> 1) - 1) & 1, kMmaTiles, n)) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem + b * T::kAccCols;
        for (int i = 0; i < nk; ++i, ++use) {
          if (!(ok = wait(full + s, phase, kMmas, use))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t d0 = operand_desc(smem_u32(smem + s * T::kStageBytes));
#pragma unroll
          for (int l = 0; l < SL; ++l) {
            if (SL > 1 && i * SL + l >= slabs) break;
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              const uint64_t da = d0 + ((l * T::kSlabBytes + 32 * k) >> 4), db = da + ((GLU ? 2 : 1) * kWeightTile >> 4);
              mma_bf16(acc, da, db, kInstrDesc<BN>, i > 0 || l > 0 || k > 0);
              if (GLU) mma_bf16(acc + BN, da + (kWeightTile >> 4), db, kInstrDesc<BN>, i > 0 || l > 0 || k > 0);
            }
          }
          mma_commit(empty + s);
          if (++s == T::kStages) s = 0, phase ^= 1;
        }
        if (!ok) break;            // accumulators that are not whole are nobody's
        mma_commit(acc_full + b);
      }
    }
  } else {
    const int quarter = warp & 3, half = warp >> 2;
    for (int tile = first, n = 0; tile < tiles; tile += step, ++n) {
      const int b = n & 1, t0 = tile % nt * BN, f0 = (tile / nt * 2 + (int)rank) * kBM;
      if (!__all_sync(0xffffffffu, wait(acc_full + b, (n >> 1) & 1, kStores, n))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      __syncwarp();
      store_tile<BN, GLU>(p, tmem + b * T::kAccCols, f0, t0, quarter, lane, turn + warp * 32 * kTileLd, half * (BN / 2), (half + 1) * (BN / 2));
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_at(in_first(acc_empty + b));
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();            // neither frees what the other may still signal
  if (__any_sync(0xffffffffu, *abort_flag)) {
    end_in_flight(rank, warp == kMmaWarp, warp == kTmaWarp && lane == 0, leader, issued, full, T::kStages, T::kStageBytes, drained, second_issued);
  }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, 1);
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kTmemCols) : "memory");
  }
}

// ---- one CTA a tile of 128 features, no cluster: for sums so short that the start is a large part of the time.
// 6 warps: 0-3 read the accumulators back, 4 issues the copies, 5 the MMAs.  Two CTAs an SM (one computes while the other
// stores), or, where the grid leaves an SM no second one, DEEP: all the stages that an SM holds
__device__ __forceinline__ void tma_load_one(void* dst, const TmaMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
               "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
template <int BN>
constexpr uint32_t kInstrDescOne = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
__device__ __forceinline__ void mma_bf16_one(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_commit_one(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

constexpr int kOneThreads = 192, kOneTmaWarp = 4, kOneMmaWarp = 5;

template <int BN, bool GLU, bool DEEP>
struct OneTile {
  static constexpr int kStageBytes = (GLU ? 2 : 1) * kWeightTile + BN * kBK * 2;
  static constexpr int kStages = DEEP ? 200 * 1024 / kStageBytes : BN == 256 ? 2 : BN == 128 ? 3 : 4;
  // of x, a copy.  64 rows as two of 32: copies that reach far past the last row are slow (24576 features, K = 2048, 17 rows: 24.8 us, so 19.7)
  static constexpr int kBoxRows = BN == 64 ? 32 : BN < 128 ? BN : 128, kBox = BN == 16 ? 0 : BN == 64 ? 1 : 3;
  static_assert(kGemmTokenBox << kBox == kBoxRows, "box");
  static constexpr int kTmemCols = (GLU ? 2 : 1) * BN < 32 ? 32 : (GLU ? 2 : 1) * BN;
  static constexpr int kSmem = kStages * kStageBytes + 1024 + 256;
  static_assert(4 * 32 * kTileLd * 2 <= kStages * kStageBytes, "bf16 outputs turn in the stages");
};

template <int BN, bool GLU, bool DEEP>
__global__ void __launch_bounds__(kOneThreads) gemm_bf16_one_kernel(const __grid_constant__ TmaMap wmap, const __grid_constant__ TmaMap xmap,
                                                                    const GemmParams p) {
  using T = OneTile<BN, GLU, DEEP>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + T::kStages * T::kStageBytes);
  uint64_t* empty = full + T::kStages;
  uint64_t* done = empty + T::kStages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t0 = blockIdx.x * BN, f0 = blockIdx.y * kBM;
  const int nk = (p.K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < T::kStages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    mbar_init(done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kOneMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(T::kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const auto wait = [&](uint64_t* bar, uint32_t parity, Role role, int use) {
    if (!EMELB_GIVE_UP(0, role, use) && mbar_wait(bar, parity, abort_flag)) return true;
    *abort_flag = 1;
    return false;
  };

  int issued = 0;
  if (warp == kOneTmaWarp && lane == 0) {
    for (int i = 0; i < nk; ++i) {
      const int s = i % T::kStages;
      if ((i >= T::kStages || EMELB_GIVE_UP(0, kCopies, i)) && !wait(empty + s, ((i / T::kStages) - 1) & 1, kCopies, i)) break;
      uint8_t* st = smem + s * T::kStageBytes;
      mbar_arrive_expect_tx(full + s, T::kStageBytes);
      tma_load_one(st, &wmap, i * kBK, f0, full + s);
      if (GLU) tma_load_one(st + kWeightTile, &wmap, i * kBK, p.M + f0, full + s);
#pragma unroll
      for (int b = 0; b < BN / T::kBoxRows; ++b)
        tma_load_one(st + (GLU ? 2 : 1) * kWeightTile + b * T::kBoxRows * kBK * 2, &xmap, i * kBK, t0 + b * T::kBoxRows, full + s);
      issued = i + 1;
    }
  } else if (warp == kOneMmaWarp && elect_one()) {
    for (int i = 0; i < nk; ++i) {
      const int s = i % T::kStages;
      if (!wait(full + s, (i / T::kStages) & 1, kMmas, i)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t st = smem_u32(smem + s * T::kStageBytes), xt = st + (GLU ? 2 : 1) * kWeightTile;
#pragma unroll
      for (int k = 0; k < kBK / 16; ++k) {
        const uint64_t db = operand_desc(xt + 32 * k);
        mma_bf16_one(tmem, operand_desc(st + 32 * k), db, kInstrDescOne<BN>, i > 0 || k > 0);
        if (GLU) mma_bf16_one(tmem + BN, operand_desc(st + kWeightTile + 32 * k), db, kInstrDescOne<BN>, i > 0 || k > 0);
      }
      mma_commit_one(empty + s);
    }
    mma_commit_one(done);
  }
  __syncwarp();
  if (warp < 4) {
    // `done` also follows MMAs that gave up: the flag, raised before, tells
    const bool ok = wait(done, 0, kStores, 0) && !*abort_flag;
    if (__all_sync(0xffffffffu, ok)) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // bf16 outputs turn in the stages, which are free: every copy has landed and been used
      store_tile<BN, GLU>(p, tmem, f0, t0, warp, lane, reinterpret_cast<__nv_bfloat16*>(smem) + warp * 32 * kTileLd, 0, BN);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*abort_flag) {
    // A wait ran out, and no role issues any more: the copies and MMAs in flight end (bounded) before their memory goes
    if (warp == kOneTmaWarp && lane == 0)
      for (int i = max(0, issued - T::kStages); i < issued; ++i)
        for (int spin = 0; spin < 1 << 16 && !mbar_try_wait(full + i % T::kStages, (i / T::kStages) & 1); ++spin) {}
    if (warp == kOneMmaWarp && lane == 0)
      for (int spin = 0; spin < 1 << 16 && !mbar_try_wait(done, 0); ++spin) {}
    __syncwarp();
  }
  if (threadIdx.x == 0 && *abort_flag && p.status) atomicExch(p.status, 1);
  if (warp == kOneMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::kTmemCols) : "memory");
  }
}

template <int BN, bool GLU, bool DEEP>
cudaError_t launch_one_stages(const TmaMap& wmap, const XMaps& x, const GemmParams& p, cudaStream_t st) {
  using T = OneTile<BN, GLU, DEEP>;
  const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_one_kernel<BN, GLU, DEEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem);
  if (e != cudaSuccess) return e;
  gemm_bf16_one_kernel<BN, GLU, DEEP><<<dim3((p.rows + BN - 1) / BN, (p.M + kBM - 1) / kBM), kOneThreads, T::kSmem, st>>>(wmap, x.box[T::kBox], p);
  return cudaGetLastError();
}

int64_t one_tiles(const GemmParams& p, int bn) { return (int64_t)((p.M + kBM - 1) / kBM) * ((p.rows + bn - 1) / bn); }

template <int BN, bool GLU>
cudaError_t launch_one(const TmaMap& wmap, const XMaps& x, const GemmParams& p, int sm_count, cudaStream_t st) {
  return one_tiles(p, BN) <= sm_count ? launch_one_stages<BN, GLU, true>(wmap, x, p, st) : launch_one_stages<BN, GLU, false>(wmap, x, p, st);
}

// rows of x a single CTA's tile: narrower ones while every one has an SM, the widest once there are more of them than SMs
int one_rows(const GemmParams& p, int sm_count) {
  if (p.rows <= 16) return 16;
  if (p.rows <= 64 || one_tiles(p, 64) <= sm_count) return 64;
  return 5 * one_tiles(p, 256) >= 6 * sm_count ? 256 : 128;
}

int64_t tiles_of(const GemmParams& p, int bn) { return (int64_t)((p.M + 2 * kBM - 1) / (2 * kBM)) * ((p.rows + bn - 1) / bn); }

// Turns x time a turn of one matrix.  Weights: us a turn of an SM pair at K = 2048 / 4096 / 8192 / 14336: 32 rows 10.6 / 16.6 / 26.8 / 42, 128 rows
// 12.6 / 18.6 / 29 / 48, 256 rows 18.7 / 27 / 45 / 72.  (64 rows cost within 3 % of 128.)
template <int BN>
int64_t turns_cost(const GemmParams& p, int pairs) {
  return (tiles_of(p, BN) + pairs - 1) / pairs * (BN == 32 ? 20 : BN == 128 ? 23 : 36);
}
int64_t pairs_cost(const GemmParams& p, int pairs) { return std::min({turns_cost<32>(p, pairs), turns_cost<128>(p, pairs), turns_cost<256>(p, pairs)}); }

// Single CTAs or pairs, us there and here, one launch behind the other in a graph.
// K to 256, to four tiles an SM: 4096 x 256 by 8 rows 3.5 / 4.5, by 200 4.5 / 6.4, by 2048 9.8 / 12.3, 136 x 136 by 100 4.5 / 5.2; beyond it the pairs' rate
// wins (8192 x 256 by 1500 18.3 / 17.1).  K to 512 likewise (8192 x 512 by 8 5.3 / 5.8, by 128 6.2 / 7.6, by 333 8.8 / 10.0, by 1000 13.2 / 13.9, by 1500 23.2 /
// 18.5), but with more than 32 rows in tiles for less than half of the SMs pairs are as fast or faster: 2048 x 512 by 100 5.3 / 5.0, by 333 5.4 / 6.7.
// K to 1024, tiles for half of the SMs to two an SM: 8192 x 1024 by 100 9.0 / 9.5, by 300 12.2 / 12.4, 2048 x 1024 by 300 8.3 / 8.8, by 1500 11.2 / 11.9; else 2048 x
// 1024 by 100 8.3 / 6.7, 8192 x 1024 by 700 18.9 / 16.2.
// Up to 64 rows of a matrix with one to two tiles an SM, which leaves most pairs idle in a last turn: 20480 x 2048 by 8 17.5 / 19.9, 32000 x 2048 by 64
// 24.1 / 25.4, 24576 x 4096 by 64 39.4 / 42.2, 23736 x 9320 by 6 76.6 / 88.9; 32000 x 4096 by 8 45.5 / 44.4, 14336 x 2048 by 32 13.8 / 13.2.
// More rows where an odd number of 128-feature tiles fills the SMs, but half of it, rounded up, not the pairs: 6256 x 8720 by 374 39.2 / 48.7, 6256 x 9616 by 1523
// 124 / 140.
// Two matrices and up to 16 rows: 512 x 2 x 256 by 16 5.1 / 5.7, 8192 x 2 x 2048 by 8 17.0 / 17.4; 14336 x 2 x 4096 by 8 41.7 / 41.9
bool one_cta(const GemmParams& p, bool glu, int sm_count) {
  if (glu) return p.rows <= 16 && p.K <= 2048;
  const int64_t tiles = one_tiles(p, std::min(one_rows(p, sm_count), 128));
  if (p.K <= 512) return tiles <= 4 * sm_count && (p.K <= 256 || p.rows <= 32 || 2 * tiles > sm_count);
  if (p.K <= 1024) return 2 * tiles > sm_count && tiles <= 2 * sm_count;
  if (p.rows <= 64) return tiles > sm_count && 2 * tiles <= (p.K <= 2048 ? 4 : 3) * sm_count;
  if (one_rows(p, sm_count) == 256) return 42 * ((one_tiles(p, 256) + sm_count - 1) / sm_count) < pairs_cost(p, std::max(sm_count / 2, 1));
  return tiles <= sm_count && 30 < pairs_cost(p, std::max(sm_count / 2, 1));
}

template <int BN, bool GLU, int SL>
cudaError_t launch_tiles(const TmaMap& wmap, const XMaps& x, const GemmParams& p, int pairs, cudaStream_t st) {
  using T = Tile<BN, GLU, SL>;
  constexpr int kBox = BN == 32 ? 0 : BN == 64 ? 1 : BN == 128 ? 2 : 3;   // of half of the rows
  static_assert(kGemmTokenBox << kBox == T::kRows, "box");
  const cudaError_t e = cudaFuncSetAttribute(gemm_bf16_kernel<BN, GLU, SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem);
  if (e != cudaSuccess) return e;
  gemm_bf16_kernel<BN, GLU, SL><<<2 * (int)std::min<int64_t>(tiles_of(p, BN), pairs), kThreads, T::kSmem, st>>>(wmap, x.box[kBox], p);
  return cudaGetLastError();
}

}  // namespace

bool encode_bf16_map(TmaMap* map, const __nv_bfloat16* base, int64_t rows, int64_t k, int64_t ld, int box_rows) {
  static_assert(sizeof(CUtensorMap) == sizeof(TmaMap), "tensor map size");
  if (reinterpret_cast<uintptr_t>(base) % 16 != 0 || ld % 8 != 0 || rows < 1 || k < 1) return false;
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess || !fn) {
      cudaGetLastError();
      return false;
    }
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  return encode(reinterpret_cast<CUtensorMap*>(map), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool encode_x_maps(XMaps* x, const __nv_bfloat16* base, int64_t rows, int64_t k, int64_t ld) {
  for (int i = 0; i < 4; ++i)
    if (!encode_bf16_map(x->box + i, base, rows, k, ld, kGemmTokenBox << i)) return false;
  return true;
}

cudaError_t launch_gemm_bf16(const LinearArgs& a, const TmaMap& wmap, const XMaps& x, float* y, __nv_bfloat16* yb, int64_t ldy, int* status,
                             int sm_count, cudaStream_t st) {
  if (yb && (ldy % 8 != 0 || reinterpret_cast<uintptr_t>(yb) % 16 != 0)) return cudaErrorInvalidValue;
  const bool glu = is_glu(a.act);
  GemmParams p{glu ? a.w.M / 2 : a.w.M, a.w.K, a.rows, a.bias, a.act, a.act_split, y, yb, ldy, status,
               a.out_scale, a.softcap, a.tail, a.tail_y, a.tail_ld};
  if (one_cta(p, glu, sm_count)) {
    if (glu) return launch_one<16, true>(wmap, x, p, sm_count, st);
    const int bn = one_rows(p, sm_count);
    if (bn == 16) return launch_one<16, false>(wmap, x, p, sm_count, st);
    if (bn == 64) return launch_one<64, false>(wmap, x, p, sm_count, st);
    return bn == 128 ? launch_one<128, false>(wmap, x, p, sm_count, st) : launch_one_stages<256, false, false>(wmap, x, p, st);
  }
  // the width with the least turns x time a turn: us a turn of two matrices at K = 2048 32 rows 14.6, 64 rows 18.7, 128 rows 22
  const int pairs = std::max(sm_count / 2, 1);
  if (glu) {
    const auto cost = [&](int bn, int weight) { return (tiles_of(p, bn) + pairs - 1) / pairs * weight; };
    const int64_t c32 = cost(32, 7), c64 = cost(64, 9), c128 = cost(128, 11);
    if (c32 <= c64 && c32 <= c128) return launch_tiles<32, true, 2>(wmap, x, p, pairs, st);
    if (c64 < c128) return launch_tiles<64, true, 1>(wmap, x, p, pairs, st);
    return launch_tiles<128, true, 1>(wmap, x, p, pairs, st);
  }
  const int64_t c32 = turns_cost<32>(p, pairs), c128 = turns_cost<128>(p, pairs), c256 = turns_cost<256>(p, pairs);
  if (c32 <= c128 && c32 <= c256) return launch_tiles<32, false, 2>(wmap, x, p, pairs, st);
  if (c128 < c256) return launch_tiles<128, false, 2>(wmap, x, p, pairs, st);
  return launch_tiles<256, false, 1>(wmap, x, p, pairs, st);
}

}  // namespace emelb
