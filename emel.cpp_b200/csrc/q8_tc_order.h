// What an MMA warp of gemm_q8_tc.cu waits for in front of a block, and in which order.  Here, without CUDA, so that a host
// program can walk every interleaving of the kernel's roles over it (tests/q8_tc_order_harness.cc).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define EMELB_ORDER_FN __host__ __device__ __forceinline__
#else
#define EMELB_ORDER_FN inline
#endif

namespace emelb {
namespace q8tc {

constexpr int kMmaWarps = 3;   // warp r issues blocks r, r + 3, ..
enum Barrier { kXFull, kDFree, kAFull };

// A parity wait tells the use it waits for from the one before it only when the one before that has ended.  A warp sees every
// use of its accumulators and of a turn's activations, but not of a pair's operands: of four pairs, one or two have no block
// of its own.  So the accumulators come first: the epilogue reads blocks in order, so once it has read block g - 3, every
// earlier pair was full, among them the one whose place block g's pair takes.  (Operands first: when the even pairs'
// producers fall behind the odd pairs', the wait for an even pair passes on the parity of the use before the last.)
// wait(barrier, index, parity) -> bool; xs, xphase: the activations' stage, fresh: parity of the accumulators
template <class Wait>
EMELB_ORDER_FN bool wait_for_block(int g, int xs, uint32_t xphase, uint32_t fresh, Wait&& wait) {
  return wait(kXFull, xs, xphase) && wait(kDFree, g % kMmaWarps, fresh) && wait(kAFull, (g >> 1) & 1, (uint32_t)(g >> 2) & 1u);
}

}  // namespace q8tc
}  // namespace emelb
