// Walks every interleaving of the roles of gemm_q8_tc.cu over its barriers: two groups of producers (even and odd pairs of
// blocks, one operand buffer each), three MMA warps, two of the epilogue's warps.  Barriers are what mbarriers are: phases
// that a count of arrivals ends, and waits on a phase's parity.  Prints the states reached and the MMAs that read operands
// of another pair, or operands that were being written.
//   harness [waits]     waits: the order of the MMA warps' waits, of the letters d (accumulators) and a (operands), instead of
//                       the kernel's own (csrc/q8_tc_order.h)
#include <cstdio>
#include <cstring>
#include <set>
#include <string>
#include <vector>

#include "../emel.cpp_b200/csrc/q8_tc_order.h"

using namespace emelb::q8tc;

namespace {

constexpr int kBlocks = 24, kEpilogue = 2;
struct State {
  signed char pair[2];        // the pair that the group works on next
  signed char writing[2];     // it has begun
  signed char content[2];     // the pair whose operands lie in the buffer; -1 while written
  signed char block[kMmaWarps], step[kMmaWarps], in_flight[kMmaWarps];   // next block, waits behind it, block whose MMAs run (-1: none)
  signed char read[kEpilogue];
  signed char a_full[2], a_free[2], d_full[kMmaWarps], d_free[kMmaWarps];   // arrivals
};

bool passes(int arrivals, int count, unsigned parity) { return ((unsigned)(arrivals / count) & 1u) != parity; }

std::string order;
struct Want { Barrier what; int index; unsigned parity; };

std::vector<Want> waits_of(int g) {
  std::vector<Want> w;
  const unsigned fresh = (unsigned)((g / kMmaWarps) & 1) ^ 1u;
  wait_for_block(g, 0, 0, fresh, [&](Barrier what, int index, uint32_t parity) {
    w.push_back(Want{what, index, parity});
    return true;
  });
  std::vector<Want> out;
  if (order.empty()) {
    for (const Want& x : w)
      if (x.what != kXFull) out.push_back(x);       // a turn's activations: every warp sees each use, not modelled
  } else {
    for (char c : order)
      for (const Want& x : w)
        if (x.what == (c == 'd' ? kDFree : kAFull)) out.push_back(x);
  }
  return out;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc > 1) order = argv[1];
  std::vector<std::vector<Want>> waits;
  for (int g = 0; g < kBlocks; ++g) waits.push_back(waits_of(g));
  State first;
  std::memset(&first, 0, sizeof first);
  for (int i = 0; i < 2; ++i) { first.pair[i] = (signed char)i; first.content[i] = -1; }
  for (int r = 0; r < kMmaWarps; ++r) { first.block[r] = (signed char)r; first.in_flight[r] = -1; }
  const auto key = [](const State& s) { return std::string(reinterpret_cast<const char*>(&s), sizeof s); };
  std::set<std::string> seen{key(first)};
  std::vector<State> todo{first};
  long long wrong = 0, ends = 0, stuck = 0;
  while (!todo.empty()) {
    const State s = todo.back();
    todo.pop_back();
    bool moved = false;
    const auto go = [&](const State& n) {
      moved = true;
      if (seen.insert(key(n)).second) todo.push_back(n);
    };
    for (int b = 0; b < 2; ++b) {
      if (s.pair[b] >= kBlocks / 2) continue;
      State n = s;
      if (!s.writing[b]) {
        if (!passes(s.a_free[b], 2, ((unsigned)(s.pair[b] >> 1) & 1u) ^ 1u)) continue;
        n.writing[b] = 1;
        n.content[b] = -1;
      } else {
        n.writing[b] = 0;
        n.content[b] = s.pair[b];
        n.a_full[b] += 1;            // four warps: the last one's arrival
        n.pair[b] += 2;
      }
      go(n);
    }
    for (int r = 0; r < kMmaWarps; ++r) {
      if (s.in_flight[r] >= 0) {     // its MMAs end
        const int g = s.in_flight[r], b = (g >> 1) & 1;
        State n = s;
        wrong += s.content[b] != (g >> 1);
        n.in_flight[r] = -1;
        n.d_full[r] += 1;
        n.a_free[b] += 1;
        go(n);
      }
      if (s.block[r] >= kBlocks) continue;
      const std::vector<Want>& w = waits[s.block[r]];
      State n = s;
      if (s.step[r] < (int)w.size()) {
        const Want& x = w[s.step[r]];
        if (!(x.what == kDFree ? passes(s.d_free[x.index], kEpilogue, x.parity) : passes(s.a_full[x.index], 1, x.parity))) continue;
        n.step[r] += 1;
      } else {
        wrong += s.content[(s.block[r] >> 1) & 1] != (s.block[r] >> 1) || s.in_flight[r] >= 0;
        n.in_flight[r] = s.block[r];
        n.block[r] += kMmaWarps;
        n.step[r] = 0;
      }
      go(n);
    }
    for (int e = 0; e < kEpilogue; ++e) {
      if (s.read[e] >= kBlocks) continue;
      const int r = s.read[e] % kMmaWarps;
      if (!passes(s.d_full[r], 1, (unsigned)(s.read[e] / kMmaWarps) & 1u)) continue;
      State n = s;
      n.read[e] += 1;
      n.d_free[r] += 1;
      go(n);
    }
    if (moved) continue;
    bool end = true;
    for (int e = 0; e < kEpilogue; ++e) end = end && s.read[e] == kBlocks;
    ++(end ? ends : stuck);
    if (wrong > 1000000) break;
  }
  std::printf("%zu %lld %lld %lld\n", seen.size(), wrong, ends, stuck);
  return 0;
}
