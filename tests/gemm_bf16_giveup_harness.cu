// Runs the kernels of gemm_bf16.cu with one role of every CTA, or of one CTA of every pair, giving up at a chosen place, as if
// a wait had run out there, and with everything else as it is: copies and MMAs in flight, the other CTA ahead or behind.  After each such launch the
// status word must be raised and the context in order, and the next, undisturbed launch must give the undisturbed bits.
// Prints the places tried and the complaints.
#include <chrono>
#include <cstdio>
#include <vector>

__device__ int g_give_up[3];   // rank, role, use
#define EMELB_GIVE_UP(rank, role, use) ((int)(rank) == g_give_up[0] && (int)(role) == g_give_up[1] && (use) == g_give_up[2])
#include "../emel.cpp_b200/csrc/gemm_bf16.cu"

namespace emelb {
namespace {

int tried = 0, complaints = 0;

__global__ void fill(__nv_bfloat16* p, int64_t n, int seed) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = __float2bfloat16_rn((float)((int)((i * 2654435761u + seed) >> 7 & 255) - 128) / 64.0f);
}

void complain(const char* what, int rank, int role, int use) {
  std::printf("rank %d role %d use %d: %s (%s)\n", rank, role, use, what, cudaGetErrorString(cudaGetLastError()));
  ++complaints;
}

struct Case {
  int outputs, K, rows;
  bool glu;
};

// tries(disturbed): disturbed(rank, role, use) launches with that give-up, false after a complaint
template <class Launch, class Tries>
void run(const Case& c, const Launch& launch_tiles_of, const Tries& tries) {
  const int M = c.glu ? 2 * c.outputs : c.outputs, K = c.K, rows = c.rows, outputs = c.outputs;
  __nv_bfloat16 *w, *x, *y;
  int* status;
  cudaMalloc(&w, (size_t)M * K * 2);
  cudaMalloc(&x, (size_t)rows * K * 2);
  cudaMalloc(&y, (size_t)rows * outputs * 2);
  cudaMalloc(&status, 4);
  cudaMemset(status, 0, 4);
  fill<<<256, 256>>>(w, (int64_t)M * K, 1);
  fill<<<256, 256>>>(x, (int64_t)rows * K, 2);
  TmaMap wmap;
  XMaps xmaps;
  if (!encode_bf16_map(&wmap, w, M, K, K, kGemmWeightBox) || !encode_x_maps(&xmaps, x, rows, K, K)) { complain("maps", -1, -1, -1); return; }
  const GemmParams p{outputs, K, rows, nullptr, c.glu ? ACT_GLU : ACT_NONE, 0, nullptr, y, outputs, status, 1.0f, 0.0f, 0x7fffffff, nullptr, 0};
  std::vector<uint16_t> want((size_t)rows * outputs), got(want.size());
  const auto launch = [&](int rank, int role, int use, std::vector<uint16_t>& out) {
    const int where[3] = {rank, role, use};
    int raised = 0;
    cudaMemcpyToSymbol(g_give_up, where, sizeof where);
    cudaMemset(y, 0xff, want.size() * 2);
    if (launch_tiles_of(wmap, xmaps, p) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) return -1;
    cudaMemcpy(out.data(), y, out.size() * 2, cudaMemcpyDeviceToHost);
    cudaMemcpy(&raised, status, 4, cudaMemcpyDeviceToHost);
    cudaMemset(status, 0, 4);
    return raised;
  };
  if (launch(-1, -1, -1, want) != 0) { complain("undisturbed", -1, -1, -1); return; }
  tries([&](int rank, int role, int use) {
    if (complaints) return;
    const auto t0 = std::chrono::steady_clock::now();
    const int raised = launch(rank, role, use, got);
    const double s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    ++tried;
    if (raised != 1) complain("status not raised", rank, role, use);
    if (s > 1.0) complain("slow", rank, role, use);
    if (raised >= 0 && (launch(-1, -1, -1, got) != 0 || got != want)) complain("the launch after it", rank, role, use);
  });
  cudaFree(w);
  cudaFree(x);
  cudaFree(y);
  cudaFree(status);
}

template <int BN, bool GLU, int SL>
void run_pairs(int outputs, int K, int rows, int pairs) {
  using T = Tile<BN, GLU, SL>;
  const int nk = ((K + kBK - 1) / kBK + SL - 1) / SL, mine = (outputs + 255) / 256 * ((rows + BN - 1) / BN) / pairs, uses = mine * nk;   // of every pair, at least
  run(Case{outputs, K, rows, GLU}, [&](const TmaMap& w, const XMaps& x, const GemmParams& p) { return launch_tiles<BN, GLU, SL>(w, x, p, pairs, nullptr); },
      [&](const auto& disturbed) {
        for (int use : {0, 1, T::kStages - 1, T::kStages, T::kStages + 1, nk - 1, nk, nk + 1, 2 * T::kStages + 3, uses - 1}) {
          if (use >= uses) continue;
          for (int rank = 0; rank < 2; ++rank) disturbed(rank, kCopies, use);
          disturbed(0, kMmas, use);
        }
        for (int tile : {2, 3, mine - 1})
          if (tile >= 2 && tile < mine) disturbed(0, kMmaTiles, tile);
        for (int tile : {0, 1, mine - 1})
          for (int rank = 0; rank < 2; ++rank) disturbed(rank, kStores, tile);
      });
}

template <int BN, bool GLU, bool DEEP>
void run_one(int outputs, int K, int rows) {
  using T = OneTile<BN, GLU, DEEP>;
  const int nk = (K + kBK - 1) / kBK;
  run(Case{outputs, K, rows, GLU}, [&](const TmaMap& w, const XMaps& x, const GemmParams& p) { return launch_one_stages<BN, GLU, DEEP>(w, x, p, nullptr); },
      [&](const auto& disturbed) {
        for (int use : {0, 1, T::kStages - 1, T::kStages, T::kStages + 1, nk - 1}) {
          if (use >= nk) continue;
          disturbed(0, kCopies, use);
          disturbed(0, kMmas, use);
        }
        disturbed(0, kStores, 0);
      });
}

}  // namespace
}  // namespace emelb

int main() {
  using namespace emelb;
  run_pairs<32, false, 2>(1024, 1000, 100, 2);
  run_pairs<128, false, 2>(1024, 1000, 500, 2);
  run_pairs<256, false, 1>(1024, 1000, 1000, 2);
  run_pairs<128, true, 1>(768, 520, 500, 3);
  run_one<16, false, true>(1000, 1000, 16);
  run_one<64, false, false>(1000, 1000, 200);
  run_one<128, false, false>(1000, 1000, 300);
  run_one<16, true, true>(520, 1000, 16);
  std::printf("%d %d\n", tried, complaints);
  return complaints != 0;
}
