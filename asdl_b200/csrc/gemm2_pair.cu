// The CTA-pair flavour of the persistent tcgen05 GEMM (see umma_gemm2_pair.cuh), in a translation
// unit of its own so that the flavours compile in parallel.
#include <algorithm>

#include "gemm2_host.h"
#include "umma_gemm2_pair.cuh"

namespace b200 {

int g2_pair_tiles(const GemmProblem2& P) {
  const int T = (P.tiles_m + 1) / 2;
  return (P.flags & G2F_SYM) ? T * (T + 1) / 2 : T * P.tiles_n;
}

// 256 x 512 tiles of a pair, where they take fewer tensor clocks (a K block of 256 x 256 takes the 620 clocks that L2 needs for it) and the
// K range is long enough for their epilogue, none of which is beside the products of the next tile.  Symmetric bf16 products, 256 x
// 256 -> 256 x 512, graph replay: 8192 x 4096 samples 118 -> 112 us (pass after pass at the power limit 137 -> 129), 8192 x 3072 101.2 -> 96.3,
// 8191 x 4032 113.9 -> 104.8, 5000 x 3333 118.1 -> 113.7; but 4096 x 4096 65.9 -> 66.3, 2048 x 4096 38.0 -> 38.8, 1600 x 4096 33.1 -> 34.7.
static int wide_tiles(const GemmProblem2& P, int pairs) {
  if (P.nsplit > 1 || P.K < 72 * G2_BK) return 0;
  const int T = (P.tiles_m + 1) / 2, narrow = g2_pair_tiles(P);
  int wide = 0;
  for (int TM = 0; TM < T; ++TM) wide += P.flags & G2F_SYM ? TM / 2 + 1 : (P.tiles_n + 1) / 2;
  const long long narrow_clocks = 620LL * ((narrow + pairs - 1) / pairs), wide_clocks = 1050LL * ((wide + pairs - 1) / pairs);
  return wide_clocks < narrow_clocks ? wide : 0;
}

template <int PARTS, int HALVES>
static void run_pair(const GemmProblem2& single, int n_work, int n_sms, cudaStream_t stream) {
  static bool attr_set_on[64] = {false};
  int dev = 0;
  B200_CUDA_CHECK(cudaGetDevice(&dev));
  bool& attr_set = attr_set_on[dev & 63];
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(umma_gemm2_pair_kernel<PARTS, HALVES>, cudaFuncAttributeMaxDynamicSharedMemorySize, G2P_SMEM_BYTES));
    attr_set = true;
  }
  const int pairs = std::max(1, std::min(n_work, n_sms / 2));
  launch_chained(umma_gemm2_pair_kernel<PARTS, HALVES>, dim3(2 * pairs), dim3(G2P_THREADS), G2P_SMEM_BYTES, stream, single, n_work);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

void g2_run_pair(const GemmProblem2& single, int n_work, int n_sms, cudaStream_t stream) {
  if (n_work <= 0) return;
  if (single.flags & G2F_SPLIT2)
    run_pair<2, 1>(single, n_work, n_sms, stream);
  else if (const int wide = wide_tiles(single, n_sms / 2))
    run_pair<1, 2>(single, wide, n_sms, stream);
  else
    run_pair<1, 1>(single, n_work, n_sms, stream);
}

}  // namespace b200
