// The "plain" flavour of the persistent tcgen05 GEMM (see umma_gemm2.cuh), in a translation
// unit of its own so that the flavours compile in parallel.
#include <algorithm>

#include "gemm2_host.h"

namespace b200 {

void g2_run_plain(const GemmProblem2& single, const GemmProblem2* probs, const GemmWork2* work, int n_work,
                 int n_sms, cudaStream_t stream, const int* prefix, int n_probs) {
  if (n_work <= 0) return;
  static bool attr_set_on[64] = {false};
  int dev = 0;
  B200_CUDA_CHECK(cudaGetDevice(&dev));
  bool& attr_set = attr_set_on[dev & 63];
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(umma_gemm2_kernel<128, 4, 2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         G2Plain::SMEM_BYTES));
    attr_set = true;
  }
  const int grid = std::min(n_work, 2 * n_sms);
  // Chained at any number of tiles.  Behind a chain two CTAs come to some SMs and none to others, and where a few more tiles than SMs
  // have the longest epilogues, symmetric ones with beta and 4-byte stores, a plain launch is up to 1.5 us faster: 153 tiles, us plainly ->
  // chained: 64 rows x 2057 17.6 -> 18.5, 64 x 2101 20.0 -> 21.5, 96 x 2101 20.3 -> 22.1, 128 x 2173 25.3 -> 25.8.  But 32 x 2101 19.8 -> 19.0,
  // 192 x 2101 21.8 -> 20.7, 256 x 2101 22.5 -> 21.6, and everything else of 150 - 168 tiles gains as at other counts: 64 x 2101 and
  // 2171 without beta 17.4 -> 17.4 and 20.8 -> 19.9, 1280 x 1793 of 64 rows 17.6 -> 16.2 and with beta 22.2 -> 21.0, 1408 x 1665 17.7 -> 16.7.
  launch_behind(g2_may_chain(probs), umma_gemm2_kernel<128, 4, 2, 1>, dim3(grid), dim3(G2Plain::THREADS), G2Plain::SMEM_BYTES, stream, single, probs, work, n_work, prefix, n_probs);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

}  // namespace b200
