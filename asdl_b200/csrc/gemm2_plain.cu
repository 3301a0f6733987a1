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
  // A chained launch fills the SMs as the kernel before leaves them, two CTAs on some and none on others, where a plain one gives each SM
  // one first.  That matters where a few more CTAs than SMs have long epilogues, of 4-byte stores: symmetric products of 64 rows with beta, us
  // plainly -> chained: n = 2101 (153 tiles) 21.6 -> 22.9; but 1801 (120) 18.0 -> 17.5, 2001 (136) 18.5 -> 17.5 (beta 0: 15.4 -> 14.4), 2177 (171) 27.6 ->
  // 27.2.
  const bool uneven = probs == nullptr && single.nsplit == 1 && single.C != nullptr &&
                      ((single.ldc & 3) != 0 || (reinterpret_cast<uintptr_t>(single.C) & 15) != 0) && n_work > n_sms && 8 * n_work <= 9 * n_sms;
  launch_behind(g2_may_chain(probs) && !uneven, umma_gemm2_kernel<128, 4, 2, 1>, dim3(grid), dim3(G2Plain::THREADS), G2Plain::SMEM_BYTES, stream, single, probs, work, n_work, prefix, n_probs);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

}  // namespace b200
