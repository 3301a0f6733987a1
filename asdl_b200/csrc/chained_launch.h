// Kernels that follow each other on a stream with a programmatic dependency: the next one is brought onto the SMs while the one
// before it finishes, and waits there before it touches memory, so the few microseconds between two kernels overlap.
//
// Every kernel launched this way calls chain_wait() before its first access to global memory, reads and writes alike.  The wait
// ends when the kernel before it has finished and its writes are visible; since that one waited in the same way, everything
// before it has finished too.  One exception: the first kernel of a chain is launched plainly, so that all older work has finished
// before any kernel of the chain is on an SM, and bn_apply and bn_dx (batchnorm.cu) read ahead of their wait what is older than
// the chain.  That holds only as long as bn_sums, the first kernel there, is launched plainly.  What a kernel of the chain has written is read by ordinary loads, not through __ldg or a
// const __restrict__ parameter: the read-only path is for data that nobody writes while the kernel is resident, and the compiler
// may move such loads ahead of the wait.  __ldcg takes its pointer from after_wait().  chain_next() lets the next kernel come as soon as all CTAs of this one have called it.
// Launched plainly -> chained, passes in turn: 8192 x 1024 bf16 samples 27.3 -> 22.9 us, 12608 x 768 fp32 samples 52.9 -> 46.9, the
// convolution factors of 32 x 256 x 14 x 14 bf16 47.7 -> 41.7 and of 128 x 64 x 32 x 32 fp32 82.6 -> 78.6, 1024 x 4096 between fp32 factors 153 -> 149.
// What a chained kernel gets of the SMs while the one before it still runs can be uneven (gemm2_plain.cu has what that costs) or short of
// L1 cache: one launch is plain for that reason (conv_gram.cu).
// A kernel that is launched plainly behind a chain waits for its end as usual; a captured chain becomes programmatic edges.
#pragma once
#include <utility>

#include "host_utils.h"

namespace b200 {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The same pointer, for loads that the compiler would move ahead of chain_wait().
template <typename T>
__device__ __forceinline__ T* after_wait(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

// `chained` false: an ordinary launch of the same kernel, whose wait then ends at once.
template <typename... Params, typename... Args>
void launch_behind(bool chained, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  config.attrs = &attribute;
  config.numAttrs = chained ? 1 : 0;
  B200_CUDA_CHECK(cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...));
}

template <typename... Params, typename... Args>
void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  launch_behind(true, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace b200
