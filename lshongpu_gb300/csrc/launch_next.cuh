// Launches whose kernel may start as the blocks of the stream's previous kernel leave (programmatic
// dependent launch): its blocks take the free places and stand at grid_ready() until every earlier
// kernel of the stream has completed and its writes are visible.  A batch of a few queries is a
// chain of ten short kernels, and the gaps between them -- one kernel's last block to the next one's
// first instruction, 1.3 to 3.4 us -- were a fifth of it.
//
// A kernel launched by launch_next begins with grid_ready(), before it reads or writes memory:
// completion of a kernel then implies completion of all before it, as with ordinary launches, and
// ordinary launches and copies before or after it wait as they always do.  No kernel lets its
// successor start before its own blocks leave: blocks that wait early hold places and shared
// memory that the kernels before them still spread over.  Measured, us a batch (ordinary launches;
// with launch_next; and with griddepcontrol.launch_dependents at each kernel's start): 1,000
// queries x 100k 106, 86, 110; one query x 1.2M 103, 91, 92; 777 x 333k (d = 37, k = 100) 155, 141,
// 180; exact, 1,000 x 100k 98, 82, 100.
#pragma once
#include "common.cuh"

namespace lshg {

__device__ __forceinline__ void grid_ready() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Counters of a later kernel, zeroed by the first kernel of a batch: a memset of its own costs an ordinary
// launch's gaps on both sides (5 us).
__device__ __forceinline__ void zero_counters(int* c, int n) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) c[i] = 0;
}

template <typename... P, typename... A>
void launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  LSHG_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

}  // namespace lshg
