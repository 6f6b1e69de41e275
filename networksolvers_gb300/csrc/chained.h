// Launches that overlap the end of the kernel before them in the stream (programmatic dependent
// launch): the next kernel's blocks are placed while the last ones of this kernel run, and wait
// for its end before they touch memory, which saves the gap between two kernels (the small
// regions of a sweep are a chain of kernels of 5 to 10 us).  Used by the site-operator products
// of few rows, the permutations, the slicing and the split products: tree TDVP step 2.10 -> 1.89
// ms, DMRG run (N = 20) 167 -> 160 ms, XXZ region step 3.19 -> 3.05 ms, expansion 24.5 -> 24.0.
// Not by the site-operator products of many rows (eigensolve at bond dimension 1024 6.61 ms with
// them, 6.50 without: their loads lose the read-only path), the 16 x 16-tile products (the
// factorization of 950 x 950 9.5 ms with them and 9.3 without; DMRG run 157) and the divide and
// conquer's kernels (XXZ region step 3.10 with them).
// A kernel launched by launch_chained starts with chained_start(); since it ends after the kernel
// before it, whatever follows sees both.
#pragma once

#include "nsg_internal.h"

#include <utility>

namespace nsg {

inline cudaLaunchAttribute chained_attribute() {
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  return a;
}

template <typename... E, typename... A>
void launch_chained(nsg_ctx* c, void (*kernel)(E...), dim3 grid, dim3 block, size_t smem, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1] = {chained_attribute()};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = c->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  NSG_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

__device__ __forceinline__ void chained_start() {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// For a __restrict__ pointer to data only read, whose loads the compiler may move past a fence:
// the pointer itself comes after the wait.
template <typename P>
__device__ __forceinline__ P* after_start(P* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}

}  // namespace nsg
