// The kernels of the far field's two passes over atoms.  Each holds every series
// length's code (kernels.cuh) and takes the compiler up to half a minute, so this
// file is compiled once per GLST_PART, all of them at the same time (build.py).
#include "kernels.cuh"

namespace glst {
namespace dev {

#if GLST_PART == 0
__global__ void __launch_bounds__(kSfThreads, 4)
k_structure_factors(const __grid_constant__ SfArgs a, uint32_t cell_base) {
  const uint32_t quads = a.n_tiles / kSfWarps;
  const uint32_t c = blockIdx.x / quads;
  sf_block(a, blockIdx.x - c * quads, cell_base + c * a.cells);
}

#elif GLST_PART == 1
__global__ void __launch_bounds__(kLrThreads, 3) k_long_range(const __grid_constant__ LrArgs a) {
  extern __shared__ float4 s_lr[];
  for (uint32_t i = threadIdx.x; i < a.tab4; i += kLrThreads) s_lr[i] = a.tab[i];
  __syncthreads();
  const uint64_t item = (uint64_t)blockIdx.x * kLrWarps + (threadIdx.x >> 5);
  const uint32_t chunk = (uint32_t)(item / a.ncell);
  if (chunk < a.n_chunks) lr_items<true>(a, (uint32_t)(item - (uint64_t)chunk * a.ncell), chunk);
}

#elif GLST_PART == 2
__global__ void __launch_bounds__(kLrThreads, 3) k_long_range_general(const __grid_constant__ LrArgs a) {
  const uint64_t item = (uint64_t)blockIdx.x * kLrWarps + (threadIdx.x >> 5);
  const uint32_t chunk = (uint32_t)(item / a.ncell);
  if (chunk < a.n_chunks) lr_items<false>(a, (uint32_t)(item - (uint64_t)chunk * a.ncell), chunk);
}

#elif GLST_PART == 3
// item (a, b) = (quad of direction tiles, first of sf.cells cells); always one
// CTA per item (inside a loop over items the moments went to local memory)
__global__ void __launch_bounds__(kSfThreads, 4) k_structure_factors_multi(const SysDesc *__restrict__ sys,
                                                                          const WorkItem *__restrict__ items,
                                                                          uint32_t n) {
  const WorkItem w = items[blockIdx.x];
  const SfArgs a = sys[w.sys].sf;
  sf_block(a, w.a, w.b);
}

#elif GLST_PART == 4
// item (a, b) = (first of kLrWarps cells, long-range chunk); out of line, as
// the structure factors
static __device__ __noinline__ void lr_item(const LrArgs &a, uint32_t cell, uint32_t chunk) { lr_items<false>(a, cell, chunk); }

__global__ void __launch_bounds__(kLrThreads, 3) k_long_range_multi(const SysDesc *__restrict__ sys,
                                                                    const WorkItem *__restrict__ items,
                                                                    uint32_t n) {
  __shared__ LrArgs s_args;
  for (uint32_t it = blockIdx.x; it < n; it += gridDim.x) {
    const WorkItem w = items[it];
    if (threadIdx.x == 0) s_args = sys[w.sys].lr;
    __syncthreads();
    const uint32_t cell = w.a + (threadIdx.x >> 5);
    if (cell < s_args.ncell) lr_item(s_args, cell, w.b);
    __syncthreads();
  }
}
#endif

}  // namespace dev
}  // namespace glst
