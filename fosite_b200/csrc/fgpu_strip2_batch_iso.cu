// fgpu_strip2_batch_iso.cu -- the strip-marching stage kernels of ensembles of isothermal 2D grids
// (fgpu_strip2.cuh).
#include "fgpu_march_inst.cuh"
#include "fgpu_strip2.cuh"

namespace fgpu {
namespace {

template <bool PRIM>
struct Strip {
  template <int LIM, bool RED, bool SRC>
  struct K {
    static constexpr auto kernel = batched_strip2_kernel<false, PRIM, kStripWarps, kStripMinBlocks, LIM, RED, SRC>;
    static constexpr size_t SMEM = Strip2Layout<Phys<2, false>::V>::smem(kStripWarps);
    static void configure() { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); }
    static void run(const StageArgs* args, const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s) {
      kernel<<<nblocks, kStripWarps * 32, SMEM, s>>>(args, maps, queue);
    }
  };
};

}  // namespace

cudaError_t strip2_batch_launch_iso(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                   const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s) {
  if (prim) launch_family<Strip<true>::K, false>(lim, red, plain, args, maps, queue, nblocks, s);
  else launch_family<Strip<false>::K, false>(lim, red, plain, args, maps, queue, nblocks, s);
  return cudaGetLastError();
}
void strip2_batch_configure_iso(bool prim, int lim) {
  if (prim) configure_family<Strip<true>::K, false>(lim);
  else configure_family<Strip<false>::K, false>(lim);
}
}  // namespace fgpu
