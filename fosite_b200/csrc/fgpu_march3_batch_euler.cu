// fgpu_march3_batch_euler.cu -- the z-marching stage kernels of ensembles of ideal-gas 3D grids
// (fgpu_march3.cuh).
#include "fgpu_march3.cuh"
#include "fgpu_march_inst.cuh"

namespace fgpu {
namespace {

template <bool PRIM>
struct March {
  template <int LIM, bool RED, bool SRC>
  struct K {
    static constexpr auto kernel = batched_march3_kernel<true, PRIM, kMarchTX, kMarchTY, 2, LIM, RED, SRC>;
    static constexpr size_t SMEM = March3Layout<Phys<3, true>::V, kMarchTX, kMarchTY>::SMEM;
    static void configure() { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); }
    static void run(const StageArgs* args, const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s) {
      kernel<<<nblocks, kMarchTX * kMarchTY, SMEM, s>>>(args, maps, queue);
    }
  };
};

}  // namespace

cudaError_t march3_batch_launch_euler(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                   const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s) {
  if (prim) launch_family<March<true>::K, true>(lim, red, plain, args, maps, queue, nblocks, s);
  else launch_family<March<false>::K, true>(lim, red, plain, args, maps, queue, nblocks, s);
  return cudaGetLastError();
}
void march3_batch_configure_euler(bool prim, int lim) {
  if (prim) configure_family<March<true>::K, true>(lim);
  else configure_family<March<false>::K, true>(lim);
}
}  // namespace fgpu
