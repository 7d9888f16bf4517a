// fgpu_strip2_euler.cu -- the strip-marching stage kernels of ideal-gas 2D meshes (fgpu_strip2.cuh).
#include "fgpu_march_inst.cuh"
#include "fgpu_strip2.cuh"

namespace fgpu {
namespace {

template <bool PRIM>
struct Strip {
  template <int LIM, bool RED, bool SRC>
  struct K {
    static constexpr auto kernel = strip2_kernel<true, PRIM, kStripWarps, kStripMinBlocks, LIM, RED, SRC>;
    static constexpr size_t SMEM = Strip2Layout<Phys<2, true>::V>::smem(kStripWarps);
    static void configure() { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); }
    static void run(int rows, cudaStream_t s, const StageArgs* A, const CUtensorMap* map, bool tma) {
      StageArgs B = *A;
      B.kchunk = rows;
      const int blocks = (strip2_warps(A->g.nx, A->g.ny, rows) + kStripWarps - 1) / kStripWarps;
      kernel<<<blocks, kStripWarps * 32, SMEM, s>>>(B, *map, tma ? 1 : 0);
    }
  };
};

}  // namespace

cudaError_t strip2_launch_euler(bool prim, int lim, int rows, cudaStream_t s, const StageArgs& A, const CUtensorMap& map,
                             bool tma) {
  const bool red = A.cfl_mode || A.last_stage || A.err_low, plain = plain_stage(A);
  if (prim) launch_family<Strip<true>::K, true>(lim, red, plain, rows, s, &A, &map, tma);
  else launch_family<Strip<false>::K, true>(lim, red, plain, rows, s, &A, &map, tma);
  return cudaGetLastError();
}
void strip2_configure_euler(bool prim, int lim) {
  if (prim) configure_family<Strip<true>::K, true>(lim);
  else configure_family<Strip<false>::K, true>(lim);
}
}  // namespace fgpu
