// fgpu_march3_iso.cu -- the z-marching stage kernels of isothermal 3D meshes (fgpu_march3.cuh).
#include "fgpu_march3.cuh"
#include "fgpu_march_inst.cuh"

namespace fgpu {
namespace {

constexpr int kMinBlocks = 2;   // resident 256-thread blocks per SM (128 registers, 89 KB shared memory each)

template <bool PRIM>
struct March {
  template <int LIM, bool RED, bool SRC>
  struct K {
    static constexpr auto kernel = march3_kernel<false, PRIM, kMarchTX, kMarchTY, kMinBlocks, LIM, RED, SRC>;
    static constexpr size_t SMEM = March3Layout<Phys<3, false>::V, kMarchTX, kMarchTY>::SMEM;
    static void configure() { cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM); }
    static void run(int kchunk, cudaStream_t s, const StageArgs* A, const CUtensorMap* map, bool tma) {
      const Grid& g = A->g;
      const dim3 grid((g.nx + kMarchTX - 1) / kMarchTX, (g.ny + kMarchTY - 1) / kMarchTY, (g.nz + kchunk - 1) / kchunk);
      kernel<<<grid, kMarchTX * kMarchTY, SMEM, s>>>(*A, *map, tma ? 1 : 0);
    }
  };
};

}  // namespace

cudaError_t march3_launch_iso(bool prim, int lim, int kchunk, cudaStream_t s, const StageArgs& A, const CUtensorMap& map,
                             bool tma) {
  const bool red = A.cfl_mode || A.last_stage || A.err_low, plain = plain_stage(A);
  if (prim) launch_family<March<true>::K, false>(lim, red, plain, kchunk, s, &A, &map, tma);
  else launch_family<March<false>::K, false>(lim, red, plain, kchunk, s, &A, &map, tma);
  return cudaGetLastError();
}
void march3_configure_iso(bool prim, int lim) {
  if (prim) configure_family<March<true>::K, false>(lim);
  else configure_family<March<false>::K, false>(lim);
}
}  // namespace fgpu
