// fgpu_march_launch.h -- host entries of the marching stage kernels (fgpu_strip2.cuh: 2D strips,
// fgpu_march3.cuh: 3D tiles).
//
// The kernel instantiations live in translation units per family and physics
// (fgpu_strip2_*.cu, fgpu_strip2_batch_*.cu, fgpu_march3_*.cu), which compile in parallel.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdlib>
#include "fgpu_kernels.cuh"

namespace fgpu {

// 3D tile: 32 x 8 cells, two 256-thread blocks per SM
constexpr int kMarchTX = 32, kMarchTY = 8;
// 2D: warps per block and resident blocks per SM (16 warps of 128 registers)
constexpr int kStripWarps = 4, kStripMinBlocks = 4;
constexpr int kStripW = 30;   // columns of a warp's strip

// Launch one stage on the marching layout.  lim: the compiled-in limiter (compiled_limiter); tma: map
// is the tensor map of the stage input (even x extent), otherwise rows are copied by element.  2D:
// rows per warp; 3D: the z extent that a block marches through (A.kchunk).
cudaError_t strip2_launch_euler(bool prim, int lim, int rows, cudaStream_t s, const StageArgs& A,
                                const CUtensorMap& map, bool tma);
cudaError_t strip2_launch_iso(bool prim, int lim, int rows, cudaStream_t s, const StageArgs& A, const CUtensorMap& map,
                              bool tma);
cudaError_t march3_launch_euler(bool prim, int lim, int kchunk, cudaStream_t s, const StageArgs& A,
                                const CUtensorMap& map, bool tma);
cudaError_t march3_launch_iso(bool prim, int lim, int kchunk, cudaStream_t s, const StageArgs& A,
                              const CUtensorMap& map, bool tma);
// Batched ensembles of 2D grids: one block per entry (grid, first warp, has a tensor map, 0) of the
// queue, the rows per warp taken from the grid's stage arguments (kchunk); args[grid] and
// maps[grid] (device arrays) the stage arguments and the tensor map of the stage input of each
// grid; lim the compiled-in limiter shared by every grid, 0 when the grids differ or read it from
// their arguments; red: some grid's stage reduces CFL / CheckData / error-norm maxima (else the
// kernel form without the reductions runs); plain: every grid's stage is a plain_stage.
cudaError_t strip2_batch_launch_euler(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                      const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s);
cudaError_t strip2_batch_launch_iso(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                    const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s);
// Batched ensembles of 3D grids: one block per entry (grid, bx, by, bz), bit 30 of the grid index
// set when it has tensor maps; the z extent of a block from the grid's stage arguments (kchunk).
cudaError_t march3_batch_launch_euler(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                      const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s);
cudaError_t march3_batch_launch_iso(bool prim, int lim, bool red, bool plain, const StageArgs* args,
                                    const CUtensorMap* maps, const int4* queue, int nblocks, cudaStream_t s);
inline int march_sms() {
  static const int sms = [] {
    int d = 0, n = 148;
    if (cudaGetDevice(&d) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
    return n > 0 ? n : 148;
  }();
  return sms;
}
// Rows per warp of 2D grids of `warp_rows` strip rows in all: as few as keep all warps resident
// in one wave (one SM holds kStripWarps * kStripMinBlocks of them), whole waves of at most 24 rows
// beyond that.  A row costs a lone warp 2.1 us and a chunk's opening about 1.5 rows, so that small
// grids want single rows (64^2 ideal-gas step: 34 / 41 / 54 us with 1 / 2 / 4 rows) and one wave is
// better than two of half the rows (186 x 390 disk: 52 / 70 us with 2 / 1 rows); 48 disks in one
// batch take 1.03 / 0.98 / 1.01 / 1.19 ms a step with 12 / 24 / 36 / 48 rows.
// FGPU_TMA_TPB fixes the count in units of 8 rows.
inline int strip_rows(long long warp_rows) {
  if (const char* e = std::getenv("FGPU_TMA_TPB")) {
    const int v = std::atoi(e);
    if (v > 0) return 8 * v;
  }
  const long long wave = (long long)march_sms() * kStripWarps * kStripMinBlocks;
  const long long waves = (warp_rows + wave * 24 - 1) / (wave * 24);
  return (int)std::max<long long>(1, (warp_rows + wave * waves - 1) / (wave * waves));
}
inline long long strip_warp_rows(const Grid& g) { return (long long)((g.nx + kStripW - 1) / kStripW) * g.ny; }
// The z extent that a block of a 3D grid marches through: two blocks a SM run at once, a block of c
// planes takes about c + 2 plane times (its opening), so the chunk that minimises waves x (c + 2).
// 90 x 75 x 61: chunks of 4 / 8 / 16 planes 571 / 535 / 835 us a Dormand-Prince step.
inline int march_chunk(const Grid& g, int copies) {
  const long long tiles = (long long)copies * ((g.nx + kMarchTX - 1) / kMarchTX) * ((g.ny + kMarchTY - 1) / kMarchTY);
  int best = 1;
  double least = 1e300;
  for (int c = 1; c <= 64 && c <= g.nz; ++c) {
    const long long waves = (tiles * ((g.nz + c - 1) / c) + 2 * march_sms() - 1) / (2 * march_sms());
    const double t = (double)waves * (c + 2);
    if (t < least) { least = t; best = c; }
  }
  return best;
}
// the limiter code a stage's kernel is compiled for: minmod, MC, van Leer; 0 when the kernel reads
// limiter and reconstruction order from the arguments (a switch per slope).  MC with theta = 1 is
// minmod: the central difference is the mean of the one-sided ones, and rounding is monotonic, so
// (qp - qm)/2 is never the smallest of the three in magnitude.
inline int compiled_limiter(int limiter, bool constant_recon, double theta) {
  if (constant_recon) return 0;
  if (limiter == LIM_MC) return theta == 1.0 ? LIM_MINMOD : LIM_MC;
  return (limiter == LIM_MINMOD || limiter == LIM_VANLEER) ? limiter : 0;
}
// opt the kernels of a limiter into their dynamic shared memory (the current device; a handle or
// batch configures those that it launches)
void strip2_configure_euler(bool prim, int lim);
void strip2_configure_iso(bool prim, int lim);
void strip2_batch_configure_euler(bool prim, int lim);
void strip2_batch_configure_iso(bool prim, int lim);
void march3_configure_euler(bool prim, int lim);
void march3_configure_iso(bool prim, int lim);
void march3_batch_configure_euler(bool prim, int lim);
void march3_batch_configure_iso(bool prim, int lim);

}  // namespace fgpu
