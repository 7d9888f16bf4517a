// fgpu_strip2.cuh -- the 2D stage kernel: every warp marches a strip of columns along y
// (sm_100a).
//
// Same right-hand side and epilogues as stage_tile (fgpu_kernels.cuh: fosite's ComputeRHS,
// timedisc_base.f90:1073-1271, fused with its consumer).  A warp owns 30 columns (lanes 1 to 30;
// lanes 0 and 31 carry the neighbours' face states) and A.kchunk rows, and works alone: no block
// barrier in the loop, so that small grids, whose time is the latency of one warp's chain, and
// large ones, where the other warps of the scheduler fill the gaps, run the same code.
//   * the rows of the strip, two halo columns on each side, arrive in the warp's ring of eight
//     row slots, one bulk tensor copy (3-D map x, y, variable) per row completing on an mbarrier;
//     strips on a periodic face, and meshes of odd x extent (rows not 16-byte aligned), fetch the
//     same row with 8-byte cp.async whose sources wrap; y ghost rows fetch the row they copy;
//   * x: the lane's own cell is reconstructed, the plus face state goes to the next lane and the
//     minus-face flux back by shuffles;
//   * y stays in registers: the plus face state and the flux of the last row;
//   * ghosts of the x faces and frame changes (FARGO) are applied once per staged point, four rows
//     at a time.
// What bounds it: the serial FP64 chains of a row (about 5 cycles an instruction for a lone warp) at
// the 16 warps an SM that 128 registers allow: 47% issue activity, 820 warp instructions a row,
// 40% of them FP64 (1024^2 ideal gas, van Leer: 65 us a stage against 130 us for the tiles of
// shared-memory slopes and fluxes, which spent as many instructions again on index arithmetic
// and barriers).  Measured against it and dropped: 20 or 24 warps an SM (96 / 80 registers: 15%
// and 65% slower, spills), both directions' fluxes interleaved (4% slower, spills), the opening
// rows in code of their own (the loop leaves the instruction cache: 2.3 times slower).
// Requirements (checked on the host): a plain or formed stage input (no k-sums in the stencil),
// no accretion rows, no interface-flux output.
#pragma once
#include <cuda.h>
#include "fgpu_bulk.cuh"
#include "fgpu_kernels.cuh"

namespace fgpu {

template <int V>
struct Strip2Layout {
  static constexpr int W = 30, RW = W + 4, NSLOT = 8;
  static constexpr int BOX = V * RW;                        // one tensor copy: [V][RW]
  static constexpr int ROW = (BOX + 15) / 16 * 16;          // slots stay 128-byte aligned
  static constexpr size_t WARP_BYTES = 8 * (size_t)NSLOT * ROW;
  static constexpr size_t smem(int warps) { return warps * (WARP_BYTES + 8 * NSLOT); }
};

// Warps of one grid: strips of 30 columns times chunks of rows
__host__ __device__ inline int strip2_strips(int nx) { return (nx + 29) / 30; }
__host__ __device__ inline int strip2_warps(int nx, int ny, int rows) {
  return strip2_strips(nx) * ((ny + rows - 1) / rows);
}

// One block: warps first .. first + NW - 1 of the grid of A (those past the last idle).
// LIM > 0: the limiter is compiled in (linear reconstruction); LIM = 0: the limiter and the
// reconstruction order are read from the arguments.  RED = false: a stage without CFL,
// CheckData or error-norm reduction, whose maxima are then dead code.  SRC = false: a stage without
// sources or frame changes (plain_stage).
template <bool EU, bool PRIM, int NW, int LIM, bool RED, bool SRC>
__device__ __forceinline__ void strip2_block(const StageArgs& A, const CUtensorMap* tmap, const bool use_tma,
                                             const int first) {
  using PH = Phys<2, EU>;
  using CE = Cells<2, EU>;
  constexpr int V = PH::V;
  using L = Strip2Layout<V>;
  constexpr int RW = L::RW, W = L::W, NSLOT = L::NSLOT;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(128) double strip2_smem[];
  __shared__ double sred[RED_STRIDE * NW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* const ring = strip2_smem + warp * (NSLOT * L::ROW);
  unsigned long long* const mbar =
      reinterpret_cast<unsigned long long*>(strip2_smem + NW * NSLOT * L::ROW) + warp * NSLOT;

  if (A.ctl && (A.ctl->stop | A.ctl->brk)) return;
  if (gated_out(A.ctl, A.gate)) return;
  const Grid& g = A.g;
  const PhysP& P = A.ph;
  const MetricP& M = A.mt;
  const double dt = A.dt_dev ? *A.dt_dev : A.dt;
  const bool roundtrip = EU && A.in.roundtrip;
  const StateRef& SR = A.rin.base ? A.rin : A.in;
  const int lim = LIM > 0 ? LIM : A.limiter;
  const bool crec = LIM > 0 ? false : A.constant_recon != 0;
  // FARGO: the stage input's frame changes (the chain of the stored state) and the subtraction of
  // the background velocity apply to every staged point
  const bool frames = SRC && (A.w_sub != nullptr || A.in.pre.n != 0);
  // the staged values are the reconstruction variables as they stand, else each staged point is
  // converted once
  const bool raw_ok = PRIM ? (SR.ready != 0) : (!roundtrip && !frames);
  const int nstrips = strip2_strips(g.nx);
  const int w = first + warp;
  const int rows = A.kchunk;
  const bool live = w < strip2_warps(g.nx, g.ny, rows);
  double cflv[4] = {0.0, 0.0, 0.0, 0.0};
  double errv = 0.0;
  int flags = 0;
  if (live) {
    const int i0 = (w % nstrips) * W;
    const int ex = min(W, g.nx - i0);
    const int ja = (w / nstrips) * rows, jb = min(g.ny, ja + rows);
    const int i = i0 + lane - 1;                 // the lane's column; box index lane + 1
    const int ip = min(i + 2, g.nx + 3);
    const bool own = lane >= 1 && lane <= ex;
    const int gxl = i0 == 0 ? 2 : 0, gxh = max(0, i0 + ex + 2 - g.nx);
    const bool tma = use_tma && !((gxl && g.bc[0] == BC_PERIODIC) || (gxh && g.bc[1] == BC_PERIODIC));

    // reconstruction variables of cell or ghost (gi, gj) from its primitive variables: the
    // CHECK_PMIN clamp, the co-moving frame last (the order of ComputeRHS:
    // AddBackgroundVelocity, CenterBoundary, SubtractBackgroundVelocity)
    auto finish = [&](double* p, int gi, int gj, double* R) {
      if (roundtrip) p[V - 1] = dmax(p[V - 1], P.pmin);
      if (PRIM) {
        if (SRC && A.w_sub) sub_velocity(p, A.w_sub[fargo_ix(g, gi, gj)], g.fdir);
#pragma unroll
        for (int v = 0; v < V; ++v) R[v] = p[v];
      } else {
        PH::p2c(p, R, P);
        if (SRC && A.w_sub) frame_change<V>(R, -1.0, A.w_sub[fargo_ix(g, gi, gj)], g.fdir);
      }
    };
    // primitive variables of the raw value u of interior cell (si, sj), real frame
    auto raw_prim = [&](double* u, int si, int sj, double* p) {
      if (PRIM && SR.ready) {
#pragma unroll
        for (int v = 0; v < V; ++v) p[v] = u[v];
      } else {
        if (SRC && SR.pre.n) apply_chain<V>(SR.pre, u, g, si, sj);
        PH::c2p(u, p, P);
      }
    };
    // a raw interior value of cell (gi, gj), in place
    auto conv = [&](double* u, int gi, int gj) {
      if (SRC && A.in.pre.n) apply_chain<V>(A.in.pre, u, g, gi, gj);
      if (PRIM || roundtrip) {
        double p[V];
        PH::c2p(u, p, P);
        finish(p, gi, gj, u);
      } else if (SRC && A.w_sub) {
        frame_change<V>(u, -1.0, A.w_sub[fargo_ix(g, gi, gj)], g.fdir);
      }
    };
    // the row that is fetched for row jr: its own, or the interior row a y ghost copies
    auto source_row = [&](int jr) {
      if (jr >= 0 && jr < g.ny) return jr;
      const bool lo = jr < 0;
      const int s = lo ? -jr : jr - (g.ny - 1), type = g.bc[lo ? 2 : 3];
      if (type == BC_PERIODIC) return lo ? g.ny - s : s - 1;
      if (type == BC_REFLECTING || type == BC_AXIS) return lo ? s - 1 : g.ny - s;
      return lo ? 0 : g.ny - 1;
    };
    auto slot = [&](int jr) { return ring + ((jr - (ja - 2)) & (NSLOT - 1)) * L::ROW; };
    auto bar = [&](int jr) { return &mbar[(jr - (ja - 2)) & (NSLOT - 1)]; };
    auto parity = [&](int jr) { return (unsigned)(((jr - (ja - 2)) / NSLOT) & 1); };
    auto issue = [&](int jr) __attribute__((always_inline)) {   // every lane
      const int src = source_row(jr);
      if (tma) {
        if (lane == 0) {
          mbar_expect_tx(bar(jr), 8u * L::BOX);
          tma_load_box<3>(slot(jr), tmap, bar(jr), i0 - 2, src, 0);
        }
      } else {
        double* const S = slot(jr);
        const double* const b = SR.base + (long long)g.nx * src;
        const int ga = wrap_index(i0 + lane - 2, g.nx, g.bc), gb = wrap_index(i0 + 30 + lane, g.nx, g.bc);
#pragma unroll
        for (int v = 0; v < V; ++v) {
          cp_async8(S + v * RW + lane, b + (long long)v * g.n + ga);
          if (lane < RW - 32) cp_async8(S + v * RW + lane + 32, b + (long long)v * g.n + gb);
        }
        cp_async_arrive(bar(jr));
      }
    };
    if (lane < NSLOT) mbar_init(&mbar[lane], tma ? 1 : 32);
    fence_proxy_async();
    __syncwarp();
    const int last = jb + 1;   // the last row fetched
    for (int jr = ja - 2; jr <= min(last, ja - 3 + NSLOT); ++jr) issue(jr);

    // the value of x ghost column lx of staged row jr (read before the row's conversion)
    auto xghost = [&](const double* S, int lx, int jr, double* R) {
      const int gi = i0 + lx - 2;
      const bool lo = gi < 0;
      const int type = g.bc[lo ? 0 : 1];
      double u[V], p[V];
      if (type == BC_ABSORBING) {
        // from the boundary cell and the next one inward (the box reaches two cells past the strip)
        const int i1 = lo ? 0 : g.nx - 1, i2 = lo ? 1 : g.nx - 2;
        double p1[V], p2[V];
#pragma unroll
        for (int v = 0; v < V; ++v) u[v] = S[v * RW + i1 - i0 + 2];
        raw_prim(u, i1, jr, p1);
#pragma unroll
        for (int v = 0; v < V; ++v) u[v] = S[v * RW + i2 - i0 + 2];
        raw_prim(u, i2, jr, p2);
        CE::absorbing_p(p1, p2, lo, 0, i1 + 2, (lo ? i2 : i1) + 2, P, M, p);
      } else {
        const int s = lo ? -gi : gi - (g.nx - 1);
        int si, lm;   // the copied cell and its box column (periodic: the wrapped value at its place)
        if (type == BC_PERIODIC) {
          si = lo ? g.nx - s : s - 1;
          lm = lx;
        } else {
          si = type == BC_NOGRAD ? (lo ? 0 : g.nx - 1) : (lo ? s - 1 : g.nx - s);
          lm = si - i0 + 2;
        }
#pragma unroll
        for (int v = 0; v < V; ++v) u[v] = S[v * RW + lm];
        raw_prim(u, si, jr, p);
        if (type == BC_REFLECTING || type == BC_AXIS) {
          p[1] = -p[1];
          if (SRC && type == BC_AXIS && M.curv) p[2] = -p[2];
        }
      }
      finish(p, gi, jr, R);
    };
    // Wait for rows r0 .. r0+3, then fill their ghost columns / convert their raw values in place
    // (four rows at once: the ghosts of an absorbing face take a warp as long for sixteen points as
    // for one).  Of the rows before and after the chunk only the lane's own column is read.
    bool lost = false;
    auto prepare = [&](int r0) __attribute__((always_inline)) {
      const int r1 = min(r0 + 4, last + 1);
#pragma unroll 1
      for (int jr = r0; jr < r1; ++jr) {
        if (!__all_sync(FULL, mbar_wait(bar(jr), parity(jr)))) lost = true;
        if (jr < ja || jr >= jb) {
          const bool outside = jr < 0 || jr >= g.ny;
          if (own && (outside || !raw_ok)) {
            double* const c = slot(jr) + lane + 1;
            double u[V], p[V];
#pragma unroll
            for (int v = 0; v < V; ++v) u[v] = c[v * RW];
            if (outside) {
              const int type = g.bc[jr < 0 ? 2 : 3];
              if (type == BC_ABSORBING) {
                CE::face_ghost_p(SR, g, P, M, 1, i, jr, 0, p);
              } else {
                raw_prim(u, i, source_row(jr), p);
                if (type == BC_REFLECTING || type == BC_AXIS) p[2] = -p[2];
              }
              finish(p, i, jr, u);
            } else {
              conv(u, i, jr);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) c[v * RW] = u[v];
            fence_proxy_async();
          }
        }
      }
      if (!raw_ok || gxl + gxh) {
        // one ghost per lane (four rows times at most four columns), from the raw values
        double G[V];
        const int gr = r0 + (lane >> 2), gc = lane & 3;
        const int glx = gc < gxl ? gc : ex + 4 - gxh + gc - gxl;
        const bool gw = lane < 16 && gr >= ja && gr < min(jb, r1) && gc < gxl + gxh;
        if (gw) xghost(slot(gr), glx, gr, G);
        __syncwarp();
        if (!raw_ok) {
          // the interior points: 32 columns of each row, then the last two of all four
#pragma unroll 1
          for (int h = 0; h < 5; ++h) {
            const int jr = h < 4 ? r0 + h : r0 + (lane >> 1), lx = h < 4 ? lane : 32 + (lane & 1);
            const int gi = i0 + lx - 2;
            if (jr >= ja && jr < min(jb, r1) && lx < ex + 4 && gi >= 0 && gi < g.nx && (h < 4 || lane < 8)) {
              double* const c = slot(jr) + lx;
              double u[V];
#pragma unroll
              for (int v = 0; v < V; ++v) u[v] = c[v * RW];
              conv(u, gi, jr);
#pragma unroll
              for (int v = 0; v < V; ++v) c[v * RW] = u[v];
            }
          }
        }
        if (gw) {
#pragma unroll
          for (int v = 0; v < V; ++v) slot(gr)[v * RW + glx] = G[v];
        }
        fence_proxy_async();
      }
      __syncwarp();
    };

    // the epilogue's arrays of a row brought into L2 by bulk prefetches, one array per lane
    const EpilogueStreams<EU, PRIM> streams(A, use_tma);
    const double* pf = nullptr;
    if (lane < V * streams.n) pf = streams.ptr(A, lane / V) + (long long)(lane % V) * g.n + i0;
    const double* pf2 = nullptr;
    if (lane + 32 < V * streams.n)
      pf2 = streams.ptr(A, (lane + 32) / V) + (long long)((lane + 32) % V) * g.n + i0;
    auto prefetch_epilogue = [&](int jr) {
      if (jr >= ja && jr < jb) {
        if (pf) bulk_prefetch_l2(pf + (long long)g.nx * jr, 8u * ex);
        if (pf2) bulk_prefetch_l2(pf2 + (long long)g.nx * jr, 8u * ex);
      }
    };

    // the column's metric factors
    // (the product build folds the inverse cell widths of the slopes into the face offsets)
    const double sx = slope_scale(A.invd[0]), sy = slope_scale(A.invd[1]);
    const double oE = M.offxE[ip] * sx, oW = M.offxW[ip] * sx, dAx = M.dAxW[ip], dAy = M.dAyS[ip];
    const double dVx = M.dydzdV[ip], dVy = M.dzdxdV[ip];
    const double csE = EU ? 0.0 : M.cs[2 * M.nxp + max(ip - 1, 0)], csW = EU ? 0.0 : M.cs[1 * M.nxp + ip];
    const double csN = EU ? 0.0 : M.cs[4 * M.nxp + ip], csS = EU ? 0.0 : M.cs[3 * M.nxp + ip];
    const int b = lane + 1;
    double RLy[V], Fym[V];   // the plus y face state of row j, the flux through j - 1/2
    int ahead = ja - 2 + NSLOT;   // the next row to fetch
    // passes ja - 4 .. ja - 1 open the chunk: the first rows prepared, the face state of row ja - 1,
    // the flux through the first y face (one copy of the code for every pass)
#pragma unroll 1
    for (int j = ja - 4; j < jb; ++j) {
      // once every lane is past row j-1 its slot takes the row NSLOT further
      __syncwarp();
      if (ahead <= last && ahead < j + NSLOT) issue(ahead++);
      prefetch_epilogue(j + 2);
      if (((j - ja) & 3) == 0) {
        prepare(j + 2);
        if (lost) break;
      }
      if (j < ja - 2) continue;
      const double* const S = slot(j) + b;
      const double *S1 = slot(j + 1) + b, *S2 = slot(j + 2) + b;
      const double oS = M.offyS[j + 1 + 2] * sy, oN = M.offyN[j + 1 + 2] * sy;
      double q0[V], rhs[V];
      {
        double RRy[V], RLn[V], Fy[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          q0[v] = S[v * RW];
          const double r1 = S1[v * RW];
          const double s = crec ? 0.0 : slope(lim, A.theta, slope_width(A.invd[1]), q0[v], r1, S2[v * RW]);
          RRy[v] = crec ? r1 : r1 + s * oS;
          RLn[v] = crec ? r1 : r1 + s * oN;
        }
        if (j >= ja - 1) {
          if (kt_flux_try<2, EU, PRIM, 1>(RLy, RRy, csN, csS, dAy, P, Fy) && own)
            kt_flux_redo<2, EU, PRIM, 1>(RLy, RRy, csN, csS, dAy, P, Fy);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          rhs[v] = dVy * (Fy[v] - Fym[v]);
          Fym[v] = Fy[v];
          RLy[v] = RLn[v];
        }
      }
      if (j < ja) continue;
      {
        double RL[V], RR[V], Fx[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double s = crec ? 0.0 : slope(lim, A.theta, slope_width(A.invd[0]), S[v * RW - 1], q0[v], S[v * RW + 1]);
          RL[v] = crec ? q0[v] : q0[v] + s * oE;
          RR[v] = crec ? q0[v] : q0[v] + s * oW;
        }
#pragma unroll
        for (int v = 0; v < V; ++v) RL[v] = __shfl_up_sync(FULL, RL[v], 1);
        if (kt_flux_try<2, EU, PRIM, 0>(RL, RR, csE, csW, dAx, P, Fx) && lane >= 1 && lane <= ex + 1)
          kt_flux_redo<2, EU, PRIM, 0>(RL, RR, csE, csW, dAx, P, Fx);
#pragma unroll
        for (int v = 0; v < V; ++v) rhs[v] = dVx * (__shfl_down_sync(FULL, Fx[v], 1) - Fx[v]) + rhs[v];
      }
      if (own) stage_cell_epilogue<2, EU, PRIM, false, SRC>(A, i, j, 0, q0, rhs, dt, cflv, errv, flags);
    }
    if (lost) {
      // a copy did not complete in time: report it and give the copies still in flight their
      // (bounded) time to land in this block's shared memory
      if (lane == 0 && A.ctl) atomicOr(&A.ctl->dev_err, 1);
      for (int jr = max(ja - 2, ahead - NSLOT); jr < min(last + 1, ahead); ++jr) mbar_wait(bar(jr), parity(jr));
      cp_async_wait_all();
    }
  }
  const bool err_out = A.last_stage || A.err_low;
  if (RED && A.ctl && (A.cfl_mode || err_out)) {
    int nv = A.cfl_mode ? (M.vis ? 4 : 1) : 0;
    double vals[4] = {cflv[0], cflv[1], cflv[2], cflv[3]};
    if (err_out && !A.cfl_mode) { vals[0] = errv; nv = 1; }
    if (nv) block_reduce_emit<NW * 32>(vals, nv, flags, err_out && !A.cfl_mode ? &A.ctl->err : A.ctl->invdt,
                                       &A.ctl->flags, sred);
  }
}

template <bool EU, bool PRIM, int NW, int MINB, int LIM, bool RED, bool SRC>
__global__ void __launch_bounds__(NW * 32, MINB)
    strip2_kernel(const __grid_constant__ StageArgs A, const __grid_constant__ CUtensorMap tmap, const int use_tma) {
  strip2_block<EU, PRIM, NW, LIM, RED, SRC>(A, &tmap, use_tma != 0, blockIdx.x * NW);
}

// Batched ensemble: block b computes warps T.y .. T.y + NW - 1 of grid T.x of the queue; args[grid]
// are the grid's stage arguments and maps[grid] the tensor map of its stage input (global
// memory, 64-byte aligned, written by the host before the launch), T.z whether it has one.
template <bool EU, bool PRIM, int NW, int MINB, int LIM, bool RED, bool SRC>
__global__ void __launch_bounds__(NW * 32, MINB)
    batched_strip2_kernel(const StageArgs* __restrict__ args, const CUtensorMap* __restrict__ maps,
                          const int4* __restrict__ queue) {
  // the grid's arguments are copied into shared memory once per block: the rows then read
  // them at fixed shared offsets instead of through global-memory address arithmetic
  __shared__ StageArgs sA;
  static_assert(sizeof(StageArgs) % 8 == 0, "argument copy by 8-byte words");
  const int4 T = queue[blockIdx.x];
  const CUtensorMap* map = maps + T.x;
  if ((threadIdx.x & 31) == 0)
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
  {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(args + T.x);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sA);
    for (int w = threadIdx.x; w < (int)(sizeof(StageArgs) / 8); w += NW * 32) dst[w] = __ldg(src + w);
  }
  __syncthreads();
  strip2_block<EU, PRIM, NW, LIM, RED, SRC>(sA, map, T.z != 0, T.y);
}

}  // namespace fgpu
