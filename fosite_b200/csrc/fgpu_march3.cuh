// fgpu_march3.cuh -- the 3D stage kernel: z-marching tiles with planes staged by bulk copies
// (sm_100a).
//
// Same right-hand side and epilogues as stage_tile (fgpu_kernels.cuh: fosite's ComputeRHS,
// timedisc_base.f90:1073-1271, fused with its consumer).  A block owns a 32 x 8 tile of x-y and
// marches a chunk of z, one thread per cell of the plane:
//   * every x-y plane of the tile, halo included, arrives in one of four plane slots by one bulk
//     tensor copy (cp.async.bulk.tensor, 4-D map x, y, z, variable) completing on an mbarrier,
//     issued a whole plane ahead; tiles on a periodic face, and meshes of odd x extent (whose
//     rows are not 16-byte aligned), fetch the same box with 8-byte cp.async whose sources wrap;
//     z ghost planes fetch the plane that they copy;
//   * a thread reconstructs its own cell in x and y, hands the plus face states to its
//     neighbours through shared memory, computes the fluxes through its own minus faces in place
//     of the states it read, and after a second barrier differences them: each slope and flux is
//     computed once, by its cell's thread, with no index arithmetic.  The tile's rim (the row and
//     column before it, the fluxes through its last faces) goes to one warp each;
//   * the z direction stays in registers (the plus face state and the flux of the last plane),
//     its flux computed right before the epilogue that consumes it;
//   * the epilogue's streams (base and earlier k of a Butcher stage, the Shu-Osher start state)
//     are brought into L2 one plane ahead by bulk prefetches, one tile row per thread.
// What bounds it: the FP64 chains and two barriers a plane at 16 warps an SM (128 registers): 44%
// issue activity, 1340 warp instructions a plane and row (2500 for the tiles whose slopes and
// fluxes were shared-memory items), 32% of them FP64.  256^3 Dormand-Prince: 11.6 ms a step against
// 14.2 ms for those tiles.
// Requirements (checked on the host): a plain or formed stage input (no k-sums in the stencil),
// no interface-flux output.
#pragma once
#include <cuda.h>
#include <type_traits>
#include "fgpu_bulk.cuh"
#include "fgpu_kernels.cuh"

namespace fgpu {

template <int V, int TX, int TY>
struct March3Layout {
  static constexpr int NSLOT = 4;
  static constexpr int RW = TX + 4, RH = TY + 4;
  static constexpr int BOX = V * RH * RW;                    // one tensor copy: [V][RH][RW]
  static constexpr int PLANE = (BOX + 15) / 16 * 16;         // slots stay 128-byte aligned
  static constexpr int NFX = V * TY * (TX + 1), NFY = V * (TY + 1) * TX;
  static constexpr size_t SMEM = 8 * ((size_t)NSLOT * PLANE + NFX + NFY + NSLOT);
};

// LIM > 0: the limiter is compiled in (linear reconstruction); LIM = 0: the limiter and the
// reconstruction order are read from the arguments.  RED = false: a stage without CFL,
// CheckData or error-norm reduction, whose maxima are then dead code.  SRC = false: a stage without
// sources (plain_stage).
template <bool EU, bool PRIM, int TX, int TY, int LIM, bool RED, bool SRC>
__device__ __forceinline__ void march3_tile(const StageArgs& A, const CUtensorMap* tmap, const bool use_tma,
                                            const int bx, const int by, const int bz) {
  using PH = Phys<3, EU>;
  using CE = Cells<3, EU>;
  constexpr int V = PH::V, NT = TX * TY;
  using L = March3Layout<V, TX, TY>;
  constexpr int RW = L::RW, RH = L::RH, RHW = RH * RW, NSLOT = L::NSLOT;
  static_assert(TX == 32 && TY >= 4, "one warp per tile row, four warps for the rim");
  extern __shared__ __align__(128) double march3_smem[];
  double* const ring = march3_smem;
  double* const FX = ring + NSLOT * L::PLANE;   // [V][TY][TX+1]  face states, then fluxes
  double* const FY = FX + L::NFX;               // [V][TY+1][TX]
  unsigned long long* const mbar = reinterpret_cast<unsigned long long*>(FY + L::NFY);
  __shared__ double sred[RED_STRIDE * (NT / 32)];
  __shared__ int abort_flag;

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
  // the staged values are the reconstruction variables as they stand, else each staged point is
  // converted once
  const bool raw_ok = PRIM ? (SR.ready != 0) : !roundtrip;
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int i0 = bx * TX, j0 = by * TY;
  const int ex = min(TX, g.nx - i0), ey = min(TY, g.ny - j0);
  const bool own = tx < ex && ty < ey;
  const int i = i0 + tx, j = j0 + ty, ip = i + 2;
  const int k0 = bz * A.kchunk, k1 = min(g.nz, k0 + A.kchunk);
  // ghost columns and rows of the staged box
  const int gxl = i0 == 0 ? 2 : 0, gxh = max(0, i0 + ex + 2 - g.nx);
  const int gyl = j0 == 0 ? 2 : 0, gyh = max(0, j0 + ey + 2 - g.ny);
  const bool xy_ghosts = (gxl | gxh | gyl | gyh) != 0;
  const bool tma = use_tma && !((gxl && g.bc[0] == BC_PERIODIC) || (gxh && g.bc[1] == BC_PERIODIC) ||
                                (gyl && g.bc[2] == BC_PERIODIC) || (gyh && g.bc[3] == BC_PERIODIC));

  // reconstruction variables from the primitive variables of a converted point / ghost
  auto finish = [&](double* p, double* R) {
    if (roundtrip) p[V - 1] = dmax(p[V - 1], P.pmin);
    if (PRIM) {
#pragma unroll
      for (int v = 0; v < V; ++v) R[v] = p[v];
    } else {
      PH::p2c(p, R, P);
    }
  };
  auto conv = [&](double* u) {   // a raw interior value, in place (PRIM or a round trip)
    double p[V];
    PH::c2p(u, p, P);
    finish(p, u);
  };
  auto raw_prim = [&](const double* u, double* p) {   // primitive variables of a raw value
    if (PRIM && SR.ready) {
#pragma unroll
      for (int v = 0; v < V; ++v) p[v] = u[v];
    } else {
      PH::c2p(u, p, P);
    }
  };
  auto ghost = [&](int d, int gi, int gj, int gk, double* R) {   // from the stored state
    double p[V];
    CE::face_ghost_p(SR, g, P, M, d, gi, gj, gk, p);
    finish(p, R);
  };
  // A face ghost of a staged plane.  Periodic faces: the wrapped raw value is at its place.
  // Faces whose ghosts copy an interior cell (reflecting, axis, no gradients): the mirror cell
  // from the same box while its values are the reconstruction variables (the arithmetic of
  // face_ghost_p on the same values).  Else from the stored state.  False: nothing to write.
  auto plane_ghost = [&](const double* S, int d, int lx, int ly, int gi, int gj, int gk, double* R) -> bool {
    const int x = d == 0 ? gi : gj, nd = d == 0 ? g.nx : g.ny;
    const bool lo = x < 0;
    const int type = g.bc[2 * d + (lo ? 0 : 1)];
    const double* src = S + ly * RW + lx;
    double u[V], p[V];
    if (type == BC_PERIODIC) {
      if (raw_ok && PRIM) return false;
#pragma unroll
      for (int v = 0; v < V; ++v) u[v] = src[v * RHW];
      raw_prim(u, p);
      finish(p, R);
      return true;
    }
    const int sdep = lo ? -x : x - (nd - 1);
    const int mirror = type == BC_NOGRAD ? (lo ? 0 : nd - 1) : (lo ? sdep - 1 : nd - sdep);
    const int lm = mirror - (d == 0 ? i0 : j0) + 2;   // the mirror's box coordinate along d
    if (raw_ok && type != BC_ABSORBING && lm >= 2 && lm <= (d == 0 ? ex : ey) + 1) {
      src = S + (d == 0 ? ly * RW + lm : lm * RW + lx);
#pragma unroll
      for (int v = 0; v < V; ++v) u[v] = src[v * RHW];
      raw_prim(u, p);
      if (type != BC_NOGRAD) {
        if (d == 0) p[1] = -p[1];
        else p[2] = -p[2];
        if (SRC && type == BC_AXIS && d == 0 && M.curv) p[2] = -p[2];
      }
      finish(p, R);
      return true;
    }
    ghost(d, gi, gj, gk, R);
    return true;
  };
  // the plane that is fetched for plane kp: its own, or the interior plane a z ghost copies
  auto source_plane = [&](int kp) {
    if (kp >= 0 && kp < g.nz) return kp;
    const bool lo = kp < 0;
    const int s = lo ? -kp : kp - (g.nz - 1), type = g.bc[lo ? 4 : 5];
    if (type == BC_PERIODIC) return lo ? g.nz - s : s - 1;
    if (type == BC_REFLECTING || type == BC_AXIS) return lo ? s - 1 : g.nz - s;
    return lo ? 0 : g.nz - 1;
  };
  // own column of plane kp as reconstruction variables, from its fetched raw values
  auto column = [&](int kp, double* u) {
    if (kp < 0 || kp >= g.nz) {
      const int type = g.bc[kp < 0 ? 4 : 5];
      if (type == BC_ABSORBING) { ghost(2, i, j, kp, u); return; }
      double p[V];
      raw_prim(u, p);
      if (type == BC_REFLECTING || type == BC_AXIS) p[3] = -p[3];
      finish(p, u);
    } else if (!raw_ok) {
      conv(u);
    }
  };

  auto slot = [&](int kp) { return ring + ((kp - (k0 - 2)) & (NSLOT - 1)) * L::PLANE; };
  auto bar = [&](int kp) { return &mbar[(kp - (k0 - 2)) & (NSLOT - 1)]; };
  auto parity = [&](int kp) { return (unsigned)(((kp - (k0 - 2)) / NSLOT) & 1); };
  // every thread calls issue: one thread the tensor copy, or all of them their share of the box
  auto issue = [&](int kp) __attribute__((always_inline)) {
    const int src = source_plane(kp);
    if (tma) {
      if (tid == 0) {
        mbar_expect_tx(bar(kp), 8u * L::BOX);
        tma_load_box<4>(slot(kp), tmap, bar(kp), i0 - 2, j0 - 2, src);
      }
    } else {
      double* const S = slot(kp);
      for (int e = tid; e < L::BOX; e += NT) {
        const int lx = e % RW, r = e / RW, ly = r % RH, v = r / RH;
        if (lx < ex + 4 && ly < ey + 4)
          cp_async8(S + e, SR.base + (long long)v * g.n +
                               CE::lin(g, wrap_index(i0 + lx - 2, g.nx, g.bc), wrap_index(j0 + ly - 2, g.ny, g.bc + 2), src));
      }
      cp_async_arrive(bar(kp));
    }
  };

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < NSLOT; ++s) mbar_init(&mbar[s], tma ? 1 : NT);
    fence_proxy_async();
  }
  __syncthreads();
  for (int kp = k0 - 2; kp < k0 - 2 + NSLOT; ++kp) issue(kp);   // up to k0 + 1 <= k1

  // wait for plane kp's copy, then fill its ghost cells / convert its raw values in place; of the
  // planes before and after the chunk only the own columns are read
  auto prepare = [&](int kp) {
    if (!mbar_wait(bar(kp), parity(kp))) abort_flag = 1;
    double* const S = slot(kp);
    if (kp < k0 || kp >= k1) {
      if (own && (!raw_ok || kp < 0 || kp >= g.nz)) {
        double* const c = S + (ty + 2) * RW + tx + 2;
        double u[V];
#pragma unroll
        for (int v = 0; v < V; ++v) u[v] = c[v * RHW];
        column(kp, u);
#pragma unroll
        for (int v = 0; v < V; ++v) c[v * RHW] = u[v];
        fence_proxy_async();
      }
      return;
    }
    if (raw_ok) {
      if (!xy_ghosts) return;
      // the ghost cells only: columns first (rows 0 .. ey-1), then rows
      const int nxg = (gxl + gxh) * ey, nyg = (gyl + gyh) * TX;
      for (int t = tid; t < nxg + nyg; t += NT) {
        int lx, ly;
        const bool xg = t < nxg;
        if (xg) {
          const int c = t / ey;
          ly = 2 + t - c * ey;
          lx = c < gxl ? c : ex + 4 - gxh + (c - gxl);
        } else {
          const int u = t - nxg, c = u / TX;
          lx = 2 + u % TX;
          ly = c < gyl ? c : ey + 4 - gyh + (c - gyl);
          if (lx >= ex + 2) continue;
        }
        double R[V];
        if (plane_ghost(S, xg ? 0 : 1, lx, ly, i0 + lx - 2, j0 + ly - 2, kp, R)) {
#pragma unroll
          for (int v = 0; v < V; ++v) S[v * RHW + ly * RW + lx] = R[v];
        }
      }
    } else {
      constexpr int NXB = (TX + 4) * TY, NYB = TX * 4;
      for (int t = tid; t < NXB + NYB; t += NT) {
        int lx, ly;
        if (t < NXB) {
          lx = t % (TX + 4);
          ly = 2 + t / (TX + 4);
          if (lx >= ex + 4 || ly >= ey + 2) continue;
        } else {
          const int u = t - NXB, q = u / TX;
          lx = 2 + u % TX;
          ly = q < 2 ? q : ey + q;
          if (lx >= ex + 2) continue;
        }
        const int gi = i0 + lx - 2, gj = j0 + ly - 2;
        const bool gx = gi < 0 || gi >= g.nx, gy = gj < 0 || gj >= g.ny;
        double R[V];
        if (gx || gy) {
          plane_ghost(S, gx ? 0 : 1, lx, ly, gi, gj, kp, R);
        } else {
#pragma unroll
          for (int v = 0; v < V; ++v) R[v] = S[v * RHW + ly * RW + lx];
          conv(R);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) S[v * RHW + ly * RW + lx] = R[v];
      }
    }
    fence_proxy_async();   // (planes that nothing is written to have returned)
  };

  // the epilogue's arrays of a plane brought into L2: one bulk prefetch per tile row and array, at
  // most two a thread (12 arrays of 5 variables and 8 rows: 480)
  const EpilogueStreams<EU, PRIM> streams(A, use_tma);
  auto prefetch_base = [&](int r) -> const double* {
    const int jr = r % TY, vq = r / TY;
    if (vq >= V * streams.n || jr >= ey) return nullptr;
    return streams.ptr(A, vq / V) + (long long)(vq % V) * g.n + CE::lin(g, i0, j0 + jr, 0);
  };
  const double* const pf = prefetch_base(tid);
  const double* const pf2 = prefetch_base(tid + NT);
  auto prefetch_epilogue = [&](int kp) {
    if (kp < k0 || kp >= k1) return;
    const long long o = (long long)g.nx * g.ny * kp;
    if (pf) bulk_prefetch_l2(pf + o, 8u * ex);
    if (pf2) bulk_prefetch_l2(pf2 + o, 8u * ex);
  };

  double cflv[4] = {0.0, 0.0, 0.0, 0.0};
  double errv = 0.0;
  int flags = 0;
  // own cell in a staged plane; its slots of the face arrays
  const int oc = (ty + 2) * RW + tx + 2;
  double* const fxw = FX + ty * (TX + 1) + tx;
  double* const fys = FY + ty * TX + tx;
  constexpr int SX = TY * (TX + 1), SY = (TY + 1) * TX;
  // z state of the own column: the plus face state of plane k, the flux through k-1/2
  double RLz[V], Fzm[V];

  // (the product build folds the inverse cell widths of the slopes into the face offsets)
  const double sx = slope_scale(A.invd[0]), sy = slope_scale(A.invd[1]), sz = slope_scale(A.invd[2]);
  // slope of the cell at box offset c along `step`
  auto cell_slope = [&](const double* S, int v, int c, int step, double invd) {   // (undivided: slope_width)
    const double* q = S + v * RHW + c;
    return crec ? 0.0 : slope(lim, A.theta, slope_width(invd), q[-step], q[0], q[step]);
  };
  // the flux through a face of direction D whose plus-side state waits at f (stride sf): tried with
  // straight-line code, redone with the checked form (bad faces are rare)
  auto flux_try = [&](auto dir, const double* f, int sf, const double* RR, double csl, double csr, double dA,
                      double* F) -> bool {
    constexpr int D = decltype(dir)::value;
    double RL[V];
#pragma unroll
    for (int v = 0; v < V; ++v) RL[v] = f[v * sf];
    return kt_flux_try<3, EU, PRIM, D>(RL, RR, csl, csr, dA, P, F);
  };
  auto flux_redo = [&](auto dir, const double* f, int sf, const double* RR, double csl, double csr, double dA,
                       double* F) {
    constexpr int D = decltype(dir)::value;
    double RL[V];
#pragma unroll
    for (int v = 0; v < V; ++v) RL[v] = f[v * sf];
    kt_flux_redo<3, EU, PRIM, D>(RL, RR, csl, csr, dA, P, F);
  };
  const std::integral_constant<int, 0> DX;
  const std::integral_constant<int, 1> DY;
  const int last = k1 + 1;   // the last plane fetched
  bool aborted = false;
  int k = k0 - 4;
  // passes k0 - 4 .. k0 - 1 open the chunk: the planes before it prepared, the z face state of
  // plane k0 - 1, the z flux through the first face (one copy of the code for every pass)
#pragma unroll 1
  for (; k < k1; ++k) {
    const double* const S = slot(k);
    double RRx[V], RRy[V];   // minus face states, then the fluxes through those faces
    if (k >= k0) {
      // ---- x and y face states of plane k: the plus states to shared memory, the minus states kept
      if (ty == 0 && tx < ex) {          // the row before the tile
        const double o = M.offyN[j0 - 1 + 2] * sy;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double s = cell_slope(S, v, RW + tx + 2, RW, A.invd[1]), q = S[v * RHW + RW + tx + 2];
          FY[v * SY + tx] = crec ? q : q + s * o;
        }
      }
      if (ty == 1 && tx < ey) {          // the column before the tile
        const double o = M.offxE[i0 - 1 + 2] * sx;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int c = (tx + 2) * RW + 1;
          const double s = cell_slope(S, v, c, 1, A.invd[0]), q = S[v * RHW + c];
          FX[v * SX + tx * (TX + 1)] = crec ? q : q + s * o;
        }
      }
      if (own) {
        const double oE = M.offxE[ip] * sx, oW = M.offxW[ip] * sx, oN = M.offyN[j + 2] * sy, oS = M.offyS[j + 2] * sy;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double q = S[v * RHW + oc];
          const double dx = cell_slope(S, v, oc, 1, A.invd[0]);
          fxw[v * SX + 1] = crec ? q : q + dx * oE;
          RRx[v] = crec ? q : q + dx * oW;
          const double dy = cell_slope(S, v, oc, RW, A.invd[1]);
          fys[v * SY + TX] = crec ? q : q + dy * oN;
          RRy[v] = crec ? q : q + dy * oS;
        }
      }
    }
    if (k >= k0 - 1) {
      __syncthreads();
      // every thread is past plane k-1: its slot takes plane k+3
      if (k + 3 <= last) issue(k + 3);
    }
    if (k >= k0) {
      // ---- fluxes through the own minus faces, in place of the plus states they consume
      if (own) {
        const double csE = EU ? 0.0 : M.cs[2 * M.nxp + ip - 1], csW = EU ? 0.0 : M.cs[1 * M.nxp + ip];
        const double csN = EU ? 0.0 : M.cs[4 * M.nxp + ip], csS = EU ? 0.0 : M.cs[3 * M.nxp + ip];
        const double dAx = M.dAxW[ip], dAy = M.dAyS[ip];
        double Fx[V], Fy[V];
        const bool bx = flux_try(DX, fxw, SX, RRx, csE, csW, dAx, Fx);
        const bool by = flux_try(DY, fys, SY, RRy, csN, csS, dAy, Fy);
        if (bx | by) {
          flux_redo(DX, fxw, SX, RRx, csE, csW, dAx, Fx);
          flux_redo(DY, fys, SY, RRy, csN, csS, dAy, Fy);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          fxw[v * SX] = RRx[v] = Fx[v];
          fys[v * SY] = RRy[v] = Fy[v];
        }
      }
      if (ty == 2 && tx < ex) {          // the last y faces
        const double o = M.offyS[j0 + ey + 2] * sy;
        const int c = (ey + 2) * RW + tx + 2;
        const double csl = EU ? 0.0 : M.cs[4 * M.nxp + ip], csr = EU ? 0.0 : M.cs[3 * M.nxp + ip], dA = M.dAyS[ip];
        double RR[V], F[V];
        double* const f = FY + ey * TX + tx;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double s = cell_slope(S, v, c, RW, A.invd[1]), q = S[v * RHW + c];
          RR[v] = crec ? q : q + s * o;
        }
        if (flux_try(DY, f, SY, RR, csl, csr, dA, F)) flux_redo(DY, f, SY, RR, csl, csr, dA, F);
#pragma unroll
        for (int v = 0; v < V; ++v) f[v * SY] = F[v];
      }
      if (ty == 3 && tx < ey) {          // the last x faces
        const int gl = i0 + ex - 1 + 2, c = (tx + 2) * RW + ex + 2;
        const double o = M.offxW[gl + 1] * sx;
        const double csl = EU ? 0.0 : M.cs[2 * M.nxp + gl], csr = EU ? 0.0 : M.cs[1 * M.nxp + gl + 1];
        const double dA = M.dAxW[gl + 1];
        double RR[V], F[V];
        double* const f = FX + tx * (TX + 1) + ex;
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double s = cell_slope(S, v, c, 1, A.invd[0]), q = S[v * RHW + c];
          RR[v] = crec ? q : q + s * o;
        }
        if (flux_try(DX, f, SX, RR, csl, csr, dA, F)) flux_redo(DX, f, SX, RR, csl, csr, dA, F);
#pragma unroll
        for (int v = 0; v < V; ++v) f[v * SX] = F[v];
      }
    }
    prepare(k + 2);
    if (k < k0 - 2) continue;
    __syncthreads();
    if (abort_flag) { aborted = true; break; }   // block-uniform: read after the barrier
    prefetch_epilogue(k + 1);
    // ---- z flux through k+1/2, divergence, sources and the stage's consumer
    if (own) {
      const double *S1 = slot(k + 1) + oc, *S2 = slot(k + 2) + oc;
      const double oB = M.offzB[k + 1 + 2] * sz, oT = M.offzT[k + 1 + 2] * sz;
      double RR[V], RLn[V], Fzp[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const double r1 = S1[v * RHW];
        const double s = crec ? 0.0 : slope(lim, A.theta, slope_width(A.invd[2]), S[v * RHW + oc], r1, S2[v * RHW]);
        RR[v] = crec ? r1 : r1 + s * oB;
        RLn[v] = crec ? r1 : r1 + s * oT;
      }
      if (k >= k0 - 1) {
        const double csT = EU ? 0.0 : M.cs[6 * M.nxp + ip], csB = EU ? 0.0 : M.cs[5 * M.nxp + ip], dAz = M.dAzB[ip];
        if (kt_flux_try<3, EU, PRIM, 2>(RLz, RR, csT, csB, dAz, P, Fzp))
          kt_flux_redo<3, EU, PRIM, 2>(RLz, RR, csT, csB, dAz, P, Fzp);
      }
      if (k >= k0) {
        // the neighbours' minus-face fluxes are this cell's plus-face fluxes (only this thread
        // reads and, for the next plane, rewrites those places: no barrier after this)
        const double dVx = M.dydzdV[ip], dVy = M.dzdxdV[ip], dVz = M.dxdydV[ip];
        double rhs[V], R0[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const double divX = dVx * (fxw[v * SX + 1] - RRx[v]);
          const double divY = dVy * (fys[v * SY + TX] - RRy[v]);
          rhs[v] = (divX + divY) + dVz * (Fzp[v] - Fzm[v]);
          R0[v] = S[v * RHW + oc];
        }
        // the z state moves on before the epilogue, which needs the registers
#pragma unroll
        for (int v = 0; v < V; ++v) { Fzm[v] = Fzp[v]; RLz[v] = RLn[v]; }
        stage_cell_epilogue<3, EU, PRIM, true, SRC>(A, i, j, k, R0, rhs, dt, cflv, errv, flags);
      } else {
#pragma unroll
        for (int v = 0; v < V; ++v) { Fzm[v] = Fzp[v]; RLz[v] = RLn[v]; }
      }
    }
  }

  if (aborted) {
    // a copy did not complete in time: report it, give the copies still in flight their
    // (bounded) time to land in this block's shared memory, leave
    if (tid == 0) {
      if (A.ctl) atomicOr(&A.ctl->dev_err, 1);
      for (int kp = max(k, k0 - 2); kp <= min(last, max(k + 3, k0 + 1)); ++kp) mbar_wait(bar(kp), parity(kp));
    }
    cp_async_wait_all();
    __syncthreads();
    return;
  }
  const bool err_out = A.last_stage || A.err_low;
  if (RED && A.ctl && (A.cfl_mode || err_out)) {
    int nv = A.cfl_mode ? (M.vis ? 4 : 3) : 0;
    double vals[4] = {cflv[0], cflv[1], cflv[2], cflv[3]};
    if (err_out && !A.cfl_mode) { vals[0] = errv; nv = 1; }
    if (nv) block_reduce_emit<NT>(vals, nv, flags, err_out && !A.cfl_mode ? &A.ctl->err : A.ctl->invdt,
                                  &A.ctl->flags, sred);
  }
}

template <bool EU, bool PRIM, int TX, int TY, int MINB, int LIM, bool RED, bool SRC>
__global__ void __launch_bounds__(TX* TY, MINB)
    march3_kernel(const __grid_constant__ StageArgs A, const __grid_constant__ CUtensorMap tmap, const int use_tma) {
  march3_tile<EU, PRIM, TX, TY, LIM, RED, SRC>(A, &tmap, use_tma != 0, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Batched ensemble: block b computes tile (T.y, T.z) of z chunk T.w of grid T.x of the queue (bit 30 of
// T.x: the grid has tensor maps); args[grid] and maps[grid] as in the 2D kernel
// (batched_strip2_kernel), the arguments copied into shared memory once per block.
template <bool EU, bool PRIM, int TX, int TY, int MINB, int LIM, bool RED, bool SRC>
__global__ void __launch_bounds__(TX* TY, MINB)
    batched_march3_kernel(const StageArgs* __restrict__ args, const CUtensorMap* __restrict__ maps,
                          const int4* __restrict__ queue) {
  __shared__ StageArgs sA;
  const int4 T = queue[blockIdx.x];
  const int grid = T.x & ~(1 << 30);
  const CUtensorMap* map = maps + grid;
  if (threadIdx.x == 0)
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
  {
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(args + grid);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sA);
    for (int w = threadIdx.x; w < (int)(sizeof(StageArgs) / 8); w += TX * TY) dst[w] = __ldg(src + w);
  }
  __syncthreads();
  march3_tile<EU, PRIM, TX, TY, LIM, RED, SRC>(sA, map, (T.x & (1 << 30)) != 0, T.y, T.z, T.w);
}

}  // namespace fgpu
