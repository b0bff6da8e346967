// Kernels of the explicit time step over the tiled level layout (layout.h).
//
// Included by one translation unit per arithmetic build:
//   kernels_fp64.cu   FP64 (multiply-adds contracted) and mixed precision
//   kernels_exact.cu  FP64 compiled with -fmad=false: operation-for-operation
//                     the reference's arithmetic
// Each includer defines IBGPU_KNS, the namespace its launchers live in.
#pragma once

#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <stdint.h>

#include "cfl.cuh"
#include "dependent.cuh"
#include "flux.cuh"
#include "cell_states.cuh"
#include "layout.h"

namespace ibgpu {
namespace IBGPU_KNS {

constexpr int kHalo = 2;
constexpr int kReg = kTile + 2 * kHalo;  // 20: tile plus a 2-cell halo
constexpr int kXFaces = kTile * (kTile + 1);
constexpr int kYFaces = (kTile + 1) * kTile;

// What a step's first stage resets (StageArgs::reset); nothing reads these
// words before the step's final stage.
__device__ __forceinline__ void step_reset(const StageArgs &a) {
  if (a.reset && blockIdx.x == 0 && threadIdx.x == 0) {
    if (a.reset & 1)
      for (int c = 0; c < 5; ++c) a.diag->res_bits[c] = 0ull;
    if (a.reset & 2) a.diag->cfl_bits = (unsigned long long)__double_as_longlong(10000.0);
  }
}

// Whether a thread evaluates its two faces as one paired flux: FP32 yes
// (f32x2 instructions); FP64 no (interleaving two scalar chains needs
// registers that cost more occupancy than the extra independence returns).
template <typename R>
constexpr bool kPairFaces = sizeof(R) == 4;

// How a stage CTA's warps share the halo.  FP64: half a record (two fields) per
// lane, two warps per side, so that every warp waits for the same loads, and
// dt through shared memory (20 steps at 2048^2 12.02 -> 11.78 ms, at 464^2
// 0.655 -> 0.640).  FP32: a record per lane, one warp per side (7.99 ms
// against 8.11 with half records: its stores are half as wide).
template <typename R>
constexpr bool kHalfHalo = sizeof(R) == 8;

// Threads of a fast-build stage CTA: FP64 adds a ninth warp that owns the
// tile's east/north edge faces and outer slopes, so every warp computes two
// faces; FP32 keeps 8 warps (its face work is cheap enough).
template <typename R>
struct StageThreads {
  static constexpr int value = sizeof(R) == 8 ? 288 : kTileCells;
};

// Resident CTAs per SM the register budget is fixed for, by arithmetic and
// block shape (the batched stage tunes between 256 and 288 threads).  FP64:
// 56 registers, 24-30 bytes of spill stores per thread.  FP32, 256 threads:
// 48 registers, which spill too (van Leer 80-108 bytes, minmod 24-56); the
// measured best all the same: 20 steps of the 2048^2 vortex 8.80 ms with six
// CTAs (40 registers), 8.35 with five, 9.14 with four.  With 288 threads four
// CTAs have 56 registers; the batched kernel then spills next to nothing (0-4
// bytes with its arguments in constant memory).  That shape is not timed for
// the single case.
template <typename R, int NT>
constexpr int stage_min_blocks() {
  return sizeof(R) == 8 ? 4 : (NT > kTileCells ? 4 : 5);
}

// Residual max-norm of a block of up to 9 warps into the step's diag: warp and
// block maxima, then one atomicMax per component and block whose result
// nobody reads, so it retires as a fire-and-forget reduction (reading the
// global value first to skip it put a memory round trip on the tail of
// every CTA: 29 us per FP64 2048^2 final stage).  Components map to
// res_max[0,1,2,4] (no z momentum in 2-D).
// Every thread of the block must call it; sred is shared scratch of 4 NT / 32
// words that no thread reads or writes any more (with the fold below, which
// uses words 64 to 64 + NT / 32, that many).
template <int NT = kTileCells>
__device__ __forceinline__ void block_resnorm(const unsigned long long (&rb)[4], DevDiag *d,
                                              unsigned long long *sred) {
  constexpr int kW = NT / 32;
  const int tid = threadIdx.x;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const unsigned long long m = warp_max_u64(rb[c]);
    if ((tid & 31) == 0) sred[c * kW + (tid >> 5)] = m;
  }
  __syncthreads();
  if (tid < 4) {
    unsigned long long m = 0ull;
#pragma unroll
    for (int w = 0; w < kW; ++w) m = sred[tid * kW + w] > m ? sred[tid * kW + w] : m;
    unsigned long long *dst = &d->res_bits[tid == 3 ? 4 : tid];
    atomicMax(dst, m);  // result unused: a reduction the CTA does not wait for
  }
}

// The next step's CFL pass folded into a final stage: the sum of each
// normal cell from the state this stage wrote (cs >= 0) or, for a normal
// cell it did not write, from the step state; the tile's smallest bound into
// diag->cfl_next_bits.  A tile has one level and a rounded quotient falls as
// its divisor grows, so the smallest bound is cfl_vol over the largest sum,
// bit for bit: one division per CTA instead of one per cell.  All threads
// call it (own = the thread owns a cell).
template <int NT>
__device__ __forceinline__ void fold_next_cfl(const StageArgs &a, const LevelConst &L,
                                              const CaseConst &cc, uint8_t fl, int64_t slot,
                                              double cs, unsigned long long *sred, int phase,
                                              bool own = true) {
  unsigned long long m = 0ull;
  if (own && (fl & CF_NORMAL)) {
    const double s =
        cs >= 0.0 ? cs : cfl_cell_sum(a.s0[F_T][slot], a.s0[F_U][slot], a.s0[F_V][slot], L, cc);
    // a NaN sum bounds nothing (std::min(CFL_dt, CFL_dt0) ignores it)
    if (s > 0.0) {
      m = (unsigned long long)__double_as_longlong(s);
      if (L.cfl_vol < 0.0) raise_error(a.diag, phase, ERR_CFL_NEG_DT, (int)slot);
    }
  }
  __syncthreads();  // sred is free again (block_resnorm read it)
  sred += 64;
  m = warp_max_u64(m);
  if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int k = 1; k < NT / 32; ++k) m = sred[k] > m ? sred[k] : m;
    const double d0 = __ddiv_rn(L.cfl_vol, __longlong_as_double((long long)m));
    if (m != 0ull && d0 >= 0.0 && d0 < 10000.0)
      atomicMin(&a.diag->cfl_next_bits, (unsigned long long)__double_as_longlong(d0));
  }
}

// One stage of the multistage update for one tile per CTA (256 threads):
// NS_Solver::ComputeFaceFlux (NS_Solver.H:704-832), ComptSource
// (NS_Solver.cpp:282-363), UpdateConsVars (:844-985) and ComptNewPrimVar
// (:3-194), plus ResinDomain's max-norm (NS_Solver.H:264-378) on the final
// stage.  Every face of the tile (and of its east/north edge) is computed
// once into shared memory from a 20x20 staged stencil region; each thread
// then gathers the four faces of its cell in the reference's summation order.
template <typename R, int LIM, bool VISC, bool FINAL>
__global__ void __launch_bounds__(kTileCells) stage_kernel(StageArgs a, CaseConst cc) {
  __shared__ R sq[4][kReg * kReg];
  __shared__ uint8_t sfl[kReg * kReg];
  __shared__ R fx[4][kXFaces];  // x-face f between cells (f%17-1, f/17) and (f%17, f/17)
  __shared__ R fy[4][kYFaces];  // y-face f between cells (f%16, f/16-1) and (f%16, f/16)

  const int tid = threadIdx.x;
  const int tile = a.tile_begin + blockIdx.x;
  const int lvl = a.tile_level[tile];
  const LevelConst &L = cc.lev[lvl];
  dep_begin();
  dep_wait();
  step_reset(a);

  // ---- stage the stencil region (tile + 2-cell halo, corners not needed)
  for (int r = tid; r < kReg * kReg; r += kTileCells) {
    int rx = r % kReg - kHalo, ry = r / kReg - kHalo;
    int ox = rx < 0 ? -1 : (rx >= kTile ? 1 : 0);
    int oy = ry < 0 ? -1 : (ry >= kTile ? 1 : 0);
    uint8_t f = 0;
    R q0 = R(0), q1 = R(0), q2 = R(0), q3 = R(0);
    if (!(ox && oy)) {
      int nb = a.tile_nb[tile * 9 + (oy + 1) * 3 + (ox + 1)];
      if (nb >= 0) {
        int64_t s = (int64_t)nb * kTileCells + (ry - oy * kTile) * kTile + (rx - ox * kTile);
        f = a.flags[s];
        if (f & CF_PRESENT) {
          const bool varying = (f & (CF_PRIM | CF_RESET)) != 0;
          const double *p0 = varying ? static_cast<const double *>(a.v.sin[0]) : a.s0[F_RHO];
          const double *p1 = varying ? static_cast<const double *>(a.v.sin[1]) : a.s0[F_U];
          const double *p2 = varying ? static_cast<const double *>(a.v.sin[2]) : a.s0[F_V];
          const double *p3 = varying ? static_cast<const double *>(a.v.sin[3]) : a.s0[F_P];
          q0 = (R)p0[s];
          q1 = (R)p1[s];
          q2 = (R)p2[s];
          q3 = (R)p3[s];
        }
      }
    }
    sfl[r] = f;
    sq[0][r] = q0;
    sq[1][r] = q1;
    sq[2][r] = q2;
    sq[3][r] = q3;
  }
  __syncthreads();

  Gas<R> g;
  g.gama = (R)cc.gama;
  g.Rg = (R)cc.Rg;
  g.Cv = (R)cc.Cv;
  g.Ma = (R)cc.Ma;
  g.gm1 = (R)cc.gm1;
  g.gamaRg = (R)cc.gamaRg;

  // ---- face fluxes
  for (int w = tid; w < kXFaces + kYFaces; w += kTileCells) {
    const bool xdir = w < kXFaces;
    int i, j, step;
    int rL1, rR1;
    if (xdir) {
      j = w / (kTile + 1);
      i = w % (kTile + 1);
      rR1 = (j + kHalo) * kReg + (i + kHalo);
      rL1 = rR1 - 1;
      step = 1;
    } else {
      int v = w - kXFaces;
      j = v / kTile;
      i = v % kTile;
      rR1 = (j + kHalo) * kReg + (i + kHalo);
      rL1 = rR1 - kReg;
      step = kReg;
    }
    const uint8_t fL = sfl[rL1], fR = sfl[rR1];
    R fm = R(0), fn = R(0), ft = R(0), fe = R(0);
    if ((fL & CF_PRESENT) && (fR & CF_PRESENT) && ((fL | fR) & CF_NORMAL)) {
      int rL2 = rL1 - step, rR2 = rR1 + step;
      const bool hasL2 = (sfl[rL2] & CF_PRESENT) != 0;
      const bool hasR2 = (sfl[rR2] & CF_PRESENT) != 0;
      // missing outer neighbour: use the other side's (NS_Solver.H:743-750)
      const int sL2 = hasL2 ? rL2 : rR2;
      const int sR2 = hasR2 ? rR2 : rL2;
      const int cn = xdir ? 1 : 2, ct = xdir ? 2 : 1;
      const R area = (R)(xdir ? L.area_x : L.area_y);
      roe_face_flux<LIM, R>(g, area,
                            sq[0][sL2], sq[cn][sL2], sq[ct][sL2], sq[3][sL2],
                            sq[0][rL1], sq[cn][rL1], sq[ct][rL1], sq[3][rL1],
                            sq[0][rR1], sq[cn][rR1], sq[ct][rR1], sq[3][rR1],
                            sq[0][sR2], sq[cn][sR2], sq[ct][sR2], sq[3][sR2],
                            fm, fn, ft, fe);
    }
    if (xdir) {
      fx[0][w] = fm;
      fx[1][w] = fn;
      fx[2][w] = ft;
      fx[3][w] = fe;
    } else {
      int v = w - kXFaces;
      fy[0][v] = fm;
      fy[1][v] = ft;
      fy[2][v] = fn;
      fy[3][v] = fe;
    }
  }
  __syncthreads();

  // ---- residual, update, primitive recovery for the thread's own cell
  const int lx = tid % kTile, ly = tid / kTile;
  const int64_t slot = (int64_t)tile * kTileCells + tid;
  const uint8_t fl = sfl[(ly + kHalo) * kReg + (lx + kHalo)];
  unsigned long long rb[4] = {0ull, 0ull, 0ull, 0ull};
  double cb = -1.0;  // the cell's sum for the next step's CFL bound, when this stage writes it
  if ((fl & CF_NORMAL) && (fl & (CF_UPDATE | CF_RESET))) {
    const int xlo = ly * (kTile + 1) + lx, xhi = xlo + 1;
    const int ylo = ly * kTile + lx, yhi = ylo + kTile;
    double res[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      double sx = (double)fx[c][xlo] - (double)fx[c][xhi];
      double sy = (double)fy[c][ylo] - (double)fy[c][yhi];
      if (VISC) {
        sx += a.vsd[(int64_t)c * a.nslots + slot];
        sy += a.vsd[(int64_t)(4 + c) * a.nslots + slot];
      }
      res[c] = sx + sy;
    }
    const double dt = a.diag->dt;
    const double level_ts = (a.v.tp * dt) * L.step_num;
    double orho = a.s0[F_RHO][slot], ou = a.s0[F_U][slot], ov = a.s0[F_V][slot],
           oe = a.s0[F_E][slot];
    double nrho, nu, nv, np, ne, nT;
    bool wrote = false;
    if (fl & CF_UPDATE) {
      // ComptOldConsVar (NS_Solver.H:392-424) then UpdateConsVars
      const double un0 = orho, un1 = orho * ou, un2 = orho * ov, un3 = orho * oe;
      const double cv0 = un0 + res[0] * level_ts / L.vol;
      const double cv1 = un1 + res[1] * level_ts / L.vol;
      const double cv2 = un2 + res[2] * level_ts / L.vol;
      const double cv3 = un3 + res[3] * level_ts / L.vol;
      if (cv0 < 0.0) raise_error(a.diag, a.phase, ERR_NEG_RHO, (int)slot);
      if (fl & CF_PRIM) {
        // Get_Prim_Vars (FlowVariables.H:50-57), FP64
        nrho = cv0;
        nu = cv1 / cv0;
        nv = cv2 / cv0;
        ne = cv3 / cv0;
        np = (ne - 0.5 * (nu * nu + nv * nv)) * cc.gm1 * nrho;
        nT = np / (nrho * cc.Rg);
        wrote = true;
      }
    }
    if (!wrote && (fl & CF_RESET)) {
      nrho = cc.initvar[0];
      nu = cc.initvar[1];
      nv = cc.initvar[2];
      np = cc.initvar[4];
      nT = cc.initvar[5];
      ne = cc.initvar[6];
      wrote = true;
    }
    if (wrote) {
      if (nT < 0.0) raise_error(a.diag, a.phase, ERR_NEG_T, (int)slot);
      if (FINAL) {
        a.s0[F_RHO][slot] = nrho;
        a.s0[F_U][slot] = nu;
        a.s0[F_V][slot] = nv;
        a.s0[F_P][slot] = np;
        a.s0[F_E][slot] = ne;
        a.s0[F_T][slot] = nT;
      } else {
        static_cast<double *>(a.v.sout[0])[slot] = nrho;
        static_cast<double *>(a.v.sout[1])[slot] = nu;
        static_cast<double *>(a.v.sout[2])[slot] = nv;
        static_cast<double *>(a.v.sout[3])[slot] = np;
      }
    }
    if (FINAL && (fl & CF_RESNORM)) {
#pragma unroll
      for (int c = 0; c < 4; ++c) rb[c] = (unsigned long long)__double_as_longlong(fabs(res[c]));
    }
    if (FINAL && a.v.cfl_next && wrote) cb = cfl_cell_sum(nT, nu, nv, L, cc);
  }
  if (FINAL) {
    __shared__ unsigned long long sred[64 + kTileCells / 32];
    block_resnorm(rb, a.diag, sred);
    if (a.v.cfl_next) fold_next_cfl<kTileCells>(a, L, cc, fl, slot, cb, sred, a.v.cfl_next - 1);
  }
}

template <>
struct SRec<float> {
  using V = float4;
  static constexpr int kPlanes = 1;
  static __device__ __forceinline__ Q4<float> ld(const V *a, int i, int) {
    const float4 t = a[i];
    return Q4<float>{t.x, t.y, t.z, t.w};
  }
  static __device__ __forceinline__ void st(V *a, int i, int, float x, float y, float z, float w) {
    a[i] = make_float4(x, y, z, w);
  }
};

template <>
struct SRec<double> {
  using V = double2;
  static constexpr int kPlanes = 2;
  static __device__ __forceinline__ Q4<double> ld(const V *a, int i, int n) {
    const double2 lo = a[i], hi = a[i + n];
    return Q4<double>{lo.x, lo.y, hi.x, hi.y};
  }
  static __device__ __forceinline__ void st(V *a, int i, int n, double x, double y, double z,
                                            double w) {
    a[i] = make_double2(x, y);
    a[i + n] = make_double2(z, w);
  }
  // half h of record i: components 2h, 2h + 1
  static __device__ __forceinline__ void st_half(V *a, int i, int n, int h, double x, double y) {
    a[i + h * n] = make_double2(x, y);
  }
};

// Whether the face between cells with flags fL | fR carries a flux.
__device__ __forceinline__ bool face_active(uint8_t fL, uint8_t fR) {
  return (fL & CF_PRESENT) && (fR & CF_PRESENT) && ((fL | fR) & CF_NORMAL);
}

// Flux (mass, x-momentum, y-momentum, energy) of one face from its states:
// normal / tangential velocity by selection (one flux evaluation even when
// the lanes of a warp mix x- and y-faces).
template <typename R>
__device__ __forceinline__ Q4<R> state_flux(const Gas<R> &g, bool xdir, R area, R halfarea,
                                            const Q4<R> &l, const Q4<R> &r) {
  R fm, fn, ft, fe;
  roe_flux_states<R>(g, area, halfarea, l.x, xdir ? l.y : l.z, xdir ? l.z : l.y, l.w, r.x,
                     xdir ? r.y : r.z, xdir ? r.z : r.y, r.w, fm, fn, ft, fe);
  return Q4<R>{fm, xdir ? fn : ft, xdir ? ft : fn, fe};
}

// Fast build of the stage (FP64 with FastMath divisions/roots, or FP32 flux
// arithmetic for the mixed mode).  Thread (tx, ty) owns cell (tx, ty): it
// limits the cell's slopes in both directions, keeps the states the cell
// gives to its west and south faces in registers and leaves those it gives
// to its east and north faces in shared memory; then it evaluates its west
// and south faces (the face's flux replaces the state it was made from, so
// one array serves both) and finally gathers the two fluxes its neighbours
// computed.  One warp adds the edge: the outer cells' states and the east
// and north faces.  The residual, update and primitive recovery run in FP64
// in every mode.
//
// What bounds it (2048^2 vortex, FP64): the latency of the CTA's chain of
// load, slopes, faces and update under four resident CTAs, with the FP64 pipe
// 55 % busy (floor 79 us a stage at 351 FP64 instructions per cell).  Cells
// held in registers instead of re-read records, states handed over instead
// of slopes, a halo addressed by whole warps (no divisions by the region
// width), limiting without branches and one test per tile for uniform tiles
// took a cell-stage from 896 to 765 instructions: 20 four-stage steps 14.58
// -> 12.27 ms FP64, 9.15 -> 8.35 ms mixed.  Measured slower: two cells per
// thread (13.8 ms, mixed 10.6: fewer warps to hide latency), persistent CTAs
// copying the next region ahead (13.3), U^n copied ahead into shared memory
// (12.5).
// NT: threads of the CTA, 256 (the edge on the first warp) or 288 (a ninth
// warp owns it); the same arithmetic either way.
// UNI: a uniform tile (it and its four side neighbours hold only leaf cells
// that recover their primitives): no presence flags, no one-sided stencils,
// every cell updated; decided once per tile so neither path tests again.
// nb: the tile this thread's halo lane reads (-1: none).
template <typename R, int LIM, bool VISC, bool FINAL, typename TI, int NT, bool UNI>
__device__ __forceinline__ void stage_tile(const StageArgs &a, const StageVar &v,
                                           const CaseConst &cc, const LevelConst &L,
                                           const int tile, const int nb, const int phase,
                                           const int fold, typename SRec<R>::V *sq, uint8_t *sfl,
                                           typename SRec<R>::V *fx, typename SRec<R>::V *fy,
                                           double *sdt) {
  using S = SRec<R>;
  using V = typename S::V;
  constexpr int kFX = kTile + 1;  // faces of a row
  constexpr int NQ = kReg * kReg, NF = kTile * kFX;
  const int tid = threadIdx.x;
  const int tx = tid & (kTile - 1), ty = (NT > kTileCells) ? ((tid >> 4) & (kTile - 1)) : (tid >> 4);
  // a cell of the tile (the ninth warp owns none)
  const bool own = (NT > kTileCells) ? tid < kTileCells : true;
  // lane of the edge warp, negative on the others
  const int et = NT > kTileCells ? tid - kTileCells : (tid < 32 ? tid : -1);

  // ---- the region: each thread its own cell, and its lane's part of the
  //      two-cell halo (kHalfHalo)
  const int rc = (ty + kHalo) * kReg + (tx + kHalo);
  Q4<R> c = {R(0), R(0), R(0), R(0)};
  uint8_t fown = 0;
  if constexpr (kHalfHalo<R>) {
    if (own) {
      const int side = tid >> 6, half = (tid >> 4) & 1;
      const int i = ((tid >> 1) & 16) + (tid & 15);  // this lane's cell of the side's 32
      int x, y, hr;  // position in the neighbour tile, record in the region
      if (side < 2) {
        x = i & 15;
        y = (side ? 0 : kTile - kHalo) + (i >> 4);
        hr = ((i >> 4) + (side ? kTile + kHalo : 0)) * kReg + x + kHalo;
      } else {
        x = (side == 2 ? kTile - kHalo : 0) + (i & 1);
        y = i >> 1;
        hr = (y + kHalo) * kReg + (i & 1) + (side == 2 ? 0 : kTile + kHalo);
      }
      const int64_t hs = (int64_t)nb * kTileCells + y * kTile + x;
      const int64_t os = (int64_t)tile * kTileCells + tid;
      const TI *in0 = static_cast<const TI *>(v.sin[0]), *in1 = static_cast<const TI *>(v.sin[1]),
               *in2 = static_cast<const TI *>(v.sin[2]), *in3 = static_cast<const TI *>(v.sin[3]);
      const TI *ha = half ? in2 : in0, *hb = half ? in3 : in1;
      R h0 = R(0), h1 = R(0);
      if (UNI) {
        // every load before the first store
        c = Q4<R>{(R)in0[os], (R)in1[os], (R)in2[os], (R)in3[os]};
        h0 = (R)ha[hs];
        h1 = (R)hb[hs];
      } else {
        // presence flags first, then the state of the present cells: the
        // stage input where the stages write it, else the step state
        fown = a.flags[os];
        const uint8_t fh = nb >= 0 ? a.flags[hs] : (uint8_t)0;
        if (fown & CF_PRESENT) {
          if (fown & (CF_PRIM | CF_RESET))
            c = Q4<R>{(R)in0[os], (R)in1[os], (R)in2[os], (R)in3[os]};
          else
            c = Q4<R>{(R)a.s0[F_RHO][os], (R)a.s0[F_U][os], (R)a.s0[F_V][os], (R)a.s0[F_P][os]};
        }
        if (fh & CF_PRESENT) {
          if (fh & (CF_PRIM | CF_RESET)) {
            h0 = (R)ha[hs];
            h1 = (R)hb[hs];
          } else {
            h0 = (R)a.s0[half ? F_V : F_RHO][hs];
            h1 = (R)a.s0[half ? F_P : F_U][hs];
          }
        }
        sfl[rc] = fown;
        if (!half) sfl[hr] = fh;
      }
      S::st(sq, rc, NQ, c.x, c.y, c.z, c.w);
      S::st_half(sq, hr, NQ, half, h0, h1);
    }
    if (tid == 0) *sdt = a.diag->dt;  // read by all after the faces
  } else {
    const int side = (NT >> 5) - 1 - (tid >> 5), i = tid & 31;
    int64_t hs = -1;  // this lane's halo cell
    int hr = 0;
    if (side < 4) {
      int x, y;  // position in the neighbour tile
      if (side < 2) {
        x = i & 15;
        y = (side ? 0 : kTile - kHalo) + (i >> 4);
        hr = ((i >> 4) + (side ? kTile + kHalo : 0)) * kReg + x + kHalo;
      } else {
        x = (side == 2 ? kTile - kHalo : 0) + (i & 1);
        y = i >> 1;
        hr = (y + kHalo) * kReg + (i & 1) + (side == 2 ? 0 : kTile + kHalo);
      }
      if (nb >= 0) hs = (int64_t)nb * kTileCells + y * kTile + x;
    }
    const int64_t os = (int64_t)tile * kTileCells + (own ? tid : 0);
    const TI *in0 = static_cast<const TI *>(v.sin[0]), *in1 = static_cast<const TI *>(v.sin[1]),
             *in2 = static_cast<const TI *>(v.sin[2]), *in3 = static_cast<const TI *>(v.sin[3]);
    Q4<R> h = {R(0), R(0), R(0), R(0)};
    if (UNI) {
      // every load before the first store
      if (own) c = Q4<R>{(R)in0[os], (R)in1[os], (R)in2[os], (R)in3[os]};
      if (side < 4) h = Q4<R>{(R)in0[hs], (R)in1[hs], (R)in2[hs], (R)in3[hs]};
    } else {
      // presence flags first, then the state of the present cells: the
      // stage input where the stages write it, else the step state
      uint8_t fh = 0;
      if (own) fown = a.flags[os];
      if (side < 4 && hs >= 0) fh = a.flags[hs];
      if (fown & CF_PRESENT) {
        if (fown & (CF_PRIM | CF_RESET))
          c = Q4<R>{(R)in0[os], (R)in1[os], (R)in2[os], (R)in3[os]};
        else
          c = Q4<R>{(R)a.s0[F_RHO][os], (R)a.s0[F_U][os], (R)a.s0[F_V][os], (R)a.s0[F_P][os]};
      }
      if (fh & CF_PRESENT) {
        if (fh & (CF_PRIM | CF_RESET))
          h = Q4<R>{(R)in0[hs], (R)in1[hs], (R)in2[hs], (R)in3[hs]};
        else
          h = Q4<R>{(R)a.s0[F_RHO][hs], (R)a.s0[F_U][hs], (R)a.s0[F_V][hs], (R)a.s0[F_P][hs]};
      }
      if (own) sfl[rc] = fown;
      if (side < 4) sfl[hr] = fh;
    }
    if (own) S::st(sq, rc, NQ, c.x, c.y, c.z, c.w);
    if (side < 4) S::st(sq, hr, NQ, h.x, h.y, h.z, h.w);
  }
  __syncthreads();

  // ---- limited slopes and the cells' face states
  Q4<R> wx = {}, wy = {}, we = {};  // own cell's state at its west / south face, edge cell's
  if (own) {
    Q4<R> hi;
    cell_states<R, LIM, NQ, kLow | kHigh>(sq, sfl, c, rc, 1, UNI, wx, hi);
    S::st(fx, ty * kFX + tx + 1, NF, hi.x, hi.y, hi.z, hi.w);
    cell_states<R, LIM, NQ, kLow | kHigh>(sq, sfl, c, rc, kReg, UNI, wy, hi);
    S::st(fy, (ty + 1) * kTile + tx, NF, hi.x, hi.y, hi.z, hi.w);
  }
  const bool xd = et < 16;  // edge lanes: east column, then north row
  const int ee = et & 15, estep = xd ? 1 : kReg;
  const int er = xd ? (ee + kHalo) * kReg + kTile + kHalo : (kTile + kHalo) * kReg + ee + kHalo;
  if (et >= 0) {
    // the cell before the first face of the row / column, and the one after
    // its last face
    const int r0 = er - (kTile + 1) * estep;
    Q4<R> lo, hi;
    cell_states<R, LIM, NQ, kHigh>(sq, sfl, S::ld(sq, r0, NQ), r0, estep, UNI, lo, hi);
    S::st(xd ? fx : fy, xd ? ee * kFX : ee, NF, hi.x, hi.y, hi.z, hi.w);
    cell_states<R, LIM, NQ, kLow>(sq, sfl, S::ld(sq, er, NQ), er, estep, UNI, we, hi);
  }
  __syncthreads();

  Gas<R> g;
  g.gama = (R)cc.gama;
  g.Rg = (R)cc.Rg;
  g.Cv = (R)cc.Cv;
  g.Ma = (R)cc.Ma;
  g.gm1 = (R)cc.gm1;
  g.gamaRg = (R)cc.gamaRg;
  g.inv_Rg = (R)cc.inv_Rg;
  g.gam_gm1 = (R)cc.gam_gm1;
  g.two_gama = (R)cc.two_gama;
  const R ax = (R)L.area_x, ay = (R)L.area_y;
  const R hax = R(0.5) * ax, hay = R(0.5) * ay;

  // ---- face fluxes: west and south face of the own cell, then the edge
  const Q4<R> none = {R(0), R(0), R(0), R(0)};
  if (own) {
    const int ix = ty * kFX + tx, iy = ty * kTile + tx;
    const bool ax_ok = UNI || face_active(sfl[rc - 1], fown);
    const bool ay_ok = UNI || face_active(sfl[rc - kReg], fown);
    if constexpr (kPairFaces<R>) {
      // both faces as the two lanes of one paired flux evaluation (f32x2
      // instructions in the mixed build)
      using P = decltype(pair(R(0), R(0)));
      const Q4<R> l = S::ld(fx, ix, NF), k = S::ld(fy, iy, NF);
      P fm, fn, ft, fe;
      roe_flux_pair<P, R>(g, pair(ax, ay), pair(l.x, k.x), pair(l.y, k.z), pair(l.z, k.y),
                          pair(l.w, k.w), pair(wx.x, wy.x), pair(wx.y, wy.z), pair(wx.z, wy.y),
                          pair(wx.w, wy.w), fm, fn, ft, fe);
      const Q4<R> fw = ax_ok ? Q4<R>{lane0(fm), lane0(fn), lane0(ft), lane0(fe)} : none;
      const Q4<R> fs = ay_ok ? Q4<R>{lane1(fm), lane1(ft), lane1(fn), lane1(fe)} : none;
      S::st(fx, ix, NF, fw.x, fw.y, fw.z, fw.w);
      S::st(fy, iy, NF, fs.x, fs.y, fs.z, fs.w);
    } else {
      Q4<R> f = state_flux<R>(g, true, ax, hax, S::ld(fx, ix, NF), wx);
      if (!ax_ok) f = none;
      S::st(fx, ix, NF, f.x, f.y, f.z, f.w);
      f = state_flux<R>(g, false, ay, hay, S::ld(fy, iy, NF), wy);
      if (!ay_ok) f = none;
      S::st(fy, iy, NF, f.x, f.y, f.z, f.w);
    }
  }
  if (et >= 0) {
    // east column (lanes 0..15) and north row (lanes 16..31) through one
    // call site, so the warp evaluates the flux once
    V *fe = xd ? fx : fy;
    const int k = xd ? ee * kFX + kTile : kTile * kTile + ee;
    Q4<R> o = state_flux<R>(g, xd, xd ? ax : ay, xd ? hax : hay, S::ld(fe, k, NF), we);
    if (!UNI && !face_active(sfl[er - estep], sfl[er])) o = none;
    S::st(fe, k, NF, o.x, o.y, o.z, o.w);
  }
  __syncthreads();

  // ---- residual, update, primitive recovery (FP64)
  const int64_t slot = (int64_t)tile * kTileCells + tid;
  const uint8_t fl = !own ? (uint8_t)0
                         : UNI ? (uint8_t)(CF_PRESENT | CF_NORMAL | CF_UPDATE | CF_PRIM | CF_RESNORM)
                               : fown;
  unsigned long long rb[4] = {0ull, 0ull, 0ull, 0ull};
  double cb = -1.0;  // the cell's sum for the next step's CFL bound, when this stage writes it
  if ((fl & CF_NORMAL) && (fl & (CF_UPDATE | CF_RESET))) {
    const Q4<R> fw = S::ld(fx, ty * kFX + tx, NF), fxh = S::ld(fx, ty * kFX + tx + 1, NF);
    const Q4<R> fs = S::ld(fy, ty * kTile + tx, NF), fyh = S::ld(fy, (ty + 1) * kTile + tx, NF);
    double res[4];
    const R sxl[4] = {fw.x, fw.y, fw.z, fw.w}, sxh[4] = {fxh.x, fxh.y, fxh.z, fxh.w};
    const R syl[4] = {fs.x, fs.y, fs.z, fs.w}, syh[4] = {fyh.x, fyh.y, fyh.z, fyh.w};
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (sizeof(R) == 4 && !VISC) {
        // mixed build: face differences in FP32 (the fluxes are FP32), one
        // conversion per component
        res[c] = (double)((sxl[c] - sxh[c]) + (syl[c] - syh[c]));
      } else {
        double sx = (sizeof(R) == 4) ? (double)(sxl[c] - sxh[c]) : (double)sxl[c] - (double)sxh[c];
        double sy = (sizeof(R) == 4) ? (double)(syl[c] - syh[c]) : (double)syl[c] - (double)syh[c];
        // frozen viscous residual of the momenta and the energy
        if (VISC && c > 0 && sizeof(R) == 4) {
          sx += a.vsd[(int64_t)(c - 1) * a.nslots + slot];
          sy += a.vsd[(int64_t)(2 + c) * a.nslots + slot];
        }
        res[c] = sx + sy;
        if (VISC && c > 0 && sizeof(R) == 8) res[c] += a.vsd[(int64_t)(c - 1) * a.nslots + slot];
      }
    }
    const double dt = kHalfHalo<R> ? *sdt : a.diag->dt;
    const double scale = (v.tp * dt) * L.step_num * L.inv_vol;
    double nrho, nu, nv, np, ne, nT;
    bool wrote = false;
    if (fl & CF_UPDATE) {
      const double orho = a.s0[F_RHO][slot], ou = a.s0[F_U][slot], ov = a.s0[F_V][slot],
                   oe = a.s0[F_E][slot];
      const double cv0 = orho + res[0] * scale;
      const double cv1 = orho * ou + res[1] * scale;
      const double cv2 = orho * ov + res[2] * scale;
      const double cv3 = orho * oe + res[3] * scale;
      if (cv0 < 0.0) raise_error(a.diag, phase, ERR_NEG_RHO, (int)slot);
      if (fl & CF_PRIM) {
        const double ir = FastMath<double>::rcp(cv0);
        nrho = cv0;
        nu = cv1 * ir;
        nv = cv2 * ir;
        ne = cv3 * ir;
        np = (ne - 0.5 * (nu * nu + nv * nv)) * cc.gm1 * nrho;
        nT = np * ir * cc.inv_Rg;
        wrote = true;
      }
    }
    if (!wrote && (fl & CF_RESET)) {
      nrho = cc.initvar[0];
      nu = cc.initvar[1];
      nv = cc.initvar[2];
      np = cc.initvar[4];
      nT = cc.initvar[5];
      ne = cc.initvar[6];
      wrote = true;
    }
    if (wrote) {
      if (nT < 0.0) raise_error(a.diag, phase, ERR_NEG_T, (int)slot);
      if (FINAL) {
        a.s0[F_RHO][slot] = nrho;
        a.s0[F_U][slot] = nu;
        a.s0[F_V][slot] = nv;
        a.s0[F_P][slot] = np;
        a.s0[F_E][slot] = ne;
        a.s0[F_T][slot] = nT;
      } else {
        // stage buffers in the arithmetic's precision (FP32 in the mixed build)
        typedef R TO;
        static_cast<TO *>(v.sout[0])[slot] = (TO)nrho;
        static_cast<TO *>(v.sout[1])[slot] = (TO)nu;
        static_cast<TO *>(v.sout[2])[slot] = (TO)nv;
        static_cast<TO *>(v.sout[3])[slot] = (TO)np;
      }
    }
    if (FINAL && (fl & CF_RESNORM)) {
#pragma unroll
      for (int c = 0; c < 4; ++c) rb[c] = (unsigned long long)__double_as_longlong(fabs(res[c]));
    }
    if (FINAL && fold && wrote) cb = cfl_cell_sum(nT, nu, nv, L, cc);
  }
  // the region is dead after the face phase: reuse it
  if (FINAL) {
    unsigned long long *sred = reinterpret_cast<unsigned long long *>(sq);
    block_resnorm<NT>(rb, a.diag, sred);
    if (fold) fold_next_cfl<NT>(a, L, cc, fl, slot, cb, sred, fold - 1, own);
  }
}

template <typename R, int LIM, bool VISC, bool FINAL, typename TI,
          int NT = StageThreads<R>::value>
__device__ __forceinline__ void stage_tile_fast(const StageArgs &a, const StageVar &v,
                                                const CaseConst &cc,
                                                const int tile, const int phase,
                                                const int fold, const int prefetch) {
  using S = SRec<R>;
  using V = typename S::V;
  constexpr int kFX = kTile + 1;  // faces of a row
  constexpr int NQ = kReg * kReg, NF = kTile * kFX;
  __shared__ V sq[S::kPlanes * NQ];
  __shared__ uint8_t sfl[NQ];
  __shared__ double sdt;
  // face (i, j) between cells i-1 and i of row j at j*17 + i, between cells
  // j-1 and j of column i at j*16 + i: the lower cell's state, then the flux
  __shared__ V fx[S::kPlanes * NF];
  __shared__ V fy[S::kPlanes * NF];

  static_assert(NT == kTileCells || NT == kTileCells + 32, "256 or 288 threads");
  const int tid = threadIdx.x;
  const int lvl = a.tile_level[tile];
  const LevelConst &L = cc.lev[lvl];
  // uniform tile: it and its four side neighbours hold only leaf cells that
  // recover their primitives, so no presence flags or one-sided stencils
  const bool uni = a.tile_uniform != nullptr && a.tile_uniform[tile] != 0;

  // this lane's side of the halo (south, north, west, east),
  // looked up beside the tile's level and uniform flag, so that the region's
  // loads wait for one round trip
  const int side = kHalfHalo<R> ? tid >> 6 : (NT >> 5) - 1 - (tid >> 5);
  const int nb = side < 4 ? __ldg(a.tile_nb + (int64_t)tile * 9 +
                                  (side == 0 ? 1 : side == 1 ? 7 : side == 2 ? 3 : 5))
                          : -1;

  dep_wait();
  {
    // U^n of the tile's own cells, which the update phase reads after the
    // faces, into L1 now (FP64 step 0.798 -> 0.779 ms)
    if (tid < 64) {
      const int fld = tid >> 4;
      const double *un = a.s0[fld == 0 ? F_RHO : (fld == 1 ? F_U : (fld == 2 ? F_V : F_E))];
      asm volatile("prefetch.global.L1 [%0];" ::"l"(un + (int64_t)tile * kTileCells + (tid & 15) * 16));
    }
  }
  if (prefetch > 0) {
    // the CTA that starts when this one ends reads this tile's input from L2
    constexpr int kLines = kTileCells * (int)sizeof(TI) / 128;  // 128-byte lines per field
    const int64_t pt = (int64_t)(tile + prefetch) * kTileCells;
    if (tid < 4 * kLines && pt < a.nslots)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const TI *>(v.sin[tid / kLines]) + pt +
                                                    (tid % kLines) * (128 / (int)sizeof(TI))));
  }

  step_reset(a);
  if (uni) stage_tile<R, LIM, VISC, FINAL, TI, NT, true>(a, v, cc, L, tile, nb, phase, fold, sq, sfl, fx, fy, &sdt);
  else stage_tile<R, LIM, VISC, FINAL, TI, NT, false>(a, v, cc, L, tile, nb, phase, fold, sq, sfl, fx, fy, &sdt);
}

// TI: element type of the stage input (the FP64 step state for the first
// stage; the stage buffers, R, after it)
template <typename R, int LIM, bool VISC, bool FINAL, typename TI>
__global__ void __launch_bounds__(StageThreads<R>::value, stage_min_blocks<R, StageThreads<R>::value>())
    stage_kernel_fast(StageArgs a, CaseConst cc) {
  dep_begin();
  stage_tile_fast<R, LIM, VISC, FINAL, TI>(a, a.v, cc, a.tile_begin + blockIdx.x, a.phase,
                                           a.v.cfl_next, a.prefetch);
}


#ifdef IBGPU_FAST_BUILD
// Constant-memory table of batched stage arguments.  A batch that fits keeps
// here, per case, its stage arguments up to the stage-dependent part
// (kStageCommonBytes), one StageVar per stage and its CaseConst up to its
// finest level, found through a per-batch header of one int4 per case
// (byte offsets of the three; w unused).  Read with a CTA-uniform index,
// these are constant-bank operands like a single-case launch's parameters,
// which keeps the batched tile body's registers, spills and argument loads
// at the single-case kernel's level.
constexpr int kBatchTableBytes = 60 * 1024;
__constant__ __align__(16) unsigned char c_batch_table[kBatchTableBytes];
#endif

// Batched stage over a work list of (case, tile) pairs of several
// independent cases (each its own mesh, state and constants).  TABLE: the
// case's arguments come from the constant-memory table, header at byte
// offset `table` (fast builds only); otherwise the stage's arguments of case
// c are args[c * nstages + stage] and its constants ccs[c] in global memory.
// phase_base holds 8 x the step's index within the run (abort ordering),
// written on the device so a captured graph can replay the launch for every
// step.  LOOP: persistent CTAs striding over the list; otherwise one CTA per
// item (no loop state, which keeps the tile body's register spills at the
// single-case kernel's level).
template <typename R, int LIM, bool VISC, bool FINAL, bool LOOP, bool TABLE, typename TI, int NT>
__global__ void __launch_bounds__(NT, stage_min_blocks<R, NT>())
    stage_kernel_batch(const StageArgs *__restrict__ args, const CaseConst *__restrict__ ccs,
                       const int2 *__restrict__ work, int nwork, int stage, int nstages,
                       const int *__restrict__ phase_base, int table) {
  // phase_base[0]: 8 x the step index; phase_base[1]: 1 when this step's
  // final stage folds in the next step's CFL pass of the cases that allow it
  dep_begin();
  dep_wait();
  const int pb = phase_base[0], fold_step = phase_base[1];
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const int2 it = work[w];
#ifdef IBGPU_FAST_BUILD
    if (TABLE) {
      const int4 h = reinterpret_cast<const int4 *>(c_batch_table + table)[it.x];
      const StageArgs &a = *reinterpret_cast<const StageArgs *>(c_batch_table + h.x);
      const StageVar &v = reinterpret_cast<const StageVar *>(c_batch_table + h.y)[stage];
      const CaseConst &cc = *reinterpret_cast<const CaseConst *>(c_batch_table + h.z);
      const int fold = (FINAL && fold_step && v.cfl_next) ? 1 + pb + 8 + 1 : 0;
      stage_tile_fast<R, LIM, VISC, FINAL, TI, NT>(a, v, cc, it.y, pb + 2 + stage, fold, 0);
    } else
#endif
    {
      const StageArgs &a = args[it.x * nstages + stage];
      const int fold = (FINAL && fold_step && a.v.cfl_next) ? 1 + pb + 8 + 1 : 0;
      stage_tile_fast<R, LIM, VISC, FINAL, TI, NT>(a, a.v, ccs[it.x], it.y, pb + 2 + stage, fold, 0);
    }
    if (!LOOP) break;
    __syncthreads();  // shared-memory reuse by the next work item
  }
}

// Input of a one-stage scheme's only stage.  That stage is first and final: it
// writes rho, u, v, p of the step state, which its neighbours' CTAs read as
// their halo, so it reads a copy of them made here (two passes over four
// fields that schemes of several stages do not take).
__device__ __forceinline__ void stage_input(const StageArgs &a, int tile) {
  dep_begin();
  dep_wait();
  const int64_t s = (int64_t)tile * kTileCells + threadIdx.x;
  constexpr int kMap[4] = {F_RHO, F_U, F_V, F_P};
#pragma unroll
  for (int f = 0; f < 4; ++f)
    static_cast<double *>(const_cast<void *>(a.v.sin[f]))[s] = a.s0[kMap[f]][s];
}
__global__ void __launch_bounds__(kTileCells) stage_input_kernel(StageArgs a) {
  stage_input(a, a.tile_begin + blockIdx.x);
}

// CFL time step over the normal cells of every level, NS_Solver::Comptdt
// (NS_Solver.cpp:196-280): a per-cell bound, a warp-shuffle and block min and
// one atomic per block (positive doubles order like their bit patterns).
__global__ void __launch_bounds__(256) cfl_kernel(CflArgs a, CaseConst cc) {
  dep_begin();
  dep_wait();
  double best = 10000.0;
  for (int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; s < a.nslots;
       s += (int64_t)gridDim.x * blockDim.x) {
    if (!(a.flags[s] & CF_NORMAL)) continue;
    const LevelConst &L = cc.lev[a.tile_level[s / kTileCells]];
    const double d0 = cfl_cell_bound(a.s0[F_T][s], a.s0[F_U][s], a.s0[F_V][s], L, cc);
    if (d0 < 0.0) raise_error(a.diag, a.phase, ERR_CFL_NEG_DT, (int)s);
    best = (d0 < best) ? d0 : best;  // std::min(CFL_dt, CFL_dt0) ignores NaN
  }
  unsigned long long b = warp_min_u64((unsigned long long)__double_as_longlong(best));
  // block minimum, then one atomic per block (result unused: not waited for)
  __shared__ unsigned long long sred[8];
  if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) b = sred[w] < b ? sred[w] : b;
    atomicMin(&a.diag->cfl_next_bits, b);
  }
}

// Per-step reset of the step's reductions (the dt and any earlier abort
// carry over between the steps of one run); for steps whose first stage does
// not do it.
__global__ void step_begin_kernel(DevDiag *d) {
  dep_begin();
  dep_wait();
  d->cfl_bits = (unsigned long long)__double_as_longlong(10000.0);
  for (int c = 0; c < 5; ++c) d->res_bits[c] = 0ull;
}

// dt = min(CFL_dt, dt*dt_ratio) (NS_Solver.cpp:263) from the bound that the
// CFL pass or the previous step's final stage accumulated, whose accumulator
// starts over.
__global__ void take_folded_cfl_kernel(DevDiag *d, CaseConst cc) {
  dep_begin();
  dep_wait();
  d->cfl_bits = d->cfl_next_bits;
  d->cfl_next_bits = (unsigned long long)__double_as_longlong(10000.0);
  double cdt = __longlong_as_double((long long)d->cfl_bits);
  double cand = d->dt * cc.dt_ratio;
  d->dt = (cand < cdt) ? cand : cdt;
}

// Scatter/gather between the caller's cell list (FlowVariables rows of 7
// doubles) and the slot SoA; alias rows (periodic copies) read their source
// slot on download and are skipped on upload.
__global__ void scatter_state_kernel(const double *rows, const int32_t *cell_slot,
                                     const uint8_t *cell_is_alias, int64_t n,
                                     double *s0_rho, double *s0_u, double *s0_v, double *s0_p,
                                     double *s0_e, double *s0_T) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    if (cell_is_alias[c]) continue;
    int64_t s = cell_slot[c];
    const double *r = rows + 7 * c;
    s0_rho[s] = r[0];
    s0_u[s] = r[1];
    s0_v[s] = r[2];
    s0_p[s] = r[4];
    s0_T[s] = r[5];
    s0_e[s] = r[6];
  }
}

__global__ void gather_state_kernel(double *rows, const int32_t *cell_slot, int64_t n,
                                    const double *s0_rho, const double *s0_u,
                                    const double *s0_v, const double *s0_p,
                                    const double *s0_e, const double *s0_T) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    int64_t s = cell_slot[c];
    double *r = rows + 7 * c;
    r[0] = s0_rho[s];
    r[1] = s0_u[s];
    r[2] = s0_v[s];
    r[3] = 0.0;
    r[4] = s0_p[s];
    r[5] = s0_T[s];
    r[6] = s0_e[s];
  }
}

// Compact rows (roe, u, v, p): the remaining fields as the reference derives
// them from those four (Get_T_ideal_gas T = p / (roe Rg), Get_E e = Cv T +
// |u|^2 / 2 with w = 0, FlowVariables.H:19-33), rounded operation by
// operation (no contraction).
__global__ void scatter_state4_kernel(const double *rows, const int32_t *cell_slot,
                                      const uint8_t *cell_is_alias, int64_t n, double Rg,
                                      double Cv, double *s0_rho, double *s0_u, double *s0_v,
                                      double *s0_p, double *s0_e, double *s0_T) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    if (cell_is_alias[c]) continue;
    int64_t s = cell_slot[c];
    const double *r = rows + 4 * c;
    const double roe = r[0], u = r[1], v = r[2], p = r[3];
    const double T = __ddiv_rn(p, __dmul_rn(roe, Rg));
    const double k = __dmul_rn(0.5, __dadd_rn(__dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v)), 0.0));
    s0_rho[s] = roe;
    s0_u[s] = u;
    s0_v[s] = v;
    s0_p[s] = p;
    s0_T[s] = T;
    s0_e[s] = __dadd_rn(__dmul_rn(Cv, T), k);
  }
}

__global__ void gather_state4_kernel(double *rows, const int32_t *cell_slot, int64_t n,
                                     const double *s0_rho, const double *s0_u,
                                     const double *s0_v, const double *s0_p) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    int64_t s = cell_slot[c];
    double *r = rows + 4 * c;
    r[0] = s0_rho[s];
    r[1] = s0_u[s];
    r[2] = s0_v[s];
    r[3] = s0_p[s];
  }
}

// ---- launchers (one set per arithmetic build)


#ifdef IBGPU_FAST_BUILD
template <typename R, int LIM, typename TI>
static void launch_stage_ti(const StageArgs &a, const CaseConst &cc, int ntiles, bool visc,
                            bool final_stage, cudaStream_t st, bool dep) {
  dim3 grid(ntiles), block(StageThreads<R>::value);
  if (visc) {
    if (final_stage) launch_dep(dep, st, grid, block, stage_kernel_fast<R, LIM, true, true, TI>, a, cc);
    else launch_dep(dep, st, grid, block, stage_kernel_fast<R, LIM, true, false, TI>, a, cc);
  } else {
    if (final_stage) launch_dep(dep, st, grid, block, stage_kernel_fast<R, LIM, false, true, TI>, a, cc);
    else launch_dep(dep, st, grid, block, stage_kernel_fast<R, LIM, false, false, TI>, a, cc);
  }
}

// in32: the stage input is the mixed build's FP32 stage buffer
template <typename R, int LIM>
static void launch_stage_t(const StageArgs &a, const CaseConst &cc, int ntiles, bool visc,
                           bool final_stage, bool in32, cudaStream_t st, bool dep) {
  if constexpr (sizeof(R) == 4) {
    if (in32) {
      launch_stage_ti<R, LIM, float>(a, cc, ntiles, visc, final_stage, st, dep);
      return;
    }
  }
  launch_stage_ti<R, LIM, double>(a, cc, ntiles, visc, final_stage, st, dep);
}
#else
template <typename R, int LIM>
static void launch_stage_t(const StageArgs &a, const CaseConst &cc, int ntiles, bool visc,
                           bool final_stage, bool, cudaStream_t st, bool dep) {
  dim3 grid(ntiles), block(kTileCells);
  if (visc) {
    if (final_stage) launch_dep(dep, st, grid, block, stage_kernel<R, LIM, true, true>, a, cc);
    else launch_dep(dep, st, grid, block, stage_kernel<R, LIM, true, false>, a, cc);
  } else {
    if (final_stage) launch_dep(dep, st, grid, block, stage_kernel<R, LIM, false, true>, a, cc);
    else launch_dep(dep, st, grid, block, stage_kernel<R, LIM, false, false>, a, cc);
  }
}
#endif

void launch_stage(const StageArgs &a, const CaseConst &cc, int ntiles, int limiter, bool visc,
                  bool final_stage, bool mixed, int stage, cudaStream_t st, bool dep) {
  if (ntiles <= 0) return;
#ifndef IBGPU_FAST_BUILD
  mixed = false;  // the exact build is FP64 only
#endif
  const bool in32 = mixed && stage > 0;
  if (mixed) {
    if (limiter == LIM_MINMOD) launch_stage_t<float, LIM_MINMOD>(a, cc, ntiles, visc, final_stage, in32, st, dep);
    else launch_stage_t<float, LIM_VANLEER>(a, cc, ntiles, visc, final_stage, in32, st, dep);
  } else {
    if (limiter == LIM_MINMOD) launch_stage_t<double, LIM_MINMOD>(a, cc, ntiles, visc, final_stage, false, st, dep);
    else launch_stage_t<double, LIM_VANLEER>(a, cc, ntiles, visc, final_stage, false, st, dep);
  }
}

void launch_stage_input(const StageArgs &a, int ntiles, cudaStream_t st, bool dep) {
  if (ntiles > 0) launch_dep(dep, st, ntiles, kTileCells, stage_input_kernel, a);
}

#ifdef IBGPU_FAST_BUILD
int stage_resident_ctas(bool mixed, int threads) {
  const bool ninth = threads > kTileCells;
  if (mixed) return ninth ? stage_min_blocks<float, kTileCells + 32>() : stage_min_blocks<float, kTileCells>();
  return ninth ? stage_min_blocks<double, kTileCells + 32>() : stage_min_blocks<double, kTileCells>();
}

// the same over a batch's work list (one-stage schemes: one StageArgs a case)
__global__ void __launch_bounds__(kTileCells)
    stage_input_batch(const StageArgs *__restrict__ args, const int2 *__restrict__ work) {
  const int2 it = work[blockIdx.x];
  stage_input(args[it.x], it.y);
}
void launch_stage_input_batch(const StageArgs *args, const int2 *work, int nwork,
                              cudaStream_t st) {
  if (nwork > 0) launch_dep(true, st, nwork, kTileCells, stage_input_batch, args, work);
}

template <typename R, int LIM, bool LOOP, bool TABLE, typename TI, int NT>
static void launch_batch_n(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                           int stage, int nstages, const int *phase_base, bool visc,
                           bool final_stage, int grid, int table, cudaStream_t st) {
  dim3 g(grid), block(NT);
  if (visc) {
    if (final_stage)
      launch_dep(true, st, g, block, stage_kernel_batch<R, LIM, true, true, LOOP, TABLE, TI, NT>, args, ccs, work, nwork, stage, nstages, phase_base, table);
    else
      launch_dep(true, st, g, block, stage_kernel_batch<R, LIM, true, false, LOOP, TABLE, TI, NT>, args, ccs, work, nwork, stage, nstages, phase_base, table);
  } else {
    if (final_stage)
      launch_dep(true, st, g, block, stage_kernel_batch<R, LIM, false, true, LOOP, TABLE, TI, NT>, args, ccs, work, nwork, stage, nstages, phase_base, table);
    else
      launch_dep(true, st, g, block, stage_kernel_batch<R, LIM, false, false, LOOP, TABLE, TI, NT>, args, ccs, work, nwork, stage, nstages, phase_base, table);
  }
}

template <typename R, int LIM, bool LOOP, bool TABLE, typename TI>
static void launch_batch_l(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                           int stage, int nstages, const int *phase_base, bool visc,
                           bool final_stage, int grid, int threads, int table, cudaStream_t st) {
  if (threads == kTileCells + 32)
    launch_batch_n<R, LIM, LOOP, TABLE, TI, kTileCells + 32>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, table, st);
  else
    launch_batch_n<R, LIM, LOOP, TABLE, TI, kTileCells>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, table, st);
}

// stage input element type: the FP64 step state for the first stage, the
// stage buffers (R) after it
template <typename R, int LIM, bool LOOP, bool TABLE>
static void launch_batch_i(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                           int stage, int nstages, const int *phase_base, bool visc,
                           bool final_stage, int grid, int threads, int table, cudaStream_t st) {
  if constexpr (sizeof(R) == 4) {
    if (stage > 0) {
      launch_batch_l<R, LIM, LOOP, TABLE, float>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
      return;
    }
  }
  launch_batch_l<R, LIM, LOOP, TABLE, double>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
}

// grid == nwork: one CTA per work item; fewer: persistent CTAs.  table >= 0:
// the arguments come from the constant-memory table.
template <typename R, int LIM>
static void launch_batch_t(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                           int stage, int nstages, const int *phase_base, bool visc,
                           bool final_stage, int grid, int threads, int table, cudaStream_t st) {
  const bool loop = grid < nwork;
  if (!loop) grid = nwork;
  if (table >= 0) {
    if (loop) launch_batch_i<R, LIM, true, true>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
    else launch_batch_i<R, LIM, false, true>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
  } else {
    if (loop) launch_batch_i<R, LIM, true, false>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, -1, st);
    else launch_batch_i<R, LIM, false, false>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, -1, st);
  }
}

void launch_stage_batch(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                        int stage, int nstages, const int *phase_base, int limiter, bool visc,
                        bool final_stage, bool mixed, int grid, int threads, int table,
                        cudaStream_t st) {
  if (nwork <= 0) return;
  if (grid < 1 || grid > nwork) grid = nwork;
  if (table >= kBatchTableBytes) table = -1;
  if (threads != kTileCells && threads != kTileCells + 32)
    threads = mixed ? StageThreads<float>::value : StageThreads<double>::value;
  if (mixed) {
    if (limiter == LIM_MINMOD) launch_batch_t<float, LIM_MINMOD>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
    else launch_batch_t<float, LIM_VANLEER>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
  } else {
    if (limiter == LIM_MINMOD) launch_batch_t<double, LIM_MINMOD>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
    else launch_batch_t<double, LIM_VANLEER>(args, ccs, work, nwork, stage, nstages, phase_base, visc, final_stage, grid, threads, table, st);
  }
}

// ---- constant-memory table: first-fit byte ranges per device
namespace {
std::mutex g_table_mu;
std::map<int, std::map<int, int>> g_table_used;  // device -> (offset -> bytes)
}  // namespace

int batch_table_reserve(int device, int bytes) {
  if (bytes <= 0 || bytes > kBatchTableBytes) return -1;
  bytes = (bytes + 15) & ~15;
  std::lock_guard<std::mutex> lk(g_table_mu);
  std::map<int, int> &used = g_table_used[device];
  int at = 0;
  for (const auto &r : used) {
    if (r.first - at >= bytes) break;
    at = r.first + r.second;
  }
  if (at + bytes > kBatchTableBytes) return -1;
  used[at] = bytes;
  return at;
}

void batch_table_release(int device, int offset) {
  if (offset < 0) return;
  std::lock_guard<std::mutex> lk(g_table_mu);
  auto d = g_table_used.find(device);
  if (d != g_table_used.end()) d->second.erase(offset);
}

cudaError_t batch_table_write(int offset, const void *src, int bytes) {
  if (offset < 0 || bytes < 0 || offset + bytes > kBatchTableBytes) return cudaErrorInvalidValue;
  return cudaMemcpyToSymbol(c_batch_table, src, (size_t)bytes, (size_t)offset,
                            cudaMemcpyHostToDevice);
}

// CFL pass of every batched case in one launch: one CTA per (case, tile)
// item of all tiles, the same per-cell bound as cfl_kernel, block minimum and
// one atomic (not waited for) into the case's diag.
__global__ void __launch_bounds__(kTileCells)
    cfl_kernel_batch(const StageArgs *__restrict__ args, const CaseConst *__restrict__ ccs,
                     const int2 *__restrict__ work, int nwork, int nstages,
                     const int *__restrict__ phase_base) {
  __shared__ unsigned long long sred[kTileCells / 32];
  dep_begin();
  dep_wait();
  const int pb = *phase_base;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const int2 it = work[w];
    const StageArgs &a = args[it.x * nstages];
    const CaseConst &cc = ccs[it.x];
    const int64_t s = (int64_t)it.y * kTileCells + threadIdx.x;
    double best = 10000.0;
    if (a.flags[s] & CF_NORMAL) {
      const LevelConst &L = cc.lev[a.tile_level[it.y]];
      const double d0 = cfl_cell_bound(a.s0[F_T][s], a.s0[F_U][s], a.s0[F_V][s], L, cc);
      if (d0 < 0.0) raise_error(a.diag, pb + 1, ERR_CFL_NEG_DT, (int)s);
      best = (d0 < best) ? d0 : best;
    }
    unsigned long long b = warp_min_u64((unsigned long long)__double_as_longlong(best));
    if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < kTileCells / 32; ++k) b = sred[k] < b ? sred[k] : b;
      atomicMin(&a.diag->cfl_bits, b);
    }
    __syncthreads();
  }
}

// dt = min(CFL_dt, dt*dt_ratio) of every batched case (one thread each)
__global__ void finalize_dt_batch(const StageArgs *__restrict__ args,
                                  const CaseConst *__restrict__ ccs, int ncases, int nstages) {
  dep_begin();
  dep_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncases) return;
  DevDiag *d = args[c * nstages].diag;
  double cdt = __longlong_as_double((long long)d->cfl_bits);
  double cand = d->dt * ccs[c].dt_ratio;
  d->dt = (cand < cdt) ? cand : cdt;
}

// the CFL bound each batched case's previous final stage accumulated
__global__ void take_folded_batch(const StageArgs *__restrict__ args,
                                  const CaseConst *__restrict__ ccs, int ncases, int nstages) {
  dep_begin();
  dep_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncases) return;
  DevDiag *d = args[c * nstages].diag;
  d->cfl_bits = d->cfl_next_bits;
  d->cfl_next_bits = (unsigned long long)__double_as_longlong(10000.0);
  double cdt = __longlong_as_double((long long)d->cfl_bits);
  double cand = d->dt * ccs[c].dt_ratio;
  d->dt = (cand < cdt) ? cand : cdt;
}
void launch_take_folded_batch(const StageArgs *args, const CaseConst *ccs, int ncases, int nstages,
                              cudaStream_t st) {
  launch_dep(true, st, (ncases + 127) / 128, 128, take_folded_batch, args, ccs, ncases, nstages);
}

// First launch of every batched step: the step's index and abort-order phase
// base (8 x the index), whether its final stage folds in the next step's CFL
// pass, and, after a run's first step, the reset of every case's reductions.
// c[0], c[1] are what the stages read; c[2] the last step's index (-1 before
// the first), c[3] the run's steps, c[4] whether the cases fold.
__global__ void batch_step_kernel(int *c, const StageArgs *__restrict__ args, int ncases,
                                  int nstages) {
  dep_begin();
  dep_wait();
  const int step = c[2] + 1;
  __syncthreads();
  if (threadIdx.x == 0) {
    c[2] = step;
    c[0] = 8 * step;
    c[1] = c[4] && step + 1 < c[3];
  }
  if (step > 0)
    for (int k = threadIdx.x; k < ncases; k += blockDim.x) {
      DevDiag *d = args[k * nstages].diag;
      d->cfl_bits = (unsigned long long)__double_as_longlong(10000.0);
      for (int j = 0; j < 5; ++j) d->res_bits[j] = 0ull;
    }
}

// dt of the listed batched cases only (the cases whose CFL pass ran)
__global__ void finalize_dt_batch_list(const StageArgs *__restrict__ args,
                                       const CaseConst *__restrict__ ccs,
                                       const int *__restrict__ list, int n, int nstages) {
  dep_begin();
  dep_wait();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int c = list[k];
  DevDiag *d = args[c * nstages].diag;
  double cdt = __longlong_as_double((long long)d->cfl_bits);
  double cand = d->dt * ccs[c].dt_ratio;
  d->dt = (cand < cdt) ? cand : cdt;
}

void launch_cfl_batch(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                      int nstages, const int *phase_base, int ncases, int grid, cudaStream_t st,
                      const int *case_list) {
  if (nwork > 0) {
    if (grid < 1 || grid > nwork) grid = nwork;
    launch_dep(true, st, grid, kTileCells, cfl_kernel_batch, args, ccs, work, nwork, nstages, phase_base);
  }
  if (case_list) {
    if (ncases > 0)
      launch_dep(true, st, (ncases + 127) / 128, 128, finalize_dt_batch_list, args, ccs, case_list,
                 ncases, nstages);
  } else if (ncases > 0) {
    launch_dep(true, st, (ncases + 127) / 128, 128, finalize_dt_batch, args, ccs, ncases, nstages);
  }
}

void launch_batch_step(int *counters, const StageArgs *args, int ncases, int nstages,
                       cudaStream_t st) {
  launch_dep(false, st, 1, 128, batch_step_kernel, counters, args, ncases, nstages);
}
#endif

void launch_cfl(const CflArgs &a, const CaseConst &cc, int nsm, cudaStream_t st, bool dep) {
  int64_t blocks = (a.nslots + 255) / 256;
  int64_t cap = (int64_t)nsm * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  launch_dep(dep, st, (unsigned)blocks, 256, cfl_kernel, a, cc);
  launch_dep(true, st, 1, 1, take_folded_cfl_kernel, a.diag, cc);
}

void launch_step_begin(DevDiag *d, cudaStream_t st, bool dep) {
  launch_dep(dep, st, 1, 1, step_begin_kernel, d);
}

void launch_take_folded_cfl(DevDiag *d, const CaseConst &cc, cudaStream_t st, bool dep) {
  launch_dep(dep, st, 1, 1, take_folded_cfl_kernel, d, cc);
}

void launch_scatter(const double *rows, const int32_t *cell_slot, const uint8_t *alias, int64_t n,
                    double *const s0[kStateFields], int nsm, cudaStream_t st) {
  int64_t blocks = (n + 255) / 256;
  if (blocks > (int64_t)nsm * 16) blocks = (int64_t)nsm * 16;
  if (blocks < 1) blocks = 1;
  scatter_state_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, cell_slot, alias, n, s0[F_RHO],
                                                         s0[F_U], s0[F_V], s0[F_P], s0[F_E],
                                                         s0[F_T]);
}

void launch_gather(double *rows, const int32_t *cell_slot, int64_t n,
                   double *const s0[kStateFields], int nsm, cudaStream_t st) {
  int64_t blocks = (n + 255) / 256;
  if (blocks > (int64_t)nsm * 16) blocks = (int64_t)nsm * 16;
  if (blocks < 1) blocks = 1;
  gather_state_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, cell_slot, n, s0[F_RHO], s0[F_U],
                                                        s0[F_V], s0[F_P], s0[F_E], s0[F_T]);
}

void launch_scatter4(const double *rows, const int32_t *cell_slot, const uint8_t *alias, int64_t n,
                     double Rg, double Cv, double *const s0[kStateFields], int nsm,
                     cudaStream_t st) {
  int64_t blocks = (n + 255) / 256;
  if (blocks > (int64_t)nsm * 16) blocks = (int64_t)nsm * 16;
  if (blocks < 1) blocks = 1;
  scatter_state4_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, cell_slot, alias, n, Rg, Cv,
                                                          s0[F_RHO], s0[F_U], s0[F_V], s0[F_P],
                                                          s0[F_E], s0[F_T]);
}

void launch_gather4(double *rows, const int32_t *cell_slot, int64_t n,
                    double *const s0[kStateFields], int nsm, cudaStream_t st) {
  int64_t blocks = (n + 255) / 256;
  if (blocks > (int64_t)nsm * 16) blocks = (int64_t)nsm * 16;
  if (blocks < 1) blocks = 1;
  gather_state4_kernel<<<(unsigned)blocks, 256, 0, st>>>(rows, cell_slot, n, s0[F_RHO], s0[F_U],
                                                         s0[F_V], s0[F_P]);
}

}  // namespace IBGPU_KNS
}  // namespace ibgpu
