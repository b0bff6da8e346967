// Ghost-fill, viscous-flux and wall-force kernels of the step (included by
// each arithmetic build after kernels.cuh, inside namespace
// ibgpu::IBGPU_KNS).  Ghost fills and forces are FP64 in every build and
// follow the reference expression by expression; the viscous flux follows
// the build's real type R.
#pragma once

#include "exactmath.cuh"

namespace ibgpu {
namespace IBGPU_KNS {

// threads of a viscous CTA: the FP64 build adds a ninth warp for the edge
template <typename R>
constexpr int visc_threads() {
#ifdef IBGPU_FAST_BUILD
  if (sizeof(R) == 8) return kTileCells + 32;
#endif
  return kTileCells;
}

// ---- coarse/fine interface ----------------------------------------------

// AMR::InterfaceRestriction -> PairRestriction_2d -> AverageCell_2d
// (AMRInterface.cpp:78-110, TwoLevelOp.H:67-87, 225-231): density-weighted
// mean of the four sons written to the coarse ghost.
__device__ __forceinline__ void restrict_pair(const PairArgs &a, const CaseConst &cc, int i) {
  double *const *q = a.s0;
  double roe = 0.0, u = 0.0, v = 0.0, e = 0.0;
  const int4 fine = reinterpret_cast<const int4 *>(a.fine)[i];
  const int sons[4] = {fine.x, fine.y, fine.z, fine.w};
  const int c = a.coarse[i];
  dep_wait();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    int f = sons[k];
    double r = q[F_RHO][f];
    roe += r;
    u += q[F_U][f] * r;
    v += q[F_V][f] * r;
    e += q[F_E][f] * r;
  }
  u /= roe;
  v /= roe;
  e /= roe;
  roe *= 0.25;
  double p = (e - 0.5 * (u * u + v * v)) * cc.gm1 * roe;
  double T = p / (roe * cc.Rg);
  q[F_RHO][c] = roe;
  q[F_U][c] = u;
  q[F_V][c] = v;
  q[F_P][c] = p;
  q[F_E][c] = e;
  q[F_T][c] = T;
}

// AMR::InterfaceProlongation -> PairProlongation_2d (TwoLevelOp.H:200-215,
// 16-22, 35-43): conserved variables of the coarse cell and its x/y
// neighbours, central gradients (q+ - q-)/2, sons at offsets -/+ 1/4,
// primitive recovery of each son.
__device__ __forceinline__ void prolong_pair(const PairArgs &a, const CaseConst &cc, int i) {
  double *const *q = a.s0;
  // neighbour order: -x, +x, -y, +y
  double U[5][4];
  const int4 nb = reinterpret_cast<const int4 *>(a.nb)[i];
  const int4 fine = reinterpret_cast<const int4 *>(a.fine)[i];
  const int cells[5] = {a.coarse[i], nb.x, nb.y, nb.z, nb.w};
  const int sons[4] = {fine.x, fine.y, fine.z, fine.w};
  dep_wait();
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    int s = cells[k];
    double r = q[F_RHO][s];
    U[k][0] = r;
    U[k][1] = r * q[F_U][s];
    U[k][2] = r * q[F_V][s];
    U[k][3] = r * q[F_E][s];
  }
  double gx[4], gy[4];
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    gx[v] = (U[2][v] - U[1][v]) * 0.5;
    gy[v] = (U[4][v] - U[3][v]) * 0.5;
  }
  const double fincrem[2] = {-0.25, 0.25};
#pragma unroll
  for (int si = 0; si < 2; ++si)
#pragma unroll
    for (int sj = 0; sj < 2; ++sj) {
      double f[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) f[v] = U[0][v] + fincrem[si] * gx[v] + fincrem[sj] * gy[v];
      double roe = f[0];
      double u = f[1] / f[0];
      double vv = f[2] / f[0];
      double e = f[3] / f[0];
      double p = (e - 0.5 * (u * u + vv * vv)) * cc.gm1 * roe;
      double T = p / (roe * cc.Rg);
      int s = sons[si * 2 + sj];
      q[F_RHO][s] = roe;
      q[F_U][s] = u;
      q[F_V][s] = vv;
      q[F_P][s] = p;
      q[F_E][s] = e;
      q[F_T][s] = T;
    }
}

// ---- domain boundary ghosts (BCValues::BCBoxTreat, BCValues.H:51-298) ----
__device__ __forceinline__ void bc_ghost(const BcArgs &a, const CaseConst &cc, int i) {
  double *const *q = a.s0;
  const int g = a.ghost[i], r = a.ref[i];
  const int type = a.type[i];
  const double *fv = a.facevar + 7 * a.face[i];
  dep_wait();
  double roe = q[F_RHO][r], u = q[F_U][r], v = q[F_V][r], p = q[F_P][r], T = q[F_T][r],
         e = q[F_E][r];
  switch (type) {
    case -50:  // outflow: copy (SetBCType_50)
      break;
    case -12:  // pressure outlet (SetBCType_12)
      p = fv[4] + a.backpressure;
      roe = p / (cc.Rg * T);
      break;
    case -13: {  // pressure inlet (SetBCType_13)
      double speed0 = sqrt(u * u + v * v);
      u = speed0 * a.cos_in;
      v = speed0 * a.sin_in;
      T = fv[5] - 0.5 * (u * u + v * v) / cc.Cp;
      p = fv[4] * pow3p5_rn(T / fv[5]);
      roe = p / (cc.Rg * T);
      e = cc.Cv * T + 0.5 * (u * u + v * v);
      break;
    }
    case -49:  // no-slip wall (SetBCType_49); -46/-42 with a static frame and faces
    case -46:
    case -42:
      u = 0.0;
      v = 0.0;
      roe = p / (cc.Rg * T);
      e = cc.Cv * T + 0.0;
      break;
    case -51: {  // slip wall (SetBCType_51)
      const double *n = a.nmv + 3 * i;
      double un = u * n[0] + v * n[1];
      u = u - un * n[0];
      v = v - un * n[1];
      double w = 0.0 - un * n[2];
      roe = p / (cc.Rg * T);
      e = cc.Cv * T + 0.5 * (u * u + v * v + w * w);
      break;
    }
    case -10:  // fixed values (SetBCType_10)
      roe = fv[0];
      u = fv[1];
      v = fv[2];
      p = fv[4];
      T = fv[5];
      e = fv[6];
      break;
    case -45:  // fixed velocity, zero-gradient pressure (SetBCType_45)
      u = fv[1];
      v = fv[2];
      T = fv[5];
      roe = p / (cc.Rg * T);
      break;
    default:
      return;
  }
  q[F_RHO][g] = roe;
  q[F_U][g] = u;
  q[F_V][g] = v;
  q[F_P][g] = p;
  q[F_E][g] = e;
  q[F_T][g] = T;
}

__global__ void restrict_kernel(PairArgs a, CaseConst cc) {
  dep_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n) restrict_pair(a, cc, i);
}
__global__ void prolong_kernel(PairArgs a, CaseConst cc) {
  dep_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.n) prolong_pair(a, cc, i);
}
__global__ void bc_kernel(BcArgs a, CaseConst cc) {
  dep_begin();
  const int i = a.begin + blockIdx.x * blockDim.x + threadIdx.x;
  if (i < a.end) bc_ghost(a, cc, i);
}

// ---- immersed-boundary ghost cells (Body::IBConditions_Image) -----------

// Image-point state, Mesh::IntpHGgcellVar (Mesh.cpp:1532-1547)
__device__ __forceinline__ void image_point(const int32_t *cells, const double *w,
                                            double *const *q, const CaseConst &cc, double &T,
                                            double &p, double &u, double &v, double &roe) {
  T = 0.0;
  p = 0.0;
  u = 0.0;
  v = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    int s = cells[k];
    T += w[k] * q[F_T][s];
    p += w[k] * q[F_P][s];
    u += w[k] * q[F_U][s];
    v += w[k] * q[F_V][s];
  }
  roe = p / (cc.Rg * T);
}

// New state of IB cell i (rho u v p e T) from the current field.
__device__ __forceinline__ void ib_cell(const IbArgs &a, const CaseConst &cc, int i,
                                        double (&o)[6]) {
  const double *f = a.cellf + 16 * i;  // signdis, hgdis, w[8], nv[3], patv[3]
  double hT, hp, hu, hv, hroe;
  image_point(a.intp + 8 * i, f + 2, a.s0, cc, hT, hp, hu, hv, hroe);
  const double signdis = f[0], hgdis = f[1];
  const double *wv = f + 13;
  double u, v, w, p, T;
  if (signdis < 0.0) {
    u = 2.0 * wv[0] - hu;
    v = 2.0 * wv[1] - hv;
    w = 2.0 * wv[2] - 0.0;
    p = hp;
    T = hT;
  } else {
    // Body::LinearDist (Body.cpp:183-204)
    double rt = signdis + hgdis;
    double r0 = signdis / rt;
    u = wv[0] + (hu - wv[0]) * r0;
    v = wv[1] + (hv - wv[1]) * r0;
    w = wv[2] + (0.0 - wv[2]) * r0;
    p = hp;
    T = hT;
  }
  double roe = p / (cc.Rg * T);
  double e = cc.Cv * T + 0.5 * (u * u + v * v + w * w);
  o[0] = roe;
  o[1] = u;
  o[2] = v;
  o[3] = p;
  o[4] = e;
  o[5] = T;
  const int phase = a.phase + (a.phase_base ? *a.phase_base : 0);
  if (hT < 0.0) raise_error(a.diag, phase, ERR_IB_NEG_T, a.cell[i]);
  if (isnan(roe) || isnan(u) || isnan(v) || isnan(p) || isnan(T) || isnan(e))
    raise_error(a.diag, phase, ERR_IB_NAN, a.cell[i]);
}

__device__ __forceinline__ void ib_put(const IbArgs &a, int i, const double (&o)[6]) {
  const int s = a.cell[i];
  a.s0[F_RHO][s] = o[0];
  a.s0[F_U][s] = o[1];
  a.s0[F_V][s] = o[2];
  a.s0[F_P][s] = o[3];
  a.s0[F_E][s] = o[4];
  a.s0[F_T][s] = o[5];
}

// The reference computes every IB cell's state before it writes any
// (Body.cpp:1361-1494).  Up to kIbBlock cells: one CTA, a barrier between the
// two halves (the airfoils have a few hundred cells: one launch instead of
// two).  More: two launches with the states in between in a.out.
constexpr int kIbBlock = 1024;
__global__ void __launch_bounds__(kIbBlock) ib_kernel(IbArgs a, CaseConst cc) {
  dep_begin();
  dep_wait();
  const int i = threadIdx.x;
  double o[6];
  if (i < a.n) ib_cell(a, cc, i, o);
  __syncthreads();
  if (i < a.n) ib_put(a, i, o);
}
__global__ void ib_compute_kernel(IbArgs a, CaseConst cc) {
  dep_begin();
  dep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  double o[6];
  ib_cell(a, cc, i, o);
  for (int k = 0; k < 6; ++k) a.out[6 * i + k] = o[k];
}
__global__ void ib_store_kernel(IbArgs a) {
  dep_begin();
  dep_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  double o[6];
  for (int k = 0; k < 6; ++k) o[k] = a.out[6 * i + k];
  ib_put(a, i, o);
}

// ---- wall forces (Body::ComptWallForce, Body.cpp:439-558) ----------------
// Per patch: image-point state, tangential shear mu*du_t/hgdis*area,
// pressure force -p n area, and their moments about the body centre.
__global__ void patch_force_kernel(ForceArgs a, CaseConst cc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  const double *f = a.patchf + 19 * i;  // pc[3], nv[3], area, hgdis, w[8], patv[3]
  double hT, hp, hu, hv, hroe;
  image_point(a.intp + 8 * i, f + 8, a.s0, cc, hT, hp, hu, hv, hroe);
  const double *pc = f, *nv = f + 3, *pv = f + 16;
  const double area = f[6], hgdis = f[7];
  const double *bc = a.body_center + 3 * a.body[i];
  double du0 = hu - pv[0], du1 = hv - pv[1], du2 = 0.0 - pv[2];
  double dx0 = pc[0] - bc[0], dx1 = pc[1] - bc[1], dx2 = pc[2] - bc[2];
  double dn = du0 * nv[0] + du1 * nv[1] + du2 * nv[2];
  du0 = (du0 - nv[0] * dn) / hgdis;
  du1 = (du1 - nv[1] * dn) / hgdis;
  du2 = (du2 - nv[2] * dn) / hgdis;
  double df0[3] = {du0 * cc.mu * area, du1 * cc.mu * area, du2 * cc.mu * area};
  double pa = -hp * area;
  double df1[3] = {nv[0] * pa, nv[1] * pa, nv[2] * pa};
  double *o = a.out + 12 * i;
  o[0] = df1[0];
  o[1] = df1[1];
  o[2] = df1[2];
  o[3] = df0[0];
  o[4] = df0[1];
  o[5] = df0[2];
  // dm = dxyz x df (Pointxyz::cross)
  o[6] = dx1 * df1[2] - dx2 * df1[1];
  o[7] = dx2 * df1[0] - dx0 * df1[2];
  o[8] = dx0 * df1[1] - dx1 * df1[0];
  o[9] = dx1 * df0[2] - dx2 * df0[1];
  o[10] = dx2 * df0[0] - dx0 * df0[2];
  o[11] = dx0 * df0[1] - dx1 * df0[0];
}

// Sums in patch order, then the reference's dimensional scaling.  Each of
// the 12 parts (pressure force, shear force, pressure moment, shear moment)
// is its own sequential sum from zero over the body's patches, as in the
// reference; the block stages the parts a chunk of patches at a time in
// shared memory and 12 threads run the 12 sums side by side (one thread
// reading them from global memory one patch after another spent some 800 ns
// per patch waiting on loads).
__global__ void __launch_bounds__(256) force_sum_kernel(ForceArgs a, CaseConst cc) {
  constexpr int kChunk = 256;
  __shared__ double part[12 * kChunk];
  __shared__ double sum[12];
  const int t = threadIdx.x;
  for (int b = 0; b < a.nbodies; ++b) {
    double acc = 0.0;
    const int i0 = a.body_begin[b], i1 = a.body_begin[b + 1];
    for (int c = i0; c < i1; c += kChunk) {
      const int m = min(kChunk, i1 - c);
      for (int k = t; k < 12 * m; k += blockDim.x) part[k] = a.out[12 * (int64_t)c + k];
      __syncthreads();
      if (t < 12)
        for (int i = 0; i < m; ++i) acc += part[12 * i + t];
      __syncthreads();  // the next chunk overwrites the parts
    }
    if (t < 12) sum[t] = acc;
    __syncthreads();
    if (t == 0) {
      double *r = a.result + 6 * b;
      for (int k = 0; k < 3; ++k) {
        double pfs = sum[k] * cc.p_ref * cc.area_ref;
        double pms = sum[6 + k] * cc.p_ref * cc.area_ref * cc.L_ref;
        double tfs = sum[3 + k] * cc.shear_ref * cc.area_ref;
        double tms = sum[9 + k] * cc.shear_ref * cc.area_ref * cc.L_ref;
        r[k] = pfs + tfs;
        r[3 + k] = pms + tms;
      }
    }
    __syncthreads();  // sum[] is rewritten for the next body
  }
}

// ---- viscous face flux (NS_Solver::ComptViscousStress) -------------------
// u, v, T of the tile and a one-cell halo (corners included) into the 18 x 18
// region, zeros and flag 0 where no cell is: a thread per own cell, the last
// four of the CTA's warps one side (lanes 0..15) and one corner (lane 16:
// south-west, north-east, north-west, south-east) each.  Waits for the
// previous kernel after the lookups that no step changes.  Returns the flags
// of the thread's own cell.
template <typename R, int NT, typename A>
__device__ __forceinline__ uint8_t visc_region(const A &a, int tile, R *su, R *sv, R *sT,
                                               uint8_t *sfl) {
  constexpr int G = kTile + 2;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool own = tid < kTileCells;
  const int rc = (((tid >> 4) & 15) + 1) * G + (tid & 15) + 1;
  const int side = NT / 32 - 1 - (tid >> 5);
  const bool halo = side < 4 && lane <= 16;
  int nb = -1, hoff = 0, hr = 0;
  if (halo) {
    int x, y;  // position relative to the tile
    if (lane < 16) {
      x = side < 2 ? lane : (side == 2 ? -1 : kTile);
      y = side < 2 ? (side ? kTile : -1) : lane;
    } else {
      x = side == 0 || side == 2 ? -1 : kTile;
      y = side == 0 || side == 3 ? -1 : kTile;
    }
    const int ox = x < 0 ? -1 : (x >= kTile ? 1 : 0), oy = y < 0 ? -1 : (y >= kTile ? 1 : 0);
    nb = a.tile_nb[(int64_t)tile * 9 + (oy + 1) * 3 + ox + 1];
    hoff = (y - oy * kTile) * kTile + x - ox * kTile;
    hr = (y + 1) * G + x + 1;
  }
  const int64_t os = (int64_t)tile * kTileCells + (own ? tid : 0);
  const uint8_t fown = own ? a.flags[os] : (uint8_t)0;
  const int64_t hs = (int64_t)nb * kTileCells + hoff;
  const uint8_t fh = nb >= 0 ? a.flags[hs] : (uint8_t)0;
  dep_wait();
  R u = R(0), v = R(0), T = R(0), hu = R(0), hv = R(0), hT = R(0);
  if (fown & CF_PRESENT) {
    u = (R)a.s0[F_U][os];
    v = (R)a.s0[F_V][os];
    T = (R)a.s0[F_T][os];
  }
  if (fh & CF_PRESENT) {
    hu = (R)a.s0[F_U][hs];
    hv = (R)a.s0[F_V][hs];
    hT = (R)a.s0[F_T][hs];
  }
  if (own) {
    su[rc] = u;
    sv[rc] = v;
    sT[rc] = T;
    sfl[rc] = fown;
  }
  if (halo) {
    su[hr] = hu;
    sv[hr] = hv;
    sT[hr] = hT;
    sfl[hr] = fh;
  }
  return fown;
}

// Expression by expression the reference: the exact build, and the mixed
// build's FP32 (whose contractions and order of summation decide roundings of
// its FP32 stage buffers, so it keeps them).
// One tile per CTA: u, v, T of the tile and a one-cell halo (corners
// included), every x- and y-face viscous flux into shared memory, then each
// leaf cell's frozen residual parts vs(high) - vs(low) per direction.
template <typename R, typename A>
__device__ __forceinline__ void viscous_tile_plain(const A &a, const CaseConst &cc, int tile) {
  constexpr int H = 1, G = kTile + 2 * H;  // 18
  __shared__ R su[G * G], sv[G * G], sT[G * G];
  __shared__ uint8_t sfl[G * G];
  __shared__ R vx[3][kXFaces];  // x-mom, y-mom, energy of x-faces
  __shared__ R vy[3][kYFaces];
  const int tid = threadIdx.x;
  const LevelConst &L = cc.lev[a.tile_level[tile]];
  visc_region<R, kTileCells>(a, tile, su, sv, sT, sfl);
  __syncthreads();
  const R ikx = (R)L.inv_dx, iky = (R)L.inv_dy;
  const R Re = (R)cc.Re, S = (R)cc.s_over_t, qk = (R)cc.qk;
  for (int w = tid; w < kXFaces + kYFaces; w += kTileCells) {
    const bool xdir = w < kXFaces;
    int rL, rR, tstep;
    if (xdir) {
      int j = w / (kTile + 1), i = w % (kTile + 1);
      rR = (j + H) * G + (i + H);
      rL = rR - 1;
      tstep = G;
    } else {
      int v = w - kXFaces;
      int j = v / kTile, i = v % kTile;
      rR = (j + H) * G + (i + H);
      rL = rR - G;
      tstep = 1;
    }
    R f1 = R(0), f2 = R(0), f3 = R(0);
    const uint8_t fL = sfl[rL], fR = sfl[rR];
    if ((fL & CF_PRESENT) && (fR & CF_PRESENT) && ((fL | fR) & CF_NORMAL)) {
      const int Lu = rL + tstep, Ru = rR + tstep, Ld = rL - tstep, Rd = rR - tstep;
      // normal difference and the 2x3-block tangential difference
      // (pfpkesai0 / pfpkesai1, NS_Solver.H:147-151)
      R dnu = su[rR] - su[rL], dnv = sv[rR] - sv[rL], dnT = sT[rR] - sT[rL];
      R dtu = R(0.25) * (su[Lu] + su[Ru] - su[Ld] - su[Rd]);
      R dtv = R(0.25) * (sv[Lu] + sv[Ru] - sv[Ld] - sv[Rd]);
      R dtT = R(0.25) * (sT[Lu] + sT[Ru] - sT[Ld] - sT[Rd]);
      R dux, duy, dvx, dvy, dTx, dTy;
      if (xdir) {
        dux = dnu * ikx; duy = dtu * iky; dvx = dnv * ikx; dvy = dtv * iky;
        dTx = dnT * ikx; dTy = dtT * iky;
      } else {
        dux = dtu * ikx; duy = dnu * iky; dvx = dtv * ikx; dvy = dnv * iky;
        dTx = dtT * ikx; dTy = dnT * iky;
      }
      R ftemp = (sT[rL] + sT[rR]) * R(0.5);
      R ft3;
      if (sizeof(R) == sizeof(double)) ft3 = (R)cube_rn((double)ftemp);
      else ft3 = ftemp * ftemp * ftemp;
      R mu0 = sqrt(ft3) * ((R(1) + S) / (ftemp + S));
      R qk0 = qk * mu0;
      R tauxx = R(2) * mu0 * (dux - (dux + dvy) / R(3)) / Re;
      R tauyy = R(2) * mu0 * (dvy - (dux + dvy) / R(3)) / Re;
      R tauxy = mu0 / Re * (duy + dvx);
      R qx = qk0 * dTx, qy = qk0 * dTy;
      R fv0 = (su[rL] + su[rR]) * R(0.5);
      R fv1 = (sv[rL] + sv[rR]) * R(0.5);
      if (xdir) {
        R area = (R)L.area_x;
        f1 = tauxx * area;
        f2 = tauxy * area;
        f3 = (fv0 * tauxx + fv1 * tauxy + qx) * area;
      } else {
        R area = (R)L.area_y;
        f1 = tauxy * area;
        f2 = tauyy * area;
        f3 = (fv0 * tauxy + fv1 * tauyy + qy) * area;
      }
    }
    if (xdir) {
      vx[0][w] = f1; vx[1][w] = f2; vx[2][w] = f3;
    } else {
      int v = w - kXFaces;
      vy[0][v] = f1; vy[1][v] = f2; vy[2][v] = f3;
    }
  }
  __syncthreads();
  const int lx = tid % kTile, ly = tid / kTile;
  const int64_t slot = (int64_t)tile * kTileCells + tid;
  if (sfl[(ly + H) * G + (lx + H)] & CF_NORMAL) {
    const int xlo = ly * (kTile + 1) + lx, xhi = xlo + 1;
    const int ylo = ly * kTile + lx, yhi = ylo + kTile;
    double *vsd = const_cast<double *>(a.vsd);  // a stage's arguments only read it
    // planes of x and y parts: the exact build has the mass's zeros too
    constexpr int x0 = sizeof(R) == 8 ? 1 : 0, y0 = sizeof(R) == 8 ? 5 : 3;
    if (sizeof(R) == 8) {
      vsd[0 * a.nslots + slot] = 0.0 - 0.0;
      vsd[4 * a.nslots + slot] = 0.0 - 0.0;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      vsd[(int64_t)(x0 + c) * a.nslots + slot] = (double)vx[c][xhi] - (double)vx[c][xlo];
      vsd[(int64_t)(y0 + c) * a.nslots + slot] = (double)vy[c][yhi] - (double)vy[c][ylo];
    }
  }
}

#ifdef IBGPU_FAST_BUILD
// The FP64 build's face: T^1.5 as T^2 times the inverse root, one reciprocal
// instead of the five divisions and the root (each some twenty FP64
// instructions), the normal stress along the face only.  n: the normal
// velocity component, t: the tangential one (the flux is the same in both
// directions with the components' roles exchanged).
__device__ __forceinline__ void viscous_face_fast(const CaseConst &cc, double area, double ikn,
                                                  double ikt, double nL, double nR, double tL,
                                                  double tR, double TL, double TR, double tn,
                                                  double tt, double &fn, double &ft, double &fe) {
  typedef FastMath<double> M;
  const double T = 0.5 * (TL + TR);
  const double T2 = T * T;  // (T = 0 has no viscosity, not 0 times an infinite root)
  const double mu = (T2 == 0.0 ? 0.0 : T2 * M::rsqrt(T)) * ((1.0 + cc.s_over_t) * M::rcp(T + cc.s_over_t)) * area;
  const double dn_n = (nR - nL) * ikn, dt_n = (tR - tL) * ikn;      // normal derivatives
  const double kt = 0.25 * ikt;
  const double dn_t = tn * kt, dt_t = tt * kt;                      // tangential derivatives
  const double m = mu * cc.inv_Re;
  fn = (m * (2.0 / 3.0)) * fma(2.0, dn_n, -dt_t);
  ft = m * (dn_t + dt_n);
  fe = fma(0.5 * (nL + nR), fn, fma(0.5 * (tL + tR), ft, (cc.qk * mu) * ((TR - TL) * ikn)));
}

// The FP64 build's tile: a thread per cell (its west and south face), a ninth
// warp for the east and north faces, whole warps for the halo sides (288
// threads); one frozen residual per component, the x and y parts added: 24
// bytes a cell written here and read by every stage instead of 64.  With the
// divisions gone it is bound by one load round trip per tile.  16 steps of
// the 914 k-row nested mesh 2.32 -> 1.96 ms, 24 of the airfoil 1.06 -> 0.92.
template <typename A>
__device__ __forceinline__ void viscous_tile_fp64(const A &a, const CaseConst &cc, int tile) {
  constexpr int G = kTile + 2, kFX = kTile + 1, NF = kTile * kFX;
  __shared__ double su[G * G], sv[G * G], sT[G * G];
  __shared__ uint8_t sfl[G * G];
  __shared__ double vx[3][NF];  // x-face i of row j at j*17 + i: x-mom, y-mom, energy
  __shared__ double vy[3][NF];  // y-face j of column i at j*16 + i
  const int tid = threadIdx.x, lane = tid & 31;
  const bool own = tid < kTileCells;
  const int tx = tid & 15, ty = (tid >> 4) & 15;
  const LevelConst &L = cc.lev[a.tile_level[tile]];
  const int rc = (ty + 1) * G + tx + 1;
  const uint8_t fown = visc_region<double, kTileCells + 32>(a, tile, su, sv, sT, sfl);
  __syncthreads();
  const double ikx = L.inv_dx, iky = L.inv_dy, ax = L.area_x, ay = L.area_y;
  // face between region cells l and l + step, tangential step ts
  auto face = [&](bool xdir, int l, double *out, int at) {
    const int step = xdir ? 1 : G, ts = xdir ? G : 1, r = l + step;
    double f[3] = {0.0, 0.0, 0.0};
    if ((sfl[l] & CF_PRESENT) && (sfl[r] & CF_PRESENT) && ((sfl[l] | sfl[r]) & CF_NORMAL)) {
      const double tu = su[l + ts] + su[r + ts] - su[l - ts] - su[r - ts],
              tv = sv[l + ts] + sv[r + ts] - sv[l - ts] - sv[r - ts];
      const double *n = xdir ? su : sv, *t = xdir ? sv : su;
      viscous_face_fast(cc, xdir ? ax : ay, xdir ? ikx : iky, xdir ? iky : ikx, n[l], n[r], t[l],
                        t[r], sT[l], sT[r], xdir ? tu : tv, xdir ? tv : tu, f[xdir ? 0 : 1],
                        f[xdir ? 1 : 0], f[2]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) out[c * NF + at] = f[c];
  };
  if (own) {
    face(true, rc - 1, &vx[0][0], ty * kFX + tx);
    face(false, rc - G, &vy[0][0], ty * kTile + tx);
  } else if (lane < 16) {
    face(true, (lane + 1) * G + kTile, &vx[0][0], lane * kFX + kTile);
  } else {
    face(false, kTile * G + (lane & 15) + 1, &vy[0][0], kTile * kTile + (lane & 15));
  }
  __syncthreads();
  if (own && (fown & CF_NORMAL)) {
    double *vsd = const_cast<double *>(a.vsd);  // a stage's arguments only read it
    const int x = ty * kFX + tx, y = ty * kTile + tx;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      vsd[(int64_t)c * a.nslots + (int64_t)tile * kTileCells + tid] =
          (vx[c][x + 1] - vx[c][x]) + (vy[c][y + kTile] - vy[c][y]);
  }
}
#endif

template <typename R>
__global__ void __launch_bounds__(visc_threads<R>()) viscous_kernel(ViscArgs a, CaseConst cc) {
  dep_begin();
  const int tile = a.tile_begin + (int)blockIdx.x;
#ifdef IBGPU_FAST_BUILD
  if constexpr (sizeof(R) == 8) viscous_tile_fp64(a, cc, tile);
  else
#endif
    viscous_tile_plain<R>(a, cc, tile);
}

#ifdef IBGPU_FAST_BUILD
// ---- the same over several cases: each block takes one block of one case
__global__ void restrict_kernel_batch(const BatchPairs *__restrict__ segs,
                                      const CaseConst *__restrict__ ccs,
                                      const int2 *__restrict__ blocks) {
  dep_begin();
  const int2 b = blocks[blockIdx.x];
  const BatchPairs &s = segs[b.x];
  const int i = b.y + threadIdx.x;
  if (i < s.a.n) restrict_pair(s.a, ccs[s.c], i);
}
__global__ void prolong_kernel_batch(const BatchPairs *__restrict__ segs,
                                     const CaseConst *__restrict__ ccs,
                                     const int2 *__restrict__ blocks) {
  dep_begin();
  const int2 b = blocks[blockIdx.x];
  const BatchPairs &s = segs[b.x];
  const int i = b.y + threadIdx.x;
  if (i < s.a.n) prolong_pair(s.a, ccs[s.c], i);
}
__global__ void bc_kernel_batch(const BatchBc *__restrict__ segs,
                                const CaseConst *__restrict__ ccs,
                                const int2 *__restrict__ blocks) {
  dep_begin();
  const int2 b = blocks[blockIdx.x];
  const BatchBc &s = segs[b.x];
  const int i = b.y + threadIdx.x;
  if (i < s.a.end) bc_ghost(s.a, ccs[s.c], i);
}
// one CTA per case (each of at most kIbBlock cells)
__global__ void __launch_bounds__(kIbBlock)
    ib_kernel_batch(const BatchIb *__restrict__ segs, const CaseConst *__restrict__ ccs) {
  dep_begin();
  dep_wait();
  const BatchIb &s = segs[blockIdx.x];
  const int i = threadIdx.x;
  double o[6];
  if (i < s.a.n) ib_cell(s.a, ccs[s.c], i, o);
  __syncthreads();
  if (i < s.a.n) ib_put(s.a, i, o);
}
template <typename R>
__global__ void __launch_bounds__(visc_threads<R>())
    viscous_kernel_batch(const StageArgs *__restrict__ args, const CaseConst *__restrict__ ccs,
                         const int2 *__restrict__ work, int nstages) {
  dep_begin();
  const int2 it = work[blockIdx.x];
  if constexpr (sizeof(R) == 8) viscous_tile_fp64(args[it.x * nstages], ccs[it.x], it.y);
  else viscous_tile_plain<R>(args[it.x * nstages], ccs[it.x], it.y);
}

void launch_pairs_batch(const BatchPairs *segs, const CaseConst *ccs, const int2 *blocks,
                        int nblocks, bool prolong, cudaStream_t st) {
  if (nblocks <= 0) return;
  launch_dep(true, st, nblocks, kBatchBlock, prolong ? prolong_kernel_batch : restrict_kernel_batch,
             segs, ccs, blocks);
}
void launch_bc_batch(const BatchBc *segs, const CaseConst *ccs, const int2 *blocks, int nblocks,
                     cudaStream_t st) {
  if (nblocks > 0) launch_dep(true, st, nblocks, kBatchBlock, bc_kernel_batch, segs, ccs, blocks);
}
bool launch_ib_batch(const BatchIb *segs, const CaseConst *ccs, int ncases, int most,
                     cudaStream_t st) {
  if (most > kIbBlock) return false;
  if (ncases > 0) launch_dep(true, st, ncases, (most + 31) / 32 * 32, ib_kernel_batch, segs, ccs);
  return true;
}
void launch_viscous_batch(const StageArgs *args, const CaseConst *ccs, const int2 *work, int nwork,
                          int nstages, bool mixed, cudaStream_t st) {
  if (nwork <= 0) return;
  if (mixed) launch_dep(true, st, nwork, visc_threads<float>(), viscous_kernel_batch<float>, args, ccs, work, nstages);
  else launch_dep(true, st, nwork, visc_threads<double>(), viscous_kernel_batch<double>, args, ccs, work, nstages);
}
#endif

// ---- launchers ---------------------------------------------------------------
void launch_restrict(const PairArgs &a, const CaseConst &cc, cudaStream_t st, bool dep) {
  if (a.n > 0) launch_dep(dep, st, (a.n + 127) / 128, 128, restrict_kernel, a, cc);
}
void launch_prolong(const PairArgs &a, const CaseConst &cc, cudaStream_t st, bool dep) {
  if (a.n > 0) launch_dep(dep, st, (a.n + 127) / 128, 128, prolong_kernel, a, cc);
}
void launch_bc(const BcArgs &a, const CaseConst &cc, cudaStream_t st, bool dep) {
  int n = a.end - a.begin;
  if (n > 0) launch_dep(dep, st, (n + 127) / 128, 128, bc_kernel, a, cc);
}
void launch_ib(const IbArgs &a, const CaseConst &cc, cudaStream_t st, bool dep) {
  if (a.n <= 0) return;
  if (a.n <= kIbBlock) {
    launch_dep(dep, st, 1, (a.n + 31) / 32 * 32, ib_kernel, a, cc);
    return;
  }
  launch_dep(dep, st, (a.n + 127) / 128, 128, ib_compute_kernel, a, cc);
  launch_dep(true, st, (a.n + 127) / 128, 128, ib_store_kernel, a);
}
void launch_forces(const ForceArgs &a, const CaseConst &cc, cudaStream_t st) {
  if (a.n > 0) patch_force_kernel<<<(a.n + 127) / 128, 128, 0, st>>>(a, cc);
  force_sum_kernel<<<1, 256, 0, st>>>(a, cc);
}
void launch_viscous(const ViscArgs &a, const CaseConst &cc, int ntiles, bool mixed,
                    cudaStream_t st, bool dep) {
  if (ntiles <= 0) return;
#ifdef IBGPU_FAST_BUILD
  if (mixed) {
    launch_dep(dep, st, ntiles, visc_threads<float>(), viscous_kernel<float>, a, cc);
    return;
  }
#endif
  launch_dep(dep, st, ntiles, visc_threads<double>(), viscous_kernel<double>, a, cc);
}

}  // namespace IBGPU_KNS
}  // namespace ibgpu
