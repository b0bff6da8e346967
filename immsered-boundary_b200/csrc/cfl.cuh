// Abort records, exact 64-bit warp reductions and the CFL bound of a cell,
// shared by the step's kernels and the allocation-free step (every operation
// separately rounded: the same bits in every build).
#pragma once

#include <cuda_runtime.h>

#include "layout.h"

namespace ibgpu {

__device__ __forceinline__ unsigned long long error_key(int phase, int check, int slot) {
  return ((unsigned long long)phase << 40) | ((unsigned long long)check << 32) | (unsigned)slot;
}
__device__ __forceinline__ void raise_error(DevDiag *d, int phase, int check, int slot) {
  atomicMin(&d->err_key, error_key(phase, check, slot));
}

// Exact maximum / minimum of a 64-bit word over the full warp with the
// 32-bit warp reductions (redux.sync): the extreme high word first, then the
// extreme low word among the lanes that hold it.  Four instructions instead
// of five rounds of two 32-bit shuffles and a 64-bit compare.
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
  const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? lo : 0xffffffffu);
  return ((unsigned long long)mh << 32) | ml;
}

// CFL bound of one normal cell, NS_Solver::Comptdt (NS_Solver.cpp:196-280),
// with every operation separately rounded so the CFL pass and the final
// stages that fold it in produce the same bits in every build: cfl_vol over
// the sum of the cell's wave speeds times face areas.
__device__ __forceinline__ double cfl_cell_sum(double T, double u, double v, const LevelConst &L,
                                               const CaseConst &cc) {
  const double c = __dsqrt_rn(__dmul_rn(cc.gamaRg, T));
  const double c0 = __dmul_rn(__dadd_rn(fabs(u), c), L.area_x);
  const double c1 = __dmul_rn(__dadd_rn(fabs(v), c), L.area_y);
  const double c2 = __dmul_rn(__dadd_rn(0.0, c), L.area_z);
  return __dadd_rn(__dadd_rn(c0, c1), c2);
}
__device__ __forceinline__ double cfl_cell_bound(double T, double u, double v, const LevelConst &L,
                                                 const CaseConst &cc) {
  return __ddiv_rn(L.cfl_vol, cfl_cell_sum(T, u, v, L, cc));
}

}  // namespace ibgpu
