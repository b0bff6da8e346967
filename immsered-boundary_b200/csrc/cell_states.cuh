// What a cell of the stage's region gives to its two faces of one direction.
// Included after the limiters of flux.cuh.
#pragma once

#include <stdint.h>

#include <cuda_runtime.h>

#include "layout.h"

namespace ibgpu {
namespace IBGPU_KNS {

// Four values of one cell (rho, u, v, p), one limited slope set, or one
// face flux (mass, x-momentum, y-momentum, energy).  In shared memory an FP32
// record is one float4; an FP64 record is split over two double2 planes
// (components 0-1 at [i], 2-3 at [i + n] for an array of n records), so a
// warp reading consecutive records moves 16-byte words at a 16-byte stride
// and every 128-bit access is conflict-free.
template <typename R>
struct Q4 {
  R x, y, z, w;
};

template <typename R>
struct SRec;

template <typename R>
__device__ __forceinline__ Q4<R> add4(const Q4<R> &a, const Q4<R> &b) {
  return Q4<R>{a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w};
}
template <typename R>
__device__ __forceinline__ Q4<R> sub4(const Q4<R> &a, const Q4<R> &b) {
  return Q4<R>{a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w};
}

// The states region cell rc (value c) gives to its two faces along `step`:
// lo to the face towards rc - step, hi to the one towards rc + step; SIDES
// says which are wanted (the region holds no cells beyond what those need).
// A cell whose neighbour on one side is missing has a flux only on the other,
// with the reference's one-sided reconstruction (its stencil then takes the
// cell two steps away on that side, NS_Solver.H:743-750); states of faces
// that carry no flux are left unset (c).
enum : int { kLow = 1, kHigh = 2 };
template <typename R, int LIM, int NQ, int SIDES>
__device__ __forceinline__ void cell_states(const typename SRec<R>::V *sq, const uint8_t *sfl,
                                            const Q4<R> &c, int rc, int step, bool uni, Q4<R> &lo,
                                            Q4<R> &hi) {
  using S = SRec<R>;
  if (uni || ((sfl[rc - step] & CF_PRESENT) && (sfl[rc + step] & CF_PRESENT))) {
    const Q4<R> m = S::ld(sq, rc - step, NQ), p = S::ld(sq, rc + step, NQ);
    const Q4<R> s = {limited_slope<LIM>(c.x - m.x, p.x - c.x),
                     limited_slope<LIM>(c.y - m.y, p.y - c.y),
                     limited_slope<LIM>(c.z - m.z, p.z - c.z),
                     limited_slope<LIM>(c.w - m.w, p.w - c.w)};
    if (SIDES & kLow) lo = sub4(c, s);
    if (SIDES & kHigh) hi = add4(c, s);
    return;
  }
  if (SIDES & kLow) lo = c;
  if (SIDES & kHigh) hi = c;
  if (sfl[rc - step] & CF_PRESENT) {
    if (SIDES & kLow) {
      const Q4<R> m = S::ld(sq, rc - step, NQ), o = S::ld(sq, rc - 2 * step, NQ);
      lo = Q4<R>{muscl_right_fast<LIM>(m.x, c.x, o.x), muscl_right_fast<LIM>(m.y, c.y, o.y),
                 muscl_right_fast<LIM>(m.z, c.z, o.z), muscl_right_fast<LIM>(m.w, c.w, o.w)};
    }
  } else if (sfl[rc + step] & CF_PRESENT) {
    if (SIDES & kHigh) {
      const Q4<R> p = S::ld(sq, rc + step, NQ), o = S::ld(sq, rc + 2 * step, NQ);
      hi = Q4<R>{muscl_left_fast<LIM>(o.x, c.x, p.x), muscl_left_fast<LIM>(o.y, c.y, p.y),
                 muscl_left_fast<LIM>(o.z, c.z, p.z), muscl_left_fast<LIM>(o.w, c.w, p.w)};
    }
  }
}

}  // namespace IBGPU_KNS
}  // namespace ibgpu
