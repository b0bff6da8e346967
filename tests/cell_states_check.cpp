// Which records of a stage's 20 x 20 region the face states of its cells read,
// for every presence pattern along the stencil: inside the region, and none of
// the corners, which hold nothing.  Built with the address sanitiser (flags)
// and without optimisation (no dead load is dropped).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#define IBGPU_KNS host
#include "layout.h"

namespace ibgpu {
namespace host {
template <int>
double limited_slope(double a, double b) { return a + b; }
template <int>
double muscl_left_fast(double a, double b, double c) { return a + b + c; }
template <int>
double muscl_right_fast(double a, double b, double c) { return a + b + c; }
}  // namespace host
}  // namespace ibgpu

#include "cell_states.cuh"

namespace {
constexpr int kHalo = 2, kReg = ibgpu::kTile + 2 * kHalo, NQ = kReg * kReg;
int g_cell, g_bad;
bool corner(int i) {
  auto out = [](int k) { return k < kHalo || k >= kReg - kHalo; };
  return out(i % kReg) && out(i / kReg);
}
}  // namespace

namespace ibgpu {
namespace host {
template <>
struct SRec<double> {
  using V = int;
  static Q4<double> ld(const V *, int i, int) {
    if (i < 0 || i >= NQ || corner(i)) {
      if (g_bad++ == 0) std::printf("cell (%d, %d) reads record %d\n", g_cell % kReg, g_cell / kReg, i);
    }
    return Q4<double>{1, 2, 3, 4};
  }
};
}  // namespace host
}  // namespace ibgpu

template <int SIDES>
void check(int rc, int step) {
  using namespace ibgpu::host;
  g_cell = rc;
  for (int pattern = 0; pattern < 16; ++pattern) {
    std::vector<uint8_t> sfl(NQ, 0);
    for (int k = 0, at = -2; at <= 2; ++at) {
      if (at == 0) continue;
      const int i = rc + at * step;
      if ((pattern >> k++ & 1) && i >= 0 && i < NQ) sfl[i] = ibgpu::CF_PRESENT;
    }
    Q4<double> lo, hi, c = {1, 1, 1, 1};
    cell_states<double, 0, NQ, SIDES>(nullptr, sfl.data(), c, rc, step, false, lo, hi);
  }
}

int main() {
  using namespace ibgpu::host;
  const int T = ibgpu::kTile;
  for (int step : {1, kReg})
    for (int ty = 0; ty < T; ++ty)
      for (int tx = 0; tx < T; ++tx) check<kLow | kHigh>((ty + kHalo) * kReg + tx + kHalo, step);
  // the edge warp: the cell after the last face of each row and column, and
  // the one before the first
  for (int e = 0; e < T; ++e)
    for (int x : {1, 0}) {
      const int step = x ? 1 : kReg;
      const int er = x ? (e + kHalo) * kReg + T + kHalo : (T + kHalo) * kReg + e + kHalo;
      check<kLow>(er, step);
      check<kHigh>(er - (T + 1) * step, step);
    }
  return g_bad != 0;
}
