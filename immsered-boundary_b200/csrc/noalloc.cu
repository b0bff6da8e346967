// ibgpu_step_periodic_noalloc: one time step of a single-level periodic
// grid without any device allocation.
//
// Who needs it: a caller that may not allocate device memory while it runs
// the solver — for instance a host application whose device memory belongs
// to another framework's pool (a multiphysics coupler that hands the solver
// buffers it owns), or a time loop that must not hit cudaMalloc/cudaFree
// because they synchronise the whole device.  Such a caller passes its own
// device buffers for the state in and out; every intermediate (the tiled
// state, the two stage buffers, the neighbour table and the step's
// diagnostics) lives in one file-scope __device__ array of fixed size, which
// each GPU that loads the library keeps until the process exits.
//
// Set-up: the first call on a device looks up the array's device address
// with cudaGetSymbolAddress and registers a static host page for the
// diagnostics (once per device, with that device current); make
// that first call before any stream capture.  All calls share the array and
// it keeps the last call's contents: calls that overlap on the GPU (two
// streams, two host threads) race and must be serialised by the caller.
#include <cstdint>
#include <cstring>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/ibgpu.h"
#include "cfl.cuh"
#include "dependent.cuh"
#include "host_internal.h"
#include "launchers.h"
#include "layout.h"

using namespace ibgpu;

namespace {

constexpr int kMaxCells = IBGPU_NOALLOC_MAX_CELLS;
constexpr int kMaxTiles = kMaxCells / kTileCells;

// byte layout of the scratch array (each part 256-byte aligned)
constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kOffDiag = 0;
constexpr size_t kOffNb = align256(kOffDiag + sizeof(DevDiag));
constexpr size_t kOffLevel = align256(kOffNb + sizeof(int32_t) * 9 * kMaxTiles);
constexpr size_t kOffUniform = align256(kOffLevel + sizeof(int32_t) * kMaxTiles);
constexpr size_t kOffDone = align256(kOffUniform + kMaxTiles);
constexpr size_t kOffTop = align256(kOffDone + sizeof(int));
constexpr size_t kOffFlags = align256(kOffTop + 2 * sizeof(unsigned long long) * kMaxTiles);
constexpr size_t kOffS0 = align256(kOffFlags + kMaxCells);
constexpr size_t kOffBuf = kOffS0 + sizeof(double) * kStateFields * kMaxCells;
constexpr size_t kScratchBytes = kOffBuf + sizeof(double) * 8 * kMaxCells;

static_assert(kMaxTiles <= kTileCells, "the last CTA reduces one tile per thread");

// zero at load; the count of finished CTAs in it returns to zero by itself
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

std::mutex g_mu;
void *g_scratch_addr[256] = {};

// Where the last kernel of a step leaves the diagnostics for the host: a
// static host page per device, registered (not allocated) on the first call,
// so that returning dt takes no copy through pageable memory.
struct alignas(4096) DiagPage {
  DevDiag d;
};
DiagPage g_diag_page[16];
DevDiag *g_diag_dev[16] = {};

__device__ __forceinline__ int64_t tiled_slot(int ix, int iy, int ntx) {
  return ((int64_t)(iy / kTile) * ntx + ix / kTile) * kTileCells + (iy % kTile) * kTile + ix % kTile;
}

// One CTA per tile: its entry of the periodic neighbour table of a row-major
// tile grid, all-leaf flags, and its cells from the caller's rows (row-major
// cells, FlowVariables layout) into the tiled SoA; with cfl also the tile's
// CFL bound and first failing cell.  The last CTA to finish sets the step's
// diagnostics and dt (NS_Solver::Comptdt) from the tiles'.  in1: null, or the
// input of a one-stage scheme's stage (rho, u, v, p, which the stage cannot
// read from the state it writes).  A small grid's
// step is launches and little else: this one stands for four (set-up, rows,
// CFL pass, dt): a step of 64 x 48 cells 74 -> 46 us, with the diagnostics
// returned through a mapped page instead of a pageable copy.
__global__ void __launch_bounds__(kTileCells)
    noalloc_load_kernel(const double *rows, int nx, int ntx, int nty, int32_t *nb, int32_t *lvl,
                        uint8_t *uniform, uint8_t *flags, double *s0, DevDiag *diag, int *done,
                        unsigned long long *top, double *in1, double dt, int cfl, CaseConst cc) {
  __shared__ unsigned long long sred[2 * (kTileCells / 32)];
  __shared__ int last;
  const int tile = blockIdx.x, tid = threadIdx.x;
  const int tx = tile % ntx, ty = tile / ntx;
  if (tid < 9) {
    const int x = (tx + tid % 3 - 1 + ntx) % ntx, y = (ty + tid / 3 - 1 + nty) % nty;
    nb[tile * 9 + tid] = y * ntx + x;
  }
  if (tid == 0) {
    lvl[tile] = 0;
    uniform[tile] = 1;
  }
  const int64_t s = (int64_t)tile * kTileCells + tid;
  flags[s] = CF_PRESENT | CF_NORMAL | CF_UPDATE | CF_PRIM | CF_RESNORM;
  const double *r =
      rows + 7 * ((int64_t)(ty * kTile + tid / kTile) * nx + tx * kTile + tid % kTile);
  const double u = r[1], v = r[2], T = r[5];
  s0[F_RHO * (int64_t)kMaxCells + s] = r[0];
  s0[F_U * (int64_t)kMaxCells + s] = u;
  s0[F_V * (int64_t)kMaxCells + s] = v;
  s0[F_P * (int64_t)kMaxCells + s] = r[4];
  s0[F_E * (int64_t)kMaxCells + s] = r[6];
  s0[F_T * (int64_t)kMaxCells + s] = T;
  if (in1) {
    in1[s] = r[0];
    in1[kMaxCells + s] = u;
    in1[2 * kMaxCells + s] = v;
    in1[3 * kMaxCells + s] = r[4];
  }
  const unsigned long long none = (unsigned long long)__double_as_longlong(10000.0);
  unsigned long long best = none, bad = ~0ull;
  // block minima of both words, valid in thread 0
  auto block_min = [&]() {
    best = warp_min_u64(best);
    bad = warp_min_u64(bad);
    if ((tid & 31) == 0) {
      sred[tid >> 5] = best;
      sred[kTileCells / 32 + (tid >> 5)] = bad;
    }
    __syncthreads();
    if (tid == 0)
      for (int w = 1; w < kTileCells / 32; ++w) {
        best = sred[w] < best ? sred[w] : best;
        bad = sred[kTileCells / 32 + w] < bad ? sred[kTileCells / 32 + w] : bad;
      }
    __syncthreads();
  };
  if (cfl) {
    const double d0 = cfl_cell_bound(T, u, v, cc.lev[0], cc);
    if (d0 < 0.0) bad = error_key(1, ERR_CFL_NEG_DT, (int)s);
    // as the CFL pass's atomic minimum of bit patterns: a negative bound (its
    // sign bit makes it large) or NaN leaves 10000
    const unsigned long long b0 = (unsigned long long)__double_as_longlong(d0);
    if (b0 < none) best = b0;
  }
  block_min();
  if (tid == 0) {
    top[2 * tile] = best;
    top[2 * tile + 1] = bad;
    __threadfence();
    last = atomicAdd(done, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  best = tid < (int)gridDim.x ? __ldcg(top + 2 * tid) : none;
  bad = tid < (int)gridDim.x ? __ldcg(top + 2 * tid + 1) : ~0ull;
  block_min();
  if (tid == 0) {
    const double cdt = __longlong_as_double((long long)best), cand = dt * cc.dt_ratio;
    diag->dt = !cfl ? dt : (cand < cdt) ? cand : cdt;
    diag->cfl_bits = best;
    for (int c = 0; c < 5; ++c) diag->res_bits[c] = 0ull;
    diag->err_key = bad;
    diag->cfl_next_bits = none;
    *done = 0;
  }
}

// tiled SoA -> caller rows
__global__ void noalloc_rows_out_kernel(const double *s0, int nx, int ny, double *rows,
                                        const DevDiag *diag, DevDiag *out, int *done) {
  dep_begin();
  dep_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *out = *diag;
    *done = 0;  // also after calls that a caller let overlap
  }
  const int64_t n = (int64_t)nx * ny;
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < n;
       c += (int64_t)gridDim.x * blockDim.x) {
    int ix = (int)(c % nx), iy = (int)(c / nx);
    int64_t s = tiled_slot(ix, iy, nx / kTile);
    double *r = rows + 7 * c;
    r[0] = s0[F_RHO * (int64_t)kMaxCells + s];
    r[1] = s0[F_U * (int64_t)kMaxCells + s];
    r[2] = s0[F_V * (int64_t)kMaxCells + s];
    r[3] = 0.0;
    r[4] = s0[F_P * (int64_t)kMaxCells + s];
    r[5] = s0[F_T * (int64_t)kMaxCells + s];
    r[6] = s0[F_E * (int64_t)kMaxCells + s];
  }
}

#define NA_CK(call)                                                       \
  do {                                                                    \
    cudaError_t e_ = (call);                                              \
    if (e_ != cudaSuccess) {                                              \
      set_last_error(std::string(#call) + ": " + cudaGetErrorString(e_)); \
      return IBGPU_E_CUDA;                                                \
    }                                                                     \
  } while (0)

int scratch_address(unsigned char **out, DevDiag **host, DevDiag **mapped) {
  int dev = 0;
  NA_CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) {
    set_last_error("device ordinal out of range");
    return IBGPU_E_ARG;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  if (!g_scratch_addr[dev]) {
    void *p = nullptr;
    NA_CK(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    if (dev < 16) {
      // left unmapped (the copy below serves) where a page cannot be pinned
      DevDiag *m = nullptr;
      if (cudaHostRegister(&g_diag_page[dev], sizeof(DiagPage), cudaHostRegisterMapped) == cudaSuccess &&
          cudaHostGetDevicePointer((void **)&m, &g_diag_page[dev], 0) == cudaSuccess)
        g_diag_dev[dev] = m;
      else
        cudaGetLastError();
    }
    g_scratch_addr[dev] = p;
  }
  *host = dev < 16 ? &g_diag_page[dev].d : nullptr;
  *mapped = dev < 16 ? g_diag_dev[dev] : nullptr;
  *out = (unsigned char *)g_scratch_addr[dev];
  return IBGPU_OK;
}

}  // namespace

extern "C" int ibgpu_step_periodic_noalloc(const ibgpu_case *cs, int ts, int nx, int ny,
                                           const double *d_rows_in, double *d_rows_out,
                                           double *dt, ibgpu_diag *diag, void *stream) {
  if (!cs || !dt || !d_rows_in || !d_rows_out || ts < 0) return IBGPU_E_ARG;
  int rc = validate_case(cs);
  if (rc) return rc;
  if (cs->nlevels != 1 || !cs->periodic_x || !cs->periodic_y || cs->viscous ||
      cs->domain_nx != nx || cs->domain_ny != ny || cs->march_step[0] != 1) {
    set_last_error("the allocation-free step takes one periodic inviscid level");
    return IBGPU_E_ARG;
  }
  if (nx <= 0 || ny <= 0 || nx % kTile || ny % kTile || (int64_t)nx * ny > kMaxCells) {
    set_last_error("grid must be a multiple of 16 per side and at most IBGPU_NOALLOC_MAX_CELLS cells");
    return IBGPU_E_ARG;
  }
  unsigned char *base = nullptr;
  DevDiag *h_page = nullptr, *m_page = nullptr;
  if ((rc = scratch_address(&base, &h_page, &m_page))) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  CaseConst cc;
  fill_case_const(cs, cc);

  DevDiag *d_diag = (DevDiag *)(base + kOffDiag);
  int32_t *d_nb = (int32_t *)(base + kOffNb);
  int32_t *d_lvl = (int32_t *)(base + kOffLevel);
  uint8_t *d_flags = base + kOffFlags;
  double *d_s0 = (double *)(base + kOffS0);
  double *d_buf = (double *)(base + kOffBuf);
  const int ntx = nx / kTile, nty = ny / kTile, ntiles = ntx * nty;
  const int64_t nslots = (int64_t)ntiles * kTileCells;

  const bool exact = cs->precision == IBGPU_FP64_EXACT;
  const bool mixed = cs->precision == IBGPU_MIXED;
  uint8_t *d_uniform = base + kOffUniform;
  int *d_done = (int *)(base + kOffDone);
  unsigned long long *d_top = (unsigned long long *)(base + kOffTop);
  launch_dep(false, st, ntiles, kTileCells, noalloc_load_kernel, d_rows_in, nx, ntx, nty, d_nb,
             d_lvl, d_uniform, d_flags, d_s0, d_diag, d_done, d_top,
             cs->nstages == 1 ? d_buf : (double *)nullptr, *dt,
             ts % cs->dt_var_step == 0 ? 1 : 0, cc);
  NA_CK(cudaGetLastError());

  StageArgs sa;
  std::memset(&sa, 0, sizeof(sa));
  sa.tile_nb = d_nb;
  sa.tile_level = d_lvl;
  sa.tile_uniform = d_uniform;
  sa.flags = d_flags;
  sa.tile_begin = 0;
  for (int f = 0; f < kStateFields; ++f) sa.s0[f] = d_s0 + (int64_t)f * kMaxCells;
  sa.vsd = nullptr;
  sa.nslots = nslots;
  sa.diag = d_diag;
  static const int map[4] = {F_RHO, F_U, F_V, F_P};
  for (int k = 0; k < cs->nstages; ++k) {
    const bool fin = k == cs->nstages - 1;
    for (int f = 0; f < 4; ++f) {
      // stage buffers (FP32 values in the mixed build, in the same regions)
      sa.v.sin[f] = (k == 0) ? (const void *)sa.s0[map[f]]
                             : (const void *)(d_buf + ((int64_t)(((k - 1) & 1) * 4 + f)) * kMaxCells);
      if (cs->nstages == 1) sa.v.sin[f] = d_buf + (int64_t)f * kMaxCells;  // the load's in1
      sa.v.sout[f] = fin ? nullptr : (void *)(d_buf + ((int64_t)((k & 1) * 4 + f)) * kMaxCells);
    }
    sa.v.tp = cs->tp[k];
    sa.phase = 2 + k;
    // the first stage follows the kernel that writes the tables a stage reads
    // before it waits: an ordinary launch
    if (exact) exact::launch_stage(sa, cc, ntiles, cs->limiter, false, fin, false, k, st, k > 0);
    else fast::launch_stage(sa, cc, ntiles, cs->limiter, false, fin, mixed, k, st, k > 0);
  }
  launch_dep(true, st, (nx * ny + 255) / 256, 256, noalloc_rows_out_kernel, d_s0, nx, ny,
             d_rows_out, d_diag, m_page ? m_page : d_diag, d_done);
  NA_CK(cudaGetLastError());

  DevDiag hd;
  if (!m_page) NA_CK(cudaMemcpyAsync(&hd, d_diag, sizeof(DevDiag), cudaMemcpyDeviceToHost, st));
  NA_CK(cudaStreamSynchronize(st));
  if (m_page) std::memcpy(&hd, h_page, sizeof(DevDiag));
  int abort_code = 0;
  if (hd.err_key != ~0ull) {
    int check = (int)((hd.err_key >> 32) & 0xff);  // one step: phases 1 (CFL), 2+k
    abort_code = check == ERR_CFL_NEG_DT ? 424 : check == ERR_NEG_T ? 37 : 523;
  }
  for (int c = 0; c < 5; ++c) {
    double v;
    std::memcpy(&v, &hd.res_bits[c], sizeof(double));
    if (v != v && !abort_code) abort_code = 268;
  }
  *dt = hd.dt;
  if (diag) {
    std::memset(diag, 0, sizeof(*diag));
    diag->dt = hd.dt;
    std::memcpy(&diag->cfl_dt, &hd.cfl_bits, sizeof(double));
    for (int c = 0; c < 5; ++c) std::memcpy(&diag->res_max[c], &hd.res_bits[c], sizeof(double));
    diag->abort_code = abort_code;
    diag->cells_marched = (int64_t)nx * ny;
    if (abort_code && abort_code != 268) {
      int slot = (int)(hd.err_key & 0xffffffffull);
      int tile = slot / kTileCells, local = slot % kTileCells;
      diag->abort_ix = (tile % ntx) * kTile + local % kTile;
      diag->abort_iy = (tile / ntx) * kTile + local / kTile;
    }
  }
  return abort_code ? IBGPU_E_ABORT : IBGPU_OK;
}
