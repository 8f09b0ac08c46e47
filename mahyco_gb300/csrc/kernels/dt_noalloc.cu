// CFL time step of a VNR state that lives in the caller's device memory,
// computed without allocating anything.
//
// Who needs it: code that owns every byte of device memory through its own
// pool (a serving process, a host solver that embeds one hydro step in its
// own time loop) or that runs while another library holds the device
// allocator, and therefore may not call cudaMalloc / cudaFree.  Those
// callers pass their own buffers for the inputs and the output; the only
// other memory the computation needs -- one partial minimum per thread
// block -- is the file-scope device array below, reserved when the library
// is loaded.
//
// The value is the one a run computes at the start of its next cycle
// (Vnr::computeDeltaT, vnr_remap/VnrRemap.cc:14-50, with the remap on:
// cfl 0.05, dt <= 1.05 * dt_n): min over cells of
// 0.05*sqrt(sum of the cell's initial sub-volumes) / (sum_p 0.25*|u_p| + c).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../internal.h"
#include "scheme_math.cuh"

namespace hydro {

// Largest state accepted: 1,048,576 cells.  A warp takes units of R x 31 cells
// (R rows, 1 to 8 by the mesh, DtGrid) and at most kDtMaxBlocks blocks are
// launched, each with one slot of the scratch (32 KiB).
constexpr long long kDtMaxCells = 1048576;
constexpr int kDtMaxBlocks = 4096;
constexpr int kDtMaxRows = 8;   // most rows of cells of a unit
constexpr int kDtCols = 31;     // columns of cells: 32 node columns a warp
constexpr int kDtMaxWarps = 16; // most warps of a block
constexpr int kDtSms = 152;     // SMs of a GB300

// One ordered-int partial minimum per block.  Every call overwrites the
// slots of the blocks it launches before the final pass reads them, so
// nothing has to be cleared between calls; two calls that overlap on the GPU
// (different streams, or the same scratch in flight) race on these slots.
static __device__ __align__(256) unsigned long long g_dt_scratch[kDtMaxBlocks];

namespace {

// Initial sub-volume sum of one cell (Vnr::initCellPos + initSubVol,
// vnr_remap/Init.cc:400-429, 495-511) from the Cartesian node coordinates
// dx*j, dy*i, with the reference's operation order.  On that mesh every
// coordinate of the four sub-volumes is a value of the column (x0, x1, their
// middle, the centre's) or of the row, so the 32 products of the reference's
// cross products are 18 different ones.
__device__ double initial_volume_sum(int i, int j, double dx, double dy) {
  const double x0 = dx * (double)j, x1 = dx * (double)(j + 1);
  const double y0 = dy * (double)i, y1 = dy * (double)(i + 1);
  // the cell's centre: (((0 + a) + b) + c) + d in node order, times 0.25
  const double xc = quarter(((plus_zero(x0) + x1) + x1) + x0);
  const double yc = quarter(((plus_zero(y0) + y0) + y1) + y1);
  // side middles: of two different nodes, and of two nodes of one coordinate
  const double xm = half(x1 + x0), x0m = half(x0 + x0), x1m = half(x1 + x1);
  const double ym = half(y1 + y0), y0m = half(y0 + y0), y1m = half(y1 + y1);
  const double xcym = xc * ym, xmyc = xm * yc;
  const double ycx0 = yc * x0m, ycx1 = yc * x1m, xcy0 = xc * y0m, xcy1 = xc * y1m;
  const double x0ym = x0 * ym, x1ym = x1 * ym, xmy0 = xm * y0, xmy1 = xm * y1;
  auto corner = [](double c12, double c23, double c34, double c41) {
    return half(((c12 + c23) + c34) + c41);
  };
  double r = plus_zero(corner(xcym - ycx0, x0m * y0 - x0ym, x0 * y0m - xmy0, xmyc - xcy0));
  r = r + corner(xcy0 - xmyc, xmy0 - y0m * x1, x1ym - y0 * x1m, ycx1 - xcym);
  r = r + corner(xcym - ycx1, x1m * y1 - x1ym, x1 * y1m - xmy1, xmyc - xcy1);
  r = r + corner(xcy1 - xmyc, xmy1 - y1m * x0, x0ym - y1 * x0m, ycx0 - xcym);
  return r;
}

// The cell's candidate, 0.05 sqrt(V) / (sum of the four nodes' 0.25 |u| +
// c), in the reference's operation order.
__device__ __noinline__ double exact_candidate(int nx, int i, int j, double dx, double dy,
                                               const double* u, const double* v,
                                               const double* c) {
  const long long n0 = (long long)i * (nx + 1) + j;
  const long long nd[4] = {n0, n0 + 1, n0 + nx + 2, n0 + nx + 1};
  double s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double a = u[nd[k]], b = v[nd[k]];
    s[k] = quarter(sqrt_ip(a * a + b * b));
  }
  const double uc = ((s[0] + s[1]) + s[2]) + s[3];  // 0.0 + s[0] = s[0] (not -0)
  const double cflsq = 0.05 * sqrt_ip(initial_volume_sum(i, j, dx, dy));
  return div_ip(cflsq, uc + c[(long long)i * nx + j]);
}

// FP32 value of a double's upper word (its sign, exponent and upper 20
// significand bits: a relative error below 2^-20); exponents outside
// [lo, 1083] (below 2^61) come back as 0 with `out` set.
__device__ __forceinline__ float upper_float(unsigned hi, unsigned lo, bool& out) {
  const unsigned e = (hi >> 20) & 0x7ffu;
  out = e - lo > 1083u - lo;
  return out ? 0.0f : __uint_as_float(((hi & 0x7fffffffu) - (896u << 20)) << 3);
}

// The minimum over cells, by a filter.  Evaluated for every cell the
// candidate costs about 150 FP64 instructions, and GB300's FP64 pipe takes
// 1.6 us per instruction and million cells (315 us at 1024 x 1000).  All
// cells of the mesh have the volume dx dy up to rounding (below 1e-8
// relative: at most 2^20 cells), so the candidates are ordered by the
// denominator sum 0.25 |u| + c up to that: it is formed in FP32 from the
// upper words (relative error below 1e-5), and the candidate itself only in
// the cells within kDtMargin of their block's largest denominator, at least
// one per block.  A cell whose sound speed is outside [2^-30, 2^61) or
// negative, or with a node velocity component of 2^61 or more (NaN and
// infinities among them), always forms it; components below 2^-126 count as
// zero beside such a sound speed.  `all`: every cell forms it (cell sizes
// for which the volumes' relative error has no such bound).
//
// The cells that form it go to a list of the block, from which all its threads
// take them in turn: where the denominators tie (a mesh at rest, a uniform
// flow) every cell is in it, and the FP64 pipe bounds the call as it does
// without a filter.  So a block has as many cells as an SM's share of the
// mesh (dt_grid).
//
// A warp takes R x 31 cells: 32 node columns, one per lane, the right
// neighbour's speed by shuffle, the loads of all its rows issued before the
// first use.  Calls back to back (GB300), every cell's candidate formed ->
// this: random fields 64 x 48 cells 18.5 -> 10.3 us, 200 x 200 30.7 -> 12.2,
// 1024 x 1000 311 -> 16.4; at rest 20.3 -> 10.3, 30.8 -> 16.4, 326 -> 197.
constexpr float kDtMargin = 1.0f - 1e-4f;

template <int R>
__device__ __forceinline__ unsigned long long block_min_candidate(
    int nx, int ny, double dx, double dy, const double* __restrict__ u,
    const double* __restrict__ v, const double* __restrict__ c, bool all) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ncol = (nx + kDtCols - 1) / kDtCols, nrow = (ny + R - 1) / R;
  const int units = ncol * nrow, nw = blockDim.x >> 5;
  const unsigned* uh = reinterpret_cast<const unsigned*>(u) + 1;
  const unsigned* vh = reinterpret_cast<const unsigned*>(v) + 1;
  const unsigned* ch = reinterpret_cast<const unsigned*>(c) + 1;
  __shared__ float warp_max[kDtMaxWarps];
  // cells that form their candidate: (warp, row, lane) of this pass
  __shared__ unsigned short list[kDtMaxWarps * R * 32];
  __shared__ int listed;
  unsigned long long best = ~0ull;
  float seen = 0.0f;  // largest denominator of the block so far
  // the trip count is the block's, not the warp's (barriers inside)
  for (int base = blockIdx.x * nw; base < units; base += gridDim.x * nw) {
    const int unit = base + warp;
    const int i0 = (unit / ncol) * R, j0 = (unit % ncol) * kDtCols, j = j0 + lane;
    const bool in = unit < units;
    float s[R + 1], D[R];
    unsigned hu[R + 1], hv[R + 1], hc[R];
#pragma unroll
    for (int r = 0; r <= R; ++r) {
      const bool node = in && j <= nx && i0 + r <= ny;
      const long long p = (long long)(i0 + r) * (nx + 1) + j;
      hu[r] = node ? __ldg(uh + 2 * p) : 0u;
      hv[r] = node ? __ldg(vh + 2 * p) : 0u;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool cell = in && lane < kDtCols && j < nx && i0 + r < ny;
      hc[r] = cell ? __ldg(ch + 2 * ((long long)(i0 + r) * nx + j)) : 0u;
    }
    unsigned odd = 0;  // rows of nodes with a component of 2^61 or more
#pragma unroll
    for (int r = 0; r <= R; ++r) {
      bool ou, ov;
      const float a = upper_float(hu[r], 897u, ou), b = upper_float(hv[r], 897u, ov);
      // out of range and not small
      const bool big = (ou && (hu[r] & 0x7ff00000u) > (1083u << 20)) ||
                       (ov && (hv[r] & 0x7ff00000u) > (1083u << 20));
      odd |= (big ? 1u : 0u) << r;
      float q;
      asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(a * a + b * b));
      s[r] = q;
    }
    odd |= __shfl_down_sync(0xffffffffu, odd, 1);
    odd |= odd >> 1;  // a cell's rows are r and r + 1
    unsigned take = 0;
    float top = 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float t = s[r] + s[r + 1];
      const float t1 = __shfl_down_sync(0xffffffffu, t, 1);
      const bool cell = in && lane < kDtCols && j < nx && i0 + r < ny;
      bool oc;
      const float fc = upper_float(hc[r], 993u, oc);
      D[r] = cell ? 0.25f * (t + t1) + fc : 0.0f;
      if (cell && (all || oc || (hc[r] >> 31) || ((odd >> r) & 1u))) take |= 1u << r;
      else top = fmaxf(top, D[r]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (lane == 0) warp_max[warp] = top;
    if (threadIdx.x == 0) listed = 0;
    __syncthreads();
    for (int w = 0; w < nw; ++w) seen = fmaxf(seen, warp_max[w]);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (D[r] > 0.0f && D[r] >= seen * kDtMargin) take |= 1u << r;
      const unsigned m = __ballot_sync(0xffffffffu, (take >> r) & 1u);
      if (m == 0) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&listed, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      if ((take >> r) & 1u)
        list[at + __popc(m & ((1u << lane) - 1u))] = (unsigned short)((warp * R + r) * 32 + lane);
    }
    __syncthreads();
    const int n = listed;
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
      const int e = list[t], w = base + (e >> 5) / R, r = (e >> 5) % R;
      const double d = exact_candidate(nx, (w / ncol) * R + r, (w % ncol) * kDtCols + (e & 31), dx,
                                       dy, u, v, c);
      if (!is_nan(d)) best = ord_bits(d) < best ? ord_bits(d) : best;
    }
    __syncthreads();  // the list, its count and the maxima are written anew
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
    best = t < best ? t : best;
  }
  __shared__ unsigned long long warp_min[kDtMaxWarps];
  if (lane == 0) warp_min[warp] = best;
  __syncthreads();
  for (int w = 0; w < nw; ++w) best = warp_min[w] < best ? warp_min[w] : best;
  return best;  // thread 0's (every thread's) block minimum
}

__device__ __forceinline__ double step_of(unsigned long long m, double dt_n) {
  // no valid candidate: the reference's reduction starts at DBL_MAX
  const double red = (m == ~0ull) ? 1.7976931348623157e308 : from_ord(m);
  return smin(red, 1.05 * dt_n);
}

template <int R>
__global__ void __launch_bounds__(kDtMaxWarps * 32)
k_dt_partial(int nx, int ny, double dx, double dy, const double* u,
             const double* v, const double* c, bool all, unsigned long long* scratch) {
  // the final pass may become resident now; it waits for this grid's end
  asm volatile("griddepcontrol.launch_dependents;");
  const unsigned long long m = block_min_candidate<R>(nx, ny, dx, dy, u, v, c, all);
  if (threadIdx.x == 0) scratch[blockIdx.x] = m;
}

// Rows of a warp's units, and the launch: blocks of equal size, one per SM, or
// k per SM where 16 warps of 8 rows do not hold an SM's share of the mesh.
// The fewest rows with which one block per SM does: where all denominators tie
// the time is that of the SM with the most cells (FP64 pipe), where one cell
// decides it hardly depends on the rows.  (Blocks of 8 warps of 8 rows at every
// size: at rest 129 us at 64 x 48 cells, 65 at 200 x 200, 227 at 1024 x 1000.)
struct DtGrid {
  int rows, warps, blocks;
};
DtGrid dt_grid(int nx, int ny) {
  const long long ncol = (nx + kDtCols - 1) / kDtCols;
  DtGrid g{1, 0, 0};
  auto units = [&] { return ncol * ((ny + g.rows - 1) / g.rows); };
  while (g.rows < kDtMaxRows && units() > kDtSms * kDtMaxWarps) g.rows *= 2;
  const long long n = units(), most = kDtSms * kDtMaxWarps;
  const long long slots = kDtSms * ((n + most - 1) / most);  // blocks of at most 16 warps
  g.warps = (int)((n + slots - 1) / slots);
  g.blocks = (int)std::min<long long>((n + g.warps - 1) / g.warps, kDtMaxBlocks);
  return g;
}

constexpr int kDtBlock = 256;
__global__ void __launch_bounds__(kDtBlock)
k_dt_final(int nblocks, double dt_n, const unsigned long long* scratch,
           double* dt_out) {
  // launched while the partial pass runs: its minima are there after this
  asm volatile("griddepcontrol.wait;" ::: "memory");
  unsigned long long best = ~0ull;
  for (int b = threadIdx.x; b < nblocks; b += kDtBlock) {
    const unsigned long long t = __ldcg(scratch + b);
    best = t < best ? t : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
    best = t < best ? t : best;
  }
  __shared__ unsigned long long warp_min[kDtBlock / 32];
  if ((threadIdx.x & 31) == 0) warp_min[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long m = warp_min[0];
    for (int w = 1; w < kDtBlock / 32; ++w) m = warp_min[w] < m ? warp_min[w] : m;
    *dt_out = step_of(m, dt_n);
  }
}

// Device address of g_dt_scratch, looked up once per device (with that
// device current) on the first call made on it, in the device's primary
// context (the CUDA runtime's); it stays valid until that context is reset,
// after which the function must not be called (documented in the header).
constexpr int kMaxDevices = 64;
unsigned long long* g_scratch_ptr[kMaxDevices];
std::mutex g_scratch_mu;

}  // namespace

}  // namespace hydro

using namespace hydro;

extern "C" int hydro_vnr_dt_noalloc(int nx, int ny, double dx, double dy,
                                    const double* d_u, const double* d_v,
                                    const double* d_c, double dt_n,
                                    double* d_dt_out, void* stream) {
  if (!d_u || !d_v || !d_c || !d_dt_out)
    return fail(-1, "hydro_vnr_dt_noalloc: null device pointer");
  if (nx < 2 || ny < 2) return fail(-2, "hydro_vnr_dt_noalloc: nx and ny must be >= 2");
  const long long ncells = (long long)nx * ny;
  if (ncells > kDtMaxCells)
    return fail(-3, "hydro_vnr_dt_noalloc: " + std::to_string(ncells) +
                        " cells exceed the fixed scratch limit of " +
                        std::to_string(kDtMaxCells) +
                        " cells");
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(-4, "hydro_vnr_dt_noalloc: no usable current device");
  unsigned long long* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_ptr[dev]) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_dt_scratch);
      if (e != cudaSuccess)
        return fail(-5, std::string("hydro_vnr_dt_noalloc: cudaGetSymbolAddress: ") +
                            cudaGetErrorString(e));
      g_scratch_ptr[dev] = static_cast<unsigned long long*>(p);
    }
    scratch = g_scratch_ptr[dev];
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the volumes' relative error is bounded where no product of coordinates
  // leaves the double range; other cell sizes take every cell exactly
  const double w = std::fabs(dx * nx), h = std::fabs(dy * ny);
  auto plain = [](double x) { return x > 1e-70 && x < 1e70; };
  const bool all = !(dx > 0.0 && dy > 0.0 && plain(dx) && plain(dy) && plain(w) && plain(h));
  const DtGrid g = dt_grid(nx, ny);
  auto partial = g.rows == 1 ? k_dt_partial<1> : g.rows == 2 ? k_dt_partial<2>
               : g.rows == 4 ? k_dt_partial<4> : k_dt_partial<8>;
  partial<<<g.blocks, g.warps * 32, 0, s>>>(nx, ny, dx, dy, d_u, d_v, d_c, all, scratch);
  // the final pass is launched ahead of the partial one's end
  // (programmatic stream serialization)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(kDtBlock);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k_dt_final, g.blocks, dt_n,
                         static_cast<const unsigned long long*>(scratch), d_dt_out);
  if (e != cudaSuccess)
    return fail(-6, std::string("hydro_vnr_dt_noalloc: launch: ") + cudaGetErrorString(e));
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return fail(-6, std::string("hydro_vnr_dt_noalloc: launch: ") + cudaGetErrorString(e));
  return 0;
}
