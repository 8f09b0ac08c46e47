// The batched launches' item loop, shared by the two schemes' kernels
// (vnr.cu, euc.cu).
#ifndef MAHYCO_GB300_ITEMS_CUH
#define MAHYCO_GB300_ITEMS_CUH

#include "../internal.h"

namespace hydro {

// Batched launches: a persistent grid walks the tile table; every thread of
// a block works on the same tile (the block reductions of some phases rely
// on it).  The tile's run view is staged in shared memory by the whole
// block, so its fields are read where they are used instead of being held
// in registers for the whole tile.  scheme >= 0: the tiles of runs of the
// other scheme are skipped (a batch may hold both; the skip is uniform over
// the block).
template <class F>
__device__ __forceinline__ void batch_items(const BatchArgs& b, const F& f, int scheme = -1) {
  __shared__ RunView sv;
  constexpr int kWords = sizeof(RunView) / sizeof(unsigned long long);
  static_assert(sizeof(RunView) % sizeof(unsigned long long) == 0, "RunView size");
  const int n = *b.ntiles;
  const int tx = threadIdx.x & ((1 << b.tw_log2) - 1);
  const int ty = threadIdx.x >> b.tw_log2;
  const int th = kBatchThreads >> b.tw_log2;
  for (int t = blockIdx.x; t < n; t += gridDim.x) {
    const Tile T = b.tiles[t];
    const unsigned long long* src =
        reinterpret_cast<const unsigned long long*>(b.views + T.inst);
    unsigned long long* dst = reinterpret_cast<unsigned long long*>(&sv);
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    if (sv.ctrl->active && (scheme < 0 || sv.scheme == scheme))
      for (int r = 0; r < b.rows; ++r) f(sv, T.i0 + ty + r * th, T.j0 + tx);
    __syncthreads();
  }
}

// Plain launches over the nodes, the boundary's apart: its nodes take a longer
// path (fewer cells, the boundary conditions), and a warp with one of them
// would run both.  The grid's first rows of blocks cover the four sides (the
// corners with the bottom and the top), each from a warp of its own, since the
// sides' conditions are different code; the others the inner nodes in tiles of
// kNodeBX x kNodeBY.
constexpr int kNodeBX = 32, kNodeBY = 4;
__host__ __device__ inline int side_warps(int n) { return (n + 31) / 32; }
__host__ __device__ inline int perimeter_rows(const RunView& v, int gx) {
  const int warps = 2 * side_warps(v.nx + 1) + 2 * side_warps(v.ny - 1);
  return ((warps + kNodeBY - 1) / kNodeBY + gx - 1) / gx;
}
inline dim3 split_node_grid(const RunView& v) {
  const int gx = (v.nx - 1 + kNodeBX - 1) / kNodeBX, gy = (v.ny - 1 + kNodeBY - 1) / kNodeBY;
  return dim3(gx, gy + perimeter_rows(v, gx));
}
template <class F>
__device__ __forceinline__ void split_node_items(const RunView& v, const F& f) {
  if (!v.ctrl->active) return;
  const int rows = perimeter_rows(v, gridDim.x), by = blockIdx.y;
  if (by < rows) {
    const int wx = side_warps(v.nx + 1), wy = side_warps(v.ny - 1);
    int w = (by * gridDim.x + blockIdx.x) * kNodeBY + threadIdx.y;  // one row of threads: a warp
    if (w < 2 * wx) {
      const bool top = w >= wx;
      const int j = (top ? w - wx : w) * 32 + threadIdx.x;
      if (j <= v.nx) f.edge_node(v, top ? v.ny : 0, j);
      return;
    }
    w -= 2 * wx;
    if (w >= 2 * wy) return;
    const bool right = w >= wy;
    const int i = 1 + (right ? w - wy : w) * 32 + threadIdx.x;
    if (i < v.ny) f.edge_node(v, i, right ? v.nx : 0);
    return;
  }
  const int i = 1 + (by - rows) * kNodeBY + threadIdx.y, j = 1 + blockIdx.x * kNodeBX + threadIdx.x;
  if (i < v.ny && j < v.nx) f.template node<true>(v, i, j);
}

}  // namespace hydro

#endif  // MAHYCO_GB300_ITEMS_CUH
