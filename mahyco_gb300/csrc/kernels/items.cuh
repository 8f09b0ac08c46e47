// The batched launches' item loop, shared by the two schemes' kernels
// (vnr.cu, euc.cu).
#ifndef MAHYCO_GB300_ITEMS_CUH
#define MAHYCO_GB300_ITEMS_CUH

#include "../internal.h"

namespace hydro {

// The lanes of a warp whose item lies inside the mesh, for votes among them
// after the others have left.  Called by whole warps (the plain and batched
// launches have blocks of 128 threads that work on one tile).
__device__ __forceinline__ unsigned lanes_inside(bool in) { return __ballot_sync(0xffffffffu, in); }

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
// would run both.  Blocks of their own cover the four sides (the corners with
// the bottom and the top), each from a warp of its own, since the sides'
// conditions are different code; the others the inner nodes in tiles of kNodeBX x
// kNodeBY.  The sides' blocks are the grid's first rows, which start first (as
// its first columns they start among the others: 17.8 us against 17.1 at 801 x 41
// cells), unless the grid would then have more than the 65535 rows of blocks a
// launch takes (meshes of fewer than 34 cells across and more than 246 000 rows):
// there they are its first columns.
constexpr int kNodeBX = 32, kNodeBY = 4;
__host__ __device__ inline int side_warps(int n) { return (n + 31) / 32; }
struct SplitGrid {
  int rows, cols;  // rows / columns of blocks for the sides; one of them is 0
};
inline dim3 split_node_grid(int nx, int ny, SplitGrid* g) {
  const int gx = (nx - 1 + kNodeBX - 1) / kNodeBX, gy = (ny - 1 + kNodeBY - 1) / kNodeBY;
  const int warps = 2 * side_warps(nx + 1) + 2 * side_warps(ny - 1);
  const int blocks = (warps + kNodeBY - 1) / kNodeBY, rows = (blocks + gx - 1) / gx;
  if (gy + rows <= 65535) *g = {rows, 0};
  else *g = {0, (blocks + gy - 1) / gy};
  return dim3(gx + g->cols, gy + g->rows);
}
// What thread (tx, ty) of block (bx, by) of a grid of gx columns has: inner(i, j)
// for an inner node, edge(i, j) for a side's.
template <class Inner, class Edge>
__host__ __device__ __forceinline__ void split_node(int nx, int ny, SplitGrid g, int gx, int bx,
                                                    int by, int tx, int ty, const Inner& inner,
                                                    const Edge& edge) {
  if (by < g.rows || bx < g.cols) {
    const int wx = side_warps(nx + 1), wy = side_warps(ny - 1);
    int w = (by * (g.cols ? g.cols : gx) + bx) * kNodeBY + ty;  // one row of threads: a warp
    if (w < 2 * wx) {
      const bool top = w >= wx;
      const int j = (top ? w - wx : w) * 32 + tx;
      if (j <= nx) edge(top ? ny : 0, j);
      return;
    }
    w -= 2 * wx;
    if (w >= 2 * wy) return;
    const bool right = w >= wy;
    const int i = 1 + (right ? w - wy : w) * 32 + tx;
    if (i < ny) edge(i, right ? nx : 0);
    return;
  }
  const int i = 1 + (by - g.rows) * kNodeBY + ty, j = 1 + (bx - g.cols) * kNodeBX + tx;
  if (i < ny && j < nx) inner(i, j);
}
template <class F>
__device__ __forceinline__ void split_node_items(const RunView& v, SplitGrid g, const F& f) {
  if (!v.ctrl->active) return;
  split_node(
      v.nx, v.ny, g, gridDim.x, blockIdx.x, blockIdx.y, threadIdx.x, threadIdx.y,
      [&](int i, int j) { f.template node<true>(v, i, j); },
      [&](int i, int j) { f.edge_node(v, i, j); });
}

}  // namespace hydro

#endif  // MAHYCO_GB300_ITEMS_CUH
