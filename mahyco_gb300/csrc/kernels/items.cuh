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
// would run both.  The grid's first columns of blocks cover the four sides
// (the corners with the bottom and the top), each from a warp of its own, since
// the sides' conditions are different code; the others the inner nodes in tiles
// of kNodeBX x kNodeBY.  Columns, because a grid has at most 65535 rows of
// blocks: the sides take none of them, so a mesh may have as many rows of cells
// as the cells' own launches hold.
constexpr int kNodeBX = 32, kNodeBY = 4;
__host__ __device__ inline int side_warps(int n) { return (n + 31) / 32; }
inline int node_rows(int ny) { return (ny - 1 + kNodeBY - 1) / kNodeBY; }
inline int perimeter_cols(int nx, int ny) {
  const int warps = 2 * side_warps(nx + 1) + 2 * side_warps(ny - 1), gy = node_rows(ny);
  return ((warps + kNodeBY - 1) / kNodeBY + gy - 1) / gy;
}
inline dim3 split_node_grid(int nx, int ny) {
  return dim3(perimeter_cols(nx, ny) + (nx - 1 + kNodeBX - 1) / kNodeBX, node_rows(ny));
}
// The node of thread (tx, ty) of block (bx, by); a side's node or an inner one.
// cols: perimeter_cols (from the host: its division would lengthen every
// thread's chain).
struct SplitNode {
  int i, j;
  bool edge, inner;
};
__host__ __device__ inline SplitNode split_node_at(int nx, int ny, int cols, int bx, int by, int tx,
                                                   int ty) {
  if (bx >= cols) {
    const int i = 1 + by * kNodeBY + ty, j = 1 + (bx - cols) * kNodeBX + tx;
    return {i, j, false, i < ny && j < nx};
  }
  const int wx = side_warps(nx + 1), wy = side_warps(ny - 1);
  int w = (by * cols + bx) * kNodeBY + ty;  // one row of threads: a warp
  if (w < 2 * wx) {
    const bool top = w >= wx;
    const int j = (top ? w - wx : w) * 32 + tx;
    return {top ? ny : 0, j, j <= nx, false};
  }
  w -= 2 * wx;
  const bool right = w >= wy;
  const int i = 1 + (right ? w - wy : w) * 32 + tx;
  return {i, right ? nx : 0, w < 2 * wy && i < ny, false};
}
template <class F>
__device__ __forceinline__ void split_node_items(const RunView& v, int cols, const F& f) {
  if (!v.ctrl->active) return;
  const SplitNode n =
      split_node_at(v.nx, v.ny, cols, blockIdx.x, blockIdx.y, threadIdx.x, threadIdx.y);
  if (n.inner) f.template node<true>(v, n.i, n.j);
  else if (n.edge) f.edge_node(v, n.i, n.j);
}

}  // namespace hydro

#endif  // MAHYCO_GB300_ITEMS_CUH
