// Every node of a mesh is visited once by the node launches' split grid, a
// side's node as one and an inner one as one, and the grid is one that can be
// launched.  Prints the number of meshes checked and of faulty ones.
#include <cstdio>
#include <vector>

#include "kernels/items.cuh"

namespace {
bool check(int nx, int ny) {
  hydro::SplitGrid sg;
  const dim3 g = hydro::split_node_grid(nx, ny, &sg);
  if (g.x < 1 || g.y < 1 || g.y > 65535u) return false;
  std::vector<unsigned char> seen((size_t)(nx + 1) * (ny + 1), 0);
  bool ok = true;
  for (unsigned by = 0; by < g.y; ++by)
    for (unsigned bx = 0; bx < g.x; ++bx)
      for (int ty = 0; ty < hydro::kNodeBY; ++ty)
        for (int tx = 0; tx < hydro::kNodeBX; ++tx) {
          auto visit = [&](int i, int j, bool edge) {
            const bool inside = i >= 0 && i <= ny && j >= 0 && j <= nx;
            const bool side = i == 0 || i == ny || j == 0 || j == nx;
            ok = ok && inside && side == edge && !seen[(size_t)i * (nx + 1) + j]++;
          };
          hydro::split_node(
              nx, ny, sg, (int)g.x, (int)bx, (int)by, tx, ty,
              [&](int i, int j) { visit(i, j, false); }, [&](int i, int j) { visit(i, j, true); });
        }
  for (unsigned char s : seen)
    ok = ok && s == 1;
  return ok;
}
}  // namespace

int main() {
  const int sizes[] = {2, 3, 4, 5, 6, 30, 31, 32, 33, 34, 63, 64, 65, 97, 128, 129, 301};
  int n = 0, bad = 0;
  for (int nx : sizes)
    for (int ny : sizes) ++n, bad += !check(nx, ny);
  // long thin meshes, to the most rows that the cells' and nodes' grids hold
  for (int nx : {2, 8, 33, 34, 100})
    for (int ny : {16383, 246700, 246800, 262139}) ++n, bad += !check(nx, ny);
  for (int ny : {2, 5, 6}) ++n, bad += !check(1000003, ny);
  std::printf("%d %d\n", n, bad);
  return bad != 0;
}
