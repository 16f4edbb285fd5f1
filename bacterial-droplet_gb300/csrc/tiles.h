// tiles.h — the tile of a z-plane that a CTA of the FP64 kernels (plain64.cu) computes and the shared memory the
// kernels take for it, in a form a host-side check shares.
#pragma once
#include <stddef.h>

namespace ttsh {

constexpr int MAXT = 256;  // threads (sites of a tile) at most

struct TileDim {
  int tx = 0, ty = 0, nx = 0, ny = 0;  // columns, rows; tiles per row and column of a plane
  int threads() const { return (tx * ty + 31) / 32 * 32; }
  size_t np() const { return (size_t)(tx + 2) * (ty + 2); }  // points of pass z and of pass x
  size_t px() const { return (size_t)tx * (ty + 2); }
};

// The tile of size N: rows of the box in nx equal parts, columns in ny, such that the FP64
// instructions per plane, counted in whole warps (3 per point of pass z, 6 of pass x, 25 of pass y
// and the pointwise terms), are fewest: 16 x 16 at N = 48, 64, 128 and 256, 10 x 25 at N = 100 (32-column
// tiles would leave 22 % of the lanes outside the box), 8 x 24 at N = 72; among tiles of one cost the widest.
// stage1 + stage2 + div + correct, us, this / a wider tile: 64^3 269 / 32 x 8 273, 256^3 14336 / 14540, 4 x 100^3 3547 /
// 25 x 10 3586, 8 x 48^3 797 / 24 x 8 830, 2 x 72^3 690 / 24 x 8 702.
inline TileDim pick_tile(int N) {
  TileDim best;
  long cost = 0;
  for (int nx = 1; nx <= N; ++nx) {
    const int tx = (N + nx - 1) / nx;
    if (tx > 64) continue;
    if (tx < 8 && tx < N) break;
    for (int ny = 1; ny <= N; ++ny) {
      const int ty = (N + ny - 1) / ny;
      if (tx * ty > MAXT) continue;
      if (ty < 4 && ty < N) break;
      auto warps = [](int points) { return (points + 31) / 32; };
      const long c = (long)nx * ny * (3 * warps((tx + 2) * (ty + 2)) + 6 * warps(tx * (ty + 2)) + 25 * warps(tx * ty));
      if (!best.tx || c < cost) {
        best.tx = tx;
        best.ty = ty;
        best.nx = nx;
        best.ny = ny;
        cost = c;
      }
    }
  }
  return best;
}

// Shared-memory values (FP64) of each kernel for a tile: below the 48 KB that a launch may take without a
// raised limit, at every size the library takes (checked by the tests).
inline size_t stage1_values(const TileDim& d) { return 2 * 4 * (d.np() + d.px()); }  // two fields at a time
inline size_t stage2_values(const TileDim& d) { return 9 * d.np() + 6 * d.px(); }    // the divergences; the Laplacians take less
inline size_t div_values(const TileDim& d) { return 6 * d.np() + 2 * d.px(); }
inline size_t correct_values(const TileDim& d) { return 4 * (d.np() + d.px()); }
inline size_t stats_values(const TileDim& d) { return 3 * d.np() + d.px(); }

}  // namespace ttsh
