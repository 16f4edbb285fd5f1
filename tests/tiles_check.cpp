// Host check of csrc/tiles.h and csrc/fftplan.h: the tiles of the FP64 kernels cover the box and fit the shared memory
// that needs no raised limit, and the sizes that the sources name have the tiles and FFT steps they name.
#include <cstdio>
#include <initializer_list>
#include <vector>

#include "fftplan.h"
#include "tiles.h"

int main() {
  int bad = 0;
  size_t most = 0;
  for (int N = 8; N <= 1024; ++N) {
    int m = N;
    for (int p : {2, 3, 5})
      while (m % p == 0) m /= p;
    if (m != 1) continue;
    const ttsh::TileDim d = ttsh::pick_tile(N);
    if (d.tx < 1 || d.threads() > ttsh::MAXT || d.tx * d.nx < N || d.ty * d.ny < N) {
      std::printf("N=%d: tile %d x %d, %d x %d of them\n", N, d.tx, d.ty, d.nx, d.ny);
      ++bad;
    }
    for (size_t v : {ttsh::stage1_values(d), ttsh::stage2_values(d), ttsh::div_values(d), ttsh::correct_values(d), ttsh::stats_values(d)})
      if (v * sizeof(double) > most) most = v * sizeof(double);
    // pass z wraps each point once: the tiles' halo may not reach two periods away
    if (d.tx * d.nx + 1 >= 2 * N || d.ty * d.ny + 1 >= 2 * N) {
      std::printf("N=%d: tiles reach too far\n", N);
      ++bad;
    }
  }
  if (most > 48 * 1024) {
    std::printf("shared memory %zu\n", most);
    ++bad;
  }
  const struct { int N, tx, ty; } tiles[] = {{48, 16, 16}, {64, 16, 16}, {128, 16, 16}, {256, 16, 16}, {100, 10, 25}, {72, 8, 24}};
  for (const auto& t : tiles) {
    const ttsh::TileDim d = ttsh::pick_tile(t.N);
    if (d.tx != t.tx || d.ty != t.ty) {
      std::printf("N=%d: tile %d x %d\n", t.N, d.tx, d.ty);
      ++bad;
    }
  }
  const struct { int N; std::vector<int> r; } steps[] = {{100, {10, 10}}, {320, {10, 8, 4}}};
  for (const auto& t : steps) {
    const ttsh::fftplan::Steps s = ttsh::fftplan::default_steps<double>(t.N);
    if (std::vector<int>(s.a, s.a + s.n) != t.r) {
      std::printf("N=%d: %d steps, first %d\n", t.N, s.n, s.a[0]);
      ++bad;
    }
  }
  std::printf("%s\n", bad ? "failed" : "ok");
  return bad != 0;
}
