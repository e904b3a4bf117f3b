// Instantiations of the tcgen05 evaluation kernels (umma.cuh, umma_rows.cuh): f32 meshes and split precision.
#include <algorithm>
#include <numeric>

#include "eval_launch.cuh"
#include "umma.cuh"
#include "umma_rows.cuh"

namespace tlg {

constexpr int kMaxItemsPerTile = kUmmaMaxGroups;

// Work items: with T tiles on a grid of C resident CTAs, each tile's n chunks go in G groups
// (G <= 8) minimising ceil(T G / C) (ceil(n / G) + 10): the rounds of items times an item's
// chunks plus its start (the gather and the first chunk's copy and MMAs, not overlapped with an
// epilogue: about ten chunks in GB300 timings of P4-P6 tetrahedra), so that a few tiles more than
// CTAs do not leave most SMs idle for a second round of whole tiles.
cudaError_t launch_umma(bool split, const UmmaArgs& args, size_t smem, cudaStream_t s) {
  auto kern = split ? umma_eval_kernel<true> : umma_eval_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  UmmaArgs a = args;
  const int64_t tiles = (a.padded + kUmmaCells - 1) / kUmmaCells;
  const int64_t ctas = persistent_grid(kern, smem, tiles * kMaxItemsPerTile * kUmmaThreads, kUmmaThreads);
  int64_t best = -1;
  for (int g = 1; g <= kUmmaMaxGroups && g <= a.chunks; ++g) {
    const int64_t per = (a.chunks + g - 1) / g;
    const int64_t cost = ((tiles * g + ctas - 1) / ctas) * (per + 10);
    if (best < 0 || cost < best) {
      best = cost;
      a.groups = g;
      a.per_group = (int)per;
    }
  }
  const int64_t grid = std::min<int64_t>(ctas, tiles * a.groups);
  kern<<<(unsigned)std::max<int64_t>(grid, 1), kUmmaThreads, smem, s>>>(a);
  return cudaGetLastError();
}

// The kernel cuts the (tile, chunk) pairs, in tile order, into equal runs, one per CTA (one CTA fits an
// SM), or with `unit` a tile's chunks into runs of whole tiles. A run costs its chunks and, for every tile that it
// touches, a start (the gather and the first MMAs) of six to eight chunks: P5 tetrahedra on an f32 mesh take
// 2.5 us a chunk and 15 us a start. So runs are equal over every SM, unless whole tiles, or whole parts of a tile
// on fewer SMs, cost less: of T tiles of n chunks on C SMs, ceil(T / C) (n + 8) where T > C, ceil(n / floor(C /
// T)) + 8 else, against r + 8 t, r = ceil(T n / C), t the most tiles that a run touches: ceil((r + n - g) / n), its
// starts multiples of g = gcd(r, n) in a tile where the runs are exactly equal, else g = 1. GB300, P4 tetrahedra
// at 125 points on an f32 mesh, us, equal runs / whole tiles: 228 tiles (r = 1.5 n) 70 / 82, 290 93 / 86, 380 (2.5 n)
// 113 / 124, 704 213 / 208; split precision 290 tiles 123 / 106, 704 276 / 258; 24 tiles, equal runs / parts of a
// tile, 20.4 / 14.3.
cudaError_t launch_umma_rows(bool split, const UmmaArgs& args, size_t smem, cudaStream_t s) {
  auto kern = split ? umma_rows_kernel<true> : umma_rows_kernel<false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  constexpr int64_t kStart = 8;
  const int threads = kRowsThreads;
  UmmaArgs a = args;
  a.unit = 1;
  const int64_t tiles = (a.padded + kRowsCells - 1) / kRowsCells, n = a.chunks;
  const int64_t ctas = persistent_grid(kern, smem, tiles * n * threads, threads);
  int64_t grid = ctas;
  if (g_grid_override <= 0) {
    const int64_t run = (tiles * n + ctas - 1) / ctas, step = tiles * n % ctas == 0 ? std::gcd(run, n) : 1;
    const int64_t cost = run + kStart * ((run + n - step + n - 1) / n);
    const int64_t rounds = (tiles + ctas - 1) / ctas, parts = std::min(n, std::max<int64_t>(ctas / tiles, 1));
    const int64_t whole = rounds > 1 ? rounds * (n + kStart) : (n + parts - 1) / parts + kStart;
    if (whole <= cost) {
      grid = rounds > 1 ? (tiles + rounds - 1) / rounds : tiles * parts;
      if (rounds > 1) a.unit = (int)n;
    }
  }
  kern<<<(unsigned)grid, threads, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace tlg
