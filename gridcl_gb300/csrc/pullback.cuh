// Pieces shared by the pull-back kernels: the basis description, the arguments, the Newton update
// and the start of the iteration (pullback.cu, pullback_poly.cuh).
#pragma once

#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "convert.cuh"
#include "eval.cuh"
#include "poly_basis.h"
#include "refcell.h"

namespace tlg {

constexpr int kBasisMaxN = 16;    // 1D nodes (degree + 1)
constexpr int kBasisMaxK = 1024;  // nodes per cell
constexpr int kPyramidMaxP = 4;   // pyramid degrees of the pull-back
constexpr int kPyramidMaxK = 55;  // (p + 1)(p + 2)(2p + 3) / 6 at p = 4

// Device copy of the basis description.
struct alignas(16) BasisData {
  int cell, p, k, n;        // cell type, degree, nodes per cell, 1D nodes (p + 1)
  const double* coef;       // pyramids: C [m][k] (m-major) after this header; else null
  double s[kBasisMaxN];     // sorted 1D nodes (tensor cells, the prism's line)
  uint8_t idx[kBasisMaxK][4];  // per node: 1D indices (tensor) or barycentric multi-index
                               // (simplex: lambda_0 .. lambda_TD; prism: alpha_0..2, line index)
};

struct PullBackArgs {
  const void* nodes;
  const uint32_t* dofmap;
  const BasisData* basis;
  const void* x;  // input points, GD components (absolute)
  void* xi;       // TD components
  void* step;     // 1 component
  int64_t first_cell, padded, out_first_cell, x_first_cell, last_cell;
  double origin[3];
  double tolerance;
  uint32_t last_node;
  int num_points, max_iterations, tile_shift, threads;
  int refinements;  // mixed precision: FP64-residual steps after the FP32 iteration (0: native)
};

template <typename F>
__device__ __forceinline__ F fmax_finite();
template <>
__device__ __forceinline__ float fmax_finite<float>() { return 3.402823466e38f; }
template <>
__device__ __forceinline__ double fmax_finite<double>() { return 1.7976931348623157e308; }

// |v| as an unsigned integer whose order is that of the magnitudes (above infinity's: NaN).
// Comparisons of doubles take the FP64 pipe, these the integer pipes.
__device__ __forceinline__ uint32_t magnitude(float v) { return __float_as_uint(v) & 0x7FFFFFFFu; }
__device__ __forceinline__ unsigned long long magnitude(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
}
__device__ __forceinline__ bool negative(float v) { return (int)__float_as_uint(v) < 0; }
__device__ __forceinline__ bool negative(double v) { return __double2hiint(v) < 0; }

// One step of a point: delta = K r, s = |delta|_inf (the largest finite value when a component
// is not finite); a point not yet frozen moves to p + delta clamped to [lo, hi] (lo < 0 < hi; NaN
// stays), records s and freezes once s <= tol (tol >= 0). K(t, g) at g * TD + t (in KT's
// precision), r and p in P's.
template <typename P, typename KT, int TD, int GD>
__device__ __forceinline__ void newton_update(P* p, const KT* K, const P* r, P& last, bool& frozen, P tol, P lo,
                                              P hi, P big) {
  P delta[TD];
  P s = big;
#pragma unroll
  for (int t = 0; t < TD; ++t) {
    P acc = P(K[t]) * r[0];
#pragma unroll
    for (int g = 1; g < GD; ++g) acc = fma(P(K[g * TD + t]), r[g], acc);
    delta[t] = acc;
    const P m = fabs(acc);
    s = t == 0 || magnitude(m) > magnitude(s) ? m : s;
  }
  if (magnitude(s) > magnitude(big)) s = big;
  if (!frozen) {
#pragma unroll
    for (int d = 0; d < TD; ++d) {
      P qd = p[d] + delta[d];
      const auto m = magnitude(qd);
      const bool below = negative(qd);
      const P edge = below ? lo : hi;
      if (m > magnitude(edge) && m <= magnitude(P(INFINITY))) qd = edge;
      p[d] = qd;
    }
    last = s;
    frozen = magnitude(s) <= magnitude(tol);
  }
}

// The vertex centroid of the reference cell, rounded to f32.
__device__ __forceinline__ void centroid_f32(int cell, float* start) {
  const float third = 1.0f / 3.0f;
  if (cell == kTriangle) start[0] = start[1] = third;
  else if (cell == kTetrahedron) start[0] = start[1] = start[2] = 0.25f;
  else if (cell == kPrism) {
    start[0] = start[1] = third;
    start[2] = 0.5f;
  } else if (cell == kPyramid) {
    start[0] = start[1] = 0.4f;
    start[2] = 0.2f;
  } else start[0] = start[1] = start[2] = 0.5f;
}

// The polynomial kernels (pullback_poly.cuh) of f32 meshes, f64 meshes and mixed precision; `found`
// is false where none is compiled for the cell, the degree and gdim.
cudaError_t launch_pull_back_poly_f32(int cell, int degree, int gd, const PullBackArgs& a, const PolyTerms& terms,
                                      cudaStream_t s, bool* found);
cudaError_t launch_pull_back_poly_f64(int cell, int degree, int gd, const PullBackArgs& a, const PolyTerms& terms,
                                      cudaStream_t s, bool* found);
cudaError_t launch_pull_back_poly_split(int cell, int degree, int gd, const PullBackArgs& a, const PolyTerms& terms,
                                        cudaStream_t s, bool* found);

}  // namespace tlg
