// The pull-back of cells of low degree (simplices P1-P3, tensor cells Q1-Q3, prisms P1-P3) on the
// polynomial form of their map. Same iteration as pullback.cu's kernels (pullback.cuh has the
// update); what differs is how X(xi) and J(xi) are formed and how the work is laid out.
//
// The map of a cell is x_0 + sum_m c_m e_m(xi), e_m the monomials of the cell's space (about the
// centre 1/2 in tensor directions, about vertex 0 on simplices), c_m = sum_k C[m][k] (x_k - x_0) with
// C = V^-1 from the host (poly_expansion; its zeros are not stored). The coefficients are formed
// once per cell; a point then costs nested multiplications: 27 multiply-adds for X and 27 for J on
// a P2 tetrahedron, 78 and 69 on a Q2 hexahedron, against the generic kernel's Lagrange products
// with divisions, indexed local arrays (local memory) and 4 K multiply-adds per coordinate.
//
// A CTA owns 16 cells. Their nodes (shifted by node 0, in the mesh's type) and then their
// coefficients go to shared memory, cell index fastest; one item per (point, cell) runs a point's
// iterations, so that lanes 0-15 and 16-31 of a warp read the coefficients of the same 16 cells
// (one 128-byte wavefront in f64) and a mesh of few cells still fills the chip: the generic kernel
// runs a cell's points one after the other in one thread. A frozen point's item ends its
// iterations (a frozen point keeps xi and its step, so the results are those of the full count;
// Newton takes 4-6 of the 16 by default).
//
// Bound by the FP64 pipe (native f64, and the residuals of mixed precision): about 115 FP64
// operations an iteration on a P2 tetrahedron. GB300, 48,000 P2 tetrahedra with 24 points, f64:
// 20.9 -> 1.26 ms (generic kernel -> this one; 1.37 with the comparisons of newton_update on the FP64 pipe);
// 35,937 Q2 hexahedra with 27 points, mixed: 9.07 -> 0.57 ms.
#pragma once

#include <algorithm>

#include "eval_launch.cuh"
#include "poly_basis.h"
#include "pullback.cuh"

namespace tlg {

struct PolyArgs {
  PullBackArgs p;
  PolyTerms t;
};

constexpr int kPolyCells = 16;  // cells of a CTA

template <int CELL, int P>
struct PolyShape {
  static constexpr int TD = CELL == kTriangle || CELL == kQuadrilateral ? 2 : 3;
  static constexpr int N = P + 1, NT = N * (N + 1) / 2;
  static constexpr int K = CELL == kTriangle        ? NT
                           : CELL == kQuadrilateral ? N * N
                           : CELL == kTetrahedron   ? N * (N + 1) * (N + 2) / 6
                           : CELL == kPrism         ? NT * N
                                                    : N * N * N;
};

// v x^a y^b z^c with the powers' tables, unit factors left out (constant indices).
template <typename F>
__device__ __forceinline__ F poly_powers(const F* px, const F* py, const F* pz, int a, int b, int c) {
  F w = px[a];
  if (b) w = a ? w * py[b] : py[b];
  if (c) w = a || b ? w * pz[c] : pz[c];
  return w;
}

// Values and, with WJ, first derivatives of sum_m c_m e_m on a simplex of dimension D (monomials
// x^a y^b z^c, |a| <= P, a fastest; the constant's and linear terms start the sums), one coordinate;
// value m at c[m * stride].
template <typename F, int D, int P, bool WJ>
__device__ __forceinline__ void poly_simplex(const F* c, int stride, const F (*pw)[P + 1], F& X, F* J) {
  int m = 0;
#pragma unroll
  for (int cc = 0; cc <= (D == 3 ? P : 0); ++cc)
#pragma unroll
    for (int b = 0; b <= P - cc; ++b)
#pragma unroll
      for (int a = 0; a <= P - cc - b; ++a) {
        const F v = c[m * stride];
        if (a + b + cc == 0) {
          X = v;
        } else {
          X = fma(v, poly_powers(pw[0], pw[1], pw[2], a, b, cc), X);
        }
        if constexpr (WJ) {
          const bool linear = a + b + cc == 1;
          if (a > 0) {
            if (linear) J[0] = v;
            else J[0] = fma(v, a > 1 ? F(a) * poly_powers(pw[0], pw[1], pw[2], a - 1, b, cc)
                                     : poly_powers(pw[0], pw[1], pw[2], 0, b, cc), J[0]);
          }
          if (b > 0) {
            if (linear) J[1] = v;
            else J[1] = fma(v, b > 1 ? F(b) * poly_powers(pw[0], pw[1], pw[2], a, b - 1, cc)
                                     : poly_powers(pw[0], pw[1], pw[2], a, 0, cc), J[1]);
          }
          if (D == 3 && cc > 0) {
            if (linear) J[2] = v;
            else J[2] = fma(v, cc > 1 ? F(cc) * poly_powers(pw[0], pw[1], pw[2], a, b, cc - 1)
                                      : poly_powers(pw[0], pw[1], pw[2], a, b, 0), J[2]);
          }
        }
        ++m;
      }
}

// X - x_0 (GD) and, with WJ, J (J(g, d) at d * GD + g) at xi from a cell's coefficients, value
// (m, g) at cs[(m * GD + g) * kPolyCells].
template <typename F, int CELL, int P, int GD, bool WJ>
__device__ __forceinline__ void poly_map(const F* cs, const F* xi, F* X, F* J) {
  constexpr int TD = PolyShape<CELL, P>::TD, N = P + 1, NT = PolyShape<CELL, P>::NT;
  constexpr int S = GD * kPolyCells;
  if constexpr (CELL == kTriangle || CELL == kTetrahedron) {
    F pw[3][P + 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      pw[d][0] = F(1);
#pragma unroll
      for (int i = 1; i <= P; ++i) pw[d][i] = d < TD ? (i > 1 ? pw[d][i - 1] * xi[d] : xi[d]) : F(1);
    }
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      F j[3];
      poly_simplex<F, TD, P, WJ>(cs + g * kPolyCells, S, pw, X[g], j);
      if constexpr (WJ)
#pragma unroll
        for (int d = 0; d < TD; ++d) J[d * GD + g] = j[d];
    }
  } else if constexpr (CELL == kPrism) {
    F pw[3][P + 1];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      pw[d][0] = F(1);
#pragma unroll
      for (int i = 1; i <= P; ++i) pw[d][i] = d < 2 ? (i > 1 ? pw[d][i - 1] * xi[d] : xi[d]) : F(1);
    }
    const F t = xi[2] - F(0.5);
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      F x = F(0), jx = F(0), jy = F(0), jz = F(0);
#pragma unroll(P > 1 ? 1 : N)  // (rolled above degree 1: the unrolled loop holds every coefficient in registers and spills)
      for (int c = P; c >= 0; --c) {
        F v, j[3];
        poly_simplex<F, 2, P, WJ>(cs + (c * NT * GD + g) * kPolyCells, S, pw, v, j);
        if (c == P) {
          x = v;
          if constexpr (WJ) {
            jx = j[0];
            jy = j[1];
          }
        } else {
          if constexpr (WJ) {
            jz = c == P - 1 ? x : fma(jz, t, x);
            jx = fma(jx, t, j[0]);
            jy = fma(jy, t, j[1]);
          }
          x = fma(x, t, v);
        }
      }
      X[g] = x;
      if constexpr (WJ) {
        J[g] = jx;
        J[GD + g] = jy;
        J[2 * GD + g] = jz;
      }
    }
  } else {  // tensor cells: nested multiplication along each direction, derivatives alongside
    F t[3];
#pragma unroll
    for (int d = 0; d < TD; ++d) t[d] = xi[d] - F(0.5);
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      F x = F(0), jx = F(0), jy = F(0), jz = F(0);
#pragma unroll(TD == 3 && P > 1 ? 1 : N)
      for (int c = TD == 3 ? P : 0; c >= 0; --c) {
        F pv = F(0), px = F(0), py = F(0);
#pragma unroll
        for (int b = P; b >= 0; --b) {
          F v = F(0), dv = F(0);
#pragma unroll
          for (int a = P; a >= 0; --a) {
            const F u = cs[((a + N * (b + N * c)) * GD + g) * kPolyCells];
            if (a == P) {
              v = u;
            } else {
              if constexpr (WJ) dv = a == P - 1 ? v : fma(dv, t[0], v);
              v = fma(v, t[0], u);
            }
          }
          if (b == P) {
            pv = v;
            px = dv;
          } else {
            if constexpr (WJ) {
              py = b == P - 1 ? pv : fma(py, t[1], pv);
              px = fma(px, t[1], dv);
            }
            pv = fma(pv, t[1], v);
          }
        }
        if (c == (TD == 3 ? P : 0)) {
          x = pv;
          jx = px;
          jy = py;
        } else {
          if constexpr (WJ) {
            jz = c == P - 1 ? x : fma(jz, t[2], x);
            jx = fma(jx, t[2], px);
            jy = fma(jy, t[2], py);
          }
          x = fma(x, t[2], pv);
        }
      }
      X[g] = x;
      if constexpr (WJ) {
        J[g] = jx;
        J[GD + g] = jy;
        if constexpr (TD == 3) J[2 * GD + g] = jz;
      }
    }
  }
}

// The CTA's cells: c0 + lane for lane < kPolyCells (clamped to the block's last cell). ys receives
// x_k - x_0 and cs the coefficients, both [.][GD][kPolyCells].
template <typename F, int CELL, int P, int GD>
__device__ __forceinline__ void poly_cells(const PolyArgs& a, int64_t c0, F* ys, F* cs) {
  constexpr int K = PolyShape<CELL, P>::K;
  const F* nodes = static_cast<const F*>(a.p.nodes);
  for (int i = threadIdx.x; i < K * kPolyCells; i += blockDim.x) {
    const int lane = i % kPolyCells, k = i / kPolyCells;
    const uint32_t* row = a.p.dofmap + min(a.p.first_cell + c0 + lane, a.p.last_cell) * K;
    const int64_t n0 = min(__ldg(row), a.p.last_node), n = min(__ldg(row + k), a.p.last_node);
#pragma unroll
    for (int g = 0; g < GD; ++g)
      ys[(k * GD + g) * kPolyCells + lane] = __ldg(nodes + n * GD + g) - __ldg(nodes + n0 * GD + g);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < K * kPolyCells; i += blockDim.x) {
    const int lane = i % kPolyCells, m = i / kPolyCells;
    F acc[GD];
#pragma unroll
    for (int g = 0; g < GD; ++g) acc[g] = F(0);
    const uint32_t end = __ldg(a.t.start + m + 1);
    for (uint32_t e = __ldg(a.t.start + m); e < end; ++e) {
      const F c = F(__ldg(&a.t.term[e].c));
      const int k = __ldg(&a.t.term[e].k);
#pragma unroll
      for (int g = 0; g < GD; ++g) acc[g] = fma(c, ys[(k * GD + g) * kPolyCells + lane], acc[g]);
    }
#pragma unroll
    for (int g = 0; g < GD; ++g) cs[(m * GD + g) * kPolyCells + lane] = acc[g];
  }
  __syncthreads();
}

// Newton in F on the coefficients cs of one cell from the reference cell's centroid, r = y - X with
// y relative to x_0: exactly the iterations of pull_back_kernel up to the one that freezes.
template <typename F, int CELL, int P, int GD>
__device__ __forceinline__ void poly_newton(const F* cs, const F* y, int iterations, F tol, F lo, F hi, F big,
                                            F* p, F& last) {
  constexpr int TD = PolyShape<CELL, P>::TD, LJ = TD * GD;
  bool frozen = false;
  for (int it = 0; it < iterations && !frozen; ++it) {
    F X[GD], J[LJ], K_[LJ], r[GD];
    poly_map<F, CELL, P, GD, true>(cs, p, X, J);
    Factors<F, TD, GD>::pinv(J, K_);
#pragma unroll
    for (int g = 0; g < GD; ++g) r[g] = y[g] - X[g];
    newton_update<F, F, TD, GD>(p, K_, r, last, frozen, tol, lo, hi, big);
  }
}

template <typename F, int CELL, int P, int GD>
__global__ void __launch_bounds__(192, 2) pull_back_poly_kernel(const __grid_constant__ PolyArgs a) {
  constexpr int TD = PolyShape<CELL, P>::TD, K = PolyShape<CELL, P>::K;
  extern __shared__ __align__(16) unsigned char smem[];
  F* ys = reinterpret_cast<F*>(smem);
  F* cs = ys + K * GD * kPolyCells;
  const F* nodes = static_cast<const F*>(a.p.nodes);
  const F* xin = static_cast<const F*>(a.p.x);
  F* xi_out = static_cast<F*>(a.p.xi);
  F* step_out = static_cast<F*>(a.p.step);
  const int nq = a.p.num_points, tmask = (1 << a.p.tile_shift) - 1;
  const F big = fmax_finite<F>();
  float start[3];
  centroid_f32(CELL, start);
  const int64_t c0 = (int64_t)blockIdx.x * kPolyCells;
  poly_cells<F, CELL, P, GD>(a, c0, ys, cs);
  for (int i = threadIdx.x; i < nq * kPolyCells; i += blockDim.x) {
    const int lane = i % kPolyCells, q = i / kPolyCells;
    const int64_t c = c0 + lane;
    if (c >= a.p.padded) continue;
    const uint32_t* row = a.p.dofmap + min(a.p.first_cell + c, a.p.last_cell) * K;
    const int64_t n0 = min(__ldg(row), a.p.last_node);
    const int64_t ox = a.p.x_first_cell + c, oo = a.p.out_first_cell + c;
    const int64_t tx = ox >> a.p.tile_shift, to = oo >> a.p.tile_shift;
    const int lx = (int)(ox & tmask), lo_ = (int)(oo & tmask);
    F y[GD];
#pragma unroll
    for (int g = 0; g < GD; ++g)
      y[g] = (xin[(((tx * nq + q) * GD + g) << a.p.tile_shift) + lx] - F(a.p.origin[g])) - __ldg(nodes + n0 * GD + g);
    F p[TD], last = big;
#pragma unroll
    for (int d = 0; d < TD; ++d) p[d] = start[d];
    poly_newton<F, CELL, P, GD>(cs + lane, y, a.p.max_iterations, F(a.p.tolerance), F(-0.1f), F(1.1f), big, p, last);
#pragma unroll
    for (int d = 0; d < TD; ++d) xi_out[(((to * nq + q) * TD + d) << a.p.tile_shift) + lo_] = p[d];
    step_out[((to * nq + q) << a.p.tile_shift) + lo_] = last;
  }
}

// Mixed precision (pull_back_split_kernel's phases): Newton in FP32 on the coefficients rounded to
// f32, then the refinements with the residual from the f64 coefficients and K from the f32 ones.
template <int CELL, int P, int GD>
__global__ void __launch_bounds__(192, 2) pull_back_poly_split_kernel(const __grid_constant__ PolyArgs a) {
  constexpr int TD = PolyShape<CELL, P>::TD, K = PolyShape<CELL, P>::K, LJ = TD * GD;
  extern __shared__ __align__(16) unsigned char smem[];
  double* ys = reinterpret_cast<double*>(smem);
  double* cs = ys + K * GD * kPolyCells;
  float* cs32 = reinterpret_cast<float*>(ys);  // over ys once the coefficients are formed
  const double* nodes = static_cast<const double*>(a.p.nodes);
  const double* xin = static_cast<const double*>(a.p.x);
  double* xi_out = static_cast<double*>(a.p.xi);
  double* step_out = static_cast<double*>(a.p.step);
  const int nq = a.p.num_points, tmask = (1 << a.p.tile_shift) - 1;
  const double big = fmax_finite<double>();
  float start[3];
  centroid_f32(CELL, start);
  const int64_t c0 = (int64_t)blockIdx.x * kPolyCells;
  poly_cells<double, CELL, P, GD>(a, c0, ys, cs);
  for (int i = threadIdx.x; i < K * GD * kPolyCells; i += blockDim.x) cs32[i] = d2f_rn(cs[i]);
  __syncthreads();
  for (int i = threadIdx.x; i < nq * kPolyCells; i += blockDim.x) {
    const int lane = i % kPolyCells, q = i / kPolyCells;
    const int64_t c = c0 + lane;
    if (c >= a.p.padded) continue;
    const uint32_t* row = a.p.dofmap + min(a.p.first_cell + c, a.p.last_cell) * K;
    const int64_t n0 = min(__ldg(row), a.p.last_node);
    const int64_t ox = a.p.x_first_cell + c, oo = a.p.out_first_cell + c;
    const int64_t tx = ox >> a.p.tile_shift, to = oo >> a.p.tile_shift;
    const int lx = (int)(ox & tmask), lo_ = (int)(oo & tmask);
    double y[GD];
    float y32[GD];
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      y[g] = (xin[(((tx * nq + q) * GD + g) << a.p.tile_shift) + lx] - a.p.origin[g]) - __ldg(nodes + n0 * GD + g);
      y32[g] = d2f_rn(y[g]);
    }
    float p32[TD], last32 = fmax_finite<float>();
#pragma unroll
    for (int d = 0; d < TD; ++d) p32[d] = start[d];
    poly_newton<float, CELL, P, GD>(cs32 + lane, y32, a.p.max_iterations, 1e-5f, -0.1f, 1.1f, fmax_finite<float>(),
                                    p32, last32);
    double p[TD], last = big;
#pragma unroll
    for (int d = 0; d < TD; ++d) p[d] = f2d_exact(p32[d]);
    bool frozen = false;
    for (int it = 0; it < a.p.refinements && !frozen; ++it) {
      float pf[TD], X32[GD], J[LJ], K_[LJ];
#pragma unroll
      for (int d = 0; d < TD; ++d) pf[d] = d2f_rn(p[d]);
      poly_map<float, CELL, P, GD, true>(cs32 + lane, pf, X32, J);
      Factors<float, TD, GD>::pinv(J, K_);
      double X[GD], r[GD], none[1], kd[LJ];
      poly_map<double, CELL, P, GD, false>(cs + lane, p, X, none);
#pragma unroll
      for (int g = 0; g < GD; ++g) r[g] = y[g] - X[g];
#pragma unroll
      for (int e = 0; e < LJ; ++e) kd[e] = f2d_exact(K_[e]);  // off the FP64 pipe
      newton_update<double, double, TD, GD>(p, kd, r, last, frozen, a.p.tolerance, double(-0.1f), double(1.1f), big);
    }
#pragma unroll
    for (int d = 0; d < TD; ++d) xi_out[(((to * nq + q) * TD + d) << a.p.tile_shift) + lo_] = p[d];
    step_out[((to * nq + q) << a.p.tile_shift) + lo_] = last;
  }
}

// Threads per CTA for nq points: the CTA size of 64 to 192 whose rounds leave the fewest idle
// threads (24 points: 384 items in 2 rounds of 192; 27: 432 in 3 of 160; 4: 64 in one of 64).
inline int poly_threads(int nq) {
  const int64_t items = (int64_t)nq * kPolyCells;
  int best = 64;
  int64_t waste = INT64_MAX;
  for (int t = 192; t >= 64; t -= 32) {
    const int64_t w = (items + t - 1) / t * t;
    if (w < waste) {
      waste = w;
      best = t;
    }
  }
  return best;
}

template <typename Kernel>
inline cudaError_t launch_poly(Kernel kern, const PolyArgs& a, size_t smem, cudaStream_t s) {
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t ctas = (a.p.padded + kPolyCells - 1) / kPolyCells;
  kern<<<(unsigned)ctas, poly_threads(a.p.num_points), smem, s>>>(a);
  return cudaGetLastError();
}

// The instantiations, each file for one precision.
#define TLG_POLY_CELLS(X)                                                                                         \
  X(kTriangle, 1, 2) X(kTriangle, 2, 2) X(kTriangle, 3, 2) X(kTriangle, 1, 3) X(kTriangle, 2, 3) X(kTriangle, 3, 3) \
  X(kQuadrilateral, 1, 2) X(kQuadrilateral, 2, 2) X(kQuadrilateral, 3, 2) X(kQuadrilateral, 1, 3)                 \
  X(kQuadrilateral, 2, 3) X(kQuadrilateral, 3, 3) X(kTetrahedron, 1, 3) X(kTetrahedron, 2, 3)                     \
  X(kTetrahedron, 3, 3) X(kHexahedron, 1, 3) X(kHexahedron, 2, 3) X(kHexahedron, 3, 3) X(kPrism, 1, 3)            \
  X(kPrism, 2, 3) X(kPrism, 3, 3)

template <int CELL, int P, int GD>
constexpr size_t poly_smem(size_t f_bytes) {
  return (size_t)2 * PolyShape<CELL, P>::K * GD * kPolyCells * f_bytes;
}

}  // namespace tlg
