// f64 evaluation on the polynomial form of a cell's map, line by line of its point set: tetrahedra
// and triangles P1-P3, hexahedra and quadrilaterals Q1-Q2, prisms P1-P2, facet rules included.
//
// GB300's FP64 pipe does one multiply-add per 16 cycles and SM for a whole warp, so the f64 fields
// cost what their FP64 operations cost. The map of a cell is x_0 + sum_abc c_abc e_a(x) e_b(y) e_c(z)
// with c the expansion of the shifted nodes x_k - x_0. Points that share z form a plane, points of
// a plane that share y a line, and contracting one direction at a time leaves
//   plane  P_ab = sum_c c_abc e_c(z),         Q_ab = sum_c c_abc e_c'(z),
//   line   A_a = sum_b P_ab e_b(y),  D_a = sum_b P_ab e_b'(y),  E_a = sum_b Q_ab e_b(y),
//   point  X = x_0 + sum_a A_a e_a(x),  J = (sum_a A_a e_a'(x), sum_a D_a e_a(x), sum_a E_a e_a(x)),
// nested multiplications with derivatives of one multiply-add per coordinate at degree 2. The
// collapsed Gauss rules are such sets with the x points of a line consecutive; in any other point
// set a line may be one point and costs what its three stages cost. On P2 tetrahedra at 24 points
// (4 x 3 x 2) a point takes 20 multiply-adds against 120 of the Lagrange sums, on Q2 hexahedra at
// 27 points 45 against 81 of the sum factorisation in the Lagrange basis, and 30 where the rule's
// middle point makes a direction's terms vanish (e_1 = e_2 = 0 at the centre); det J and K take 36
// more (det J by the first column's cofactors, which K needs anyway).
//
// A CTA owns 16 or 32 cells, one or two tiles of the output. Shared memory holds, cell index fastest (a
// half-warp reads one 128-byte row), the shifted nodes, the coefficients and the planes' sums; the
// threads share each stage, and one item per (line, cell) does the line's points. A mesh of 3,072
// cells thus spreads over 192 CTAs with two to nine items per cell in flight, where one thread per
// cell used 24 SMs of 152.
//
// The shift makes the sums relative to the cell's size instead of the mesh's, so the errors are
// no larger than the Lagrange sums' on absolute coordinates: 64^3 x 6 P2 tetrahedra against 64-bit
// references det J 1.8e-14 -> 1.7e-16, x 8.1e-17 -> 8.0e-17.
//
// Bound by the FP64 pipe (91 % active on P2 tetrahedra). GB300, x, J, det J and K, ms (one thread per
// cell with Lagrange sums, or sum factorisation in the Lagrange basis, -> this kernel): 1,572,864 P2
// tetrahedra at 24 points 10.92 -> 4.38; 226,981 Q2 hexahedra at 27 points 1.49 -> 0.89; 3,072 P1
// tetrahedra at 14 points 0.053 -> 0.033 (now the host's call).
#pragma once

#include <algorithm>
#include <cstdint>

#include "eval.cuh"
#include "eval_launch.cuh"
#include "poly_basis.h"
#include "refcell.h"

namespace tlg {

// The mesh's and the table's side of a launch. tab: PolyTerm terms by row and row starts, the same
// by column, PolyNode planes, lines, points (poly_basis.h); its first tab_bytes are staged.
struct PolyCells {
  const double* nodes;
  const uint32_t* dofmap;
  const unsigned char* tab;
  int* err;
  int64_t first_cell, last_cell;
  uint32_t last_node, tab_bytes, off_starts;
};

struct PolyEvalArgs {
  PolyCells cells;
  const uint32_t* flags;
  const double* refn;  // [Q][TD] reference normals (facet rules)
  double* out[6];
  int64_t padded, out_first_cell, last_flag;
  double origin[3];
  uint32_t off_planes, off_lines, off_points, mask;
  int num_points, num_planes, tile_shift;
  int rule_global;  // only the terms and row starts are staged, the rule is read from global memory
  int batch;  // planes whose sums are held at a time
};

// The exponents a cell's polynomial has: with a simplex in (x, y) a + b <= P, with a simplex in
// (x, y, z) a + b + c <= P; else every exponent up to P.
template <int CELL, int P>
struct PolySpace {
  static constexpr int TD = CELL == kTriangle || CELL == kQuadrilateral ? 2 : 3;
  static constexpr bool kTri = CELL == kTriangle || CELL == kTetrahedron || CELL == kPrism;  // simplex in (x, y)
  static constexpr bool kTet = CELL == kTetrahedron;
  static constexpr bool kTensor = CELL == kHexahedron || CELL == kQuadrilateral;
  static constexpr int N = P + 1;
  static constexpr int AB = kTri ? N * (N + 1) / 2 : N * N;         // P_ab
  static constexpr int QAB = kTet ? P * (P + 1) / 2 : AB;           // Q_ab
  static constexpr int K = TD == 2 ? AB : kTet ? N * (N + 1) * (N + 2) / 6 : AB * N;
  static constexpr int PLANE = TD == 2 ? 0 : AB + QAB;              // sums of a plane and coordinate
  // Highest exponent of b beside a in P_ab and Q_ab, and of c beside (a, b).
  __host__ __device__ static constexpr int pb(int a) { return kTri ? P - a : P; }
  __host__ __device__ static constexpr int qb(int a) { return kTet ? P - 1 - a : pb(a); }
  __host__ __device__ static constexpr int cc(int a, int b) { return kTet ? P - a - b : P; }
  static constexpr int DA = kTri ? P - 1 : P;  // highest a of D_a
  static constexpr int EA = kTet ? P - 1 : P;  // of E_a
  // Positions: P_ab (a fastest), Q_ab, c_abc.
  __host__ __device__ static constexpr int pi(int a, int b) { return kTri ? b * N - b * (b - 1) / 2 + a : b * N + a; }
  __host__ __device__ static constexpr int qi(int a, int b) { return kTet ? b * P - b * (b - 1) / 2 + a : pi(a, b); }
  __host__ __device__ static constexpr int ci(int a, int b, int c) {
    if constexpr (!kTet) {
      return c * AB + pi(a, b);
    } else {
      int m = 0;
      for (int l = 0; l < c; ++l) m += (P - l + 1) * (P - l + 2) / 2;
      return m + b * (P - c + 1) - b * (b - 1) / 2 + a;
    }
  }
};

// sum_{i <= D} A[i] e_i at a node: e_0 = 1, e_1 = t, e_2 = t s1 (s1 = t or 2 t), e_i = t^i at degree
// 3; and its derivative (e_2' = s2).
struct PolyAt {
  double t, s1, s2;
  bool mid;
  __device__ __forceinline__ PolyAt(const PolyNode& n) : t(n.t), s1(n.s1), s2(n.s2), mid(n.mid != 0) {}
};
// AT_MID: t = 0, only the first term is left.
template <int D, bool AT_MID = false>
__device__ __forceinline__ double poly_val(const double* A, const PolyAt& u) {
  if constexpr (D == 0 || AT_MID) return A[0];
  else if constexpr (D == 1) return fma(A[1], u.t, A[0]);
  else if constexpr (D == 2) return fma(fma(A[2], u.s1, A[1]), u.t, A[0]);
  else return fma(fma(fma(A[3], u.t, A[2]), u.t, A[1]), u.t, A[0]);
}
template <int D, bool AT_MID = false>
__device__ __forceinline__ double poly_der(const double* A, const PolyAt& u) {
  static_assert(D >= 1 && D <= 3, "degrees 1-3");
  if constexpr (D == 1 || AT_MID) {
    return A[1];
  } else if constexpr (D == 2) {
    return fma(A[2], u.s2, A[1]);
  } else {
    const double d = fma(A[3], u.t, A[2]);  // the derivative alongside the nested value
    return fma(fma(A[3], u.t, d), u.t, fma(d, u.t, A[1]));
  }
}
// The same with the degree a constant only after unrolling.
template <int P, bool AT_MID>
__device__ __forceinline__ double poly_val_n(int deg, const double* A, const PolyAt& u) {
  if (deg == 0) return A[0];
  if (deg == 1) return poly_val<1, AT_MID>(A, u);
  if (P >= 2 && deg == 2) return poly_val<P >= 2 ? 2 : 1, AT_MID>(A, u);
  return poly_val<P, AT_MID>(A, u);
}
template <int P, bool AT_MID>
__device__ __forceinline__ double poly_der_n(int deg, const double* A, const PolyAt& u) {
  if (deg == 0) return 0.0;
  if (deg == 1) return A[1];
  if (P >= 2 && deg == 2) return poly_der<P >= 2 ? 2 : 1, AT_MID>(A, u);
  return poly_der<P, AT_MID>(A, u);
}

// Whether v is infinite or NaN (an integer test: a comparison of doubles takes the FP64 pipe), and a NaN.
__device__ __forceinline__ bool poly_bad(double v) { return (__double2hiint(v) & 0x7FF00000) == 0x7FF00000; }
__device__ __forceinline__ double poly_nan() { return __hiloint2double(0x7FF80000, 0); }

// The three stages of one item, each with its middle point's form: P_ab and Q_ab of a plane and
// coordinate (strides between the coefficients of c and the sums of o), the line's A, D and E from
// them, and X and J at a point.
template <int CELL, int P, int STRIDE, bool AT_MID, int OSTRIDE = STRIDE>
__device__ __forceinline__ void poly_plane(const double* c, const PolyAt& z, bool want_j, double* o) {
  using S = PolySpace<CELL, P>;
  [[maybe_unused]] bool bad = false;
#pragma unroll
  for (int b = 0; b <= P; ++b)
#pragma unroll
    for (int x = 0; x <= (S::kTri ? P - b : P); ++x) {
      double v[P + 1];
#pragma unroll
      for (int l = 0; l <= P; ++l)
        if (l <= S::cc(x, b) && (!AT_MID || l < 2)) v[l] = c[S::ci(x, b, l) * STRIDE];
      o[S::pi(x, b) * OSTRIDE] = poly_val_n<P, AT_MID>(S::cc(x, b), v, z);
      if (want_j && S::cc(x, b) > 0) o[(S::AB + S::qi(x, b)) * OSTRIDE] = poly_der_n<P, AT_MID>(S::cc(x, b), v, z);
      if constexpr (AT_MID && !S::kTensor) bad = bad || poly_bad(v[1]);
    }
  // (Nodes of a prism's outer layers that are not finite, as poly_coefficients does for tensor cells.)
  if constexpr (AT_MID && !S::kTensor)
    if (bad) o[S::pi(0, 0) * OSTRIDE] = o[S::pi(1, 0) * OSTRIDE] = o[S::pi(0, 1) * OSTRIDE] = poly_nan();
}

template <int CELL, int P, int GD, int STRIDE, bool AT_MID>
__device__ __forceinline__ void poly_line(const double* sums, const PolyAt& y, bool want_j, double (*A)[P + 1],
                                          double (*D)[PolySpace<CELL, P>::DA + 1],
                                          double (*E)[PolySpace<CELL, P>::EA + 1]) {
  using S = PolySpace<CELL, P>;
#pragma unroll
  for (int g = 0; g < GD; ++g) {
#pragma unroll
    for (int x = 0; x <= P; ++x) {
      double v[P + 1];
#pragma unroll
      for (int b = 0; b <= P; ++b)
        if (b <= S::pb(x) && (!AT_MID || b < 2)) v[b] = sums[(S::pi(x, b) * GD + g) * STRIDE];
      A[g][x] = poly_val_n<P, AT_MID>(S::pb(x), v, y);
      if (x <= S::DA) D[g][x] = poly_der_n<P, AT_MID>(S::pb(x), v, y);
    }
    if constexpr (S::TD == 3) {
      if (want_j) {
#pragma unroll
        for (int x = 0; x <= S::EA; ++x) {
          double v[P + 1];
#pragma unroll
          for (int b = 0; b <= P; ++b)
            if (b <= S::qb(x) && (!AT_MID || b < 1)) v[b] = sums[((S::AB + S::qi(x, b)) * GD + g) * STRIDE];
          E[g][x] = poly_val_n<P, AT_MID>(S::qb(x), v, y);
        }
      }
    }
  }
}

template <int CELL, int P, int GD, bool AT_MID>
__device__ __forceinline__ void poly_point(const PolyAt& x, bool want_x, bool want_j, const double (*A)[P + 1],
                                           const double (*D)[PolySpace<CELL, P>::DA + 1],
                                           const double (*E)[PolySpace<CELL, P>::EA + 1], double* xp, double* j) {
  using S = PolySpace<CELL, P>;
#pragma unroll
  for (int g = 0; g < GD; ++g) {
    if (want_x) xp[g] = poly_val<P, AT_MID>(A[g], x);
    if (want_j) {
      j[g] = poly_der<P, AT_MID>(A[g], x);
      j[GD + g] = poly_val<S::DA, AT_MID>(D[g], x);
      if constexpr (S::TD == 3) j[2 * GD + g] = poly_val<S::EA, AT_MID>(E[g], x);
    }
  }
}

// The CTA's cells c0 .. c0 + W - 1: the rule and expansion staged (stage_issue's copy, begun here),
// the nodes, and the coefficients c_abc in cs [K][GD][W] (tensor cells: ys itself). Returns whether
// the table arrived; a barrier of the CTA.
template <int CELL, int P, int GD, int W>
__device__ __forceinline__ bool poly_coefficients(const PolyCells& a, int64_t c0, unsigned char* smem, uint64_t* bar,
                                                  double* ys, double* cs) {
  using S = PolySpace<CELL, P>;
  constexpr int TD = S::TD, K = S::K, N = S::N;
  constexpr bool TENSOR = S::kTensor;
  stage_issue(a.tab, smem, a.tab_bytes, bar, a.err);
  const PolyTerm* terms = reinterpret_cast<const PolyTerm*>(smem);
  const uint32_t* starts = reinterpret_cast<const uint32_t*>(smem + a.off_starts);
  const int tid = threadIdx.x, nt = blockDim.x;
  // The nodes, while the table is on its way: x_k - x_0 at k (tensor cells: x_k).
  for (int i = tid; i < K * W; i += nt) {
    const int lane = i % W, k = i / W;
    const uint32_t* row = a.dofmap + min(a.first_cell + c0 + lane, a.last_cell) * K;
    const int64_t n0 = min(__ldg(row), a.last_node), n = min(__ldg(row + k), a.last_node);
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      const double v = __ldg(a.nodes + n * GD + g);
      ys[(k * GD + g) * W + lane] = TENSOR ? v : __dsub_rn(v, __ldg(a.nodes + n0 * GD + g));
    }
  }
  if (!stage_wait(bar, a.err)) return false;
  if constexpr (TENSOR) {
    // Lattice order first (node starts[m] at lattice position m), one (g, cell) per thread; then
    // a direction at a time, in place: (u_0, u_1) -> (u_0, u_1 - u_0) or (u_0, u_1, u_2) -> (u_1,
    // u_2 - u_0, u_0 - 2 u_1 + u_2). Coordinates that are not differences yet (the lines through
    // index 0 of the directions done) are differenced first, so that every rounding is relative to
    // the cell's size; the constant, the coordinate of node starts[REF], becomes 0.
    for (int i = tid; i < GD * W; i += nt) {
      double u[K];
#pragma unroll
      for (int m = 0; m < K; ++m) u[m] = ys[(int)starts[m] * (GD * W) + i];
#pragma unroll
      for (int d = 0; d < TD; ++d) {
        const int st = d == 0 ? 1 : d == 1 ? N : N * N;
#pragma unroll
        for (int l = 0; l < K / N; ++l) {
          const int o = l % st + l / st * (st * N);
          const bool raw = l % st == 0;
          if constexpr (N == 2) {
            u[o + st] = __dsub_rn(u[o + st], u[o]);
          } else {
            const double p = u[o], q = u[o + st], r = u[o + 2 * st];
            u[o] = q;
            if (raw) {
              const double dp = __dsub_rn(p, q), dr = __dsub_rn(r, q);
              u[o + st] = __dsub_rn(dr, dp);
              u[o + 2 * st] = __dadd_rn(dp, dr);
            } else {
              u[o + st] = __dsub_rn(r, p);
              u[o + 2 * st] = fma(-2.0, q, __dadd_rn(p, r));
            }
          }
        }
      }
      u[0] = 0.0;
      // A node that is not finite makes the whole coordinate so, as the Lagrange sums do (0 times NaN): at a
      // middle point, which takes the low coefficients only, too. Every node is in the highest coefficient.
      if (N == 3 && poly_bad(u[K - 1])) {
        u[0] = u[1] = u[N] = poly_nan();
        if constexpr (TD == 3) u[N * N] = poly_nan();
      }
#pragma unroll
      for (int m = 0; m < K; ++m) cs[m * (GD * W) + i] = u[m];
    }
  } else {
    for (int i = tid; i < K * W; i += nt) {
      const int lane = i % W, m = i / W;
      double acc[GD];
#pragma unroll
      for (int g = 0; g < GD; ++g) acc[g] = 0.0;
      for (uint32_t e = starts[m]; e < starts[m + 1]; ++e) {
        const double c = terms[e].c;
        const int k = terms[e].k;
#pragma unroll
        for (int g = 0; g < GD; ++g) acc[g] = fma(c, ys[(k * GD + g) * W + lane], acc[g]);
      }
#pragma unroll
      for (int g = 0; g < GD; ++g) cs[(m * GD + g) * W + lane] = acc[g];
    }
  }
  __syncthreads();

  return true;
}

// det J and, with want_k, K of a volume cell's J (codimension 0): K's rows by cofactors (K(t, g) at
// TD g + t), det J by the first column's, which are row 0 of K.
template <int D>
__device__ __forceinline__ void poly_square(const double* j, bool want_k, double& dj, double* kk) {
  using M = Factors<double, D, D>;
  if constexpr (D == 3) {
    kk[0] = M::cross(j[4], j[8], j[7], j[5]);
    kk[3] = M::cross(j[6], j[5], j[3], j[8]);
    kk[6] = M::cross(j[3], j[7], j[6], j[4]);
    dj = fma(j[2], kk[6], fma(j[1], kk[3], __dmul_rn(j[0], kk[0])));
    if (want_k) {
      kk[1] = M::cross(j[7], j[2], j[1], j[8]);
      kk[4] = M::cross(j[0], j[8], j[6], j[2]);
      kk[7] = M::cross(j[6], j[1], j[0], j[7]);
      kk[2] = M::cross(j[1], j[5], j[4], j[2]);
      kk[5] = M::cross(j[3], j[2], j[0], j[5]);
      kk[8] = M::cross(j[0], j[4], j[3], j[1]);
      const double inv = __drcp_rn(dj);
#pragma unroll
      for (int r = 0; r < 9; ++r) kk[r] = __dmul_rn(kk[r], inv);
    }
  } else {
    dj = M::detj(j);
    if (want_k) M::pinv(j, kk);
  }
}

// W: cells of a CTA, 16 or 32.
template <int CELL, int P, int GD, int W>
__global__ void __launch_bounds__(W == 32 ? 288 : 192, 2) eval_poly_kernel(const __grid_constant__ PolyEvalArgs a) {
  using S = PolySpace<CELL, P>;
  constexpr int TD = S::TD, K = S::K, N = S::N;
  constexpr bool MID = !S::kTri && P == 2;  // x, y about the centre
  constexpr bool MIDZ = !S::kTet && P == 2;
  constexpr bool TENSOR = S::kTensor;
  constexpr bool AFFINE = S::kTri && TD == (S::kTet ? 3 : 2) && P == 1;
  constexpr int REF = TENSOR && N == 3 ? K / 2 : 0;  // lattice position of the constant's node
  using M = Factors<double, TD, GD>;
  __shared__ uint64_t bar;
  extern __shared__ __align__(16) unsigned char smem[];
  double* ys = reinterpret_cast<double*>(smem + a.cells.tab_bytes);  // [K][GD][W]: nodes, tensor cells in place
  double* cs = TENSOR ? ys : ys + K * GD * W;                  // coefficients
  double* pl = cs + K * GD * W;                                // [batch][PLANE][GD][W]
  const unsigned char* rule = a.rule_global ? a.cells.tab : smem;
  const PolyNode* planes = reinterpret_cast<const PolyNode*>(rule + a.off_planes);
  const PolyNode* lines = reinterpret_cast<const PolyNode*>(rule + a.off_lines);
  const PolyNode* points = reinterpret_cast<const PolyNode*>(rule + a.off_points);
  const uint32_t* starts = reinterpret_cast<const uint32_t*>(smem + a.cells.off_starts);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int64_t c0 = (int64_t)blockIdx.x * W;
  if (!poly_coefficients<CELL, P, GD, W>(a.cells, c0, smem, &bar, ys, cs)) return;
  const uint32_t mask = a.mask;
  const bool want_x = (mask & kOutPoints) != 0, want_j = (mask & ~kOutPoints) != 0;
  const bool want_k = (mask & (kOutPinv | kOutFacetNormals)) != 0;
  const int nq = a.num_points, tmask = (1 << a.tile_shift) - 1;
  for (int p0 = 0; p0 < a.num_planes; p0 += a.batch) {
    const int np = min(a.batch, a.num_planes - p0);
    if constexpr (TD == 3) {
      // P_ab and Q_ab of the batch's planes: one (plane, coordinate, cell) per item.
      if (p0 > 0) __syncthreads();
      for (int i = tid; i < np * GD * W; i += nt) {
        const int e = i % (GD * W), p = i / (GD * W);
        const PolyAt z(planes[p0 + p]);
        const double* c = cs + e;
        double* o = pl + (size_t)p * (S::PLANE * GD * W) + e;
        if (MIDZ && z.mid) poly_plane<CELL, P, GD * W, MIDZ>(c, z, want_j, o);
        else poly_plane<CELL, P, GD * W, false>(c, z, want_j, o);
      }
      __syncthreads();
    }
    const int l0 = planes[p0].first, nl = planes[p0 + np - 1].first + planes[p0 + np - 1].count - l0;
    for (int i = tid; i < nl * W; i += nt) {
      const int lane = i % W;
      const int64_t c = c0 + lane;
      if (c >= a.padded) continue;
      const PolyNode& ln = lines[l0 + i / W];
      const PolyAt y(ln);
      const double* sums = TD == 3 ? pl + (size_t)(ln.plane - p0) * (S::PLANE * GD * W) + lane : cs + lane;
      double A[GD][N], D[GD][S::DA + 1], E[GD][S::EA + 1];
      if (MID && y.mid) poly_line<CELL, P, GD, W, MID>(sums, y, want_j, A, D, E);
      else poly_line<CELL, P, GD, W, false>(sums, y, want_j, A, D, E);
      const uint32_t* row = a.cells.dofmap + min(a.cells.first_cell + c, a.cells.last_cell) * K;
      const int64_t n0 = min(__ldg(row + (TENSOR ? starts[REF] : 0)), a.cells.last_node);
      double xo[GD];
#pragma unroll
      for (int g = 0; g < GD; ++g) xo[g] = __dadd_rn(__ldg(a.cells.nodes + n0 * GD + g), a.origin[g]);
      double sign = 1.0;
      if ((mask & kOutNormals) && a.flags != nullptr && a.last_flag >= 0)
        sign = (__ldg(a.flags + min(a.cells.first_cell + c, a.last_flag)) & 1u) ? -1.0 : 1.0;
      const int64_t o = a.out_first_cell + c;
      const int64_t tile = o >> a.tile_shift;
      const int ol = (int)(o & tmask);
      double j[TD * GD], kk[TD * GD], nrm[3], dj = 0.0;
      for (int e = 0; e < ln.count; ++e) {
        const PolyNode& pt = points[ln.first + e];
        const PolyAt x(pt);
        const int q = pt.first;
        const bool new_j = want_j && (!AFFINE || e == 0);  // an affine cell's J, det J, K: once
        double xp[GD];
        if (MID && x.mid) poly_point<CELL, P, GD, MID>(x, want_x, new_j, A, D, E, xp, j);
        else poly_point<CELL, P, GD, false>(x, want_x, new_j, A, D, E, xp, j);
        if (want_x) {
#pragma unroll
          for (int g = 0; g < GD; ++g) xp[g] = __dadd_rn(xp[g], xo[g]);
          store_point(a.out[0], tile, q, nq, GD, ol, a.tile_shift, xp, GD);
        }
        if (!want_j) continue;
        if (new_j) {
          if constexpr (TD == GD) {
            poly_square<TD>(j, want_k, dj, kk);
          } else {
            // One cross product and length for the area element and the normal (the operations
            // of Factors::detj and Factors::normal).
            if (mask & (kOutDetJ | kOutNormals)) {
              double v[3];
              M::surface_normal(j, v);
              dj = __dsqrt_rn(M::dot3(v, v));
              if (mask & kOutNormals)
#pragma unroll
                for (int g = 0; g < 3; ++g) nrm[g] = __ddiv_rn(__dmul_rn(sign, v[g]), dj);
            }
            if (want_k) M::pinv(j, kk);
          }
        }
        if (mask & kOutJacobian) store_point(a.out[1], tile, q, nq, TD * GD, ol, a.tile_shift, j, TD * GD);
        if (mask & kOutDetJ) store_point(a.out[2], tile, q, nq, 1, ol, a.tile_shift, &dj, 1);
        if (mask & kOutPinv) store_point(a.out[3], tile, q, nq, TD * GD, ol, a.tile_shift, kk, TD * GD);
        if constexpr (TD == GD) {
          if (mask & kOutFacetNormals) {
            double n[GD], rn[TD];
#pragma unroll
            for (int t = 0; t < TD; ++t) rn[t] = __ldg(a.refn + (int64_t)q * TD + t);
            M::facet_normal(kk, rn, n);
            store_point(a.out[5], tile, q, nq, GD, ol, a.tile_shift, n, GD);
          }
        }
        if constexpr (TD + 1 == GD) {
          if (mask & kOutNormals) store_point(a.out[4], tile, q, nq, GD, ol, a.tile_shift, nrm, GD);
        }
      }
    }
  }
}

// Planes per batch: their sums within 1.5 KiB per cell.
template <int CELL, int P, int GD>
inline int poly_batch(int planes) {
  constexpr int bytes = PolySpace<CELL, P>::PLANE * GD * 8;  // of a plane and cell
  if (bytes == 0 || planes < 1) return std::max(planes, 1);
  const int most = std::max(1, std::min(planes, 1536 / std::max(bytes, 1)));
  const int batches = (planes + most - 1) / most;
  return (planes + batches - 1) / batches;  // batches of equal size
}

// Threads per CTA for `items` (line, cell) items in flight: one round of them up to `most`
// threads, beyond that the size whose rounds leave the fewest threads idle.
inline int poly_line_threads(int items, int most) {
  if (items <= most) return std::max(64, (items + 31) / 32 * 32);
  int best = most, waste = INT32_MAX;
  for (int t = most; t >= 96; t -= 32) {
    const int w = (items + t - 1) / t * t;
    if (w < waste) {
      waste = w;
      best = t;
    }
  }
  return best;
}

template <int CELL, int P, int GD, int W>
inline cudaError_t launch_poly_width(PolyEvalArgs a, int lines, cudaStream_t s) {
  using S = PolySpace<CELL, P>;
  constexpr bool tensor = CELL == kHexahedron || CELL == kQuadrilateral;
  auto kern = eval_poly_kernel<CELL, P, GD, W>;
  a.batch = poly_batch<CELL, P, GD>(a.num_planes);
  const size_t value_bytes = (size_t)GD * W * 8;
  const size_t smem = a.cells.tab_bytes + (size_t)(tensor ? 1 : 2) * S::K * value_bytes +
                      (S::TD == 3 ? (size_t)a.batch * S::PLANE * value_bytes : 0);
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t ctas = (a.padded + W - 1) / W;
  const int in_batch = (int)((int64_t)lines * std::min(a.batch, a.num_planes) / std::max(a.num_planes, 1));
  kern<<<(unsigned)ctas, poly_line_threads(std::max(in_batch, 1) * W, W == 32 ? 288 : 192), smem, s>>>(a);
  return cudaGetLastError();
}

// SMs of the device, queried once per thread.
inline int poly_sms() {
  static thread_local int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return sms;
}

// Cells of a CTA: 16; 32 for the cells whose kernels leave out a middle point's terms (tensor
// directions at degree 2), so that a warp is one line and its lanes agree on the branch, once the
// 32-cell CTAs fill the SMs twice (Q2 hexahedra at 27 points, ms with 32 / 16 cells: 226,981 cells
// 0.89 / 1.12, 20,000 0.107 / 0.123, 10,000 0.067 / 0.070).
template <int CELL, int P, int GD>
inline cudaError_t launch_poly_cell(const PolyEvalArgs& a, int lines, cudaStream_t s) {
  if constexpr (P == 2 && (CELL == kHexahedron || CELL == kPrism || CELL == kQuadrilateral)) {
    if (a.padded >= (int64_t)64 * poly_sms()) return launch_poly_width<CELL, P, GD, 32>(a, lines, s);
  }
  return launch_poly_width<CELL, P, GD, 16>(a, lines, s);
}

// Defined in eval_poly.cu: `found` is false where no kernel is compiled for the cell.
cudaError_t launch_eval_poly(int cell, int degree, int gd, const PolyEvalArgs& a, int lines, cudaStream_t s,
                             bool* found);

}  // namespace tlg
