// FP32 evaluation of hexahedra Q1-Q2 (f32 meshes, and split precision: f64 meshes, f32 fields) on the
// polynomial form of their map, line by line of the point set (eval_poly.cuh has the form), one cell per
// thread in persistent CTAs.
//
// The paired kernel (eval_pair_kernel) sums the 27 Lagrange terms at every point: 312 paired multiply-adds
// and 78 table loads of its 810 instructions per pair of points on Q2 hexahedra at 27 points, at 36 % of
// the issue slots. Here the cell's coordinates become coefficients once (differences in place in the thread's
// shared-memory slots), and contracted plane by plane and line by line a point takes 21 multiply-adds, a
// line 45, a plane 81, none of them where a coordinate is the centre (e_1 = e_2 = 0: the middle point of odd
// Gauss rules); the rule is the same for every thread, so these branches do not diverge. Every coefficient is
// a difference of shifted coordinates, so that the sums' errors stay below those of the Lagrange sums: det J
// of 100,000 curved cells 1.8e-7 -> 1.3e-7 against 64 bits.
//
// Spread over a CTA by stages as the f64 kernel (16 or 32 cells, one item per line and pair of cells) the same
// arithmetic waited for each CTA's gather: 0.47 ms against the paired kernel's 0.36 on 500,000 cells.
//
// GB300, x, J, det J and K, ms (paired kernel -> this one): Q2 at 27 points, 500,000 cells in f32 0.288 -> 0.239,
// in split precision 0.356 -> 0.334 (the FP64 subtractions of the 81 coordinates are a quarter of it); at 64
// points, 190,000 cells, split 0.282 -> 0.232; Q1 at 8 points, 1,500,000 cells, split 0.243 -> 0.216.
#pragma once

#include <cstdint>
#include <type_traits>

#include "eval.cuh"
#include "eval_launch.cuh"

namespace tlg {

// A plane, line or point of the rule (poly_basis.h's PolyNode) in f32.
struct PolyNodeF {
  float t, s1, s2;
  int mid, first, count, plane, pad;
};
static_assert(sizeof(PolyNodeF) == 32, "table stride");

struct HexLineArgs {
  const void* nodes;
  const uint32_t* dofmap;
  const unsigned char* tab;  // staged: lattice [K] u32, planes, lines, points (PolyNodeF)
  const double* dphi64;      // split: the f64 derivative table [Q][K][3] of the recompute
  float* out[4];             // points, jacobian, detj, pinv
  int* err;
  unsigned long long* recomputed;
  int64_t first_cell, padded, range_cells, out_first_cell, last_cell;
  double origin[3];
  float cond_limit;
  uint32_t last_node, tab_bytes, off_planes, off_lines, off_points, mask;
  int num_points, num_planes, tile_shift;
};

// sum A_i e_i and its derivative at a node of a tensor direction, P = 1 or 2; AT_MID: t = 0.
template <int P, bool AT_MID>
__device__ __forceinline__ float hex_val(const float* A, const PolyNodeF& u) {
  if constexpr (AT_MID) return A[0];
  else if constexpr (P == 1) return __fmaf_rn(A[1], u.t, A[0]);
  else return __fmaf_rn(__fmaf_rn(A[2], u.s1, A[1]), u.t, A[0]);
}
template <int P, bool AT_MID>
__device__ __forceinline__ float hex_der(const float* A, const PolyNodeF& u) {
  if constexpr (AT_MID || P == 1) return A[1];
  else return __fmaf_rn(A[2], u.s2, A[1]);
}

// P_ab and Q_ab of a plane (m = a + N b, per coordinate) from the slots c[(m + N^2 l) * 3 + g).
template <int P, int T, bool AT_MID>
__device__ __forceinline__ void hex_plane(const float* c, const PolyNodeF& z, float (*p)[(P + 1) * (P + 1)],
                                          float (*q)[(P + 1) * (P + 1)]) {
  constexpr int N = P + 1;
#pragma unroll
  for (int m = 0; m < N * N; ++m)
#pragma unroll
    for (int g = 0; g < 3; ++g) {
      float v[N];
#pragma unroll
      for (int l = 0; l < (AT_MID ? 2 : N); ++l) v[l] = c[((m + l * N * N) * 3 + g) * T];
      p[g][m] = hex_val<P, AT_MID>(v, z);
      q[g][m] = hex_der<P, AT_MID>(v, z);
    }
}

template <int P, bool AT_MID>
__device__ __forceinline__ void hex_line(const float (*p)[(P + 1) * (P + 1)], const float (*q)[(P + 1) * (P + 1)],
                                         const PolyNodeF& y, float (*A)[P + 1], float (*D)[P + 1], float (*E)[P + 1]) {
  constexpr int N = P + 1;
#pragma unroll
  for (int g = 0; g < 3; ++g)
#pragma unroll
    for (int x = 0; x < N; ++x) {
      float v[N], w[N];
#pragma unroll
      for (int b = 0; b < N; ++b) {
        v[b] = p[g][b * N + x];
        w[b] = q[g][b * N + x];
      }
      A[g][x] = hex_val<P, AT_MID>(v, y);
      D[g][x] = hex_der<P, AT_MID>(v, y);
      E[g][x] = hex_val<P, AT_MID>(w, y);
    }
}

template <int P, bool AT_MID>
__device__ __forceinline__ void hex_point(const PolyNodeF& x, const float (*A)[P + 1], const float (*D)[P + 1],
                                          const float (*E)[P + 1], float* xp, float* j) {
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    xp[g] = hex_val<P, AT_MID>(A[g], x);
    j[g] = hex_der<P, AT_MID>(A[g], x);
    j[3 + g] = hex_val<P, AT_MID>(D[g], x);
    j[6 + g] = hex_val<P, AT_MID>(E[g], x);
  }
}

// CTAs per SM: 4 at Q1, 3 at Q2 (split precision, 2,000,000 Q2 cells: 3 / 4 CTAs, the latter with 116 bytes of
// spills, 1.24 / 1.28 ms; 1,500,000 Q1 cells 0.245 / 0.216). SHIFT: log2 of the tile at compile time (4), or -1: a.tile_shift.
template <bool SPLIT, int P, int SHIFT>
__global__ void __launch_bounds__(kEvalThreads, P == 1 ? 4 : 3) eval_hexline_kernel(const __grid_constant__ HexLineArgs a) {
  using B = Ar<float>;
  using M = Factors<float, 3, 3>;
  using NT = typename std::conditional<SPLIT, double, float>::type;
  constexpr int N = P + 1, K = N * N * N, T = kEvalThreads, REF = P == 2 ? K / 2 : 0;
  constexpr bool MID = P == 2;
  __shared__ uint64_t bar;
  extern __shared__ __align__(16) unsigned char smem[];
  if (!stage_table(a.tab, smem, a.tab_bytes, &bar, a.err)) return;
  float* xs = reinterpret_cast<float*>(smem + a.tab_bytes) + threadIdx.x;
  const uint32_t* lattice = reinterpret_cast<const uint32_t*>(smem);
  const PolyNodeF* planes = reinterpret_cast<const PolyNodeF*>(smem + a.off_planes);
  const PolyNodeF* lines = reinterpret_cast<const PolyNodeF*>(smem + a.off_lines);
  const PolyNodeF* points = reinterpret_cast<const PolyNodeF*>(smem + a.off_points);
  const NT* nodes = static_cast<const NT*>(a.nodes);
  const uint32_t mask = a.mask;
  const int nq = a.num_points, shift = SHIFT >= 0 ? SHIFT : a.tile_shift;
  // (An infinite limit leaves NaN only above it.)
  const float lim = a.cond_limit <= 3.402823466e38f ? fminf(9.0f * a.cond_limit * a.cond_limit, 3.402823466e38f)
                                                    : a.cond_limit;

  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < a.padded; c += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t* row = a.dofmap + min(a.first_cell + c, a.last_cell) * K;
    // The coordinates (split: relative to node 0) to the slots in lattice order; the constant's node plus the
    // origin (split: as an f32 pair; f32: the origin and the node).
    double x0[3];
    if constexpr (SPLIT) {
      const int64_t n0 = min(__ldg(row), a.last_node);
#pragma unroll
      for (int g = 0; g < 3; ++g) x0[g] = __ldg(nodes + n0 * 3 + g);
    }
    float xh[3], xl[3];
#pragma unroll
    for (int l0 = 0; l0 < K; l0 += N * N) {
      uint32_t n[N * N];
#pragma unroll
      for (int l = 0; l < N * N; ++l) n[l] = min(__ldg(row + lattice[l0 + l]), a.last_node);
#pragma unroll
      for (int l = 0; l < N * N; ++l)
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          const NT v = __ldg(nodes + (int64_t)n[l] * 3 + g);
          if constexpr (SPLIT) xs[((l0 + l) * 3 + g) * T] = d2f_rn(v - x0[g]);
          else xs[((l0 + l) * 3 + g) * T] = v;
          if (l0 + l == REF) {
            if constexpr (SPLIT) {
              const double o = v + a.origin[g];
              xh[g] = d2f_rn(o);
              xl[g] = d2f_rn(o - f2d_exact(xh[g]));
            } else {
              xh[g] = (float)a.origin[g];
              xl[g] = v;
            }
          }
        }
    }
    // Coefficients in place: (u_0, u_1) -> (u_0, u_1 - u_0), (u_0, u_1, u_2) -> (u_1, u_2 - u_0, u_0 - 2 u_1 + u_2)
    // along each direction, coordinates that are not differences yet differenced first; the constant becomes 0.
#pragma unroll 1
    for (int g = 0; g < 3; ++g) {
      float u[K];
#pragma unroll
      for (int m = 0; m < K; ++m) u[m] = xs[(m * 3 + g) * T];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const int st = d == 0 ? 1 : d == 1 ? N : N * N;
#pragma unroll
        for (int l = 0; l < K / N; ++l) {
          const int o = l % st + l / st * (st * N);
          if constexpr (N == 2) {
            u[o + st] = B::sub(u[o + st], u[o]);
          } else {
            const float p = u[o], q = u[o + st], r = u[o + 2 * st];
            u[o] = q;
            if (l % st == 0) {
              const float dp = B::sub(p, q), dr = B::sub(r, q);
              u[o + st] = B::sub(dr, dp);
              u[o + 2 * st] = B::add(dp, dr);
            } else {
              u[o + st] = B::sub(r, p);
              u[o + 2 * st] = B::fma(-2.0f, q, B::add(p, r));
            }
          }
        }
      }
      u[0] = 0.0f;
      // (A node that is not finite reaches every point, as in poly_coefficients.)
      if (MID && (__float_as_uint(u[K - 1]) & 0x7F800000u) == 0x7F800000u)
        u[0] = u[1] = u[N] = u[N * N] = __uint_as_float(0x7FC00000u);
#pragma unroll
      for (int m = 0; m < K; ++m) xs[(m * 3 + g) * T] = u[m];
    }
    const int64_t o = a.out_first_cell + c;
    const int64_t tq = (o >> shift) * nq;
    const int lane = (int)(o & ((1 << shift) - 1));
    float* out[4];
    const int len[4] = {3, 9, 1, 9};
#pragma unroll
    for (int f = 0; f < 4; ++f) out[f] = a.out[f] ? a.out[f] + ((tq * len[f]) << shift) + lane : nullptr;

    for (int ip = 0; ip < a.num_planes; ++ip) {
      const PolyNodeF z = planes[ip];
      const int first = lines[z.first].first;  // of the plane's points (at most 64 in split precision)
      unsigned long long flagged = 0;
      float p[3][N * N], q[3][N * N];
      if (MID && z.mid) hex_plane<P, T, MID>(xs, z, p, q);
      else hex_plane<P, T, false>(xs, z, p, q);
      for (int il = z.first; il < z.first + z.count; ++il) {
        const PolyNodeF y = lines[il];
        float A[3][N], D[3][N], E[3][N];
        if (MID && y.mid) hex_line<P, MID>(p, q, y, A, D, E);
        else hex_line<P, false>(p, q, y, A, D, E);
        for (int e = y.first; e < y.first + y.count; ++e) {
          const PolyNodeF x = points[e];
          const int at = x.first << shift;
          float xp[3], j[9], k[9];
          if (MID && x.mid) hex_point<P, MID>(x, A, D, E, xp, j);
          else hex_point<P, false>(x, A, D, E, xp, j);
          if (mask & kOutPoints) {
            float* s = out[0] + (int64_t)at * 3;
#pragma unroll
            for (int g = 0; g < 3; ++g) s[g << shift] = B::add(xh[g], B::add(xl[g], xp[g]));
          }
          if (!(mask & ~kOutPoints)) continue;
          if (mask & kOutJacobian) {
            float* s = out[1] + (int64_t)at * 9;
#pragma unroll
            for (int r = 0; r < 9; ++r) s[r << shift] = j[r];
          }
          if (!SPLIT && !(mask & (kOutDetJ | kOutPinv))) continue;
          // K's rows by cofactors (K(t, g) at 3 g + t), det J by the first column's.
          k[0] = M::cross(j[4], j[8], j[7], j[5]);
          k[3] = M::cross(j[6], j[5], j[3], j[8]);
          k[6] = M::cross(j[3], j[7], j[6], j[4]);
          const float dj = B::fma(j[2], k[6], B::fma(j[1], k[3], B::mul(j[0], k[0])));
          if (mask & kOutDetJ) out[2][at] = dj;
          if (!SPLIT && !(mask & kOutPinv)) continue;
          k[1] = M::cross(j[7], j[2], j[1], j[8]);
          k[4] = M::cross(j[0], j[8], j[6], j[2]);
          k[7] = M::cross(j[6], j[1], j[0], j[7]);
          k[2] = M::cross(j[1], j[5], j[4], j[2]);
          k[5] = M::cross(j[3], j[2], j[0], j[5]);
          k[8] = M::cross(j[0], j[4], j[3], j[1]);
          const float inv = B::rcp(dj);
#pragma unroll
          for (int r = 0; r < 9; ++r) k[r] = B::mul(k[r], inv);
          if (mask & kOutPinv) {
            float* s = out[3] + (int64_t)at * 9;
#pragma unroll
            for (int r = 0; r < 9; ++r) s[r << shift] = k[r];
          }
          if constexpr (SPLIT) {
            // |J|_F |K|_F / 3 against the limit, both squared (an overflow counts as above it).
            float jj = B::mul(j[0], j[0]), kk = B::mul(k[0], k[0]);
#pragma unroll
            for (int r = 1; r < 9; ++r) {
              jj = B::fma(j[r], j[r], jj);
              kk = B::fma(k[r], k[r], kk);
            }
            if (!(B::mul(jj, kk) <= lim)) flagged |= 1ull << (e - first);
          }
        }
      }
      if constexpr (SPLIT) {
        // The plane's near-degenerate points again in FP64, over the values stored (a call beside the plane's
        // sums and the point's values would cost their registers).
        if (!(mask & (kOutJacobian | kOutDetJ | kOutPinv))) flagged = 0;
        for (; flagged; flagged &= flagged - 1) {
          const int qi = points[first + __ffsll((long long)flagged) - 1].first, at = qi << shift;
          recompute_f64<3, 3, K>(static_cast<const double*>(a.nodes), row, a.last_node, a.dphi64 + (int64_t)qi * K * 3,
                                 (mask & kOutJacobian) ? out[1] + (int64_t)at * 9 : nullptr,
                                 (mask & kOutDetJ) ? out[2] + at : nullptr,
                                 (mask & kOutPinv) ? out[3] + (int64_t)at * 9 : nullptr, 1 << shift);
          if (a.recomputed && c < a.range_cells) atomicAdd(a.recomputed, 1ull);
        }
      }
    }
  }
}

// Defined in eval_hexline.cu: f32 meshes (split = false) or split precision, degree 1 or 2.
cudaError_t launch_eval_hexline(bool split, int degree, const HexLineArgs& a, cudaStream_t s, bool* found);

}  // namespace tlg
