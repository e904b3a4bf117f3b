// Double-float evaluation (df.cuh: f64 nodes and fields, arithmetic on the FP32 pipe) of volume cells
// on the polynomial form of their map, line by line of the point set: tetrahedra P1-P3, hexahedra
// Q1-Q2 and prisms P1-P2 in 3D. The decomposition is eval_poly.cuh's; the pipes share it:
//  - FP64, once per cell and plane: the shifted nodes, the coefficients and the planes' sums P_ab, Q_ab
//    (5 to 25 operations a point), then split into double-floats in shared memory by integer
//    operations and a conversion (df_split_int);
//  - FP32, per line and point: A, D, E, then X and J as double-float sums (DfAcc), det J and K. On a P2
//    tetrahedron a point takes 18 double-float terms and a line 15 against 63 per point of the
//    monomial sums that one thread ran over a whole cell; a Q2 hexahedron 36 and a third of 45.
// A thread works on two neighbouring cells (the paired FP32 instructions hold one cell each, the
// point's table values are the same for both), so that an odd number of points or lines wastes
// nothing and the two cells' values leave as one 16-byte store. A CTA owns 16 cells; its items are
// (plane, coordinate, cell), (line, coordinate, pair) and (point, pair), the stages' results in shared
// memory. (One item per line and pair with the line's sums in registers took 255 registers: six warps
// per SM, issue 31 % active, 3.04 ms on the P2 tetrahedra below.)
//
// X adds the cell's offset in FP64. f64 bit patterns are assembled by df_to_f64_fast, ten integer
// operations and an FFMA; it does not take zero mantissas, magnitudes outside [2^-81, 2^127) and NaN. Zeros and
// powers of two, which axis-aligned and straight cells have at every point, are mended in place (df_mend);
// the others send three components of the thread's field through df_to_f64 out of line. J leaves three
// components at a time as K does: nine at a time with the mending spilled. Q2 hexahedra, 140,608 cells at 27
// points, axis-aligned / curved, all four factors: 0.69 / 0.41 ms when every special value went out of line,
// 0.485 / 0.408 so (three lanes per cell: 0.50 either way); mending every value without a branch cost the
// curved cells 8 %.
//
// Bound by the issue slots (50 % of them used at 16 warps per SM: dependent double-float chains, and 80-90 %
// hits in the instruction cache) with the FP64 pipe 40 % and the integer pipe 32 % active. GB300, x, J, det J
// and K, ms, the former kernels (one thread or three lanes per cell) -> this one: P2 tetrahedra, 1,572,864
// cells at 24 points 3.04 -> 1.91; Q2 hexahedra, 500,000 at 27 points 1.74 -> 1.36; P3 tetrahedra, 180,000 at
// 64 points 2.36 -> 0.88; 1,000 P2 tetrahedra at 27 points 0.073 -> 0.032 (the host's call).
#pragma once

#include <cstdint>

#include "df.cuh"
#include "eval_poly.cuh"

namespace tlg {

// A coordinate value's powers as (head, tail): e_1 = t, e_2, e_3 and e_2', e_3' (poly_basis.h).
struct PolyDfNode {
  float2 t, e2, e3, s2, s3;
  int first, count, plane, mid;
};
static_assert(sizeof(PolyDfNode) == 56, "table stride");

struct PolyDfArgs {
  PolyCells cells;  // the f64 section: expansion, planes
  const unsigned char* dftab;  // PolyDfNode lines, points (read from global memory where dftab_bytes = 0)
  double* out[4];              // points, jacobian, detj, pinv
  int64_t padded, out_first_cell;
  double origin[3];
  uint32_t off_planes, off_dfpoints, dftab_bytes, mask;
  int num_points, num_planes, rule_global;
  int plane_lines;  // the most lines of a plane
  int batch, chunk, alias;  // planes, and of their lines those, held at a time
  int wide;  // every output is 16-byte aligned: two cells per store
};

// v as h + l, h the nearest f32 (ties away from zero) and l the nearest f32 to the rest, for v in the
// f32 normal range (|v| from 2^-70 up); `special` is set for other values (zero, tiny, huge, NaN), whose
// h and l are not valid.
__device__ __forceinline__ void df_split_int(double v, float& h, float& l, bool& special) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned long long r = b + 0x10000000ull;  // half of the 29 mantissa bits below h's
  const uint32_t bh = (uint32_t)(b >> 32), x = (uint32_t)(r >> 29);
  special = special || ((uint32_t)(r >> 32) & 0x7FFFFFFFu) - (953u << 20) >= ((1150u - 953u) << 20);
  // f64 exponent e + 1023 -> f32 e + 127: the low eight bits differ by 128.
  h = __uint_as_float((bh & 0x80000000u) | ((x ^ 0x40000000u) & 0x7FFFFFFFu));
  // The rest: v's low 29 bits as a signed integer in units of 2^-52 of v's binade (h's may be the next), here
  // times 8, by a power of two with v's sign.
  const uint32_t scale = (((bh << 3) & 0xFF800000u) - (951u << 23)) | (bh & 0x80000000u);
  l = __fmul_rn(__int2float_rn((int)((uint32_t)b << 3)), __uint_as_float(scale));
}

// df_to_f64 for h with a nonzero mantissa and 2^-81 <= |h| < 2^127 (else `special` is set and the
// value is not valid): the f64 of h plus n = l / (64 ulp64(h)), rounded, in its mantissa.
__device__ __forceinline__ double df_to_f64_fast(float h, float l, bool& special) {
  const uint32_t hb = __float_as_uint(h);
  special = special || (hb << 9) == 0u || (hb << 1) - (46u << 24) >= (208u << 24);
  // 2^(173 - e) with h's sign, 1.5 * 2^23 + n: its low bits are n.
  const float scale = __uint_as_float((300u << 23) - (hb & 0xFF800000u));
  const uint32_t n6 = (__float_as_uint(__fmaf_rn(l, scale, 12582912.0f)) << 6) + 0x30000000u;  // 64 n
  const uint32_t lo = hb << 29;
  const uint32_t hi = (uint32_t)((int)hb >> 3) & 0x8FFFFFFFu;
  const uint64_t bits = (((uint64_t)(hi + (896u << 20)) << 32) | lo) + (uint64_t)(int64_t)(int)n6;
  return __longlong_as_double((long long)bits);
}

// df_to_f64_fast's value d of (h, l) mended where h is a zero or a power of two in range, which axis-aligned
// and straight cells have everywhere; `rest` is set for the other special values.
__device__ __forceinline__ void df_mend(float h, double& d, bool& rest) {
  const uint32_t hb = __float_as_uint(h), mag = hb << 1;
  rest = rest || (mag != 0u && mag - (46u << 24) >= (208u << 24));
  // 64 n, d's low word as h's mantissa is zero: a power of two whose magnitude l lowers lands in the binade
  // below, whose ulp is half.
  const int n6 = __double2loint(d);
  if ((hb << 9) == 0u && n6 < 0) d = __longlong_as_double(__double_as_longlong(d) + n6);
  if (mag == 0u) d = __hiloint2double((int)hb, 0);
}

using Dp = DF<float2>;

// The n entries (h0, h1, l0, l1) of t as the two f64 (hi, lo words), in place; out of line, as it would
// double the kernel's code for values that are rare (tiny, huge, not finite).
static __device__ __noinline__ void df_pairs_slow(float4* t, int n) {
  for (int c = 0; c < n; ++c) {
    const double x = df_to_f64(t[c].x, t[c].z), y = df_to_f64(t[c].y, t[c].w);
    t[c] = make_float4(__int_as_float(__double2hiint(x)), __int_as_float(__double2loint(x)),
                       __int_as_float(__double2hiint(y)), __int_as_float(__double2loint(y)));
  }
}

// LEN components of both cells of a pair as f64, and their stores at p[c * 16], p[c * 16 + 1].
template <int LEN>
__device__ __forceinline__ void df_pair_to_f64(const Dp* v, double2* d) {
  bool special = false;
#pragma unroll
  for (int c = 0; c < LEN; ++c) {
    d[c].x = df_to_f64_fast(v[c].h.x, v[c].l.x, special);
    d[c].y = df_to_f64_fast(v[c].h.y, v[c].l.y, special);
  }
  if (__builtin_expect(special, 0)) {
    bool rest = false;
#pragma unroll
    for (int c = 0; c < LEN; ++c) {
      df_mend(v[c].h.x, d[c].x, rest);
      df_mend(v[c].h.y, d[c].y, rest);
    }
    if (__builtin_expect(rest, 0)) {
      float4 t[LEN];
#pragma unroll
      for (int c = 0; c < LEN; ++c) t[c] = make_float4(v[c].h.x, v[c].h.y, v[c].l.x, v[c].l.y);
      df_pairs_slow(t, LEN);
#pragma unroll
      for (int c = 0; c < LEN; ++c) {
        d[c].x = __hiloint2double(__float_as_int(t[c].x), __float_as_int(t[c].y));
        d[c].y = __hiloint2double(__float_as_int(t[c].z), __float_as_int(t[c].w));
      }
    }
  }
}
template <int LEN>
__device__ __forceinline__ void df_store_pair(double* p, const double2* d, bool wide) {
  if (wide) {
#pragma unroll
    for (int c = 0; c < LEN; ++c) *reinterpret_cast<double2*>(p + c * 16) = d[c];
  } else {
#pragma unroll
    for (int c = 0; c < LEN; ++c) {
      p[c * 16] = d[c].x;
      p[c * 16 + 1] = d[c].y;
    }
  }
}
template <int LEN>
__device__ __forceinline__ void df_put_pair(double* p, const Dp* v, bool wide) {
  double2 d[LEN];
  df_pair_to_f64<LEN>(v, d);
  df_store_pair<LEN>(p, d, wide);
}

// sum_{i <= D} A[i] e_i and its derivative at a node; AT_MID: t = 0, one term is left.
template <int D, bool AT_MID = false>
__device__ __forceinline__ Dp df_val(const Dp* A, const PolyDfNode& u) {
  if constexpr (D == 0 || AT_MID) {
    return A[0];
  } else {
    using B = Ar<float2>;
    DfAcc<float2> s;
    s.s = A[0].h;
    s.c = A[0].l;
    s.add(A[1].h, A[1].l, B::splat(u.t.x), B::splat(u.t.y));
    if constexpr (D >= 2) s.add(A[2].h, A[2].l, B::splat(u.e2.x), B::splat(u.e2.y));
    if constexpr (D >= 3) s.add(A[3].h, A[3].l, B::splat(u.e3.x), B::splat(u.e3.y));
    return s.value();
  }
}
template <int D, bool AT_MID = false>
__device__ __forceinline__ Dp df_der(const Dp* A, const PolyDfNode& u) {
  if constexpr (D == 1 || AT_MID) {
    return A[1];
  } else {
    using B = Ar<float2>;
    DfAcc<float2> s;
    s.s = A[1].h;
    s.c = A[1].l;
    s.add(A[2].h, A[2].l, B::splat(u.s2.x), B::splat(u.s2.y));
    if constexpr (D >= 3) s.add(A[3].h, A[3].l, B::splat(u.s3.x), B::splat(u.s3.y));
    return s.value();
  }
}
template <int P, bool AT_MID>
__device__ __forceinline__ Dp df_val_n(int deg, const Dp* A, const PolyDfNode& u) {
  if (deg == 0) return A[0];
  if (deg == 1) return df_val<1, AT_MID>(A, u);
  if (P >= 2 && deg == 2) return df_val<P >= 2 ? 2 : 1, AT_MID>(A, u);
  return df_val<P, AT_MID>(A, u);
}
template <int P, bool AT_MID>
__device__ __forceinline__ Dp df_der_n(int deg, const Dp* A, const PolyDfNode& u) {
  if (deg == 1) return A[1];
  if (P >= 2 && deg == 2) return df_der<P >= 2 ? 2 : 1, AT_MID>(A, u);
  return df_der<P, AT_MID>(A, u);
}

// Positions of a line's sums: A_a, D_a, E_a.
template <int CELL, int P>
struct DfLine {
  using S = PolySpace<CELL, P>;
  static constexpr int D0 = P + 1, E0 = D0 + S::DA + 1, COUNT = E0 + S::EA + 1;
};

__device__ __forceinline__ Dp df_entry(const float4* s) {
  const float4 v = *s;
  Dp r;
  r.h = make_float2(v.x, v.y);
  r.l = make_float2(v.z, v.w);
  return r;
}

// One coordinate of a line's A, D, E from its plane's sums: entry e of the pair at s[e * STRIDE], sum
// m to o[m * STRIDE].
template <int CELL, int P, int STRIDE>
__device__ __forceinline__ void df_line(const float4* s, const PolyDfNode& y, bool want_j, float4* o) {
  using S = PolySpace<CELL, P>;
  using L = DfLine<CELL, P>;
  auto put = [&](int m, const Dp& v) { o[m * STRIDE] = make_float4(v.h.x, v.h.y, v.l.x, v.l.y); };
#pragma unroll
  for (int x = 0; x <= P; ++x) {
    Dp v[P + 1];
#pragma unroll
    for (int b = 0; b <= P; ++b)
      if (b <= S::pb(x)) v[b] = df_entry(s + S::pi(x, b) * STRIDE);
    put(x, df_val_n<P, false>(S::pb(x), v, y));
    if (want_j && x <= S::DA) put(L::D0 + x, df_der_n<P, false>(S::pb(x), v, y));
  }
  if (want_j)
#pragma unroll
    for (int x = 0; x <= S::EA; ++x) {
      Dp v[P + 1];
#pragma unroll
      for (int b = 0; b <= P; ++b)
        if (b <= S::qb(x)) v[b] = df_entry(s + (S::AB + S::qi(x, b)) * STRIDE);
      put(L::E0 + x, df_val_n<P, false>(S::qb(x), v, y));
    }
}

template <int CELL, int P>
__global__ void __launch_bounds__(128, 4) eval_dfpoly_kernel(const __grid_constant__ PolyDfArgs a) {
  using S = PolySpace<CELL, P>;
  using L = DfLine<CELL, P>;
  constexpr int W = 16, K = S::K, N = S::N, COL = 3 * W, PAIRS = W / 2, ROW = 3 * PAIRS;
  constexpr bool MIDZ = !S::kTet && P == 2, TENSOR = S::kTensor;
  constexpr int REF = TENSOR && N == 3 ? K / 2 : 0;
  using A = Ar<Dp>;
  using M = Factors<Dp, 3, 3>;
  __shared__ uint64_t bar;
  __shared__ __align__(16) double xo[COL];  // x_0 + origin, [g][cell]
  extern __shared__ __align__(16) unsigned char smem[];
  // pl [batch][PLANE][3][PAIRS] and, over the nodes and coefficients where one batch holds every plane,
  // ls [lines of the batch][COUNT][3][PAIRS]: float4 (h0, h1, l0, l1).
  float4* pl = reinterpret_cast<float4*>(smem + a.cells.tab_bytes + a.dftab_bytes);
  double* ys = reinterpret_cast<double*>(pl + (size_t)a.batch * (S::PLANE * ROW));
  double* cs = TENSOR ? ys : ys + K * COL;
  float4* ls = reinterpret_cast<float4*>(a.alias ? ys : cs + K * COL);
  const unsigned char* dfrule = a.dftab_bytes ? smem + a.cells.tab_bytes : a.dftab;
  const PolyNode* planes = reinterpret_cast<const PolyNode*>((a.rule_global ? a.cells.tab : smem) + a.off_planes);
  const PolyDfNode* lines = reinterpret_cast<const PolyDfNode*>(dfrule);
  const PolyDfNode* points = reinterpret_cast<const PolyDfNode*>(dfrule + a.off_dfpoints);
  const uint32_t* starts = reinterpret_cast<const uint32_t*>(smem + a.cells.off_starts);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int64_t c0 = (int64_t)blockIdx.x * W;
  for (uint32_t i = tid; i < a.dftab_bytes / 8; i += nt)
    reinterpret_cast<uint2*>(smem + a.cells.tab_bytes)[i] = __ldg(reinterpret_cast<const uint2*>(a.dftab) + i);
  if (!poly_coefficients<CELL, P, 3, W>(a.cells, c0, smem, &bar, ys, cs)) return;
  for (int i = tid; i < COL; i += nt) {
    const uint32_t* row = a.cells.dofmap + min(a.cells.first_cell + c0 + i % W, a.cells.last_cell) * K;
    const int64_t n0 = min(__ldg(row + (TENSOR ? starts[REF] : 0)), a.cells.last_node);
    xo[i] = __dadd_rn(__ldg(a.cells.nodes + n0 * 3 + i / W), a.origin[i / W]);
  }

  const uint32_t mask = a.mask;
  const bool want_x = (mask & kOutPoints) != 0, want_j = (mask & ~kOutPoints) != 0, wide = a.wide != 0;
  const int nq = a.num_points;
  for (int p0 = 0; p0 < a.num_planes; p0 += a.batch) {
    const int np = min(a.batch, a.num_planes - p0);
    for (int i = tid; i < np * COL; i += nt) {
      const int e = i % COL, p = i / COL, lane = e % W, g = e / W;
      const PolyAt z(planes[p0 + p]);
      double v[S::PLANE];
      if (MIDZ && z.mid) poly_plane<CELL, P, COL, MIDZ, 1>(cs + e, z, want_j, v);
      else poly_plane<CELL, P, COL, false, 1>(cs + e, z, want_j, v);
      float* o = reinterpret_cast<float*>(pl + ((size_t)p * (S::PLANE * 3) + g) * PAIRS + lane / 2) + lane % 2;
#pragma unroll
      for (int m = 0; m < S::PLANE; ++m) {
        if (m >= S::AB && !want_j) continue;
        float h, l;
        bool special = false;
        df_split_int(v[m], h, l, special);
        if (__builtin_expect(special, 0)) {
          const int hi = __double2hiint(v[m]);
          if (((hi << 1) | __double2loint(v[m])) == 0) {  // zero
            h = __int_as_float(hi);
            l = 0.0f;
          } else {
            df_split(v[m], h, l);
          }
        }
        o[m * (ROW * 4)] = h;
        o[m * (ROW * 4) + 2] = l;
      }
    }
    __syncthreads();
    const int b0 = planes[p0].first, b1 = planes[p0 + np - 1].first + planes[p0 + np - 1].count;
    for (int l0 = b0; l0 < b1; l0 += a.chunk) {
      const int nl = min(a.chunk, b1 - l0);
      if (l0 > b0) __syncthreads();
      for (int i = tid; i < nl * ROW; i += nt) {
        const int col = i % ROW, l = i / ROW;
        const PolyDfNode& ln = lines[l0 + l];
        df_line<CELL, P, ROW>(pl + (size_t)(ln.plane - p0) * (S::PLANE * ROW) + col, ln, want_j,
                              ls + (size_t)l * (L::COUNT * ROW) + col);
      }
      __syncthreads();
      const int q0 = lines[l0].first, npts = lines[l0 + nl - 1].first + lines[l0 + nl - 1].count - q0;
      for (int i = tid; i < npts * PAIRS; i += nt) {
        const int pair = i % PAIRS;
        const int64_t c = c0 + 2 * pair;
        if (c >= a.padded) continue;
        const PolyDfNode& x = points[q0 + i / PAIRS];
        const float4* s = ls + (size_t)(x.plane - l0) * (L::COUNT * ROW) + pair;
        const int64_t o = a.out_first_cell + c;
        const int64_t q = o / 16 * nq + x.first;
        const int l16 = (int)(o % 16);
        Dp xp[3], j[9];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
          const float4* sg = s + g * PAIRS;
          Dp v[N];
#pragma unroll
          for (int m = 0; m < N; ++m) v[m] = df_entry(sg + m * ROW);
          if (want_x) xp[g] = df_val<P>(v, x);
          if (!want_j) continue;
          j[g] = df_der<P>(v, x);
#pragma unroll
          for (int m = 0; m <= S::DA; ++m) v[m] = df_entry(sg + (L::D0 + m) * ROW);
          j[3 + g] = df_val<S::DA>(v, x);
#pragma unroll
          for (int m = 0; m <= S::EA; ++m) v[m] = df_entry(sg + (L::E0 + m) * ROW);
          j[6 + g] = df_val<S::EA>(v, x);
        }
        if (want_x) {
          double2 d[3];
          df_pair_to_f64<3>(xp, d);
#pragma unroll
          for (int g = 0; g < 3; ++g) {
            const double2 off = reinterpret_cast<const double2*>(xo)[g * PAIRS + pair];
            d[g].x = __dadd_rn(d[g].x, off.x);
            d[g].y = __dadd_rn(d[g].y, off.y);
          }
          df_store_pair<3>(a.out[0] + q * 48 + l16, d, wide);
        }
        if (!want_j) continue;
        if (mask & kOutJacobian) {
          double* pj = a.out[1] + q * 144 + l16;
          df_put_pair<3>(pj, j, wide);
          df_put_pair<3>(pj + 48, j + 3, wide);
          df_put_pair<3>(pj + 96, j + 6, wide);
        }
        if (!(mask & (kOutDetJ | kOutPinv))) continue;
        // Row 0 of the cofactors gives det J; K leaves three entries (a component g) at a time.
        Dp r0[3];
        r0[0] = M::cross(j[4], j[8], j[7], j[5]);
        r0[1] = M::cross(j[6], j[5], j[3], j[8]);
        r0[2] = M::cross(j[3], j[7], j[6], j[4]);
        const Dp dj = A::fma(j[2], r0[2], A::fma(j[1], r0[1], A::mul(j[0], r0[0])));
        if (mask & kOutDetJ) df_put_pair<1>(a.out[2] + q * 16 + l16, &dj, wide);
        if (mask & kOutPinv) {
          const Dp inv = A::rcp(dj);
          double* pk = a.out[3] + q * 144 + l16;
          Dp k[3];
          k[0] = A::mul(r0[0], inv);
          k[1] = A::mul(M::cross(j[7], j[2], j[1], j[8]), inv);
          k[2] = A::mul(M::cross(j[1], j[5], j[4], j[2]), inv);
          df_put_pair<3>(pk, k, wide);
          k[0] = A::mul(r0[1], inv);
          k[1] = A::mul(M::cross(j[0], j[8], j[6], j[2]), inv);
          k[2] = A::mul(M::cross(j[3], j[2], j[0], j[5]), inv);
          df_put_pair<3>(pk + 48, k, wide);
          k[0] = A::mul(r0[2], inv);
          k[1] = A::mul(M::cross(j[6], j[1], j[0], j[7]), inv);
          k[2] = A::mul(M::cross(j[0], j[4], j[3], j[1]), inv);
          df_put_pair<3>(pk + 96, k, wide);
        }
      }
    }
    if (p0 + a.batch < a.num_planes) __syncthreads();
  }
}

template <int CELL, int P>
inline cudaError_t launch_dfpoly_cell(PolyDfArgs a, int lines, cudaStream_t s) {
  using S = PolySpace<CELL, P>;
  using L = DfLine<CELL, P>;
  auto kern = eval_dfpoly_kernel<CELL, P>;
  const size_t value = (size_t)3 * 16 * 8, nodes = (size_t)(S::kTensor ? 1 : 2) * S::K * value;
  const int planes = std::max(a.num_planes, 1);
  // Planes held at a time, and lines: those whose sums keep seven CTAs on an SM (30 KiB each; the registers
  // allow 16 warps).
  auto in_batch = [&](int n) { return (int)std::min<int64_t>(lines, (int64_t)n * a.plane_lines); };
  auto bytes = [&](int n, int l) {
    const size_t sums = (size_t)l * L::COUNT * value, head = a.cells.tab_bytes + a.dftab_bytes + n * S::PLANE * value;
    return head + (n >= planes ? std::max(nodes, sums) : nodes + sums);
  };
  a.batch = planes;
  while (a.batch > 1 && bytes(a.batch, in_batch(a.batch)) > 30 * 1024) a.batch = std::min(a.batch - 1, (a.batch + 1) / 2);
  a.chunk = in_batch(a.batch);
  while (a.chunk > 8 && bytes(a.batch, a.chunk) > 64 * 1024) a.chunk = (a.chunk + 1) / 2;
  a.alias = a.batch >= planes ? 1 : 0;
  const size_t smem = bytes(a.batch, a.chunk);
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t ctas = (a.padded + 15) / 16;
  // CTAs of 64 threads (few threads at a barrier, many CTAs), or of 96 where a batch's (point, pair)
  // items then idle fewer: P2 tetrahedra at 24 points 64 / 96 / 128 threads 0.99 / 1.04 / 1.13 ms (786,432
  // cells), Q2 hexahedra at 27 points 1.67 / 1.37 / 1.51 (500,000).
  const int64_t items = ((int64_t)a.num_points * a.batch + planes - 1) / planes * 8;
  const int threads = (items + 63) / 64 * 64 <= (items + 95) / 96 * 96 ? 64 : 96;
  kern<<<(unsigned)ctas, threads, smem, s>>>(a);
  return cudaGetLastError();
}

// Defined in eval_dfpoly.cu: `found` is false where no kernel is compiled for the cell.
cudaError_t launch_eval_dfpoly(int cell, int degree, const PolyDfArgs& a, int lines, cudaStream_t s, bool* found);

}  // namespace tlg
