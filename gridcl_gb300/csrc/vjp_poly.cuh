// The f64 adjoint (vjp.cuh has its formulas) of volume cells on the polynomial form of their map
// (eval_poly.cuh): tetrahedra P1-P3, hexahedra Q1-Q2 and prisms P1-P2 in 3D, triangles P1-P3 and
// quadrilaterals Q1-Q2 in the plane.
//
// The forward stages are eval_poly_kernel's, so the fused forward fields have its bits. The
// cotangents run through the same stages transposed:
//   point  A~_a += e_a(x) x~ + e_a'(x) J~_0,  D~_a += e_a(x) J~_1,  E~_a += e_a(x) J~_2,
//   line   P~_ab += e_b(y) A~_a + e_b'(y) D~_a,  Q~_ab += e_b(y) E~_a,
//   plane  c~_abc += e_c(z) P~_ab + e_c'(z) Q~_ab,
//   cell   L(k) = sum_m C[m][k] c~_m,
// J~ = K^T (d~ det J - K~ K^T). One item per (line, cell) walks the line's points with the line's
// sums and their cotangents in registers; the cotangents then go through shared memory to one item
// per (b, coordinate, cell) and to the rows. Every sum runs in the order of the lines, the planes
// and the expansion's terms: deterministic.
//
// Bound by the FP64 pipe. Per point of a Q2 hexahedron at 27 points about 200 FP64 operations with
// the forward fields, against 360 of the sum factorisation in the Lagrange basis with one cell per
// thread (255 registers and spills). GB300, forward and adjoint with the node sums, ms:
// 110,592 Q2 hexahedra at 27 points 1.82 -> 1.26; 60,000 cells: P2 tetrahedra at 24 points 2.12 -> 0.52,
// P2 prisms at 21 points 2.28 -> 0.79, Q1 hexahedra at 8 points 0.257 -> 0.191; 1,000 P1 tetrahedra at 8
// points 0.074 -> 0.054. FP64 pipe 86 % active on the hexahedra.
#pragma once

#include "eval_poly.cuh"
#include "vjp.cuh"

namespace tlg {

struct VjpPolyArgs {
  PolyCells cells;
  const double* ct[3];  // cotangents: points, detj, pinv (tile 16) or null
  double* out[4];       // fused forward fields: points, jacobian, detj, pinv, or null
  double* local;        // contributions [cell][K][R]
  int64_t padded, out_first_cell, range_end;
  double origin[3];
  uint32_t off_planes, off_lines, off_points, off_tterms, off_tstarts;  // (tterms, tstarts: by column)
  int num_points, num_planes, rule_global;
  int plane_lines;  // the most lines of a plane
  int batch, chunk;  // planes whose sums are held, lines whose cotangents are held at a time
  int alias;         // a batch's lines are one round of items: their cotangents go over the planes' sums
};

// e_i and e_i' of a node, i <= P (the products with t formed once).
template <int P>
struct PolyE {
  double e[P + 1], d[P + 1];
  __device__ __forceinline__ PolyE(const PolyAt& u) {
    e[0] = 1.0;
    d[0] = 0.0;
    e[1] = u.t;
    d[1] = 1.0;
    if constexpr (P >= 2) {
      e[2] = __dmul_rn(u.t, u.s1);
      d[2] = u.s2;
    }
    if constexpr (P >= 3) {
      e[3] = __dmul_rn(e[2], u.t);
      d[3] = __dmul_rn(3.0, e[2]);
    }
  }
};

template <int CELL, int P>
struct VjpPolyShape {
  using S = PolySpace<CELL, P>;
  static constexpr int GD = S::TD, R = GD == 3 ? 4 : GD;
  // A line's cotangents per coordinate: A~ (P + 1), D~, and in 3D E~.
  static constexpr int NB = P + 1 + S::DA + 1 + (S::TD == 3 ? S::EA + 1 : 0);
};

// A point's part of the line's cotangents. AT_MID: t = 0, where only e_0 and e_1' are left.
template <int CELL, int P, bool AT_MID>
__device__ __forceinline__ void poly_point_bar(const PolyAt& x, bool has_x, const double* xb, const double* jb,
                                               double (*A)[P + 1], double (*D)[PolySpace<CELL, P>::DA + 1],
                                               double (*E)[PolySpace<CELL, P>::EA + 1]) {
  using S = PolySpace<CELL, P>;
  constexpr int GD = S::TD;
  if constexpr (AT_MID) {
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      if (has_x) A[g][0] = __dadd_rn(A[g][0], xb[g]);
      A[g][1] = __dadd_rn(A[g][1], jb[g]);
      D[g][0] = __dadd_rn(D[g][0], jb[GD + g]);
      if constexpr (GD == 3) E[g][0] = __dadd_rn(E[g][0], jb[2 * GD + g]);
    }
  } else {
    const PolyE<P> u(x);
#pragma unroll
    for (int g = 0; g < GD; ++g) {
      if (has_x) {
        A[g][0] = __dadd_rn(A[g][0], xb[g]);
#pragma unroll
        for (int a = 1; a <= P; ++a) A[g][a] = fma(u.e[a], xb[g], A[g][a]);
      }
      A[g][1] = __dadd_rn(A[g][1], jb[g]);
#pragma unroll
      for (int a = 2; a <= P; ++a) A[g][a] = fma(u.d[a], jb[g], A[g][a]);
      D[g][0] = __dadd_rn(D[g][0], jb[GD + g]);
#pragma unroll
      for (int a = 1; a <= S::DA; ++a) D[g][a] = fma(u.e[a], jb[GD + g], D[g][a]);
      if constexpr (GD == 3) {
        E[g][0] = __dadd_rn(E[g][0], jb[2 * GD + g]);
#pragma unroll
        for (int a = 1; a <= S::EA; ++a) E[g][a] = fma(u.e[a], jb[2 * GD + g], E[g][a]);
      }
    }
  }
}

template <int CELL, int P, int W>
__global__ void __launch_bounds__(192, 2) vjp_poly_kernel(const __grid_constant__ VjpPolyArgs a) {
  using S = PolySpace<CELL, P>;
  using V = VjpPolyShape<CELL, P>;
  constexpr int TD = S::TD, GD = TD, K = S::K, N = S::N, R = V::R, NB = V::NB, LJ = TD * GD;
  constexpr bool MID = !S::kTri && P == 2, MIDZ = !S::kTet && P == 2, TENSOR = S::kTensor;
  constexpr int REF = TENSOR && N == 3 ? K / 2 : 0;
  constexpr int COL = GD * W;  // (coordinate, cell) columns
  __shared__ uint64_t bar;
  extern __shared__ __align__(16) unsigned char smem[];
  double* ys = reinterpret_cast<double*>(smem + a.cells.tab_bytes);
  double* cs = TENSOR ? ys : ys + K * COL;
  double* cb = cs + K * COL;            // c~ [K][GD][W]
  double* pl = cb + K * COL;            // [batch][PLANE][GD][W]
  double* lb = TD == 3 && !a.alias ? pl + (size_t)a.batch * (S::PLANE * COL) : pl;  // [chunk][NB][GD][W]
  const unsigned char* rule = a.rule_global ? a.cells.tab : smem;
  const PolyNode* planes = reinterpret_cast<const PolyNode*>(rule + a.off_planes);
  const PolyNode* lines = reinterpret_cast<const PolyNode*>(rule + a.off_lines);
  const PolyNode* points = reinterpret_cast<const PolyNode*>(rule + a.off_points);
  const uint32_t* starts = reinterpret_cast<const uint32_t*>(smem + a.cells.off_starts);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int64_t c0 = (int64_t)blockIdx.x * W;
  for (int i = tid; i < K * COL; i += nt) cb[i] = 0.0;
  if (!poly_coefficients<CELL, P, GD, W>(a.cells, c0, smem, &bar, ys, cs)) return;

  const int nq = a.num_points;
  const bool has_x = a.ct[0] != nullptr, want_x = a.out[0] != nullptr;
  for (int p0 = 0; p0 < a.num_planes; p0 += a.batch) {
    const int np = min(a.batch, a.num_planes - p0);
    if constexpr (TD == 3) {
      for (int i = tid; i < np * COL; i += nt) {
        const int e = i % COL, p = i / COL;
        const PolyAt z(planes[p0 + p]);
        double* o = pl + (size_t)p * (S::PLANE * COL) + e;
        if (MIDZ && z.mid) poly_plane<CELL, P, COL, MIDZ>(cs + e, z, true, o);
        else poly_plane<CELL, P, COL, false>(cs + e, z, true, o);
      }
      __syncthreads();
    }
    const int l0 = planes[p0].first, l1 = planes[p0 + np - 1].first + planes[p0 + np - 1].count;
    for (int lc = l0; lc < l1; lc += a.chunk) {
      const int nl = min(a.chunk, l1 - lc);
      for (int i0 = 0; i0 < nl * W; i0 += nt) {
        const int i = i0 + tid, lane = i % W;
        const int64_t c = c0 + lane;
        const bool active = i < nl * W && c < a.padded;
        double Ab[GD][N], Db[GD][S::DA + 1], Eb[GD][S::EA + 1];
        if (active) {
          const PolyNode& ln = lines[lc + i / W];
          const PolyAt y(ln);
          const double* sums = TD == 3 ? pl + (size_t)(ln.plane - p0) * (S::PLANE * COL) + lane : cs + lane;
          double A[GD][N], D[GD][S::DA + 1], E[GD][S::EA + 1];
          if (MID && y.mid) poly_line<CELL, P, GD, W, MID>(sums, y, true, A, D, E);
          else poly_line<CELL, P, GD, W, false>(sums, y, true, A, D, E);
#pragma unroll
          for (int g = 0; g < GD; ++g) {
#pragma unroll
            for (int x = 0; x < N; ++x) Ab[g][x] = 0.0;
#pragma unroll
            for (int x = 0; x <= S::DA; ++x) Db[g][x] = 0.0;
#pragma unroll
            for (int x = 0; x <= S::EA; ++x) Eb[g][x] = 0.0;
          }
          const int64_t o = a.out_first_cell + c;
          const int64_t tq = o / 16 * nq;
          const int l16 = (int)(o % 16);
          double xo[GD];
          if (want_x) {
            const uint32_t* row = a.cells.dofmap + min(a.cells.first_cell + c, a.cells.last_cell) * K;
            const int64_t n0 = min(__ldg(row + (TENSOR ? starts[REF] : 0)), a.cells.last_node);
#pragma unroll
            for (int g = 0; g < GD; ++g) xo[g] = __dadd_rn(__ldg(a.cells.nodes + n0 * GD + g), a.origin[g]);
          }
          for (int e = 0; e < ln.count; ++e) {
            const PolyNode& pt = points[ln.first + e];
            const PolyAt x(pt);
            const int64_t q = tq + pt.first;
            // The cotangents first: they arrive while the forward stage runs.
            double xb[GD], kb[LJ], db = 0.0;
            if (has_x)
#pragma unroll
              for (int g = 0; g < GD; ++g) xb[g] = __ldg(a.ct[0] + (q * GD + g) * 16 + l16);
            if (a.ct[1]) db = __ldg(a.ct[1] + q * 16 + l16);
            if (a.ct[2])
#pragma unroll
              for (int r = 0; r < LJ; ++r) kb[r] = __ldg(a.ct[2] + (q * LJ + r) * 16 + l16);
            double xp[GD], j[LJ], kk[LJ], dj;
            if (MID && x.mid) poly_point<CELL, P, GD, MID>(x, want_x, true, A, D, E, xp, j);
            else poly_point<CELL, P, GD, false>(x, want_x, true, A, D, E, xp, j);
            poly_square<TD>(j, true, dj, kk);
            if (want_x)
#pragma unroll
              for (int g = 0; g < GD; ++g) a.out[0][(q * GD + g) * 16 + l16] = __dadd_rn(xp[g], xo[g]);
            if (a.out[1])
#pragma unroll
              for (int r = 0; r < LJ; ++r) a.out[1][(q * LJ + r) * 16 + l16] = j[r];
            if (a.out[2]) a.out[2][q * 16 + l16] = dj;
            if (a.out[3])
#pragma unroll
              for (int r = 0; r < LJ; ++r) a.out[3][(q * LJ + r) * 16 + l16] = kk[r];
            // J~(g, d) = sum_t K(t, g) (delta_td d~ det J - sum_h K~(t, h) K(d, h)).
            const double s = __dmul_rn(db, dj);
            double jb[LJ];
            if (a.ct[2]) {
              double m[LJ];  // (t, d) at t TD + d
#pragma unroll
              for (int t = 0; t < TD; ++t)
#pragma unroll
                for (int d = 0; d < TD; ++d) {
                  double v = t == d ? s : 0.0;
#pragma unroll
                  for (int h = 0; h < GD; ++h)
                    v = t != d && h == 0 ? __dmul_rn(-kb[t], kk[d]) : fma(-kb[h * TD + t], kk[h * TD + d], v);
                  m[t * TD + d] = v;
                }
#pragma unroll
              for (int d = 0; d < TD; ++d)
#pragma unroll
                for (int g = 0; g < GD; ++g) {
                  double v = __dmul_rn(kk[g * TD], m[d]);
#pragma unroll
                  for (int t = 1; t < TD; ++t) v = fma(kk[g * TD + t], m[t * TD + d], v);
                  jb[d * GD + g] = v;
                }
            } else {
#pragma unroll
              for (int d = 0; d < TD; ++d)
#pragma unroll
                for (int g = 0; g < GD; ++g) jb[d * GD + g] = __dmul_rn(s, kk[g * TD + d]);
            }
            // A cotangent that is not finite reaches every node of the cell, as through the Lagrange functions (0
            // times NaN), also from a middle point, whose low coefficients only some nodes are in: the highest
            // coefficient is in every node's row.
            if constexpr (TENSOR && N == 3) {
#pragma unroll
              for (int g = 0; g < GD; ++g) {
                bool bad = has_x && poly_bad(xb[g]);
#pragma unroll
                for (int d = 0; d < TD; ++d) bad = bad || poly_bad(jb[d * GD + g]);
                if (bad) cb[((K - 1) * GD + g) * W + lane] = poly_nan();
              }
            }
            if (MID && x.mid) poly_point_bar<CELL, P, MID>(x, has_x, xb, jb, Ab, Db, Eb);
            else poly_point_bar<CELL, P, false>(x, has_x, xb, jb, Ab, Db, Eb);
          }
        }
        if (a.alias) __syncthreads();  // every item has read its plane's sums
        if (!active) continue;
        double* out = lb + (size_t)(i / W) * (NB * COL) + lane;
#pragma unroll
        for (int g = 0; g < GD; ++g) {
          int r = 0;
#pragma unroll
          for (int x = 0; x < N; ++x) out[(r++ * GD + g) * W] = Ab[g][x];
#pragma unroll
          for (int x = 0; x <= S::DA; ++x) out[(r++ * GD + g) * W] = Db[g][x];
          if constexpr (TD == 3)
#pragma unroll
            for (int x = 0; x <= S::EA; ++x) out[(r++ * GD + g) * W] = Eb[g][x];
        }
      }
      __syncthreads();
      // The chunk's lines into c~, one (b, coordinate, cell) per item.
      for (int i = tid; i < N * COL; i += nt) {
        const int col = i % COL, b = i / COL;
        const int pa = S::kTri ? P - b : P, qa = S::kTet ? P - 1 - b : pa;  // highest a of P~_ab, Q~_ab
        for (int p = p0; p < p0 + np; ++p) {
          const int f0 = max(planes[p].first, lc), f1 = min(planes[p].first + planes[p].count, lc + nl);
          if (f0 >= f1) continue;
          double Pb[N], Qb[N];
#pragma unroll
          for (int x = 0; x < N; ++x) Pb[x] = Qb[x] = 0.0;
          for (int l = f0; l < f1; ++l) {
            const PolyNode& ln = lines[l];
            const PolyAt y(ln);
            const double* in = lb + (size_t)(l - lc) * (NB * COL) + col;
            const double* dl = in + N * COL;
            const double* el = dl + (S::DA + 1) * COL;
            if (b == 0) {
#pragma unroll
              for (int x = 0; x < N; ++x) Pb[x] = __dadd_rn(Pb[x], in[x * COL]);
              if constexpr (TD == 3)
#pragma unroll
                for (int x = 0; x <= S::EA; ++x) Qb[x] = __dadd_rn(Qb[x], el[x * COL]);
            } else if (MID && ln.mid) {  // e_b = 0, e_1' = 1, e_2' = 0
              if (b == 1)
#pragma unroll
                for (int x = 0; x <= S::DA; ++x) Pb[x] = __dadd_rn(Pb[x], dl[x * COL]);
            } else {
              const PolyE<P> u(y);
              double eb = u.e[1], de = u.d[1];
#pragma unroll
              for (int m = 2; m <= P; ++m) {
                eb = b == m ? u.e[m] : eb;
                de = b == m ? u.d[m] : de;
              }
#pragma unroll
              for (int x = 0; x < N; ++x)
                if (x <= pa) {
                  Pb[x] = fma(eb, in[x * COL], Pb[x]);
                  if (x <= S::DA) Pb[x] = b == 1 ? __dadd_rn(Pb[x], dl[x * COL]) : fma(de, dl[x * COL], Pb[x]);
                }
              if constexpr (TD == 3)
#pragma unroll
                for (int x = 0; x <= S::EA; ++x)
                  if (x <= qa) Qb[x] = fma(eb, el[x * COL], Qb[x]);
            }
          }
          if constexpr (TD == 3) {
            const PolyAt z(planes[p]);
            const PolyE<P> u(z);
#pragma unroll
            for (int x = 0; x < N; ++x)
              if (x <= pa) {
#pragma unroll
                for (int l = 0; l < N; ++l) {
                  if (S::kTet && l > P - x - b) continue;
                  double* v = cb + S::ci(x, b, l) * COL + col;
                  if (l == 0) *v = __dadd_rn(*v, Pb[x]);
                  else if (MIDZ && z.mid) {
                    if (l == 1) *v = __dadd_rn(*v, Qb[x]);
                  } else {
                    const double w = fma(u.e[l], Pb[x], *v);
                    *v = l == 1 ? __dadd_rn(w, Qb[x]) : fma(u.d[l], Qb[x], w);
                  }
                }
              }
          } else {
#pragma unroll
            for (int x = 0; x < N; ++x)
              if (x <= pa) {
                double* v = cb + S::pi(x, b) * COL + col;
                *v = __dadd_rn(*v, Pb[x]);
              }
          }
        }
      }
      __syncthreads();
    }
  }
  // The rows L(k) = sum_m C[m][k] c~_m.
  if constexpr (TENSOR) {
    // The transposed directions, in place: (q_0, q_1) of (u_0, u_1 - u_0), or (r, s, t) of (u_1, u_2 -
    // u_0, u_0 - 2 u_1 + u_2).
    for (int i = tid; i < COL; i += nt) {
      double u[K];
#pragma unroll
      for (int m = 0; m < K; ++m) u[m] = cb[m * COL + i];
#pragma unroll
      for (int d = TD - 1; d >= 0; --d) {
        const int st = d == 0 ? 1 : d == 1 ? N : N * N;
#pragma unroll
        for (int l = 0; l < K / N; ++l) {
          const int o = l % st + l / st * (st * N);
          if constexpr (N == 2) {
            u[o] = __dsub_rn(u[o], u[o + st]);
          } else {
            const double p = u[o], q = u[o + st], r = u[o + 2 * st];
            u[o] = __dsub_rn(r, q);
            u[o + st] = fma(-2.0, r, p);
            u[o + 2 * st] = __dadd_rn(r, q);
          }
        }
      }
#pragma unroll
      for (int m = 0; m < K; ++m) cb[m * COL + i] = u[m];
    }
    __syncthreads();
  }
  const PolyTerm* tterms = reinterpret_cast<const PolyTerm*>(smem + a.off_tterms);
  const uint32_t* tstarts = reinterpret_cast<const uint32_t*>(smem + a.off_tstarts);
  for (int i = tid; i < K * W; i += nt) {
    const int lane = i % W, k = i / W;
    const int64_t cell = a.cells.first_cell + c0 + lane;
    if (cell >= a.range_end) continue;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    int node = k;
    if constexpr (TENSOR) {
      node = (int)starts[k];
#pragma unroll
      for (int g = 0; g < GD; ++g) v[g] = cb[(k * GD + g) * W + lane];
    } else {
      for (uint32_t e = tstarts[k]; e < tstarts[k + 1]; ++e) {
        const double c = tterms[e].c;
        const int m = tterms[e].k;
#pragma unroll
        for (int g = 0; g < GD; ++g) v[g] = fma(c, cb[(m * GD + g) * W + lane], v[g]);
      }
    }
    double* row = a.local + (cell * K + node) * R;
    if constexpr (R == 4) Vec4<double>::put(row, v[0], v[1], v[2], v[3]);
    else
#pragma unroll
      for (int g = 0; g < GD; ++g) row[g] = v[g];
  }
}

template <int CELL, int P, int W>
inline cudaError_t launch_vjp_poly_width(VjpPolyArgs a, int lines, cudaStream_t s) {
  using S = PolySpace<CELL, P>;
  using V = VjpPolyShape<CELL, P>;
  auto kern = vjp_poly_kernel<CELL, P, W>;
  // Planes and lines held at a time: as many as keep three CTAs on an SM (72 KiB each); a batch whose
  // lines are one round of items puts their cotangents over the planes' sums.
  const size_t col = (size_t)V::GD * W * 8, fixed = a.cells.tab_bytes + (size_t)(S::kTensor ? 2 : 3) * S::K * col;
  const size_t plane = S::TD == 3 ? S::PLANE * col : 0, line = V::NB * col, budget = 72 * 1024;
  const int planes = std::max(a.num_planes, 1);
  auto in_batch = [&](int n) { return S::TD == 3 ? (int)std::min<int64_t>(lines, (int64_t)n * a.plane_lines) : lines; };
  auto bytes = [&](int n, int l) {
    const bool over = l * W <= 192 && l >= in_batch(n);
    return fixed + (over ? std::max(n * plane, l * line) : n * plane + l * line);
  };
  a.batch = 1;
  while (S::TD == 3 && a.batch < planes && bytes(a.batch + 1, in_batch(a.batch + 1)) <= budget) ++a.batch;
  if (S::TD == 3) {  // batches of equal size
    const int batches = (planes + a.batch - 1) / a.batch;
    a.batch = (planes + batches - 1) / batches;
  }
  a.chunk = in_batch(a.batch);
  while (a.chunk > 2 && bytes(a.batch, a.chunk) > budget) --a.chunk;
  a.alias = S::TD == 3 && a.chunk * W <= 192 && a.chunk >= in_batch(a.batch) ? 1 : 0;
  const size_t smem = bytes(a.batch, a.chunk);
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return e;
  const int64_t ctas = (a.padded + W - 1) / W;
  kern<<<(unsigned)ctas, poly_line_threads(a.chunk * W, 192), smem, s>>>(a);
  return cudaGetLastError();
}

// Defined in vjp_poly.cu: `found` is false where no kernel is compiled for the cell.
cudaError_t launch_vjp_poly(int cell, int degree, const VjpPolyArgs& a, int lines, cudaStream_t s, bool* found);

}  // namespace tlg
