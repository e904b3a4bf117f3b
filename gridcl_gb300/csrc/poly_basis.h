// Polynomial (monomial) form of a cell's map: the expansion of the Lagrange functions and the
// line structure of a point set, host side, shared by the pull-back's and the f64 evaluation's
// polynomial kernels.
#pragma once

#include <cstdint>
#include <vector>

namespace tlg {

// C by rows: row m's nonzero terms are term[start[m] .. start[m + 1]).
struct PolyTerm {
  double c;
  int k, pad;
};
struct PolyTerms {
  const uint32_t* start;
  const PolyTerm* term;
};

// A coordinate value with what it heads: a plane (z; its lines), a line (y; its points, its plane)
// or a point (x; `first` its index in the point set, `plane` its line). t is the value about the direction's centre,
// e_2(t) = t s1, e_2'(t) = s2; mid: t = 0 (an integer, as a comparison of doubles takes the FP64 pipe).
struct PolyNode {
  double t, s1, s2;
  int first, count, plane, mid;
};
static_assert(sizeof(PolyNode) == 40 && sizeof(PolyTerm) == 16, "table strides");

// The bases of a direction. Simplex directions: t^i about vertex 0. Tensor directions (all of
// tensor cells, z of prisms): kCentred t^i about 1/2; kLine about 1/2 with e_2 = 2 t^2 at degree 2
// (so that the coefficients of three nodes are u_1, u_2 - u_0, u_0 - 2 u_1 + u_2), t^i about 0 at
// degree 1.
enum PolyBasis { kCentred, kLine };

// C [m][k] (m-major) with Lagrange function k = sum_m C[m][k] e_m, e_m = e_a(x) e_b(y) e_c(z), a
// fastest, |a| <= degree on simplices, a + b <= degree on prisms: C = V^-1, V[j][m] = e_m(node j),
// by Gauss-Jordan with partial pivoting, checked by V C = I to 1e-12. Empty for other cells or
// when the check fails.
std::vector<double> poly_expansion(int cell, int degree, const std::vector<double>& nodes, PolyBasis basis);

// The point set in planes (equal z; one plane in 2D) of lines (equal y) of points, in order of
// first appearance; lines of more than kPolyLine points in near-equal parts. Empty when a coordinate is
// not finite: such a point shares no line (NaN has no order), and its values are the tabulation's.
constexpr int kPolyLine = 4;
struct PolyRule {
  std::vector<PolyNode> planes, lines, points;
};
PolyRule poly_rule(int cell, int degree, const double* points, int64_t npoints);

}  // namespace tlg
