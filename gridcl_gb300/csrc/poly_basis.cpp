#include "poly_basis.h"

#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <utility>

#include "refcell.h"

namespace tlg {

namespace {

bool simplex_direction(int cell, int d) {
  return cell == kTriangle || cell == kTetrahedron || (cell == kPrism && d < 2);
}

// e_i(t) and the node values of a direction at x.
PolyNode poly_node(int cell, int degree, int d, double x, PolyBasis basis) {
  PolyNode n = {};
  const bool tensor = !simplex_direction(cell, d);
  n.t = x - (tensor && (basis == kCentred || degree > 1) ? 0.5 : 0.0);
  const double s = tensor && basis == kLine && degree == 2 ? 2.0 : 1.0;
  n.s1 = s * n.t;
  n.s2 = 2.0 * s * n.t;
  n.mid = n.t == 0.0 ? 1 : 0;
  return n;
}

double poly_e(const PolyNode& n, int i) {
  if (i == 0) return 1.0;
  if (i == 1) return n.t;
  if (i == 2) return n.t * n.s1;
  return std::pow(n.t, i);
}

}  // namespace

std::vector<double> poly_expansion(int cell, int degree, const std::vector<double>& nodes, PolyBasis basis) {
  const int td = tdim(cell);
  if (degree < 1 || degree > 3 || td < 2 || cell == kPyramid) return {};
  const bool simplex = cell == kTriangle || cell == kTetrahedron, prism = cell == kPrism;
  std::vector<std::array<int, 3>> ex;
  for (int c = 0; c <= (td == 3 ? degree : 0); ++c)
    for (int b = 0; b <= degree - (simplex ? c : 0); ++b)
      for (int a = 0; a <= degree - (simplex ? b + c : prism ? b : 0); ++a) ex.push_back({a, b, c});
  const size_t k = ex.size();
  if (nodes.size() != k * td) return {};
  std::vector<double> V(k * k), w(k * 2 * k, 0.0);
  for (size_t j = 0; j < k; ++j) {
    PolyNode n[3];
    for (int d = 0; d < td; ++d) n[d] = poly_node(cell, degree, d, nodes[j * td + d], basis);
    for (size_t m = 0; m < k; ++m) {
      double v = 1.0;
      for (int d = 0; d < td; ++d) v *= poly_e(n[d], ex[m][d]);
      V[j * k + m] = w[j * 2 * k + m] = v;
    }
    w[j * 2 * k + k + j] = 1.0;
  }
  for (size_t c = 0; c < k; ++c) {
    size_t piv = c;
    for (size_t r = c + 1; r < k; ++r)
      if (std::fabs(w[r * 2 * k + c]) > std::fabs(w[piv * 2 * k + c])) piv = r;
    if (std::fabs(w[piv * 2 * k + c]) < 1e-12) return {};
    if (piv != c)
      for (size_t e = 0; e < 2 * k; ++e) std::swap(w[piv * 2 * k + e], w[c * 2 * k + e]);
    const double inv = 1.0 / w[c * 2 * k + c];
    for (size_t e = 0; e < 2 * k; ++e) w[c * 2 * k + e] *= inv;
    for (size_t r = 0; r < k; ++r) {
      const double f = w[r * 2 * k + c];
      if (r == c || f == 0.0) continue;
      for (size_t e = 0; e < 2 * k; ++e) w[r * 2 * k + e] -= f * w[c * 2 * k + e];
    }
  }
  std::vector<double> C(k * k);
  for (size_t m = 0; m < k; ++m)
    for (size_t i = 0; i < k; ++i) {
      // Most entries are small multiples of 1/8: the elimination's errors rounded off.
      const double v = w[m * 2 * k + k + i], r = std::round(8.0 * v) / 8.0;
      C[m * k + i] = std::fabs(v - r) < 1e-11 ? r : v;
    }
  for (size_t j = 0; j < k; ++j)
    for (size_t i = 0; i < k; ++i) {
      double v = 0.0;
      for (size_t m = 0; m < k; ++m) v += V[j * k + m] * C[m * k + i];
      if (!(std::fabs(v - (i == j ? 1.0 : 0.0)) < 1e-12)) return {};
    }
  return C;
}

PolyRule poly_rule(int cell, int degree, const double* points, int64_t npoints) {
  const int td = tdim(cell);
  for (int64_t i = 0; i < npoints * td; ++i)
    if (!std::isfinite(points[i])) return {};
  // Planes by z, lines by (z, y), in order of first appearance.
  struct Line {
    double y;
    std::vector<int> q;
  };
  struct Plane {
    double z;
    std::vector<Line> lines;
  };
  std::vector<Plane> planes;
  std::map<double, size_t> plane_of;
  std::map<std::pair<double, double>, size_t> line_of;
  for (int64_t q = 0; q < npoints; ++q) {
    const double* p = points + q * td;
    const double z = td == 3 ? p[2] : 0.0;
    const auto pi = plane_of.emplace(z, planes.size());
    if (pi.second) planes.push_back({z, {}});
    Plane& pl = planes[pi.first->second];
    const auto li = line_of.emplace(std::make_pair(z, p[1]), pl.lines.size());
    if (li.second) pl.lines.push_back({p[1], {}});
    pl.lines[li.first->second].q.push_back((int)q);
  }
  PolyRule r;
  for (size_t i = 0; i < planes.size(); ++i) {
    PolyNode pn = poly_node(cell, degree, 2, planes[i].z, kLine);
    pn.first = (int)r.lines.size();
    for (const Line& l : planes[i].lines) {
      const int n = (int)l.q.size(), parts = (n + kPolyLine - 1) / kPolyLine;
      for (int s = 0, at = 0; s < parts; ++s) {
        const int len = (n - at + parts - s - 1) / (parts - s);
        PolyNode ln = poly_node(cell, degree, 1, l.y, kLine);
        ln.first = (int)r.points.size();
        ln.count = len;
        ln.plane = (int)i;
        for (int e = 0; e < len; ++e) {
          PolyNode pt = poly_node(cell, degree, 0, points[l.q[at + e] * td], kLine);
          pt.first = l.q[at + e];
          pt.plane = (int)r.lines.size();
          r.points.push_back(pt);
        }
        r.lines.push_back(ln);
        at += len;
      }
    }
    pn.count = (int)r.lines.size() - pn.first;
    r.planes.push_back(pn);
  }
  return r;
}

}  // namespace tlg
