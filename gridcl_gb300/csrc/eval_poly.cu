// Instantiations of the f64 polynomial evaluation.
#include "eval_poly.cuh"

namespace tlg {

cudaError_t launch_eval_poly(int cell, int degree, int gd, const PolyEvalArgs& a, int lines, cudaStream_t s,
                             bool* found) {
  *found = true;
#define TLG_X(CELL, P, GD) \
  if (cell == CELL && degree == P && gd == GD) return launch_poly_cell<CELL, P, GD>(a, lines, s);
  TLG_X(kTetrahedron, 1, 3)
  TLG_X(kTetrahedron, 2, 3)
  TLG_X(kTetrahedron, 3, 3)
  TLG_X(kHexahedron, 1, 3)
  TLG_X(kHexahedron, 2, 3)
  TLG_X(kPrism, 1, 3)
  TLG_X(kPrism, 2, 3)
  TLG_X(kTriangle, 1, 2)
  TLG_X(kTriangle, 2, 2)
  TLG_X(kTriangle, 3, 2)
  TLG_X(kTriangle, 1, 3)
  TLG_X(kTriangle, 2, 3)
  TLG_X(kTriangle, 3, 3)
  TLG_X(kQuadrilateral, 1, 2)
  TLG_X(kQuadrilateral, 2, 2)
  TLG_X(kQuadrilateral, 1, 3)
  TLG_X(kQuadrilateral, 2, 3)
#undef TLG_X
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
