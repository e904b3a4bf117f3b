// Instantiations of the double-float polynomial evaluation.
#include "eval_dfpoly.cuh"

namespace tlg {

cudaError_t launch_eval_dfpoly(int cell, int degree, const PolyDfArgs& a, int lines, cudaStream_t s, bool* found) {
  *found = true;
#define TLG_X(CELL, P) \
  if (cell == CELL && degree == P) return launch_dfpoly_cell<CELL, P>(a, lines, s);
  TLG_X(kTetrahedron, 1)
  TLG_X(kTetrahedron, 2)
  TLG_X(kTetrahedron, 3)
  TLG_X(kHexahedron, 1)
  TLG_X(kHexahedron, 2)
  TLG_X(kPrism, 1)
  TLG_X(kPrism, 2)
#undef TLG_X
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
