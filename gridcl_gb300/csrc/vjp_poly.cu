// Instantiations of the f64 polynomial adjoint.
#include "vjp_poly.cuh"

namespace tlg {

// 32 cells per CTA for the cells whose kernels leave out a middle point's terms, as the evaluation
// (launch_poly_cell), 16 for the others and on meshes that do not fill the SMs with 32.
template <int CELL, int P>
static cudaError_t launch_cell(const VjpPolyArgs& a, int lines, cudaStream_t s) {
  if constexpr (P == 2 && (CELL == kHexahedron || CELL == kPrism || CELL == kQuadrilateral)) {
    if (a.padded >= (int64_t)64 * poly_sms()) return launch_vjp_poly_width<CELL, P, 32>(a, lines, s);
  }
  return launch_vjp_poly_width<CELL, P, 16>(a, lines, s);
}

cudaError_t launch_vjp_poly(int cell, int degree, const VjpPolyArgs& a, int lines, cudaStream_t s, bool* found) {
  *found = true;
#define TLG_X(CELL, P) \
  if (cell == CELL && degree == P) return launch_cell<CELL, P>(a, lines, s);
  TLG_X(kTetrahedron, 1)
  TLG_X(kTetrahedron, 2)
  TLG_X(kTetrahedron, 3)
  TLG_X(kHexahedron, 1)
  TLG_X(kHexahedron, 2)
  TLG_X(kPrism, 1)
  TLG_X(kPrism, 2)
  TLG_X(kTriangle, 1)
  TLG_X(kTriangle, 2)
  TLG_X(kTriangle, 3)
  TLG_X(kQuadrilateral, 1)
  TLG_X(kQuadrilateral, 2)
#undef TLG_X
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
