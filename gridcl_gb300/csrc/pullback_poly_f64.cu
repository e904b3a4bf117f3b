// The polynomial pull-back kernels of f64 meshes.
#include "pullback_poly.cuh"

namespace tlg {

cudaError_t launch_pull_back_poly_f64(int cell, int degree, int gd, const PullBackArgs& p, const PolyTerms& terms,
                                      cudaStream_t s, bool* found) {
  const PolyArgs a = {p, terms};
  *found = true;
#define TLG_X(CELL, P, GD) \
  if (cell == CELL && degree == P && gd == GD) \
    return launch_poly(pull_back_poly_kernel<double, CELL, P, GD>, a, poly_smem<CELL, P, GD>(sizeof(double)), s);
  TLG_POLY_CELLS(TLG_X)
#undef TLG_X
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
