// The polynomial pull-back kernels of mixed precision (f64 meshes).
#include "pullback_poly.cuh"

namespace tlg {

cudaError_t launch_pull_back_poly_split(int cell, int degree, int gd, const PullBackArgs& p, const PolyTerms& terms,
                                        cudaStream_t s, bool* found) {
  const PolyArgs a = {p, terms};
  *found = true;
#define TLG_X(CELL, P, GD) \
  if (cell == CELL && degree == P && gd == GD) \
    return launch_poly(pull_back_poly_split_kernel<CELL, P, GD>, a, poly_smem<CELL, P, GD>(sizeof(double)), s);
  TLG_POLY_CELLS(TLG_X)
#undef TLG_X
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
