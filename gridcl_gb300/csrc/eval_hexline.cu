// Instantiations of the FP32 line kernel of hexahedra.
#include "eval_hexline.cuh"

namespace tlg {

template <bool SPLIT, int P>
static cudaError_t launch_degree(const HexLineArgs& a, cudaStream_t s) {
  const size_t smem = a.tab_bytes + (size_t)(P + 1) * (P + 1) * (P + 1) * 3 * kEvalThreads * 4;
  // One step per CTA for f32 Q1 where a cell stores 120 values and more (1,331,000 cells at 8 points, ms,
  // persistent / one step: four factors 0.174 / 0.152, at 6 points 0.133 / 0.125, but det J alone 0.051 / 0.060, det J and K 0.091 / 0.096; at 27
  // points det J and K 0.259 / 0.224); f32 Q2 at 27 points is even (500,000 cells 0.239 / 0.232, 100,000 0.061 /
  // 0.065), split precision slower (Q2 0.338 / 0.352, Q1 0.216 / 0.261).
  const int len[4] = {3, 9, 1, 9};
  int64_t values = 0;
  for (int i = 0; i < 4; ++i)
    if ((a.mask >> i) & 1u) values += (int64_t)a.num_points * len[i];
  if (a.tile_shift == 4)
    return launch_persistent(eval_hexline_kernel<SPLIT, P, 4>, a, a.padded, smem, s, P == 1 && !SPLIT && values >= 120);
  if constexpr (!SPLIT) return launch_persistent(eval_hexline_kernel<SPLIT, P, -1>, a, a.padded, smem, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_eval_hexline(bool split, int degree, const HexLineArgs& a, cudaStream_t s, bool* found) {
  *found = true;
  if (degree == 1) return split ? launch_degree<true, 1>(a, s) : launch_degree<false, 1>(a, s);
  if (degree == 2) return split ? launch_degree<true, 2>(a, s) : launch_degree<false, 2>(a, s);
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
