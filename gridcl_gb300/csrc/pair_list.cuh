// The paired-FP32 kernels' (element, precision) list, shared by the translation units that
// instantiate them (eval_pair.cu: plain; eval_pair_meas.cu: with the per-cell measure).
#pragma once
#include "eval_launch.cuh"

namespace tlg {

// One step per CTA (launch_persistent): volume cells on f32 meshes where J is wanted and a cell stores at least
// 120 values (18 nodes and more with det J alone: 18 points), so that its start and the CTA's table copy are small beside the
// rest; and in split precision from P2 on where the FP64 subtractions (3 K per cell) are at most 6 % of the
// values stored. GB300, ms, persistent / one step:
// split P2 tetrahedra 24 points 1,572,864 cells 0.640 / 0.539 (5.7 %), 27 points 440,000 0.204 / 0.183, 64 points
// 187,000 0.198 / 0.180; P3 24 points 300,000 0.161 / 0.169 (11 %); P2 prisms 27 points 300,000 0.164 / 0.173
// (9 %); P1 tetrahedra 8 points 1,000,000 0.138 / 0.144; f32 P1 tetrahedra 8 points 1,500,000 0.193 / 0.164, P2
// 24 points 1,000,000 0.388 / 0.329, P3 64 points 150,000 0.166 / 0.145, P2 prisms 27 points 0.141 / 0.126, P3 27
// points det J alone 280,000 0.075 / 0.069; but of 280,000 f32 cells P1 8 points det J alone 0.0108 / 0.0123, points
// alone 0.0085 / 0.0104, det J and K 0.0202 / 0.0213 (6 points four factors, 1,500,000 cells: 0.143 / 0.125), P2 4
// points four factors 0.0249 / 0.0269, P3 125 points alone
// 0.167 / 0.180; f32 P2 triangles 9 points 800,000 0.049 / 0.053 and split P2 triangles 0.128 / 0.131.
inline bool pair_one_step(bool split, int td, int k, const PairArgs& a) {
  if (td != 3) return false;
  const int len[6] = {3, 9, 1, 9, 3, 3};
  int64_t values = 0;
  for (int i = 0; i < 6; ++i)
    if ((a.mask >> i) & 1u) values += (int64_t)a.num_points * len[i];
  if (!split)
    return (a.mask & ~(uint32_t)(kOutPoints | kOutCellMeasure)) && (values >= 120 || (k >= 18 && a.num_points >= 18));
  return k >= 10 && 3 * k * 100 <= 6 * values;
}

template <bool SPLIT, bool MEAS>
static cudaError_t launch_pair(int td, int gd, int k, const PairArgs& a, size_t smem, cudaStream_t s,
                               bool* found) {
  *found = true;
  const bool step = pair_one_step(SPLIT, td, k, a);
#define TLG_PAIR(TD, GD, K) \
  if (td == TD && gd == GD && k == K) return launch_persistent(eval_pair_kernel<SPLIT, TD, GD, K, MEAS>, a, a.padded, smem, s, step);
  // Tetrahedra P1-P3, hexahedra Q1-Q2, prisms P1-P2.
  TLG_PAIR(3, 3, 4)
  TLG_PAIR(3, 3, 10)
  TLG_PAIR(3, 3, 20)
  TLG_PAIR(3, 3, 8)
  TLG_PAIR(3, 3, 27)
  TLG_PAIR(3, 3, 6)
  TLG_PAIR(3, 3, 18)
  // Pyramids P1-P3.
  TLG_PAIR(3, 3, 5)
  TLG_PAIR(3, 3, 14)
  TLG_PAIR(3, 3, 30)
  // Triangles P1-P4 and quadrilaterals Q1-Q2, planar and embedded in 3D.
  TLG_PAIR(2, 2, 3)
  TLG_PAIR(2, 2, 6)
  TLG_PAIR(2, 2, 10)
  TLG_PAIR(2, 2, 15)
  TLG_PAIR(2, 2, 4)
  TLG_PAIR(2, 2, 9)
  TLG_PAIR(2, 3, 3)
  TLG_PAIR(2, 3, 6)
  TLG_PAIR(2, 3, 10)
  TLG_PAIR(2, 3, 15)
  TLG_PAIR(2, 3, 4)
  TLG_PAIR(2, 3, 9)
#undef TLG_PAIR
  *found = false;
  return cudaSuccess;
}

}  // namespace tlg
