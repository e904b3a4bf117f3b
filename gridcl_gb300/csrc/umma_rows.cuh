// Blackwell tensor-core evaluation (tcgen05) with one accumulator row per cell: the contraction of
// umma.cuh, X^T Phi with TF32 heads and tails and FP32 accumulators in tensor memory, for volume cells
// whose coordinates fit shared memory as heads and tails of 128 cells (to 56 nodes, 64 on f32 meshes).
//
// Per tile of 128 cells and coordinate g, two A operands (128 rows = cells, K = nodes): the TF32 heads
// of the coordinates relative to the cell's first node, and their tails. The B operand holds a chunk of
// 8 points x (phi, dphi_0..2) twice, as heads (columns 0-31) and as tails (columns 32-63; the table's
// two blocks are adjacent 8-row blocks of the canonical layout, so one N = 64 descriptor spans them).
// A_tail B, then A_head B accumulate into 64 columns per coordinate: the smaller products first, so
// that the sums round at the size of the heads' products only. x and J of a point are the sums of a
// row's head column and tail column.
//
// Bound: every partial product of a cell lands in the lane that stores the cell, so the epilogue (one
// thread per cell, eight warps of four points a chunk) needs no exchange and no CTA-wide barrier. Warps
// wait for a chunk's accumulators (mbarrier), load them, release the buffer (mbarrier, one arrival per
// warp) and finish their points; a ninth warp issues the table copies and the MMAs, a chunk
// ahead of the epilogue. N = 64 because the MMAs of this shape are bound by reading A (66 cycles for
// 128 x 32 x 8, counted on the 32-column kernel): one pass over A serves both halves of B.
// The kernel of umma.cuh (heads in rows 0-63, tails in rows 64-127, summed over two warps through
// shared memory, two CTA barriers per chunk) remains for cells of more nodes, whose tails do not fit
// beside the heads, and of fewer (forced strategies; two of its CTAs fit an SM).
//
// GB300, ms, that kernel / this one (all four factors): P5 tetrahedra, 216 points, 24,576 cells, f32 0.255
// / 0.133 (a floor of 0.071 by bytes), split 0.287 / 0.178; 19,456 cells (a tile per SM) 0.174 / 0.083, split
// 0.195 / 0.099; P4, 125 points, 90,000 cells, f32 0.438 / 0.219, split 0.505 / 0.285; 3,000 cells 0.023 /
// 0.017. Error against 64 bits on the first: 1.4e-6 / 9.6e-7 (fewer products meet in one accumulator). What
// is left there: a chunk takes 2.5 us, 2.0 of them the 42 MMAs (with one output alone), a tile's start 15 us.
// On the way, same case: one thread issuing behind a thread-index test, a coordinate after the other, work
// items in groups as in the other kernel 0.178; a converged warp electing the issuing lane, coordinates
// interleaved, equal runs 0.149, all with sixteen epilogue warps of 96 registers and one node quad a round
// of the gather (two spilled: 0.155); eight warps of 168 registers with two quads 0.139, four 0.133. Split:
// sixteen warps (spills) 0.312, eight 0.216, two quads 0.191, equal runs 0.178; three quads spill: 0.197.
//
// Tensor memory: 2 buffers x 3 coordinates x 64 columns, 512 allocated; the launch asks for at least 152
// KB of shared memory, so that no other CTA of a tensor-memory kernel shares the SM and the allocation
// never waits. Every wait is bounded: on expiry a warp does nothing more until the CTA's next barrier,
// where all leave; the CTA records the error, waits (bounded) for what it has in flight, frees its tensor
// memory and returns.
#pragma once

#include "umma.cuh"

namespace tlg {

constexpr int kRowsCells = 128;                      // cells per tile
// Epilogue warps (a quarter of them per lane quarter, two points at a time), and the issuing warp.
constexpr int kRowsEpiWarps = 8;
constexpr int kRowsThreads = kRowsEpiWarps * 32 + 32;
constexpr int kRowsN = 2 * kUmmaN;                   // columns per coordinate: heads, tails
constexpr int kRowsTmemCols = 512;
constexpr int kRowsMinNodes = 28;                    // fewer nodes: the kernel of umma.cuh
constexpr size_t kRowsMinSmem = (size_t)152 * 1024;

// Shared memory: A (3 x head and tail x 128 x kpad), B (2 buffers x head and tail x 32 x kpad), 6
// mbarriers, the tensor-memory address and the queue's count, split: the queue, 1 KiB of alignment.
inline size_t umma_rows_smem_bytes(int kpad, bool split) {
  return 1024 + (size_t)6 * kRowsCells * kpad * 4 + (size_t)4 * kUmmaN * kpad * 4 + 64 + (split ? kUmmaFix * 4 : 0);
}

// The 8 head and 8 tail columns of two points for each coordinate (this thread's lane), one wait for all.
__device__ __forceinline__ void tmem_ld_rows(uint32_t t, float (*h)[8], float (*l)[8]) {
  uint32_t r[48];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%48];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%49];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16, %17, %18, %19, %20, %21, %22, %23}, [%50];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24, %25, %26, %27, %28, %29, %30, %31}, [%51];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%32, %33, %34, %35, %36, %37, %38, %39}, [%52];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%40, %41, %42, %43, %44, %45, %46, %47}, [%53];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
      : "r"(t), "r"(t + 32u), "r"(t + 64u), "r"(t + 96u), "r"(t + 128u), "r"(t + 160u)
      : "memory");
#pragma unroll
  for (int g = 0; g < 3; ++g)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      h[g][i] = __uint_as_float(r[g * 16 + i]);
      l[g][i] = __uint_as_float(r[g * 16 + 8 + i]);
    }
}

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xFFFFFFFF;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// Split precision: J, det J, K and facet normals of cell `cr` of the range at point q from the f64 nodes and
// derivative table, stored. (A call of its own: inlined, its f64 values spill the epilogue's registers.)
static __device__ __noinline__ void umma_recompute_point(const UmmaArgs& a, int64_t cr, int q) {
  constexpr int TD = 3, GD = 3, LJ = 9;
  const int64_t cell = min(a.first_cell + cr, a.last_cell);
  float j[LJ], k[LJ], dj;
  recompute_f64_rt<TD, GD>(static_cast<const double*>(a.nodes), a.dofmap + cell * a.k, a.k, a.last_node,
                           a.dphi64 + (int64_t)q * a.k * TD, j, &dj, k, 1);
  const int64_t tile = (a.out_first_cell + cr) >> 4;
  const int lane = (int)((a.out_first_cell + cr) & 15), nq = a.num_points;
  if (a.mask & kOutJacobian) store_point(static_cast<float*>(a.out[1]), tile, q, nq, LJ, lane, 4, j, LJ);
  if (a.mask & kOutDetJ) store_point(static_cast<float*>(a.out[2]), tile, q, nq, 1, lane, 4, &dj, 1);
  if (a.mask & kOutPinv) store_point(static_cast<float*>(a.out[3]), tile, q, nq, LJ, lane, 4, k, LJ);
  if (a.mask & kOutFacetNormals) {
    float n[GD];
    Factors<float, TD, GD>::facet_normal(k, a.refn + q * TD, n);
    store_point(static_cast<float*>(a.out[5]), tile, q, nq, GD, lane, 4, n, GD);
  }
  if (a.recomputed && cr < a.range_cells) atomicAdd(a.recomputed, 1ull);
}

// Defined in umma.cu: the kernel of the precision, on a persistent grid.
cudaError_t launch_umma_rows(bool split, const UmmaArgs& a, size_t smem, cudaStream_t s);

template <bool SPLIT>
__global__ void __launch_bounds__(kRowsThreads, 1) umma_rows_kernel(const __grid_constant__ UmmaArgs a) {
  constexpr int TD = 3, GD = 3, LJ = 9;
  constexpr int kEpi = kRowsEpiWarps, kPart = kEpi / 4;  // kPart warps share a lane quarter
  using A = Ar<float>;
  using M = Factors<float, TD, GD>;
  using NT = typename std::conditional<SPLIT, double, float>::type;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t raw_s = (uint32_t)__cvta_generic_to_shared(smem_raw);
  unsigned char* smem = smem_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
  const int kpad = a.kpad, K = a.k, nq = a.num_points;
  const uint32_t a_bytes = (uint32_t)kRowsCells * kpad * 4u;    // one coordinate's heads or tails
  const uint32_t bbytes = (uint32_t)kRowsN * kpad * 4u;         // one B chunk, heads and tails
  const uint32_t sbo = (uint32_t)kpad * 32u;                    // 8-row blocks
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * a_bytes + 2 * bbytes);  // B[2], MMA[2], free[2]
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 6);
  uint32_t* fix_n = tslot + 1;                                  // queued points of this item
  uint32_t* fix = reinterpret_cast<uint32_t*>(bars + 8);        // [kUmmaFix]: (cell << 16) | point
  const uint32_t a_s = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t b_s = a_s + 6 * a_bytes;
  const uint32_t bar_b = (uint32_t)__cvta_generic_to_shared(bars), bar_m = bar_b + 16, bar_f = bar_b + 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int polls = (a.err && a.err[1] > 0) ? a.err[1] : (1 << 22);
  const bool issue_copies = !(a.err && a.err[2] == 1);
  const NT* nodes = static_cast<const NT*>(a.nodes);
  const uint32_t mask = a.mask;
  // The (tile, chunk) pairs in tile order are cut into equal runs of units, one per CTA; an item is a run's
  // part of one tile.
  const int64_t units = (a.padded + kRowsCells - 1) / kRowsCells * a.chunks / a.unit;
  const int64_t first = units * blockIdx.x / gridDim.x * a.unit, last = units * (blockIdx.x + 1) / gridDim.x * a.unit;
  const int run = (int)(last - first);
  const bool issuer = __shfl_sync(0xFFFFFFFFu, warp, 0) == kEpi;  // the issuing warp

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(tslot)),
                 "r"((uint32_t)kRowsTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 6; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar_b + 8 * i), "r"(i < 4 ? 1 : kEpi)
                   : "memory");
    *fix_n = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  const uint32_t tmem = *tslot;

  // Chunk number n of the run uses B and accumulator buffer n & 1, and the barriers' phase n >> 1. The
  // issuing warp's copies run ahead of its MMAs (`loaded` chunks so far).
  int loaded = 0, load_chunk = (int)(first % a.chunks);
  bool pend_b[2] = {false, false}, pend_m[2] = {false, false};  // in flight, and the phases they end
  uint32_t phase_b[2] = {0u, 0u}, phase_m[2] = {0u, 0u};
  auto load_next = [&]() {
    if (loaded >= run) return;
    const int buf = loaded & 1;
    if (issue_copies) {
      if (elect_one()) umma_load_b(a, b_s + buf * bbytes, bar_b + 8 * buf, load_chunk, bbytes);
      __syncwarp();
      pend_b[buf] = true;
      phase_b[buf] = (uint32_t)(loaded >> 1) & 1u;
    }
    ++loaded;
    load_chunk = load_chunk + 1 == a.chunks ? 0 : load_chunk + 1;
  };
  if (issuer) {
    load_next();
    load_next();
  }
  // The issuing warp (all lanes wait, one issues): the MMAs of chunk n, after its tables landed and its
  // accumulators were read; then, once the MMAs before them (of the other B buffer) are done, the copy
  // into that buffer.
  auto issue = [&](int n) -> bool {
    const int buf = n & 1;
    const uint32_t ph = (uint32_t)(n >> 1) & 1u;
    if (!__all_sync(0xFFFFFFFFu, umma_wait(bar_b + 8 * buf, ph, polls))) return false;
    pend_b[buf] = false;
    if (n >= 2 && !__all_sync(0xFFFFFFFFu, umma_wait(bar_f + 8 * buf, ph ^ 1u, polls))) return false;
    tmem_fence_after();
    constexpr uint32_t kIdesc = umma_idesc(128, kRowsN);
    const uint64_t bd = umma_desc(b_s + buf * bbytes, 128u, sbo);
    if (elect_one()) {
      // The coordinates innermost: consecutive MMAs accumulate into different columns and overlap.
      const int steps = kpad / 8;
      const uint32_t d = tmem + (uint32_t)(buf * GD * kRowsN);
      const uint64_t step_a = 2 * a_bytes >> 4;  // the next coordinate's operand
      // (a k-step of 8 nodes is 256 bytes on, 16 in the descriptors' units)
      uint64_t ad = umma_desc(a_s + a_bytes, 128u, sbo), b = bd;
#pragma unroll 2
      for (int s = 0; s < steps; ++s, ad += 16, b += 16)
#pragma unroll
        for (int g = 0; g < GD; ++g) umma_tf32(d + g * kRowsN, ad + g * step_a, b, kIdesc, s > 0);
      ad = umma_desc(a_s, 128u, sbo), b = bd;
#pragma unroll 2
      for (int s = 0; s < steps; ++s, ad += 16, b += 16)
#pragma unroll
        for (int g = 0; g < GD; ++g) umma_tf32(d + g * kRowsN, ad + g * step_a, b, kIdesc, 1u);
      umma_commit(bar_m + 8 * buf);
    }
    __syncwarp();
    pend_m[buf] = true;
    phase_m[buf] = ph;
    if (n >= 1) {
      const int ob = buf ^ 1;
      if (!__all_sync(0xFFFFFFFFu, umma_wait(bar_m + 8 * ob, (uint32_t)((n - 1) >> 1) & 1u, polls))) return false;
      pend_m[ob] = false;
      load_next();
    }
    return true;
  };

  // Warp w reads tensor-memory lane quarter w % 4 (its cells) and finishes points 2 (w / 4) and
  // 2 (w / 4) + 1 of each chunk.
  const int c = (warp & 3) * 32 + lane;  // this thread's cell in the tile
  const int own0 = 2 * (warp >> 2);
  bool ok = true;  // the same for all lanes of an epilogue warp
  int seq = 0;
  while (seq < run) {
    const int64_t tile = (first + seq) / a.chunks;
    const int chunk0 = (int)((first + seq) - tile * a.chunks);
    const int nchunks = min(a.chunks - chunk0, run - seq);
    const int64_t cr = tile * kRowsCells + c;  // cell index in the range
    const int64_t cell = min(a.first_cell + cr, a.last_cell);
    const bool store = cr < a.padded;
    float xh[GD], xl[GD];
    if (warp < kEpi && ok) {
      // Gather: thread (cell c, node quads warp / 4 (mod kPart)) writes heads and tails, four nodes of a
      // coordinate as one 16-byte row of a core matrix. Every warp has seen the item's last MMAs
      // complete, so that A is free.
      const uint32_t* row = a.dofmap + cell * K;
      NT x0[GD];
      const uint32_t n0 = min(__ldg(row), a.last_node);
#pragma unroll
      for (int g = 0; g < GD; ++g) x0[g] = __ldg(nodes + (int64_t)n0 * GD + g);
      // The next quads' indices are loaded ahead, so that a round waits for its coordinates only; as many
      // quads a round as the registers hold. (Beyond the cell's nodes: its first node, its coordinates
      // taken as zero.)
      constexpr int kQuads = SPLIT ? 2 : 4;
      auto load_indices = [&](int kq, uint32_t (*n)[4]) {
#pragma unroll
        for (int h = 0; h < kQuads; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k = 4 * (kq + h * kPart) + i;
            n[h][i] = k < K ? min(__ldg(row + k), a.last_node) : n0;
          }
      };
      uint32_t n[kQuads][4];
      load_indices(warp >> 2, n);
      for (int kq = warp >> 2; kq < kpad / 4; kq += kQuads * kPart) {
        NT v[kQuads][GD][4];
#pragma unroll
        for (int h = 0; h < kQuads; ++h)
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int g = 0; g < GD; ++g) v[h][g][i] = __ldg(nodes + (int64_t)n[h][i] * GD + g);
        load_indices(kq + kQuads * kPart, n);
#pragma unroll
        for (int h = 0; h < kQuads; ++h) {
          const int kh = kq + h * kPart;
          if (kh >= kpad / 4) break;
          const uint32_t off = (uint32_t)(c >> 3) * sbo + (uint32_t)kh * 128u + (c & 7) * 16u;
#pragma unroll
          for (int g = 0; g < GD; ++g) {
            uint32_t hd[4], tl[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float y;
              if constexpr (SPLIT) y = d2f_rn(v[h][g][i] - x0[g]);
              else y = v[h][g][i] - x0[g];
              if (4 * kh + i >= K) y = 0.0f;
              hd[i] = umma_tf32_head(y);
              tl[i] = umma_tf32_head(y - __uint_as_float(hd[i]));
            }
            *reinterpret_cast<uint4*>(smem + 2 * g * a_bytes + off) = make_uint4(hd[0], hd[1], hd[2], hd[3]);
            *reinterpret_cast<uint4*>(smem + (2 * g + 1) * a_bytes + off) = make_uint4(tl[0], tl[1], tl[2], tl[3]);
          }
        }
      }
      // This thread's first node plus the origin (split: as an f32 pair).
#pragma unroll
      for (int g = 0; g < GD; ++g) {
        if constexpr (SPLIT) {
          const double v = x0[g] + a.origin[g];
          xh[g] = d2f_rn(v);
          xl[g] = d2f_rn(v - f2d_exact(xh[g]));
        } else {
          xh[g] = x0[g];
          xl[g] = (float)a.origin[g];
        }
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tmem_fence_before();
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    tmem_fence_after();

    if (issuer) {
      for (int j = 0; j < nchunks && ok; ++j) ok = issue(seq + j);
    }
    if (warp < kEpi) {
      const int64_t o = a.out_first_cell + cr;
      const int64_t tile_idx = o >> 4;
      const int tl = (int)(o & 15);
      for (int j = 0; j < nchunks; ++j) {
        const int buf = (seq + j) & 1;
        const bool done = umma_wait(bar_m + 8 * buf, (uint32_t)((seq + j) >> 1) & 1u, polls);
        // (the tensor-memory loads are warp-collective)
        ok = __all_sync(0xFFFFFFFFu, done);
        if (!ok) break;
        tmem_fence_after();
#pragma unroll 1
        for (int own = own0; own < kUmmaPoints; own += 2 * kPart) {
          float u[GD][8], ul[GD][8];  // column 4 p + r of two points: r = 0 phi, 1 + d dphi_d
          const int q0 = (chunk0 + j) * kUmmaPoints + own;
          __syncwarp();  // (after the recomputes of some lanes)
          if (q0 < nq)
            tmem_ld_rows(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(buf * GD * kRowsN + 4 * own), u, ul);
          if (own + 2 * kPart >= kUmmaPoints) {  // the last of this warp's: the buffer is free
            tmem_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_f + 8 * buf);
          }
          if (q0 >= nq) continue;
#pragma unroll
          for (int g = 0; g < GD; ++g)
#pragma unroll
            for (int i = 0; i < 8; ++i) u[g][i] = A::add(u[g][i], ul[g][i]);
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            const int q = q0 + p;
            if (q >= nq) continue;  // the same for the whole warp
            float x[GD], jm[LJ];
#pragma unroll
            for (int g = 0; g < GD; ++g) {
              x[g] = u[g][4 * p];
#pragma unroll
              for (int d = 0; d < TD; ++d) jm[d * GD + g] = u[g][4 * p + 1 + d];
            }
            if ((mask & kOutPoints) && store) {
              float xp[GD];
#pragma unroll
              for (int g = 0; g < GD; ++g)
                xp[g] = SPLIT ? A::add(xh[g], A::add(xl[g], x[g])) : A::add(A::add(x[g], xh[g]), xl[g]);
              store_point(static_cast<float*>(a.out[0]), tile_idx, q, nq, GD, tl, 4, xp, GD);
            }
            if ((mask & ~kOutPoints) == 0) continue;
            float kk[LJ];
            M::pinv(jm, kk);
            float dj = M::detj(jm);
            bool deferred = false;
            if constexpr (SPLIT) {
              // Ill-conditioned points get J, det J, K and facet normals from FP64: at the end of the item
              // by way of its queue, beyond the queue's capacity here.
              const float kap = M::condition(jm, kk);
              if (store && !(kap <= a.cond_limit) && (mask & (kOutJacobian | kOutDetJ | kOutPinv))) {
                const uint32_t slot = atomicAdd(fix_n, 1u);
                if (slot < (uint32_t)kUmmaFix) fix[slot] = ((uint32_t)c << 16) | (uint32_t)q;
                else umma_recompute_point(a, cr, q);
                deferred = true;
              }
            }
            if (!store || deferred) continue;
            if (mask & kOutJacobian) store_point(static_cast<float*>(a.out[1]), tile_idx, q, nq, LJ, tl, 4, jm, LJ);
            if (mask & kOutDetJ) store_point(static_cast<float*>(a.out[2]), tile_idx, q, nq, 1, tl, 4, &dj, 1);
            if (mask & kOutPinv) store_point(static_cast<float*>(a.out[3]), tile_idx, q, nq, LJ, tl, 4, kk, LJ);
            if (mask & kOutFacetNormals) {
              float n[GD];
              M::facet_normal(kk, a.refn + q * TD, n);
              store_point(static_cast<float*>(a.out[5]), tile_idx, q, nq, GD, tl, 4, n, GD);
            }
          }
        }
      }
    }
    seq += nchunks;
    if constexpr (SPLIT) {
      // The item's queued points, one per thread: J, det J, K (and facet normals) from FP64.
      __syncthreads();
      const int nfix = min((int)*fix_n, kUmmaFix);
      if (nfix > 0) {  // the same for the CTA
        __syncthreads();
        if (tid == 0) *fix_n = 0;  // the next item's gather ends with a barrier
        for (int e = tid; e < nfix; e += kRowsThreads)  // the issuing warp too
          umma_recompute_point(a, tile * kRowsCells + (fix[e] >> 16), (int)(fix[e] & 0xFFFFu));
      }
    }
  }
  if (__syncthreads_or(!ok) && issuer && lane == 0) {
    // A wait expired: record it, and let what is in flight land (bounded).
    if (a.err) atomicExch(a.err, 1);
    for (int b = 0; b < 2; ++b) {
      if (pend_m[b]) umma_wait(bar_m + 8 * b, phase_m[b], polls);
      if (pend_b[b]) umma_wait(bar_b + 8 * b, phase_b[b], polls);
    }
  }
  tmem_fence_before();
  __syncthreads();
  tmem_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)kRowsTmemCols)
                 : "memory");
}

}  // namespace tlg
