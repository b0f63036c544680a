// The gradient and Adam arithmetic shared by the optimiser's kernels (optimizer.cu, grad_tiles.cu): the per-pair terms of
// src/gradient.rs:120-147 and the step of src/adam.rs:45-57, and the tiled form of an iteration.
#pragma once

#include "engine.cuh"

namespace pacmap {

struct Sched {
  float w_nn, w_mn, w_fp, lr_t;
};

constexpr int GRAD_G = 8;  // lanes per row

// What one iteration reads and writes: y_cur -> y_next, m and v in place (grad_only: none of them written).
struct GradArgs {
  const float* y_cur;
  float *y_next, *m, *v;
  const uint32_t *rp, *col;
  uint64_t n;
  const uint32_t* long_rows;
  uint32_t n_long;
  const Sched* sched;
  float a1, a2;
  float *row_loss, *grad_out;  // may be null
  int grad_only;
};

// y of partner j (DIM consecutive floats; one 8-byte load for 2-D).
template <int DIM>
__device__ __forceinline__ void load_y(const float* __restrict__ y, uint32_t j, float (&out)[DIM]) {
  if constexpr (DIM == 2) {
    const float2 v = *reinterpret_cast<const float2*>(y + static_cast<uint64_t>(j) * 2);
    out[0] = v.x;
    out[1] = v.y;
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) out[c] = y[static_cast<uint64_t>(j) * DIM + c];
  }
}

// The force of partner yj on yi (per-pair arithmetic of gradient.rs:120-147) and the pair's loss.
template <int DIM, bool REPULSIVE>
__device__ __forceinline__ void pair_term(const float (&yi)[DIM], const float (&yj)[DIM], float c1, float c2, float w,
                                          float (&term)[DIM], float& loss, bool want_loss) {
  float df[DIM];
  float dsq = 1.0f;
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    df[c] = __fsub_rn(yi[c], yj[c]);
    dsq = __fadd_rn(dsq, __fmul_rn(df[c], df[c]));
  }
  const float tt = __fadd_rn(c1, dsq);
  const float w1 = __fmul_rn(w, __fdiv_rn(c2, __fmul_rn(tt, tt)));
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    const float gterm = __fmul_rn(w1, df[c]);
    term[c] = REPULSIVE ? -gterm : gterm;
  }
  if (want_loss)
    loss = REPULSIVE ? __fmul_rn(w, __fdiv_rn(1.0f, __fadd_rn(1.0f, dsq))) : __fmul_rn(w, __fdiv_rn(dsq, tt));
}

// One segment (one pair type) of a row: lane gl of a G-lane group takes entries s + gl, s + gl + G, ...
// in that order, with the partner index and y of the next entry loaded ahead (two-deep pipeline; four entries in
// flight need 74 registers instead of 48 and made the 1M x 128 iterations 2 % slower).
// The type's constants (c1, c2, weight, sign) are fixed for the whole segment.
template <int DIM, bool REPULSIVE>
__device__ __forceinline__ void accumulate_segment(const float* __restrict__ y, const uint32_t* __restrict__ col,
                                                   uint32_t s, uint32_t e, int gl, int G, const float (&yi)[DIM],
                                                   float c1, float c2, float w, float (&acc)[DIM], float& lacc,
                                                   bool want_loss) {
  uint32_t j = s + static_cast<uint32_t>(gl);
  if (j >= e) return;
  const uint32_t g = static_cast<uint32_t>(G);
  uint32_t ja = col[j];
  uint32_t jb = j + g < e ? col[j + g] : 0u;
  float ya[DIM];
  load_y<DIM>(y, ja, ya);
  for (; j < e; j += g) {
    float yb[DIM];
    if (j + g < e) load_y<DIM>(y, jb, yb);
    const uint32_t jc = j + 2 * g < e ? col[j + 2 * g] : 0u;
    float term[DIM], loss = 0.0f;
    pair_term<DIM, REPULSIVE>(yi, ya, c1, c2, w, term, loss, want_loss);
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], term[c]);
    if (want_loss) lacc += loss;
#pragma unroll
    for (int c = 0; c < DIM; ++c) ya[c] = yb[c];
    jb = jc;
  }
}

// Adam (adam.rs:45-57) of one coordinate: updates m and v, returns the new y.
__device__ __forceinline__ float adam_coord(float g, float yi, float* __restrict__ m, float* __restrict__ v, float a1,
                                            float a2, float lr_t) {
  float mm = *m, vv = *v;
  mm = __fadd_rn(mm, __fmul_rn(a1, __fsub_rn(g, mm)));
  vv = __fadd_rn(vv, __fmul_rn(a2, __fsub_rn(__fmul_rn(g, g), vv)));
  const float step = __fdiv_rn(__fmul_rn(lr_t, mm), __fadd_rn(__fsqrt_rn(vv), 1e-7f));
  *m = mm;
  *v = vv;
  return __fsub_rn(yi, step);
}

// What row i's gradient g leads to: the Adam step (not with grad_only) and grad_out; yi is the row's y. Up to four
// coordinates everything is loaded before anything is stored: the compiler cannot know that y_next, m and v are apart, and
// keeps each load behind the stores before it, so that a row's step was a chain of DIM round trips to memory. Rows of 48
// near and far entries: 400,000 in 2-D 119 us an iteration coordinate by coordinate, 97 so; 30,000 in 3-D 22.5 and 15.9;
// 100,000 in 4-D 59 and 54. Above four the registers of the loads cost as much as the chain (5-D 197 us one by one for
// 300,000 rows, 8-D 327 against 338 together).
template <int DIM>
__device__ __forceinline__ void finish_row(const GradArgs& p, uint64_t i, const float (&g)[DIM], const float (&yi)[DIM],
                                           float lr_t) {
  if constexpr (DIM <= 4) {
    if (!p.grad_only) {
      float m[DIM], v[DIM], y[DIM];
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        m[c] = p.m[i * DIM + c];
        v[c] = p.v[i * DIM + c];
      }
#pragma unroll
      for (int c = 0; c < DIM; ++c) y[c] = adam_coord(g[c], yi[c], &m[c], &v[c], p.a1, p.a2, lr_t);
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        p.y_next[i * DIM + c] = y[c];
        p.m[i * DIM + c] = m[c];
        p.v[i * DIM + c] = v[c];
      }
    }
    if (p.grad_out) {
#pragma unroll
      for (int c = 0; c < DIM; ++c) p.grad_out[i * DIM + c] = g[c];
    }
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      if (!p.grad_only)
        p.y_next[i * DIM + c] = adam_coord(g[c], yi[c], p.m + i * DIM + c, p.v + i * DIM + c, p.a1, p.a2, lr_t);
      if (p.grad_out) p.grad_out[i * DIM + c] = g[c];
    }
  }
}

// out[i] = sum of in[0..i) for i < len (the total must fit in 32 bits).
void exclusive_scan_u32(Ctx& c, const uint32_t* d_in, uint64_t len, uint32_t* d_out);

// ---- grad_tiles.cu ----
// The neighbour and far entries of a CSR regrouped by (partner tile, window of rows) for partners in shared memory.
struct TileGrad {
  uint32_t tiles = 0, tile_pts = 0, windows = 0, ctas = 0;
  DevBuf<uint32_t> unit_off;    // per unit (tile, window, 32 rows): its first word of idx
  DevBuf<uint16_t> meta;        // per (unit, lane): the row within the window and its entries in the tile
  DevBuf<uint32_t> idx;         // four partners per 8 bytes: index within the tile, bit 15 set for far pairs
  DevBuf<uint32_t> cta_units;   // the units of each block
  DevBuf<float> partial;        // tiles x n x dim
  DevBuf<float> partial_loss;   // tiles x n, when losses are asked for
  DevBuf<uint32_t> long_rows;   // rows left to grad_adam_long_kernel
  uint32_t n_long = 0;
};
// Builds it when the problem's sizes favour it and the device has the memory (else false, nothing built); the same lists
// get the same answer unless memory runs out. losses: some iteration wants its loss.
bool build_tile_grad(Ctx& c, const Csr& csr, uint64_t n, uint64_t dim, bool losses, TileGrad& out);
// One iteration of every row but the long ones (which p.long_rows must name), on stream s: two launches. mid: the
// iteration's mid-near weight is not 0. With p.row_loss the rows' losses too; y, m and v are the same bits either way.
void launch_tile_grad(const TileGrad& tg, const GradArgs& p, uint64_t dim, int itr, bool mid, cudaStream_t s);
// out = num / x as the tiled gradient divides (tests).
void debug_divide(Ctx& c, float num, const float* d_x, uint64_t n, float* d_out);

}  // namespace pacmap
