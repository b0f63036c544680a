// The optimiser -- src/lib.rs:736-843 (pacmap), src/gradient.rs:35-151, src/adam.rs:35-60 (file lines),
// src/weights.rs:52-81.
//
// K7 build_csr: every pair (i, j), i != j, of the three lists becomes two entries -- partner j in the
//    segment (i, type) and partner i in the segment (j, type) -- via a counting sort, then each segment
//    is sorted by partner. When the lists are grouped by point (the generated ones are), a mid-near or
//    far segment is point i's own partners in pair order followed by the points that drew i, sorted:
//    only that second part is placed by atomics and sorted (a neighbour segment is sorted whole). A pair's
//    contribution to each endpoint is bit-identical whichever endpoint lists it (the squared distance and
//    the weight use |y_i - y_j| only), so the sorted segments fix one deterministic summation order with
//    no floating-point atomics. (The reference's rayon reduce, gradient.rs:53-70, has no fixed order at
//    all.)
// K8 grad_adam_kernel: one group of G = 8 lanes per point sums its segments (NN c=10, MN c=10000, FP
//    repulsive c=1, exactly the per-pair f32 arithmetic of gradient.rs:120-147), reduces across the
//    group in a fixed butterfly, and applies the Adam step (adam.rs:45-57) to that point at once:
//    y is ping-ponged between two buffers because other points read y_j during the iteration.
//    Phase 3 has w_mn = 0: the MN segments are skipped (0 * finite = 0 adds nothing).
//    Rows of more than 1,024 entries go to grad_adam_long_kernel beside it, a warp each. From 65,536 rows in 2-D
//    and 3-D the near and far partners come from tiles of y in shared memory instead (grad_tiles.cu).
// K9 optimize_device: while all rows fit the GPU at once (18,944 in 1-D and 2-D, 14,208 in 3-D, 9,472 in 4-D and 5-D, 4,736
//    above, on 148 SMs) all iterations run in one launch (grad_adam_resident_kernel); above, with losses asked for, or with
//    a row of more than 1,024 entries, they are captured into one CUDA graph (one to three kernel nodes per iteration,
//    snapshot copies as memcpy nodes). The per-iteration (w_nn, w_mn, w_fp, lr_t) schedule lives in a device table
//    computed with the reference's f32 formulas.
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>

#include "arrivals.h"
#include "engine.cuh"
#include "grad.cuh"
#include "ptx.cuh"

namespace pacmap {
namespace {

// ------------------------------------------------------------------------------------------------
// K7: CSR build
// ------------------------------------------------------------------------------------------------
__global__ void csr_count_kernel(const uint32_t* __restrict__ pairs, uint64_t P, int type, uint64_t n,
                                 uint32_t* __restrict__ cnt, uint32_t* __restrict__ err) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t p = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P; p += stride) {
    const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    if (a >= n || b >= n) {
      atomicOr(err, DEV_ERR_PAIR_INDEX);
      continue;
    }
    if (a == b) continue;
    atomicAdd(&cnt[static_cast<uint64_t>(a) * 3 + type], 1u);
    atomicAdd(&cnt[static_cast<uint64_t>(b) * 3 + type], 1u);
  }
}

__global__ void csr_fill_kernel(const uint32_t* __restrict__ pairs, uint64_t P, int type, uint64_t n,
                                uint32_t* __restrict__ cursor, uint32_t* __restrict__ col) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t p = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P; p += stride) {
    const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    if (a >= n || b >= n || a == b) continue;
    col[atomicAdd(&cursor[static_cast<uint64_t>(a) * 3 + type], 1u)] = b;
    col[atomicAdd(&cursor[static_cast<uint64_t>(b) * 3 + type], 1u)] = a;
  }
}

// The generated pair lists hold each point's pairs together (rows i*k .. i*k + k - 1 start with i). Then
// a segment's forward entries (partners of its own pairs) are written in pair order without atomics, and
// only the reverse entries (points that drew it) are placed by atomics and sorted.
__global__ void grouped_check_kernel(const uint32_t* __restrict__ pairs, uint64_t P, uint32_t k,
                                     uint32_t* __restrict__ flag) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  bool ok = true;
  for (uint64_t p = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P; p += stride)
    ok = ok && pairs[2 * p] == static_cast<uint32_t>(p / k);
  if (!__all_sync(0xFFFFFFFFu, ok) && (threadIdx.x & 31) == 0) *flag = 0u;
}

// Forward counts of grouped lists: segment (i, type) gets the partners j != i of point i's k pairs. One
// warp per point, its pairs read in coalesced chunks of 32.
__global__ void __launch_bounds__(256) csr_fwd_count_kernel(const uint32_t* __restrict__ pairs, uint64_t n,
                                                            uint32_t k, int type, uint32_t* __restrict__ fwd,
                                                            uint32_t* __restrict__ cnt, uint32_t* __restrict__ err) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31;
  if (i >= n) return;
  uint32_t c = 0;
  bool bad = false;
  for (uint32_t q = lane; q < k; q += 32) {
    const uint32_t j = pairs[2 * (i * k + q) + 1];
    bad |= j >= n;
    c += (j < n && j != i) ? 1u : 0u;
  }
  c = __reduce_add_sync(0xFFFFFFFFu, c);
  if (__any_sync(0xFFFFFFFFu, bad) && lane == 0) atomicOr(err, DEV_ERR_PAIR_INDEX);
  if (lane == 0) {
    fwd[i * 3 + type] = c;
    cnt[i * 3 + type] = c;
  }
}

__global__ void csr_rev_count_kernel(const uint32_t* __restrict__ pairs, uint64_t P, int type, uint64_t n,
                                     uint32_t* __restrict__ cnt) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t p = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; p < P; p += stride) {
    const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    if (b < n && a != b) atomicAdd(&cnt[static_cast<uint64_t>(b) * 3 + type], 1u);
  }
}

// The forward entries of point i's segment in pair order, one warp per point (coalesced reads and writes).
__global__ void __launch_bounds__(256) csr_fwd_fill_kernel(const uint32_t* __restrict__ pairs, uint64_t n,
                                                           uint32_t k, int type, const uint32_t* __restrict__ rp,
                                                           uint32_t* __restrict__ col) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31;
  if (i >= n) return;
  uint32_t pos = rp[i * 3 + type];
  for (uint32_t q0 = 0; q0 < k; q0 += 32) {
    const uint32_t q = q0 + lane;
    const uint32_t j = q < k ? pairs[2 * (i * k + q) + 1] : 0xFFFFFFFFu;
    const bool keep = q < k && j < n && j != i;
    const unsigned bal = __ballot_sync(0xFFFFFFFFu, keep);
    if (keep) col[pos + __popc(bal & ((1u << lane) - 1u))] = j;
    pos += __popc(bal);
  }
}

// Reverse entries: pair (a, b) puts a into b's segment at a cursor taken by atomicAdd. Four pairs per round
// have their atomics in flight together (a thread would otherwise wait one round trip per pair); the
// order inside a segment is the atomics' and is sorted afterwards.
__global__ void csr_rev_fill_kernel(const uint32_t* __restrict__ pairs, uint64_t P, int type, uint64_t n,
                                    uint32_t* __restrict__ cursor, uint32_t* __restrict__ col) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  uint64_t p = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  for (; p + 3 * stride < P; p += 4 * stride) {
    uint32_t a[4], b[4], pos[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      a[k] = pairs[2 * (p + k * stride)];
      b[k] = pairs[2 * (p + k * stride) + 1];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      pos[k] = (b[k] < n && a[k] != b[k]) ? atomicAdd(&cursor[static_cast<uint64_t>(b[k]) * 3 + type], 1u) : 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (b[k] < n && a[k] != b[k]) col[pos[k]] = a[k];
  }
  for (; p < P; p += stride) {
    const uint32_t a = pairs[2 * p], b = pairs[2 * p + 1];
    if (b < n && a != b) col[atomicAdd(&cursor[static_cast<uint64_t>(b) * 3 + type], 1u)] = a;
  }
}

__global__ void add_offsets_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t len,
                                   uint32_t* __restrict__ out) {
  const uint64_t s = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s < len) out[s] = a[s] + b[s];
}

// Exclusive scan of u32 counts (the host checks that the total fits in u32).
constexpr int SCAN_T = 256, SCAN_PER = 8, SCAN_TILE = SCAN_T * SCAN_PER;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* tmp, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) tmp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < (SCAN_T / 32) ? tmp[lane] : 0u;
    uint32_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < (SCAN_T / 32)) tmp[lane] = wi - w;
    if (lane == (SCAN_T / 32) - 1) tmp[SCAN_T / 32] = wi;
  }
  __syncthreads();
  const uint32_t res = tmp[warp] + incl - v;
  total = tmp[SCAN_T / 32];
  __syncthreads();
  return res;
}

__global__ void __launch_bounds__(SCAN_T) scan_tiles_kernel(const uint32_t* __restrict__ in, uint64_t len,
                                                            uint32_t* __restrict__ out, uint32_t* __restrict__ sums) {
  __shared__ uint32_t tmp[SCAN_T / 32 + 1];
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * SCAN_TILE + threadIdx.x * SCAN_PER;
  uint32_t v[SCAN_PER], s = 0;
#pragma unroll
  for (int q = 0; q < SCAN_PER; ++q) {
    v[q] = (base + q < len) ? in[base + q] : 0u;
    s += v[q];
  }
  uint32_t total;
  uint32_t run = block_exclusive_scan(s, tmp, total);
#pragma unroll
  for (int q = 0; q < SCAN_PER; ++q) {
    if (base + q < len) out[base + q] = run;
    run += v[q];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_T) scan_sums_kernel(uint32_t* __restrict__ sums, uint64_t len) {
  __shared__ uint32_t tmp[SCAN_T / 32 + 1];
  uint32_t carry = 0;
  for (uint64_t b0 = 0; b0 < len; b0 += SCAN_T) {
    const uint64_t i = b0 + threadIdx.x;
    const uint32_t v = i < len ? sums[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_exclusive_scan(v, tmp, total);
    if (i < len) sums[i] = carry + ex;
    carry += total;
  }
}

__global__ void scan_add_kernel(uint32_t* __restrict__ out, uint64_t len, const uint32_t* __restrict__ sums) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < len) out[i] += sums[i / SCAN_TILE];
}

// Segment sort: one warp per segment of <= 1024 entries in shared memory; longer segments are
// listed for a block-level pass.
constexpr int SEG_WARPS = 8, SEG_SMALL = 1024, SEG_MID = 32768;

template <typename T>
__device__ __forceinline__ void bitonic_sort_range(T* s, int len, int tid, int nthreads, bool block) {
  for (int size = 2; size <= len; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (block) __syncthreads(); else __syncwarp();
      for (int t = tid; t < (len >> 1); t += nthreads) {
        const int i = 2 * t - (t & (stride - 1));
        const int j = i + stride;
        const bool up = ((i & size) == 0);
        const T a = s[i], b = s[j];
        if ((a > b) == up) {
          s[i] = b;
          s[j] = a;
        }
      }
    }
  }
  if (block) __syncthreads(); else __syncwarp();
}

// skip (may be null): the first skip[s] entries of segment s are already in their final order. The
// neighbour segments (type 0) are sorted whole all the same: a point and its neighbour are often each
// other's neighbours, and sorting puts the two entries of such a pair side by side, where the gradient
// kernel's lanes read the partner's coordinates in one request instead of two.
__device__ __forceinline__ uint32_t seg_skip(const uint32_t* __restrict__ skip, uint64_t sidx) {
  return (skip && sidx % 3 != 0) ? skip[sidx] : 0u;
}

__global__ void __launch_bounds__(SEG_WARPS * 32) seg_sort_small_kernel(const uint32_t* __restrict__ rp,
                                                                        const uint32_t* __restrict__ skip,
                                                                        uint32_t* __restrict__ col, uint64_t nseg,
                                                                        uint32_t* __restrict__ big,
                                                                        uint32_t* __restrict__ nbig) {
  __shared__ uint32_t buf[SEG_WARPS][SEG_SMALL];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint64_t sidx = static_cast<uint64_t>(blockIdx.x) * SEG_WARPS + warp; sidx < nseg;
       sidx += static_cast<uint64_t>(gridDim.x) * SEG_WARPS) {
    const uint32_t b = rp[sidx] + seg_skip(skip, sidx), e = rp[sidx + 1];
    const int len = static_cast<int>(e - b);
    if (len <= 1) continue;
    if (len > SEG_SMALL) {
      if (lane == 0) big[atomicAdd(nbig, 1u)] = static_cast<uint32_t>(sidx);
      continue;
    }
    if (len <= 128) {  // in registers: up to 4 keys per lane
      auto sort_regs = [&](auto tag) {
        constexpr int R = decltype(tag)::value;
        uint32_t v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int t = r * 32 + lane;
          v[r] = t < len ? col[b + t] : 0xFFFFFFFFu;
        }
        warp_sort_regs_u32<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int t = r * 32 + lane;
          if (t < len) col[b + t] = v[r];
        }
      };
      if (len <= 32) sort_regs(std::integral_constant<int, 1>());
      else if (len <= 64) sort_regs(std::integral_constant<int, 2>());
      else sort_regs(std::integral_constant<int, 4>());
      continue;
    }
    const int P = next_pow2(len);
    for (int t = lane; t < P; t += 32) buf[warp][t] = t < len ? col[b + t] : 0xFFFFFFFFu;
    bitonic_sort_range<uint32_t>(buf[warp], P, lane, 32, false);
    for (int t = lane; t < len; t += 32) col[b + t] = buf[warp][t];
    __syncwarp();
  }
}

__global__ void __launch_bounds__(1024) seg_sort_mid_kernel(const uint32_t* __restrict__ rp,
                                                            const uint32_t* __restrict__ skip,
                                                            uint32_t* __restrict__ col,
                                                            const uint32_t* __restrict__ big, uint32_t nbig) {
  extern __shared__ uint32_t mbuf[];
  for (uint32_t q = blockIdx.x; q < nbig; q += gridDim.x) {
    const uint32_t sidx = big[q];
    const uint32_t b = rp[sidx] + seg_skip(skip, sidx), e = rp[sidx + 1];
    const int len = static_cast<int>(e - b);
    if (len > SEG_MID) continue;
    const int P = next_pow2(len);
    __syncthreads();
    for (int t = threadIdx.x; t < P; t += blockDim.x) mbuf[t] = t < len ? col[b + t] : 0xFFFFFFFFu;
    bitonic_sort_range<uint32_t>(mbuf, P, threadIdx.x, blockDim.x, true);
    for (int t = threadIdx.x; t < len; t += blockDim.x) col[b + t] = mbuf[t];
  }
}

// Segments beyond shared memory: a bitonic network over a power-of-two global scratch, one block.
__global__ void __launch_bounds__(1024) seg_sort_huge_kernel(uint32_t* __restrict__ col, uint32_t b, uint32_t len,
                                                             uint32_t* __restrict__ scratch, uint32_t P) {
  for (uint32_t t = threadIdx.x; t < P; t += blockDim.x) scratch[t] = t < len ? col[b + t] : 0xFFFFFFFFu;
  bitonic_sort_range<uint32_t>(scratch, static_cast<int>(P), threadIdx.x, blockDim.x, true);
  for (uint32_t t = threadIdx.x; t < len; t += blockDim.x) col[b + t] = scratch[t];
}

// ------------------------------------------------------------------------------------------------
// Initialisation
// ------------------------------------------------------------------------------------------------
constexpr int INIT_MAX_DIM = 16;
constexpr int STD_BLOCKS = 256;

// Per-block partial sums of (v - mean)^2 in f64, one row of partials per block (fixed order).
__global__ void __launch_bounds__(256) var_partial_kernel(const float* __restrict__ v, uint64_t n, int dim,
                                                          const float* __restrict__ mean,
                                                          double* __restrict__ partial) {
  __shared__ double red[256];
  for (int cc = 0; cc < dim; ++cc) {
    double s = 0.0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
      const double df = static_cast<double>(v[i * dim + cc]) - static_cast<double>(mean[cc]);
      s += df * df;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) partial[static_cast<uint64_t>(blockIdx.x) * dim + cc] = red[0];
    __syncthreads();
  }
}

__global__ void std_final_kernel(const double* __restrict__ partial, int nblocks, int dim, uint64_t n,
                                 float* __restrict__ sd) {
  const int cc = threadIdx.x;
  if (cc >= dim) return;
  double s = 0.0;
  for (int b = 0; b < nblocks; ++b) s += partial[static_cast<uint64_t>(b) * dim + cc];
  sd[cc] = static_cast<float>(sqrt(s / static_cast<double>(n)));
}

__global__ void zscore_kernel(const float* __restrict__ v, uint64_t total, int dim, const float* __restrict__ mean,
                              const float* __restrict__ sd, float* __restrict__ y) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride) {
    const int cc = static_cast<int>(t % dim);
    const float a = __fmul_rn(__fsub_rn(v[t], mean[cc]), 0.0001f);
    y[t] = __fdiv_rn(a, sd[cc]);
  }
}

__global__ void random_init_kernel(uint64_t total, uint64_t seed, float* __restrict__ y) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride) {
    const uint64_t q = t >> 1;
    uint32_t w[4];
    philox4x32_10(static_cast<uint32_t>(q), static_cast<uint32_t>(q >> 32), 0u, TAG_INIT, static_cast<uint32_t>(seed),
                  static_cast<uint32_t>(seed >> 32), w);
    const double u1 = (static_cast<double>(w[0] >> 8) + 1.0) * (1.0 / 16777216.0);
    const double u2 = static_cast<double>(w[1] >> 8) * (1.0 / 16777216.0);
    const double r = sqrt(-2.0 * log(u1));
    const double a = 6.283185307179586476925286766559 * u2;
    y[t] = static_cast<float>((t & 1) ? r * sin(a) : r * cos(a));
  }
}

// ------------------------------------------------------------------------------------------------
// K8: fused gradient + Adam
// ------------------------------------------------------------------------------------------------
// The same segment by a whole warp, for rows of more than GRAD_LONG entries: each lane forms the terms of its own
// entries (LONG_U x 32 in flight), and lane l then adds, from the four lanes l % 8 + 8 r in turn, the entries
// that lane l % 8 of an eight-lane group would have added, in the same order: the sums are the same bits. (Entry t of
// the segment belongs to lane t % 8 in both.)
constexpr uint32_t GRAD_LONG = 1024;
constexpr int LONG_U = 4;
template <int DIM, bool REPULSIVE>
__device__ __forceinline__ void accumulate_segment_warp(const float* __restrict__ y, const uint32_t* __restrict__ col,
                                                        uint32_t s, uint32_t e, int lane, const float (&yi)[DIM],
                                                        float c1, float c2, float w, float (&acc)[DIM], float& lacc,
                                                        bool want_loss) {
  const uint32_t ln = static_cast<uint32_t>(lane), gl = ln & 7u;
  uint32_t nj[LONG_U];
#pragma unroll
  for (int u = 0; u < LONG_U; ++u) nj[u] = s + u * 32 + ln < e ? col[s + u * 32 + ln] : 0u;
  for (uint32_t b = s; b < e; b += LONG_U * 32) {
    float ya[LONG_U][DIM];
#pragma unroll
    for (int u = 0; u < LONG_U; ++u) load_y<DIM>(y, nj[u], ya[u]);  // past the end: point 0, not added below
#pragma unroll
    for (int u = 0; u < LONG_U; ++u) {
      const uint32_t t = b + (LONG_U + u) * 32 + ln;
      nj[u] = t < e ? col[t] : 0u;
    }
#pragma unroll
    for (int u = 0; u < LONG_U; ++u) {
      float term[DIM], loss = 0.0f;
      pair_term<DIM, REPULSIVE>(yi, ya[u], c1, c2, w, term, loss, want_loss);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool in = b + u * 32 + gl + 8 * r < e;
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
          const float tv = __shfl_sync(0xFFFFFFFFu, term[c], gl + 8 * r);
          if (in) acc[c] = __fadd_rn(acc[c], tv);
        }
        if (want_loss) {
          const float lv = __shfl_sync(0xFFFFFFFFu, loss, gl + 8 * r);
          if (in) lacc += lv;
        }
      }
    }
  }
}

// A row's forces: the NN, MN (skipped when w_mn = 0) and FP segments in turn (c = 10, 10000 and 1 in the
// denominators, FP repulsive). WARP: the whole warp on one row, else the G lanes of a group.
template <int DIM, bool WARP>
__device__ __forceinline__ void accumulate_row(const float* __restrict__ y, const uint32_t* __restrict__ col,
                                               uint32_t s0, uint32_t s1, uint32_t s2, uint32_t s3, bool use_mn,
                                               int gl, int G, const float (&yi)[DIM], const Sched& sc,
                                               float (&acc)[DIM], float& lacc, bool want_loss) {
  if constexpr (WARP) {
    accumulate_segment_warp<DIM, false>(y, col, s0, s1, gl, yi, 10.0f, 20.0f, sc.w_nn, acc, lacc, want_loss);
    if (use_mn)
      accumulate_segment_warp<DIM, false>(y, col, s1, s2, gl, yi, 10000.0f, 20000.0f, sc.w_mn, acc, lacc, want_loss);
    accumulate_segment_warp<DIM, true>(y, col, s2, s3, gl, yi, 1.0f, 2.0f, sc.w_fp, acc, lacc, want_loss);
  } else {
    accumulate_segment<DIM, false>(y, col, s0, s1, gl, G, yi, 10.0f, 20.0f, sc.w_nn, acc, lacc, want_loss);
    if (use_mn)
      accumulate_segment<DIM, false>(y, col, s1, s2, gl, G, yi, 10000.0f, 20000.0f, sc.w_mn, acc, lacc, want_loss);
    accumulate_segment<DIM, true>(y, col, s2, s3, gl, G, yi, 1.0f, 2.0f, sc.w_fp, acc, lacc, want_loss);
  }
}

// One row's iteration by the lanes gl of an eight-lane group (gmask: its lanes), or by a whole warp.
template <int DIM, bool WARP>
__device__ __forceinline__ void grad_adam_row(const GradArgs& p, const Sched& sc, uint64_t i, uint32_t s0, uint32_t s1,
                                              uint32_t s2, uint32_t s3, int gl, unsigned gmask) {
  constexpr int G = GRAD_G;
  const bool want_loss = p.row_loss != nullptr;
  float yi[DIM], acc[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    yi[c] = p.y_cur[i * DIM + c];
    acc[c] = 0.0f;
  }
  float lacc = 0.0f;
  accumulate_row<DIM, WARP>(p.y_cur, p.col, s0, s1, s2, s3, sc.w_mn != 0.0f, gl, G, yi, sc, acc, lacc, want_loss);
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], __shfl_xor_sync(gmask, acc[c], o, G));
    if (want_loss) lacc += __shfl_xor_sync(gmask, lacc, o, G);
  }
  if (gl == 0) {
    finish_row<DIM>(p, i, acc, yi, sc.lr_t);
    if (want_loss) p.row_loss[i] = lacc;
  }
}

template <int DIM>
__global__ void __launch_bounds__(256) grad_adam_kernel(const GradArgs p, int itr) {
  const Sched sc = p.sched[itr];
  const int gl = threadIdx.x & (GRAD_G - 1);
  const uint64_t groups = static_cast<uint64_t>(gridDim.x) * (blockDim.x / GRAD_G);
  const unsigned gmask = ((1u << GRAD_G) - 1u) << ((threadIdx.x & 31) & ~(GRAD_G - 1));
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / GRAD_G) + threadIdx.x / GRAD_G; i < p.n;
       i += groups) {
    const uint32_t s0 = p.rp[3 * i], s1 = p.rp[3 * i + 1], s2 = p.rp[3 * i + 2], s3 = p.rp[3 * i + 3];
    if (s3 - s0 > GRAD_LONG) continue;  // grad_adam_long_kernel's
    grad_adam_row<DIM, false>(p, sc, i, s0, s1, s2, s3, gl, gmask);
  }
}

// Rows of more than GRAD_LONG entries (points that thousands of others drew as neighbour), a warp each, beside
// grad_adam_kernel: walked by eight lanes, one such row outlasted all others together (60,000 image-like rows,
// near-black images in up to ~7,000 lists: 120 us an iteration with eight lanes and two entries in flight, 54 us with
// the warp). A kernel of its own: its registers in the other one cost the 1M x 128 fit 2 to 15 %.
template <int DIM>
__global__ void __launch_bounds__(256) grad_adam_long_kernel(const GradArgs p, int itr) {
  const uint32_t q = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (q >= p.n_long) return;
  const uint64_t i = p.long_rows[q];
  const Sched sc = p.sched[itr];
  grad_adam_row<DIM, true>(p, sc, i, p.rp[3 * i], p.rp[3 * i + 1], p.rp[3 * i + 2], p.rp[3 * i + 3], threadIdx.x & 31,
                           0xFFFFFFFFu);
}

// ------------------------------------------------------------------------------------------------
// All iterations in one launch, for problems whose rows fit the GPU at once
// ------------------------------------------------------------------------------------------------
// y of a partner, which another block may have written before the last grid_arrive_wait: an ordinary load (L1 serves
// repeated partners; the barrier's acquire keeps it from serving an earlier iteration's), never a read-only one.
template <int DIM>
__device__ __forceinline__ void load_y_shared(const float* y, uint32_t j, float (&out)[DIM]) {
  if constexpr (DIM == 2) {
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];"
                 : "=f"(out[0]), "=f"(out[1])
                 : "l"(y + static_cast<uint64_t>(j) * 2)
                 : "memory");
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c)
      asm volatile("ld.global.f32 %0, [%1];" : "=f"(out[c]) : "l"(y + static_cast<uint64_t>(j) * DIM + c) : "memory");
  }
}

// accumulate_segment with RES_U entries of a lane in flight (the iteration is bound by latency here, not by the
// gathers' rate).
constexpr int RES_U = 4;
template <int DIM, bool REPULSIVE>
__device__ __forceinline__ void accumulate_resident(const float* y, const uint32_t* __restrict__ col, uint32_t s,
                                                    uint32_t e, int gl, const float (&yi)[DIM], float c1,
                                                    float c2, float w, float (&acc)[DIM]) {
  constexpr uint32_t G = GRAD_G;
  for (uint32_t j = s + static_cast<uint32_t>(gl); j < e; j += RES_U * G) {
    uint32_t nj[RES_U];
    float ya[RES_U][DIM];
#pragma unroll
    for (int u = 0; u < RES_U; ++u) nj[u] = j + u * G < e ? __ldg(col + j + u * G) : 0u;
#pragma unroll
    for (int u = 0; u < RES_U; ++u)
      if (j + u * G < e) load_y_shared<DIM>(y, nj[u], ya[u]);
#pragma unroll
    for (int u = 0; u < RES_U; ++u) {
      if (j + u * G >= e) break;
      float term[DIM], loss;
      pair_term<DIM, REPULSIVE>(yi, ya[u], c1, c2, w, term, loss, false);
#pragma unroll
      for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], term[c]);
    }
  }
}

struct ResidentArgs {
  float* y[2];  // iteration itr0 reads y[0]
  float *m, *v;
  const uint32_t *rp, *col;
  uint32_t n;
  const Sched* sched;
  const int* snap_slot;  // per iteration from itr0 on: the snapshot to write, or -1; may be null
  float* snap;
  int itr0, itr1;
  float a1, a2;
  uint32_t *arrived, *err;
  uint32_t absent;  // blocks waited for that do not exist: 0 (1: the test hook, whose waits run out)
};

// Waits until every block of the (cooperative) grid, and `absent` more, has arrived `round` times. False when it gave up
// (2 s); a block that gives up does not arrive again, so the others give up at their next wait.
__device__ __forceinline__ bool grid_arrive_wait(uint32_t* arrived, uint32_t round, uint32_t absent, uint32_t* err) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
    const uint32_t want = arrivals_wanted(round, gridDim.x) + absent;
    const uint64_t t0 = globaltimer();
    uint32_t seen;
    int good = 1;
    for (uint32_t it = 1;; ++it) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
      if (arrivals_reached(seen, want)) break;
      if ((it & 255u) == 0 && globaltimer() - t0 > WAIT_LIMIT_NS) {
        good = 0;
        break;
      }
    }
    if (!good) atomicOr(err, DEV_ERR_TIMEOUT);
    ok = good;
  }
  __syncthreads();
  return ok != 0;
}

// One row per eight lanes for all iterations: its y, m and v stay in registers (every lane of the group computes the same
// Adam step), its partner indices in L1, and the blocks meet once per iteration. The sums are those of
// grad_adam_kernel. Bound by that meeting and the latency of the gathers from L2: 2,000 rows in 2-D 4.4 us an iteration
// against 8.1 for a graph node each, 9,000 rows 5.2 against 9.0, 18,000 rows 8.4 against 12.1; nothing to capture either
// (0.5 ms a fit).
template <int DIM>
__global__ void __launch_bounds__(256, DIM <= 2 ? 4 : (DIM == 3 ? 3 : 1)) grad_adam_resident_kernel(const ResidentArgs p) {
  const int gl = threadIdx.x & (GRAD_G - 1);
  const unsigned gmask = ((1u << GRAD_G) - 1u) << ((threadIdx.x & 31) & ~(GRAD_G - 1));
  const uint32_t i = blockIdx.x * (256 / GRAD_G) + threadIdx.x / GRAD_G;
  const bool row = i < p.n;
  const uint64_t at = static_cast<uint64_t>(i) * DIM;
  uint32_t s[4] = {};
  float yi[DIM] = {}, m[DIM] = {}, v[DIM] = {};
  if (row) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = p.rp[3 * static_cast<uint64_t>(i) + q];
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      yi[c] = p.y[0][at + c];
      m[c] = p.m[at + c];
      v[c] = p.v[at + c];
    }
  }
  for (int itr = p.itr0; itr < p.itr1; ++itr) {
    const int from = (itr - p.itr0) & 1;
    const Sched sc = p.sched[itr];
    if (row) {
      const float* y = p.y[from];
      float acc[DIM] = {};
      accumulate_resident<DIM, false>(y, p.col, s[0], s[1], gl, yi, 10.0f, 20.0f, sc.w_nn, acc);
      if (sc.w_mn != 0.0f)
        accumulate_resident<DIM, false>(y, p.col, s[1], s[2], gl, yi, 10000.0f, 20000.0f, sc.w_mn, acc);
      accumulate_resident<DIM, true>(y, p.col, s[2], s[3], gl, yi, 1.0f, 2.0f, sc.w_fp, acc);
#pragma unroll
      for (int o = GRAD_G / 2; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], __shfl_xor_sync(gmask, acc[c], o, GRAD_G));
      const int slot = p.snap_slot ? p.snap_slot[itr - p.itr0] : -1;
#pragma unroll
      for (int c = 0; c < DIM; ++c) {
        yi[c] = adam_coord(acc[c], yi[c], &m[c], &v[c], p.a1, p.a2, sc.lr_t);
        if (gl == 0) {
          p.y[from ^ 1][at + c] = yi[c];
          if (slot >= 0) p.snap[static_cast<uint64_t>(slot) * p.n * DIM + at + c] = yi[c];
        }
      }
    }
    if (itr + 1 < p.itr1 && !grid_arrive_wait(p.arrived, static_cast<uint32_t>(itr + 1 - p.itr0), p.absent, p.err))
      return;
  }
  if (row && gl == 0) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) {
      p.m[at + c] = m[c];
      p.v[at + c] = v[c];
    }
  }
}

// The rows with more than GRAD_LONG entries, in any order (each is summed by itself).
__global__ void long_rows_kernel(const uint32_t* __restrict__ rp, uint64_t n, uint32_t* __restrict__ rows,
                                 uint32_t* __restrict__ count) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n && rp[3 * i + 3] - rp[3 * i] > GRAD_LONG) rows[atomicAdd(count, 1u)] = static_cast<uint32_t>(i);
}

// Sum of the per-row losses in a fixed order (one block of 1,024 threads); each pair was counted at both endpoints.
__global__ void __launch_bounds__(1024) loss_reduce_kernel(const float* __restrict__ row_loss, uint64_t n,
                                                           float* __restrict__ out) {
  __shared__ double red[1024];
  double s = 0.0;
  // A thread's additions are one chain in this order; LOSS_AHEAD loads are in flight ahead of them.
  constexpr int LOSS_AHEAD = 16;
  uint64_t i = threadIdx.x;
  for (; i + (LOSS_AHEAD - 1) * 1024ull < n; i += LOSS_AHEAD * 1024ull) {
    float v[LOSS_AHEAD];
#pragma unroll
    for (int q = 0; q < LOSS_AHEAD; ++q) v[q] = row_loss[i + q * 1024ull];
#pragma unroll
    for (int q = 0; q < LOSS_AHEAD; ++q) s += v[q];
  }
  for (; i < n; i += 1024) s += row_loss[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 512; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = static_cast<float>(0.5 * red[0]);
}

using GradFn = void (*)(const GradArgs, int);
using ResidentFn = void (*)(const ResidentArgs);
struct GradFns {
  GradFn rows, long_rows;
  ResidentFn resident;
};

GradFns pick_grad_kernel(uint64_t dim) {
  switch (dim) {
    case 1: return {grad_adam_kernel<1>, grad_adam_long_kernel<1>, grad_adam_resident_kernel<1>};
    case 2: return {grad_adam_kernel<2>, grad_adam_long_kernel<2>, grad_adam_resident_kernel<2>};
    case 3: return {grad_adam_kernel<3>, grad_adam_long_kernel<3>, grad_adam_resident_kernel<3>};
    case 4: return {grad_adam_kernel<4>, grad_adam_long_kernel<4>, grad_adam_resident_kernel<4>};
    case 5: return {grad_adam_kernel<5>, grad_adam_long_kernel<5>, grad_adam_resident_kernel<5>};
    case 6: return {grad_adam_kernel<6>, grad_adam_long_kernel<6>, grad_adam_resident_kernel<6>};
    case 7: return {grad_adam_kernel<7>, grad_adam_long_kernel<7>, grad_adam_resident_kernel<7>};
    case 8: return {grad_adam_kernel<8>, grad_adam_long_kernel<8>, grad_adam_resident_kernel<8>};
    default: return {};
  }
}

// compiler-rt __powisf2 (Rust f32::powi with a run-time exponent).
float powi_f32(float a, int b) {
  const bool recip = b < 0;
  float r = 1.0f;
  while (true) {
    if (b & 1) r *= a;
    b /= 2;
    if (b == 0) break;
    a *= a;
  }
  return recip ? 1.0f / r : r;
}

// weights.rs:52-81 and adam.rs:45-47 (file lines) in the reference's f32 arithmetic.
Sched schedule_at(uint64_t itr, uint64_t p1, uint64_t p2, float lr) {
  Sched s;
  if (itr < p1) {
    const float progress = static_cast<float>(itr) / static_cast<float>(p1);
    const float a = (1.0f - progress) * 1000.0f;
    const float b = progress * 3.0f;
    s.w_mn = a + b;
    s.w_nn = 2.0f;
    s.w_fp = 1.0f;
  } else if (itr < p1 + p2) {
    s.w_mn = 3.0f;
    s.w_nn = 3.0f;
    s.w_fp = 1.0f;
  } else {
    s.w_mn = 0.0f;
    s.w_nn = 1.0f;
    s.w_fp = 1.0f;
  }
  const int t = static_cast<int>(itr + 1);
  const float sq = std::sqrt(1.0f - powi_f32(0.999f, t));
  const float q = 1.0f - powi_f32(0.9f, t);
  s.lr_t = (lr * sq) / q;
  return s;
}

}  // namespace

void exclusive_scan_u32(Ctx& c, const uint32_t* d_in, uint64_t len, uint32_t* d_out) {
  const uint64_t tiles = ceil_div(len, SCAN_TILE);
  DevBuf<uint32_t> sums(c, tiles);
  scan_tiles_kernel<<<static_cast<unsigned>(tiles), SCAN_T, 0, c.stream>>>(d_in, len, d_out, sums.get());
  PM_LAUNCHED();
  scan_sums_kernel<<<1, SCAN_T, 0, c.stream>>>(sums.get(), tiles);
  PM_LAUNCHED();
  scan_add_kernel<<<ceil_div(len, 256), 256, 0, c.stream>>>(d_out, len, sums.get());
  PM_LAUNCHED();
}

void build_csr(Ctx& c, uint64_t n, const uint32_t* d_pnn, uint64_t n_nn, const uint32_t* d_pmn, uint64_t n_mn,
               const uint32_t* d_pfp, uint64_t n_fp, Csr& out, bool grouped_known) {
  PM_REQUIRE(n < (1ull << 32), PACMAP_ERR_UNSUPPORTED, "pair indices are u32: n must be < 2^32");
  PM_REQUIRE(2 * (n_nn + n_mn + n_fp) < 0xFFFFFFFFull, PACMAP_ERR_UNSUPPORTED, "more than 2^31 pairs");
  const uint64_t nseg = 3 * n;
  DevBuf<uint32_t> cnt(c, nseg + 1);
  PM_CUDA(cudaMemsetAsync(cnt.get(), 0, (nseg + 1) * sizeof(uint32_t), c.stream));
  const uint32_t* lists[3] = {d_pnn, d_pmn, d_pfp};
  const uint64_t sizes[3] = {n_nn, n_mn, n_fp};
  auto grid_for = [&](uint64_t items) {
    return static_cast<unsigned>(std::min<uint64_t>(ceil_div(items, 256), c.sm_count * 16ull));
  };
  // Are the lists grouped by point (every generated list is)? Then forward entries need no atomics.
  bool grouped = n > 0;
  for (int t = 0; t < 3 && grouped; ++t) grouped = sizes[t] % n == 0 && sizes[t] / n < (1ull << 31);
  DevBuf<uint32_t> flag, fwd;
  if (grouped && !grouped_known) {
    flag.alloc(c, 1);
    const uint32_t one = 1u;
    PM_CUDA(cudaMemcpyAsync(flag.get(), &one, sizeof(uint32_t), cudaMemcpyHostToDevice, c.stream));
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      grouped_check_kernel<<<grid_for(sizes[t]), 256, 0, c.stream>>>(lists[t], sizes[t],
                                                                     static_cast<uint32_t>(sizes[t] / n), flag.get());
      PM_LAUNCHED();
    }
    uint32_t h = 0;
    PM_CUDA(cudaMemcpyAsync(&h, flag.get(), sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaStreamSynchronize(c.stream));
    grouped = h != 0;
  }
  if (grouped) {
    fwd.alloc(c, nseg);
    PM_CUDA(cudaMemsetAsync(fwd.get(), 0, nseg * sizeof(uint32_t), c.stream));
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_fwd_count_kernel<<<ceil_div(n, 8), 256, 0, c.stream>>>(lists[t], n, static_cast<uint32_t>(sizes[t] / n), t,
                                                                fwd.get(), cnt.get(), c.d_err);
      PM_LAUNCHED();
    }
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_rev_count_kernel<<<grid_for(sizes[t]), 256, 0, c.stream>>>(lists[t], sizes[t], t, n, cnt.get());
      PM_LAUNCHED();
    }
  } else {
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_count_kernel<<<grid_for(sizes[t]), 256, 0, c.stream>>>(lists[t], sizes[t], t, n, cnt.get(), c.d_err);
      PM_LAUNCHED();
    }
  }
  c.check_errors("pair lists");
  out.row_ptr.alloc(c, nseg + 1);
  exclusive_scan_u32(c, cnt.get(), nseg + 1, out.row_ptr.get());
  uint32_t total = 0;
  PM_CUDA(cudaMemcpyAsync(&total, out.row_ptr.get() + nseg, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  out.entries = total;
  out.entries_mn = std::min<uint64_t>(total, 2 * n_mn);
  out.col.alloc(c, std::max<uint64_t>(total, 1));
  if (grouped) {
    // forward entries in pair order; reverse entries after them by atomics (cursor = row_ptr + forward)
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_fwd_fill_kernel<<<ceil_div(n, 8), 256, 0, c.stream>>>(lists[t], n, static_cast<uint32_t>(sizes[t] / n), t,
                                                               out.row_ptr.get(), out.col.get());
      PM_LAUNCHED();
    }
    add_offsets_kernel<<<ceil_div(nseg, 256), 256, 0, c.stream>>>(out.row_ptr.get(), fwd.get(), nseg, cnt.get());
    PM_LAUNCHED();
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_rev_fill_kernel<<<grid_for(sizes[t]), 256, 0, c.stream>>>(lists[t], sizes[t], t, n, cnt.get(),
                                                                    out.col.get());
      PM_LAUNCHED();
    }
  } else {
    // cursor = row_ptr (reuse the count buffer)
    PM_CUDA(cudaMemcpyAsync(cnt.get(), out.row_ptr.get(), (nseg + 1) * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                            c.stream));
    for (int t = 0; t < 3; ++t) {
      if (!sizes[t]) continue;
      csr_fill_kernel<<<grid_for(sizes[t]), 256, 0, c.stream>>>(lists[t], sizes[t], t, n, cnt.get(), out.col.get());
      PM_LAUNCHED();
    }
  }
  // sort what the atomics placed: whole segments, or (grouped) the reverse part after the forward entries
  const uint32_t* skip = grouped ? fwd.get() : nullptr;
  DevBuf<uint32_t> big(c, nseg + 1);
  PM_CUDA(cudaMemsetAsync(big.get() + nseg, 0, sizeof(uint32_t), c.stream));
  const unsigned g = static_cast<unsigned>(std::min<uint64_t>(ceil_div(nseg, SEG_WARPS), c.sm_count * 8ull));
  seg_sort_small_kernel<<<g, SEG_WARPS * 32, 0, c.stream>>>(out.row_ptr.get(), skip, out.col.get(), nseg, big.get(),
                                                           big.get() + nseg);
  PM_LAUNCHED();
  // at most 2 pairs / GRAD_LONG rows can be long
  out.long_rows.alloc(c, total / GRAD_LONG + 2);
  uint32_t* n_long = out.long_rows.get() + total / GRAD_LONG + 1;
  PM_CUDA(cudaMemsetAsync(n_long, 0, sizeof(uint32_t), c.stream));
  long_rows_kernel<<<ceil_div(n, 256), 256, 0, c.stream>>>(out.row_ptr.get(), n, out.long_rows.get(), n_long);
  PM_LAUNCHED();
  uint32_t nbig = 0;
  PM_CUDA(cudaMemcpyAsync(&nbig, big.get() + nseg, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaMemcpyAsync(&out.n_long, n_long, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  if (nbig > 0) {
    const size_t smem = SEG_MID * sizeof(uint32_t);
    PM_CUDA(cudaFuncSetAttribute(seg_sort_mid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(smem)));
    seg_sort_mid_kernel<<<std::min<uint32_t>(nbig, c.sm_count * 2), 1024, smem, c.stream>>>(
        out.row_ptr.get(), skip, out.col.get(), big.get(), nbig);
    PM_LAUNCHED();
    // Segments longer than shared memory (points that appear in > 32768 pairs of one type).
    std::vector<uint32_t> hb(nbig), hrp(nseg + 1), hskip;
    PM_CUDA(cudaMemcpyAsync(hb.data(), big.get(), nbig * sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaMemcpyAsync(hrp.data(), out.row_ptr.get(), (nseg + 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                            c.stream));
    if (skip) {
      hskip.resize(nseg);
      PM_CUDA(cudaMemcpyAsync(hskip.data(), skip, nseg * sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
    }
    PM_CUDA(cudaStreamSynchronize(c.stream));
    DevBuf<uint32_t> scratch;
    for (uint32_t q = 0; q < nbig; ++q) {
      const uint32_t b = hrp[hb[q]] + ((skip && hb[q] % 3 != 0) ? hskip[hb[q]] : 0u), len = hrp[hb[q] + 1] - b;
      if (len <= static_cast<uint32_t>(SEG_MID)) continue;
      const uint32_t P = static_cast<uint32_t>(next_pow2(static_cast<int>(len)));
      if (scratch.count < P) scratch.alloc(c, P);
      seg_sort_huge_kernel<<<1, 1024, 0, c.stream>>>(out.col.get(), b, len, scratch.get(), P);
      PM_LAUNCHED();
    }
  }
}

void init_value_device(Ctx& c, const float* d_v, uint64_t n, uint64_t dim, float* d_y) {
  PM_REQUIRE(n > 0, PACMAP_ERR_EMPTY_ARRAY_MEAN, "Failed to calculate mean axis: the array is empty");
  PM_REQUIRE(dim <= INIT_MAX_DIM, PACMAP_ERR_UNSUPPORTED, "embedding dimensions above 16 are not supported");
  if (dim == 0) return;
  DevBuf<float> mean(c, dim), sd(c, dim);
  DevBuf<double> partial(c, static_cast<size_t>(STD_BLOCKS) * dim);
  column_mean_seq(c, d_v, n, dim, 0.0f, 1.0f, mean.get());
  var_partial_kernel<<<STD_BLOCKS, 256, 0, c.stream>>>(d_v, n, static_cast<int>(dim), mean.get(), partial.get());
  PM_LAUNCHED();
  std_final_kernel<<<1, 32, 0, c.stream>>>(partial.get(), STD_BLOCKS, static_cast<int>(dim), n, sd.get());
  PM_LAUNCHED();
  const uint64_t total = n * dim;
  zscore_kernel<<<static_cast<unsigned>(std::min<uint64_t>(ceil_div(total, 256), c.sm_count * 16ull)), 256, 0,
                  c.stream>>>(d_v, total, static_cast<int>(dim), mean.get(), sd.get(), d_y);
  PM_LAUNCHED();
}

void init_random_device(Ctx& c, uint64_t n, uint64_t dim, uint64_t seed, float* d_y) {
  const uint64_t total = n * dim;
  if (!total) return;
  random_init_kernel<<<static_cast<unsigned>(std::min<uint64_t>(ceil_div(total, 256), c.sm_count * 16ull)), 256, 0,
                       c.stream>>>(total, seed, d_y);
  PM_LAUNCHED();
}

namespace {
// A second stream that joins a capture: fork() makes it wait for the main stream, join() the main stream for it.
// Both record their event while capturing, so the events only shape the graph.
struct Branch {
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2] = {};
  explicit Branch(bool on) {
    if (!on) return;
    cudaError_t e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    for (auto& x : ev)
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      release();
      PM_CUDA(e);
    }
  }
  bool fork(cudaStream_t main) {
    return cudaEventRecord(ev[0], main) == cudaSuccess && cudaStreamWaitEvent(stream, ev[0], 0) == cudaSuccess;
  }
  bool join(cudaStream_t main) {
    return cudaEventRecord(ev[1], stream) == cudaSuccess && cudaStreamWaitEvent(main, ev[1], 0) == cudaSuccess;
  }
  void release() {
    for (auto& x : ev)
      if (x) cudaEventDestroy(x);
    if (stream) cudaStreamDestroy(stream);
    stream = nullptr;
  }
  ~Branch() { release(); }
  Branch(const Branch&) = delete;
  Branch& operator=(const Branch&) = delete;
};

// The blocks of the resident form when all rows fit the GPU at once, eight lanes each, and none is a long one, else 0.
unsigned resident_blocks(Ctx& c, const Csr& csr, uint64_t n, ResidentFn fn) {
  if (csr.n_long > 0 || n >= (1ull << 24)) return 0;
  int per_sm = 0;
  PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 256, 0));
  const unsigned blocks = ceil_div(n, 256 / GRAD_G);
  return blocks <= static_cast<unsigned>(c.sm_count * per_sm) ? blocks : 0;
}

// optimize_device in the resident form; false when the rows do not fit, or when the call wants what only the other path
// gives (losses, the last gradient).
bool optimize_resident(Ctx& c, const Csr& csr, const OptimizeArgs& a, ResidentFn fn, const Sched* sched,
                       float* const (&bufs)[2], float a1, float a2) {
  if (a.h_loss || a.d_grad_last) return false;
  const unsigned blocks = resident_blocks(c, csr, a.n, fn);
  if (blocks == 0) return false;
  const uint64_t iters = a.itr_end - a.itr_begin;
  DevBuf<uint32_t> arrived(c, 1);
  static_assert(ARRIVALS_START == 0xFFFFFFFFu, "set byte by byte");
  PM_CUDA(cudaMemsetAsync(arrived.get(), 0xFF, sizeof(uint32_t), c.stream));
  DevBuf<int> slots;
  std::vector<int> hslots;
  if (a.d_snap && a.snapshots) {
    hslots.assign(iters, -1);
    for (uint64_t t = 0; t < iters; ++t)
      for (uint64_t q = 0; q < a.n_snapshots; ++q)
        if (a.snapshots[q] == a.itr_begin + t + 1) {
          hslots[t] = static_cast<int>(q);
          break;
        }
    upload(c, slots, hslots.data(), iters);
  }
  ResidentArgs ra{};
  ra.y[0] = bufs[0];
  ra.y[1] = bufs[1];
  ra.m = a.d_m;
  ra.v = a.d_v;
  ra.rp = csr.row_ptr.get();
  ra.col = csr.col.get();
  ra.n = static_cast<uint32_t>(a.n);
  ra.sched = sched;
  ra.snap_slot = slots.get();
  ra.snap = a.d_snap;
  ra.itr0 = static_cast<int>(a.itr_begin);
  ra.itr1 = static_cast<int>(a.itr_end);
  ra.a1 = a1;
  ra.a2 = a2;
  ra.arrived = arrived.get();
  ra.err = c.d_err;
  ra.absent = stall_optimizer_hook() ? 1 : 0;
  void* params[] = {&ra};
  PM_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(fn), dim3(blocks), dim3(256), params, 0, c.stream));
  count_launch();
  if (bufs[iters & 1] != a.d_y)
    PM_CUDA(cudaMemcpyAsync(a.d_y, bufs[iters & 1], a.n * a.dim * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  last_graph_setup_ms() = 0.0;
  return true;
}
}  // namespace

double& last_graph_setup_ms() {
  static thread_local double v = 0.0;
  return v;
}

void optimize_device(Ctx& c, const Csr& csr, const OptimizeArgs& a) {
  const uint64_t n = a.n, dim = a.dim;
  if (a.itr_end <= a.itr_begin || n == 0 || dim == 0) return;
  PM_REQUIRE(dim <= 8, PACMAP_ERR_UNSUPPORTED, "the optimiser supports embedding dimensions 1..8");
  const GradFns fns = pick_grad_kernel(dim);
  if (a.h_loss && a.last_loss_only && a.itr_end - a.itr_begin > 1 && resident_blocks(c, csr, n, fns.resident) > 0) {
    // the iterations before the last without losses, in the resident form
    OptimizeArgs b = a;
    b.itr_end = a.itr_end - 1;
    b.h_loss = nullptr;
    b.d_grad_last = nullptr;
    optimize_device(c, csr, b);
    b = a;
    b.itr_begin = a.itr_end - 1;
    optimize_device(c, csr, b);
    return;
  }
  const uint64_t total_iters = a.p1 + a.p2 + a.p3;
  const uint64_t sched_len = std::max<uint64_t>(total_iters, a.itr_end);
  std::vector<Sched> hs(sched_len);
  for (uint64_t t = 0; t < sched_len; ++t) hs[t] = schedule_at(t, a.p1, a.p2, a.lr);
  DevBuf<Sched> sched(c, sched_len);
  PM_CUDA(cudaMemcpyAsync(sched.get(), hs.data(), sched_len * sizeof(Sched), cudaMemcpyHostToDevice, c.stream));
  const float a1 = 1.0f - 0.9f, a2 = 1.0f - 0.999f;

  DevBuf<float> yb(c, n * dim);
  DevBuf<float> row_loss, loss_dev;
  const uint64_t iters = a.itr_end - a.itr_begin;
  const uint64_t losses = a.last_loss_only ? 1 : iters;
  if (a.h_loss) {
    row_loss.alloc(c, n);
    loss_dev.alloc(c, losses);
  }
  // The tiles of y are copied 16 bytes at a time and the points of two coordinates loaded by 8. A caller's buffer that
  // starts off the 16-byte grid is worked on in a copy, so that its address does not choose the form of an iteration
  // (whose sums differ in their last digits).
  const bool on_grid = (reinterpret_cast<uintptr_t>(a.d_y) & 15u) == 0;
  DevBuf<float> ya;
  if (!on_grid) {
    ya.alloc(c, n * dim);
    PM_CUDA(cudaMemcpyAsync(ya.get(), a.d_y, n * dim * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
  }
  float* bufs[2] = {on_grid ? a.d_y : ya.get(), yb.get()};
  if (optimize_resident(c, csr, a, fns.resident, sched.get(), bufs, a1, a2)) return;
  int per_sm = 0;
  PM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fns.rows, 256, 0));
  const unsigned grid = static_cast<unsigned>(std::max<uint64_t>(
      1, std::min<uint64_t>(ceil_div(n, 256 / GRAD_G), static_cast<uint64_t>(c.sm_count) * std::max(per_sm, 1))));
  GradArgs ga{};
  ga.m = a.d_m;
  ga.v = a.d_v;
  ga.rp = csr.row_ptr.get();
  ga.col = csr.col.get();
  ga.n = n;
  ga.long_rows = csr.long_rows.get();
  ga.n_long = csr.n_long;
  ga.sched = sched.get();
  ga.a1 = a1;
  ga.a2 = a2;
  // Many rows: the partners through shared memory, tile by tile.
  TileGrad tg;
  const bool tiled = build_tile_grad(c, csr, n, dim, a.h_loss != nullptr, tg);
  if (tiled) {
    ga.long_rows = tg.long_rows.get();
    ga.n_long = tg.n_long;
  }
  Branch branch(ga.n_long > 0);  // the long rows run beside the others

  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  const auto setup_t0 = std::chrono::steady_clock::now();
  PM_CUDA(cudaStreamBeginCapture(c.stream, cudaStreamCaptureModeThreadLocal));
  uint64_t launches = 0;
  bool capture_ok = true;
  std::string capture_msg;
  for (uint64_t itr = a.itr_begin; itr < a.itr_end; ++itr) {
    const int src = static_cast<int>((itr - a.itr_begin) & 1), dst = src ^ 1;
    ga.y_cur = bufs[src];
    ga.y_next = bufs[dst];
    const bool last = itr + 1 == a.itr_end, want_loss = a.h_loss && (last || !a.last_loss_only);
    ga.grad_out = last ? a.d_grad_last : nullptr;
    ga.row_loss = want_loss ? row_loss.get() : nullptr;
    if (ga.n_long > 0) {
      capture_ok = branch.fork(c.stream) && capture_ok;
      fns.long_rows<<<ceil_div(ga.n_long, 8), 256, 0, branch.stream>>>(ga, static_cast<int>(itr));
      ++launches;
    }
    if (tiled) {
      launch_tile_grad(tg, ga, dim, static_cast<int>(itr), hs[itr].w_mn != 0.0f, c.stream);
      launches += 2;
    } else {
      fns.rows<<<grid, 256, 0, c.stream>>>(ga, static_cast<int>(itr));
      ++launches;
    }
    if (ga.n_long > 0) capture_ok = branch.join(c.stream) && capture_ok;
    if (want_loss) {
      loss_reduce_kernel<<<1, 1024, 0, c.stream>>>(row_loss.get(), n,
                                                   loss_dev.get() + (a.last_loss_only ? 0 : itr - a.itr_begin));
      ++launches;
    }
    if (a.d_snap && a.snapshots) {
      for (uint64_t sidx = 0; sidx < a.n_snapshots; ++sidx) {
        if (a.snapshots[sidx] == itr + 1) {
          if (cudaMemcpyAsync(a.d_snap + sidx * n * dim, bufs[dst], n * dim * sizeof(float), cudaMemcpyDeviceToDevice,
                              c.stream) != cudaSuccess) {
            capture_ok = false;
            capture_msg = "snapshot copy";
          }
          break;
        }
      }
    }
  }
  const cudaError_t end_err = cudaStreamEndCapture(c.stream, &graph);
  if (!capture_ok || end_err != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    throw Fail{PACMAP_ERR_CUDA, "graph capture failed: " + capture_msg + " " + cudaGetErrorString(end_err)};
  }
  const cudaError_t inst = cudaGraphInstantiate(&exec, graph, 0);
  last_graph_setup_ms() =
      std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - setup_t0).count();
  if (inst != cudaSuccess) {
    cudaGraphDestroy(graph);
    throw Fail{PACMAP_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(inst)};
  }
  const cudaError_t lerr = cudaGraphLaunch(exec, c.stream);
  count_launch(launches);
  cudaGraphExecDestroy(exec);
  cudaGraphDestroy(graph);
  PM_CUDA(lerr);
  if (bufs[iters & 1] != a.d_y)
    PM_CUDA(cudaMemcpyAsync(a.d_y, bufs[iters & 1], n * dim * sizeof(float), cudaMemcpyDeviceToDevice, c.stream));
  if (a.h_loss) {
    PM_CUDA(cudaMemcpyAsync(a.h_loss, loss_dev.get(), losses * sizeof(float), cudaMemcpyDeviceToHost, c.stream));
  }
  PM_CUDA(cudaStreamSynchronize(c.stream));
}

void gradient_device(Ctx& c, const Csr& csr, const float* d_y, uint64_t n, uint64_t dim, float w_nn, float w_mn,
                     float w_fp, float* d_grad, float* h_loss) {
  if (n == 0 || dim == 0) return;
  PM_REQUIRE(dim <= 8, PACMAP_ERR_UNSUPPORTED, "the optimiser supports embedding dimensions 1..8");
  const GradFns fns = pick_grad_kernel(dim);
  const Sched hs{w_nn, w_mn, w_fp, 0.0f};
  DevBuf<Sched> sched(c, 1);
  DevBuf<float> row_loss(c, n), loss_dev(c, 1);
  PM_CUDA(cudaMemcpyAsync(sched.get(), &hs, sizeof(Sched), cudaMemcpyHostToDevice, c.stream));
  const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(ceil_div(n, 256 / GRAD_G), c.sm_count * 8ull));
  GradArgs ga{};
  ga.y_cur = d_y;
  ga.rp = csr.row_ptr.get();
  ga.col = csr.col.get();
  ga.n = n;
  ga.long_rows = csr.long_rows.get();
  ga.n_long = csr.n_long;
  ga.sched = sched.get();
  ga.row_loss = row_loss.get();
  ga.grad_out = d_grad;
  ga.grad_only = 1;
  fns.rows<<<grid, 256, 0, c.stream>>>(ga, 0);
  PM_LAUNCHED();
  if (csr.n_long > 0) {
    fns.long_rows<<<ceil_div(csr.n_long, 8), 256, 0, c.stream>>>(ga, 0);
    PM_LAUNCHED();
  }
  loss_reduce_kernel<<<1, 1024, 0, c.stream>>>(row_loss.get(), n, loss_dev.get());
  PM_LAUNCHED();
  PM_CUDA(cudaMemcpyAsync(h_loss, loss_dev.get(), sizeof(float), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
}

}  // namespace pacmap
