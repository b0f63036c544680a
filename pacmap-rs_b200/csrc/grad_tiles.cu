// The gradient of many points with the partners' coordinates in shared memory.
//
// grad_adam_kernel (optimizer.cu) gathers every partner's y from L2, one 32-byte sector request per 8-byte partner, and
// runs at the rate of those requests (0.96 ms an iteration for 1,000,000 points in 2-D, 240 to 280 million gathers).
// Here the points are cut into tiles of up to 29,052 (2-D; 19,364 in 3-D: what 227 KB of shared memory hold beside the
// unused places' point). An iteration is two kernels:
//   tile_force_kernel  each block keeps one tile's y in shared memory and goes over the rows that have partners there
//                      (neighbour and far pairs), a lane per row, writing the row's sum over the tile's partners;
//   tile_adam_kernel   eight lanes per row add the row's tile sums in a fixed order, gather its mid-near partners as
//                      grad_adam_kernel does (they are few, and none in the last phase), and take the Adam step.
// The regrouped lists are built once per fit (build_tile_grad): rows in windows of 128, within each (tile, window)
// sorted by their number of entries and cut into units of 32, each row's entries in CSR order. A unit runs to its longest
// row: for entries spread at random it goes over 1.1 places per entry at 48 entries per row and tile, 1.2 at 20, 1.36 at 7
// (1,000,000 rows), and stores 1.1, 1.25 and 1.5.
// No atomics on floats: the sums and their order are the same on every call (another order than grad_adam_kernel's).
#include <algorithm>

#include "grad.cuh"
#include "ptx.cuh"

namespace pacmap {
namespace {

constexpr int WIN = 128;             // rows per window
constexpr int WIN_UNITS = WIN / 32;  // units per (tile, window)
constexpr int BUILD_T = 256;
constexpr int FORCE_T = 1024;
constexpr int MAX_TILES = 64;
constexpr uint32_t ROW_MAX = 511;    // entries of a row: 9 bits in meta; longer rows get a warp each
constexpr int TILE_SMEM = 232448;

// The rule of build_tile_grad, from 65,536 rows on (smaller fits keep grad_adam_kernel's order of sums to the bit). An
// iteration of the last phase, tiled against grad_adam_kernel, in us, lists in random order of rows, 2-D (3-D):
//   65,536 rows with 144 near and far entries each 29 (39) against 44 (66); 100,000 with 144 41 (51) / 67 (97);
//   200,000 with 192 80 (108) / 167 (243); 400,000 with 192 170 (252) / 320 (482); 1,000,000 with 240 734 (1177) / 961 (1463).
// Two fixed costs bound it from below: of a row in each tile (a unit's time whatever its entries), paid from 3 to 4.5
// entries per row and tile on (1,000,000 rows, 2-D: 4.1 entries 592 / 599, 2.7 507 / 433), and of the second kernel and the
// tiles' loads, paid from 24 to 50 entries per row on (65,536 rows, 2-D: 36 entries 18.4 / 18.8, with neighbours close by in
// memory 19.2 / 17.1). Building the lists takes 0.1 ms at 100,000 rows and 3 at 1,000,000. The number of iterations is no
// part of the rule: the sums' order, and with it their last digits, would depend on how a caller cuts a schedule into calls.
constexpr uint64_t TILE_MIN_ROWS = 65536;
constexpr double TILE_MIN_ROW_ENTRIES = 48.0;
double tile_min_entries(uint64_t dim) { return dim == 2 ? 4.5 : 4.0; }

__device__ __forceinline__ uint32_t div_magic(uint32_t col, uint64_t magic) {
  return static_cast<uint32_t>((col * magic) >> 40);  // col / tile_pts for col < 2^24, tile_pts < 2^15
}

// Goes over the neighbour and far entries of the window's rows (a warp per row, in order) and calls
// f(row in window, tile, rank of the entry within (row, tile), index within the tile, far). cnt[tile][row] (shared,
// zeroed) ends up with the entries per (row, tile).
template <typename F>
__device__ __forceinline__ void for_window_entries(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ col,
                                                   uint64_t n, uint64_t row0, uint32_t tile_pts, uint64_t magic,
                                                   uint16_t (*cnt)[WIN], F&& f) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < WIN; r += BUILD_T / 32) {
    const uint64_t i = row0 + r;
    if (i >= n) break;
    const uint32_t s0 = rp[3 * i], s1 = rp[3 * i + 1], s2 = rp[3 * i + 2], s3 = rp[3 * i + 3];
    if (s3 - s0 > ROW_MAX) continue;
    for (int type = 0; type < 2; ++type) {
      const uint32_t b = type ? s2 : s0, e = type ? s3 : s1;
      for (uint32_t q = b; q < e; q += 32) {
        const bool in = q + lane < e;
        const uint32_t j = in ? col[q + lane] : 0u;
        const uint32_t t = in ? div_magic(j, magic) : 0xFFFFFFFFu;
        const unsigned same = __match_any_sync(0xFFFFFFFFu, t);
        const uint32_t base = in ? cnt[t][r] : 0u;
        const int before = __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (in && before == 0) cnt[t][r] = static_cast<uint16_t>(base + __popc(same));
        __syncwarp();
        if (in) f(r, t, base + before, j - t * tile_pts, type);
      }
    }
  }
}

// Per (tile, window): the rows sorted by entries, descending (ties by row, descending), into units of 32; meta and the
// 8-byte words each unit needs (four entries per word and lane).
__global__ void __launch_bounds__(BUILD_T) tile_count_kernel(const uint32_t* __restrict__ rp,
                                                             const uint32_t* __restrict__ col, uint64_t n,
                                                             uint32_t tiles, uint32_t tile_pts, uint64_t magic,
                                                             uint32_t windows, uint16_t* __restrict__ meta,
                                                             uint32_t* __restrict__ words) {
  extern __shared__ __align__(16) unsigned char tsm[];
  uint16_t(*cnt)[WIN] = reinterpret_cast<uint16_t(*)[WIN]>(tsm);
  for (uint32_t e = threadIdx.x; e < tiles * WIN; e += BUILD_T) cnt[e / WIN][e % WIN] = 0;
  __syncthreads();
  for_window_entries(rp, col, n, static_cast<uint64_t>(blockIdx.x) * WIN, tile_pts, magic, cnt,
                     [](int, uint32_t, uint32_t, uint32_t, int) {});
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (uint32_t t = warp; t < tiles; t += BUILD_T / 32) {
    uint32_t key[WIN_UNITS];
#pragma unroll
    for (int q = 0; q < WIN_UNITS; ++q) {
      const int r = q * 32 + lane;
      key[q] = ((ROW_MAX - cnt[t][r]) << 7) | static_cast<uint32_t>(WIN - 1 - r);
    }
    warp_sort_regs_u32<WIN_UNITS>(key);
    const uint64_t unit0 = (static_cast<uint64_t>(t) * windows + blockIdx.x) * WIN_UNITS;
#pragma unroll
    for (int q = 0; q < WIN_UNITS; ++q) {
      const uint32_t c = ROW_MAX - (key[q] >> 7), r = WIN - 1 - (key[q] & (WIN - 1));
      meta[(unit0 + q) * 32 + lane] = static_cast<uint16_t>(r | (c << 7));
      if (lane == 0) words[unit0 + q] = 32 * ((c + 3) / 4);
    }
  }
}

// Every place names the point after the tile's until tile_fill_kernel fills it.
__global__ void tile_clear_kernel(uint32_t* __restrict__ idx, uint64_t words, uint32_t none) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < words; t += stride) idx[t] = none;
}

__global__ void __launch_bounds__(BUILD_T) tile_fill_kernel(const uint32_t* __restrict__ rp,
                                                            const uint32_t* __restrict__ col, uint64_t n,
                                                            uint32_t tiles, uint32_t tile_pts, uint64_t magic,
                                                            uint32_t windows, const uint16_t* __restrict__ meta,
                                                            const uint32_t* __restrict__ unit_off,
                                                            uint16_t* __restrict__ idx) {
  extern __shared__ __align__(16) unsigned char tsm[];
  uint16_t(*cnt)[WIN] = reinterpret_cast<uint16_t(*)[WIN]>(tsm);
  uint8_t(*slot)[WIN] = reinterpret_cast<uint8_t(*)[WIN]>(tsm + static_cast<size_t>(tiles) * WIN * 2);
  for (uint32_t e = threadIdx.x; e < tiles * WIN; e += BUILD_T) {
    const uint32_t t = e / WIN, place = e % WIN;
    cnt[t][place] = 0;
    slot[t][meta[(static_cast<uint64_t>(t) * windows + blockIdx.x) * WIN + place] & (WIN - 1)] =
        static_cast<uint8_t>(place);
  }
  __syncthreads();
  for_window_entries(rp, col, n, static_cast<uint64_t>(blockIdx.x) * WIN, tile_pts, magic, cnt,
                     [&](int r, uint32_t t, uint32_t rank, uint32_t local, int far) {
                       const uint32_t p = slot[t][r];
                       const uint64_t unit = (static_cast<uint64_t>(t) * windows + blockIdx.x) * WIN_UNITS + (p >> 5);
                       const uint64_t word = unit_off[unit] + (rank >> 2) * 32 + (p & 31);
                       idx[4 * word + (rank & 3)] = static_cast<uint16_t>(local | (far ? 0x8000u : 0u));
                     });
}

__global__ void tile_long_rows_kernel(const uint32_t* __restrict__ rp, uint64_t n, uint32_t* __restrict__ rows,
                                      uint32_t* __restrict__ count) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n && rp[3 * i + 3] - rp[3 * i] > ROW_MAX) rows[atomicAdd(count, 1u)] = static_cast<uint32_t>(i);
}

// Equal shares of the work for the blocks: entries' words plus UNIT_WORDS per unit for its fixed cost.
constexpr uint64_t UNIT_WORDS = 64;
__global__ void tile_shares_kernel(const uint32_t* __restrict__ unit_off, uint64_t units, uint32_t ctas,
                                   uint32_t* __restrict__ cta_units) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > ctas) return;
  const uint64_t total = unit_off[units] + UNIT_WORDS * units, want = total * b / ctas;
  uint64_t lo = 0, hi = units;  // the first unit whose work before it is >= want
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (unit_off[mid] + UNIT_WORDS * mid >= want) hi = mid;
    else lo = mid + 1;
  }
  cta_units[b] = b == ctas ? static_cast<uint32_t>(units) : static_cast<uint32_t>(lo);
}

// x, at most `most`; NaN stays NaN (fminf would give `most`).
__device__ __forceinline__ float min_or_nan(float x, float most) {
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(most));
  return x;
}

// num / x for x >= 1, without a branch: an approximate reciprocal, one Newton step, and a correction of the quotient by
// its exact remainder (P. W. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM
// J. Res. Dev. 34, 1990): correctly rounded up to x = 2^126 (tested against the / operator for every mantissa of x),
// 0 beyond, where the quotient is below 1e-36; NaN for NaN, as a division. The compiler's division checks its operands
// and branches, which kept two entries' divisions from overlapping.
__device__ __forceinline__ float div_by(float num, float x) {
  x = min_or_nan(x, 3.402823466e+38f);  // infinity would make the remainder NaN
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  y = fmaf(fmaf(-x, y, 1.0f), y, y);
  const float q = num * y;
  return fmaf(fmaf(-x, q, num), y, q);
}

// The coordinates of the place after a tile's points, which unused places of a unit name. Whatever finite yi is, that place
// adds nothing: numbers of this size lie 2^76 apart, so a coordinate's difference is 0 or so large that t^2 is infinite
// and the factor 0 (or all differences are 0); and no difference overflows, which would make 0 times it NaN.
constexpr float NOWHERE = 1e30f;

// One entry of a row (gradient.rs:120-147): the partner's y from shared memory, its term added to acc. The per-pair
// factor is w c2 / t^2 with t = c1 + 1 + |dy|^2; near pairs have w c2 = 20 w_nn and c1 = 10, far ones (bit 15 of e)
// repel: -2 w_fp and 1. Multiplications and additions are fused here, which rounds less often than the separate ones.
// LOSS: its loss too, w_nn d / (10 + d) or w_fp / (1 + d) with d = 1 + |dy|^2, added to lacc; none is the unused places'
// point, which has no loss. The arithmetic of the force is the same with and without.
template <int DIM, bool LOSS>
__device__ __forceinline__ void add_entry(const float* ys, uint32_t e, bool far, const float (&yi)[DIM],
                                          float near_num, float far_num, float (&acc)[DIM], uint32_t none, float w_nn,
                                          float w_fp, float& lacc) {
  float df[DIM];
  if constexpr (DIM == 2) {
    const float2 v = reinterpret_cast<const float2*>(ys)[e];
    df[0] = yi[0] - v.x;
    df[1] = yi[1] - v.y;
  } else {
#pragma unroll
    for (int c = 0; c < DIM; ++c) df[c] = yi[c] - ys[e * DIM + c];
  }
  float t = far ? 2.0f : 11.0f;
#pragma unroll
  for (int c = 0; c < DIM; ++c) t = fmaf(df[c], df[c], t);
  const float w1 = div_by(far ? far_num : near_num, t * t);
#pragma unroll
  for (int c = 0; c < DIM; ++c) acc[c] = fmaf(w1, df[c], acc[c]);
  if constexpr (LOSS) {
    float dsq = 1.0f;
#pragma unroll
    for (int c = 0; c < DIM; ++c) dsq = fmaf(df[c], df[c], dsq);
    dsq = min_or_nan(dsq, 1.2676506e30f);  // 2^100: both losses are at their limits there, and div_by is exact enough
    const float part = div_by(far ? 1.0f : dsq, (far ? 1.0f : 10.0f) + dsq);
    if (e != none) lacc = fmaf(far ? w_fp : w_nn, part, lacc);
  }
}

// The two entries of w, side by side and added in order.
template <int DIM, bool LOSS>
__device__ __forceinline__ void add_two(const float* ys, uint32_t w, const float (&yi)[DIM], float near_num,
                                        float far_num, float (&acc)[DIM], uint32_t none, float w_nn, float w_fp,
                                        float& lacc) {
  add_entry<DIM, LOSS>(ys, w & 0x7FFFu, (w & 0x8000u) != 0, yi, near_num, far_num, acc, none, w_nn, w_fp, lacc);
  add_entry<DIM, LOSS>(ys, (w >> 16) & 0x7FFFu, static_cast<int32_t>(w) < 0, yi, near_num, far_num, acc, none, w_nn,
                       w_fp, lacc);
}

struct ForceArgs {
  const float* y;
  float *partial, *partial_loss;  // partial_loss: LOSS only
  const uint32_t *unit_off, *cta_units;
  const uint2* idx;
  const uint16_t* meta;
  uint32_t n, tile_pts, windows;
  const Sched* sched;
};

// A unit: 32 rows of one window, a lane each, over their partners in one tile. Bound by the instructions per entry
// (about 25; a two-wide form of the arithmetic was slower: its operands cost two more shared loads and the packing) and
// per unit, and by the latency of the list words, which are two units ahead. 200,000 rows in 2-D: 72 us for 36 million
// entries. LOSS writes the row's loss over the tile's partners too, for the iterations whose loss is asked for: an instantiation
// of its own, so that the others do not carry it, with the same sums of forces.
template <int DIM, bool LOSS>
__global__ void __launch_bounds__(FORCE_T, 1) tile_force_kernel(const ForceArgs p, int itr) {
  extern __shared__ __align__(16) float ys[];
  const float w_nn = p.sched[itr].w_nn, w_fp = p.sched[itr].w_fp, near_num = 20.0f * w_nn, far_num = -2.0f * w_fp;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t per_tile = p.windows * WIN_UNITS;
  uint32_t u = p.cta_units[blockIdx.x];
  const uint32_t uend = p.cta_units[blockIdx.x + 1];
  while (u < uend) {
    const uint32_t t = u / per_tile, ue = min(uend, (t + 1) * per_tile);
    const uint32_t first = t * p.tile_pts, floats = min(p.tile_pts, p.n - first) * DIM;
    const float* src = p.y + static_cast<uint64_t>(first) * DIM;  // 16-byte aligned: tile_pts is a multiple of 4
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < floats / 4; e += FORCE_T) cp_async16(ys + 4 * e, src + 4 * e);
    for (uint32_t e = (floats & ~3u) + threadIdx.x; e < floats; e += FORCE_T) ys[e] = src[e];
    if (threadIdx.x < DIM) ys[p.tile_pts * DIM + threadIdx.x] = NOWHERE;
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // While a unit is summed, the next one's first entries and its rows' y are on their way, and the place and rows of
    // the one after that. A warp takes every STEP-th unit: always the same quarter of a window.
    constexpr uint32_t STEP = FORCE_T / 32;
    static_assert(STEP % WIN_UNITS == 0, "a warp's units are the same quarter of their windows");
    uint32_t unit = u + warp;
    const uint32_t* offp = p.unit_off + unit;
    const uint16_t* metap = p.meta + static_cast<uint64_t>(unit) * 32 + lane;
    uint32_t row0 = (unit / WIN_UNITS - t * p.windows) * WIN;
    float* outp = p.partial + (static_cast<uint64_t>(t) * p.n + row0) * DIM;
    float* lossp = LOSS ? p.partial_loss + static_cast<uint64_t>(t) * p.n + row0 : nullptr;
    const float* yrow = p.y + static_cast<uint64_t>(row0) * DIM;
    // the first two words of a row's entries in the tile
    const uint2 none = make_uint2(p.tile_pts * 0x10001u, p.tile_pts * 0x10001u);
    auto first_words = [&](uint32_t o, uint32_t c, uint2& a, uint2& b) {
      const uint2* q = p.idx + o + lane;
      a = c > 0 ? __ldcs(q) : none;
      b = c > 4 ? __ldcs(q + 32) : none;
    };
    uint32_t off = 0, mt = 0, off2 = 0, mt2 = 0;
    uint2 wa = none, wb = none;
    float yi[DIM] = {};
    if (unit < ue) {
      off = *offp;
      mt = *metap;
      first_words(off, mt >> 7, wa, wb);
      const uint32_t r = min(row0 + (mt & (WIN - 1)), p.n - 1) - row0;
#pragma unroll
      for (int d = 0; d < DIM; ++d) yi[d] = yrow[r * DIM + d];
    }
    if (unit + STEP < ue) {
      off2 = offp[STEP];
      mt2 = metap[STEP * 32];
    }
    while (unit < ue) {
      const uint32_t c = mt >> 7, r = mt & (WIN - 1), most = __shfl_sync(0xFFFFFFFFu, c, 0);  // lane 0: the longest row
      const bool real = row0 + r < p.n;
      const uint2* words = p.idx + off + lane + 64;
      uint2 na = none, nb = none;
      float yi_n[DIM] = {}, acc[DIM] = {}, lacc = 0.0f;
      yrow += STEP / WIN_UNITS * WIN * DIM;
      row0 += STEP / WIN_UNITS * WIN;
      if (unit + STEP < ue) {
        first_words(off2, mt2 >> 7, na, nb);
        const uint32_t rn = min(row0 + (mt2 & (WIN - 1)), p.n - 1) - row0;
#pragma unroll
        for (int d = 0; d < DIM; ++d) yi_n[d] = yrow[rn * DIM + d];
      }
      off = off2;
      mt = mt2;
      if (unit + 2 * STEP < ue) {
        off2 = offp[2 * STEP];
        mt2 = metap[2 * STEP * 32];
      }
      for (uint32_t k = 0; k < most; k += 4) {
        const uint2 wk = k + 8 < c ? __ldcs(words) : none;
        words += 32;
        add_two<DIM, LOSS>(ys, wa.x, yi, near_num, far_num, acc, p.tile_pts, w_nn, w_fp, lacc);
        if (k + 2 < most) add_two<DIM, LOSS>(ys, wa.y, yi, near_num, far_num, acc, p.tile_pts, w_nn, w_fp, lacc);
        wa = wb;
        wb = wk;
      }
      if (real) {
        if constexpr (DIM == 2) {
          *reinterpret_cast<float2*>(outp + r * 2) = make_float2(acc[0], acc[1]);
        } else {
#pragma unroll
          for (int d = 0; d < DIM; ++d) outp[r * DIM + d] = acc[d];
        }
        if constexpr (LOSS) lossp[r] = lacc;
      }
      outp += STEP / WIN_UNITS * WIN * DIM;
      if constexpr (LOSS) lossp += STEP / WIN_UNITS * WIN;
      offp += STEP;
      metap += STEP * 32;
      unit += STEP;
      wa = na;
      wb = nb;
#pragma unroll
      for (int d = 0; d < DIM; ++d) yi[d] = yi_n[d];
    }
    u = ue;
  }
}

// A row's tile sums (lane gl of eight adds tiles gl, gl + 8, ... in order), its mid-near pairs, the lanes' sums
// pairwise, and the Adam step. Without the mid-near part (MID: their weight is not 0) a kernel of its own, 32 registers
// a thread against 39: an iteration of the last phase at 1,000,000 rows 777 -> 750 us in 2-D, 1,320 -> 1,272 in 3-D.
// With it the gathers' rate binds: four or eight partners in flight per lane instead of two changed nothing at
// 1,000,000 rows. LOSS: the row's loss into p.row_loss, from the tiles' and the mid-near pairs', by the same lanes.
template <int DIM, bool MID, bool LOSS>
__global__ void __launch_bounds__(256) tile_adam_kernel(const GradArgs p, const float* __restrict__ partial,
                                                        const float* __restrict__ partial_loss, uint32_t tiles, int itr) {
  const Sched sc = p.sched[itr];
  const int gl = threadIdx.x & (GRAD_G - 1);
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * (blockDim.x / GRAD_G) + threadIdx.x / GRAD_G;
  if (i >= p.n) return;
  const unsigned gmask = ((1u << GRAD_G) - 1u) << ((threadIdx.x & 31) & ~(GRAD_G - 1));
  const uint32_t s0 = p.rp[3 * i], s1 = p.rp[3 * i + 1], s2 = p.rp[3 * i + 2], s3 = p.rp[3 * i + 3];
  if (s3 - s0 > ROW_MAX) return;  // grad_adam_long_kernel's
  float yi[DIM], acc[DIM];
#pragma unroll
  for (int c = 0; c < DIM; ++c) {
    yi[c] = p.y_cur[i * DIM + c];
    acc[c] = 0.0f;
  }
  float lacc = 0.0f;
  // A row without near and far pairs has only unused places, whose sums are NaN when its y is not finite.
  const uint32_t used = s0 == s1 && s2 == s3 ? 0u : tiles;
#pragma unroll 4
  for (uint32_t t = gl; t < used; t += GRAD_G) {
    const float* src = partial + (static_cast<uint64_t>(t) * p.n + i) * DIM;
    float v[DIM];
    if constexpr (DIM == 2) {
      const float2 q = __ldcs(reinterpret_cast<const float2*>(src));
      v[0] = q.x;
      v[1] = q.y;
    } else {
#pragma unroll
      for (int c = 0; c < DIM; ++c) v[c] = __ldcs(src + c);
    }
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], v[c]);
    if constexpr (LOSS) lacc += __ldcs(partial_loss + static_cast<uint64_t>(t) * p.n + i);
  }
  if constexpr (MID)
    accumulate_segment<DIM, false>(p.y_cur, p.col, s1, s2, gl, GRAD_G, yi, 10000.0f, 20000.0f, sc.w_mn, acc, lacc, LOSS);
#pragma unroll
  for (int o = GRAD_G / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int c = 0; c < DIM; ++c) acc[c] = __fadd_rn(acc[c], __shfl_xor_sync(gmask, acc[c], o, GRAD_G));
    if constexpr (LOSS) lacc += __shfl_xor_sync(gmask, lacc, o, GRAD_G);
  }
  if (gl != 0) return;
  if constexpr (LOSS) p.row_loss[i] = lacc;
  finish_row<DIM>(p, i, acc, yi, sc.lr_t);
}

using ForceFn = void (*)(const ForceArgs, int);
ForceFn force_kernel(uint64_t dim, bool loss) {
  if (dim == 2) return loss ? tile_force_kernel<2, true> : tile_force_kernel<2, false>;
  return loss ? tile_force_kernel<3, true> : tile_force_kernel<3, false>;
}

using AdamFn = void (*)(const GradArgs, const float*, const float*, uint32_t, int);
template <bool LOSS>
AdamFn adam_kernel(uint64_t dim, bool mid) {
  if (dim == 2) return mid ? tile_adam_kernel<2, true, LOSS> : tile_adam_kernel<2, false, LOSS>;
  return mid ? tile_adam_kernel<3, true, LOSS> : tile_adam_kernel<3, false, LOSS>;
}

// The lists for `tiles` tiles; false when too many rows are long ones.
bool build_lists(Ctx& c, const Csr& csr, uint64_t n, uint64_t dim, uint64_t tiles, bool losses, TileGrad& out) {
  out.tiles = static_cast<uint32_t>(tiles);
  out.tile_pts = static_cast<uint32_t>(((n + tiles - 1) / tiles + 3) / 4 * 4);
  out.windows = ceil_div(n, WIN);
  out.ctas = static_cast<uint32_t>(c.sm_count);
  const uint64_t magic = ((1ull << 40) + out.tile_pts - 1) / out.tile_pts;
  const uint64_t units = tiles * out.windows * WIN_UNITS;
  // long rows first: too many of them, and the other form is the better one
  out.long_rows.alloc(c, csr.entries / ROW_MAX + 2);
  uint32_t* count = out.long_rows.get() + csr.entries / ROW_MAX + 1;
  PM_CUDA(cudaMemsetAsync(count, 0, sizeof(uint32_t), c.stream));
  tile_long_rows_kernel<<<ceil_div(n, 256), 256, 0, c.stream>>>(csr.row_ptr.get(), n, out.long_rows.get(), count);
  PM_LAUNCHED();
  DevBuf<uint32_t> words(c, units + 1);
  PM_CUDA(cudaMemsetAsync(words.get() + units, 0, sizeof(uint32_t), c.stream));
  out.meta.alloc(c, units * 32);
  out.unit_off.alloc(c, units + 1);
  const size_t smem_count = static_cast<size_t>(tiles) * WIN * 2;
  const size_t smem_fill = smem_count + static_cast<size_t>(tiles) * WIN;
  tile_count_kernel<<<out.windows, BUILD_T, smem_count, c.stream>>>(csr.row_ptr.get(), csr.col.get(), n, out.tiles,
                                                                    out.tile_pts, magic, out.windows, out.meta.get(),
                                                                    words.get());
  PM_LAUNCHED();
  exclusive_scan_u32(c, words.get(), units + 1, out.unit_off.get());
  uint32_t total = 0;
  PM_CUDA(cudaMemcpyAsync(&out.n_long, count, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaMemcpyAsync(&total, out.unit_off.get() + units, sizeof(uint32_t), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  if (out.n_long > n / 64) return false;
  out.idx.alloc(c, std::max<uint64_t>(2ull * total, 2));
  tile_clear_kernel<<<c.sm_count * 8, 256, 0, c.stream>>>(out.idx.get(), 2ull * total, out.tile_pts * 0x10001u);
  PM_LAUNCHED();
  tile_fill_kernel<<<out.windows, BUILD_T, smem_fill, c.stream>>>(csr.row_ptr.get(), csr.col.get(), n, out.tiles,
                                                                  out.tile_pts, magic, out.windows, out.meta.get(),
                                                                  out.unit_off.get(),
                                                                  reinterpret_cast<uint16_t*>(out.idx.get()));
  PM_LAUNCHED();
  out.cta_units.alloc(c, out.ctas + 1);
  tile_shares_kernel<<<ceil_div(out.ctas + 1, 128), 128, 0, c.stream>>>(out.unit_off.get(), units, out.ctas,
                                                                       out.cta_units.get());
  PM_LAUNCHED();
  out.partial.alloc(c, tiles * n * dim);
  if (losses) out.partial_loss.alloc(c, tiles * n);
  for (const bool loss : {false, true})
    PM_CUDA(cudaFuncSetAttribute(force_kernel(dim, loss), cudaFuncAttributeMaxDynamicSharedMemorySize, TILE_SMEM));
  return true;
}

}  // namespace

bool build_tile_grad(Ctx& c, const Csr& csr, uint64_t n, uint64_t dim, bool losses, TileGrad& out) {
  if ((dim != 2 && dim != 3) || n < TILE_MIN_ROWS || n >= (1ull << 24)) return false;
  const uint64_t fit = (TILE_SMEM / (4 * dim) - 1) / 4 * 4;  // a tile's points and NOWHERE
  const uint64_t tiles = (n + fit - 1) / fit;
  const double per_row = static_cast<double>(csr.entries) / static_cast<double>(n);
  const double near_far = static_cast<double>(csr.entries - csr.entries_mn) / static_cast<double>(n);
  if (tiles > MAX_TILES || per_row > 0.8 * ROW_MAX || near_far < TILE_MIN_ROW_ENTRIES ||
      near_far < tile_min_entries(dim) * static_cast<double>(tiles))
    return false;
  // The lists and the tiles' sums take 1 GB at 1,000,000 rows, which grad_adam_kernel does without.
  bool built = false;
  if (!try_scratch([&] { built = build_lists(c, csr, n, dim, tiles, losses, out); }) || !built) out = TileGrad();
  return built;
}

void launch_tile_grad(const TileGrad& tg, const GradArgs& p, uint64_t dim, int itr, bool mid, cudaStream_t s) {
  ForceArgs f{};
  f.y = p.y_cur;
  f.partial = tg.partial.get();
  f.partial_loss = tg.partial_loss.get();
  f.unit_off = tg.unit_off.get();
  f.idx = reinterpret_cast<const uint2*>(tg.idx.get());
  f.cta_units = tg.cta_units.get();
  f.meta = tg.meta.get();
  f.n = static_cast<uint32_t>(p.n);
  f.tile_pts = tg.tile_pts;
  f.windows = tg.windows;
  f.sched = p.sched;
  const size_t smem = static_cast<size_t>(tg.tile_pts + 1) * dim * sizeof(float);
  const unsigned rows = ceil_div(p.n, 256 / GRAD_G);
  const bool loss = p.row_loss != nullptr;
  force_kernel(dim, loss)<<<tg.ctas, FORCE_T, smem, s>>>(f, itr);
  const AdamFn adam = loss ? adam_kernel<true>(dim, mid) : adam_kernel<false>(dim, mid);
  adam<<<rows, 256, 0, s>>>(p, tg.partial.get(), tg.partial_loss.get(), tg.tiles, itr);
}

namespace {
__global__ void debug_divide_kernel(float num, const float* __restrict__ x, uint64_t n, float* __restrict__ out) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < n; t += stride)
    out[t] = div_by(num, x[t]);
}
}  // namespace

void debug_divide(Ctx& c, float num, const float* d_x, uint64_t n, float* d_out) {
  debug_divide_kernel<<<c.sm_count * 8, 256, 0, c.stream>>>(num, d_x, n, d_out);
  PM_LAUNCHED();
}

}  // namespace pacmap
