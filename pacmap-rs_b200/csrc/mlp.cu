// The learned initialiser (no reference analogue; it lets a shortened schedule replace the plain one): an MLP
// d -> 512 -> 512 -> dim (ReLU) with BF16 weights and activations and FP32 accumulation, trained with
// AdamW on (preprocessed x, PaCMAP embedding) pairs and applied to new data as Initialization::Value
// (src/lib.rs:753-766 rescales it to std 1e-4, so only its geometry matters).
//
// Every GEMM of the forward and backward pass is one hand-written tcgen05 kernel, C = A . B^T with
// both operands K-major BF16 (TMA, 128-byte swizzle, FP32 accumulator in TMEM) and a
// fused epilogue: bias + ReLU -> BF16, ReLU backprop through the stored activation -> BF16, or FP32.
// Operands needed in the other orientation (X^T, H^T, dZ^T, W^T) come from a BF16 transpose kernel.
// FP32 master weights, AdamW (decoupled weight decay), BF16 copies refreshed after each step.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "engine.cuh"
#include "mlp.cuh"
#include "tcgen05.cuh"

namespace pacmap {
namespace {

constexpr int MLP_H = 512;
constexpr int GEMM_THREADS = 192;  // warp 0 TMA, warp 1 MMA + TMEM owner, warps 2..5 epilogue
// Operand pipeline depth. Two stages (66 KB at BN = 128) leave room for three blocks per SM, which overlap each
// other's waits and epilogues; a grid of at most one block per SM has nobody to overlap with and hides the copies
// behind six stages instead.
constexpr int GEMM_STAGES_MANY = 2, GEMM_STAGES_FEW = 6;
constexpr int A_STAGE = 128 * 128;  // 128 rows x 64 bf16

enum Epi : int { EPI_F32 = 0, EPI_BIAS_RELU = 1, EPI_DRELU = 2 };

struct GemmOut {
  float* out_f32;
  __nv_bfloat16* out_bf16;
  const float* bias;
  const __nv_bfloat16* aux;  // the forward activation H (ReLU'(Z) = H > 0)
  int ld_out, ld_aux, m_valid, n_valid;
};

struct alignas(8) GemmShared {
  uint64_t full[GEMM_STAGES_FEW];
  uint64_t empty[GEMM_STAGES_FEW];
  uint64_t done;
  uint32_t tmem_base;
  int abort_flag;
};

template <int BN>
__host__ __device__ constexpr int tmem_cols() {
  return BN <= 32 ? 32 : (BN <= 64 ? 64 : (BN <= 128 ? 128 : 256));
}

template <int BN, int EPI, int GEMM_STAGES>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_tn_kernel(const __grid_constant__ CUtensorMap amap,
                                                                  const __grid_constant__ CUtensorMap bmap, int K,
                                                                  GemmOut o, uint32_t* __restrict__ err) {
  constexpr int B_STAGE = BN * 128;
  extern __shared__ __align__(1024) unsigned char gemm_raw[];
  // aligned by offsetting the shared array itself, so every access keeps the shared address space
  unsigned char* base = gemm_raw + ((1024u - (smem_u32(gemm_raw) & 1023u)) & 1023u);
  unsigned char* a_s = base;
  unsigned char* b_s = base + GEMM_STAGES * A_STAGE;
  GemmShared* sh = reinterpret_cast<GemmShared*>(b_s + GEMM_STAGES * B_STAGE);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * 128, n0 = blockIdx.y * BN;
  const int nk = K / 64;
  if (threadIdx.x == 0) {
    for (int s = 0; s < GEMM_STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    mbar_init(&sh->done, 1);
    sh->abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)),
                 "r"(tmem_cols<BN>()));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sh->tmem_base;
  volatile int* abort_flag = &sh->abort_flag;
  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int kb = 0; kb < nk; ++kb) {
        const int s = kb % GEMM_STAGES;
        if (kb >= GEMM_STAGES && !mbar_wait(&sh->empty[s], ((kb / GEMM_STAGES) + 1) & 1, abort_flag)) break;
        mbar_expect_tx(&sh->full[s], A_STAGE + B_STAGE);
        tma_load_2d(a_s + s * A_STAGE, &amap, &sh->full[s], kb * 64, m0);
        tma_load_2d(b_s + s * B_STAGE, &bmap, &sh->full[s], kb * 64, n0);
        issued = kb + 1;
      }
      if (issued < nk) {
        atomicOr(err, DEV_ERR_TIMEOUT);
        sh->abort_flag = 1;
      }
      for (int kb = (issued > GEMM_STAGES ? issued - GEMM_STAGES : 0); kb < issued; ++kb) {
        const uint64_t t0 = globaltimer();
        while (!mbar_try_wait(&sh->full[kb % GEMM_STAGES], (kb / GEMM_STAGES) & 1) && globaltimer() - t0 < WAIT_LIMIT_NS) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = idesc_f16_mn(true, BN);
      bool ok = true;
      for (int kb = 0; kb < nk; ++kb) {
        const int s = kb % GEMM_STAGES;
        if (!mbar_wait(&sh->full[s], (kb / GEMM_STAGES) & 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint64_t ad = sdesc_sw128(smem_u32(a_s + s * A_STAGE));
        const uint64_t bd = sdesc_sw128(smem_u32(b_s + s * B_STAGE));
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) umma_f16(tmem, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
        umma_commit(&sh->empty[s]);
      }
      if (!ok) {
        atomicOr(err, DEV_ERR_TIMEOUT);
        sh->abort_flag = 1;
      }
      umma_commit(&sh->done);
      // Every issued MMA has completed before the tensor memory is released (bounded, whatever the abort
      // flag: the epilogue's own wait gives up at once on abort).
      const uint64_t t0 = globaltimer();
      while (!mbar_try_wait(&sh->done, 0) && globaltimer() - t0 < WAIT_LIMIT_NS) {
      }
    }
  } else {
    const int quad = warp & 3;
    const int row = m0 + quad * 32 + lane;
    if (mbar_wait(&sh->done, 0, abort_flag) && !*abort_flag) {
      tc_fence_after();
      const uint32_t taddr = tmem + (static_cast<uint32_t>(quad * 32) << 16);
      constexpr int CH = BN < 32 ? BN : 32;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += CH) {
        float v[32];
        if constexpr (CH == 32) {
          tmem_ld32(taddr + c0, v);
        } else {
          float w[16];
          tmem_ld16(taddr + c0, w);
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = w[i];
        }
        if (row < o.m_valid) {
          if (EPI != EPI_F32 && CH == 32 && n0 + c0 + 32 <= o.n_valid && (o.ld_out % 8) == 0 &&
              (EPI != EPI_DRELU || (o.ld_aux % 8) == 0)) {
            // 32 bf16 of this row: four 16-byte stores (and four 16-byte loads of the activation)
            const size_t off = static_cast<size_t>(row) * o.ld_out + n0 + c0;
            uint4* dst = reinterpret_cast<uint4*>(o.out_bf16 + off);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t w[4];
              uint4 hv = make_uint4(0u, 0u, 0u, 0u);
              if (EPI == EPI_DRELU)
                hv = *reinterpret_cast<const uint4*>(o.aux + static_cast<size_t>(row) * o.ld_aux + n0 + c0 + 8 * q);
              const uint32_t hw[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                float lo = v[8 * q + 2 * e], hi = v[8 * q + 2 * e + 1];
                if (EPI == EPI_BIAS_RELU) {
                  lo += o.bias[n0 + c0 + 8 * q + 2 * e];
                  hi += o.bias[n0 + c0 + 8 * q + 2 * e + 1];
                  lo = lo > 0.0f ? lo : 0.0f;
                  hi = hi > 0.0f ? hi : 0.0f;
                } else {
                  const float hl = __uint_as_float(hw[e] << 16), hh = __uint_as_float(hw[e] & 0xFFFF0000u);
                  lo = hl > 0.0f ? lo : 0.0f;
                  hi = hh > 0.0f ? hi : 0.0f;
                }
                w[e] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(lo))) |
                       (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
              }
              dst[q] = make_uint4(w[0], w[1], w[2], w[3]);
            }
          } else {
#pragma unroll
            for (int i = 0; i < CH; ++i) {
              const int col = n0 + c0 + i;
              if (col >= o.n_valid) continue;
              float a = v[i];
              const size_t off = static_cast<size_t>(row) * o.ld_out + col;
              if (EPI == EPI_F32) {
                if (o.bias) a += o.bias[col];
                o.out_f32[off] = a;
              } else if (EPI == EPI_BIAS_RELU) {
                a += o.bias[col];
                o.out_bf16[off] = __float2bfloat16_rn(a > 0.0f ? a : 0.0f);
              } else {
                const float h = __bfloat162float(o.aux[static_cast<size_t>(row) * o.ld_aux + col]);
                o.out_bf16[off] = __float2bfloat16_rn(h > 0.0f ? a : 0.0f);
              }
            }
          }
        }
      }
    } else {
      atomicOr(err, DEV_ERR_TIMEOUT);
      sh->abort_flag = 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols<BN>()));
}

// f32 rows (optionally gathered through `rows`) -> bf16 [rows_pad][cols_pad], zero padded, eight columns per thread and
// 16-byte store (cols_pad a multiple of 8). mean (may be null): the rows are preprocessed on the way, x' = (x - mn) / mx -
// mean, in preprocess_x's f32 arithmetic. One pass over the rows and one 32-bit division per eight elements: 1,000,000 x 128
// took 322 us with a 64-bit division per element, 113 so.
__global__ void __launch_bounds__(256) cast_pad_kernel(const float* __restrict__ src, const uint32_t* __restrict__ rows,
                                                       uint64_t n_rows, int cols, int ld_src, uint64_t rows_pad,
                                                       int cols_pad, __nv_bfloat16* __restrict__ dst, float mn, float mx,
                                                       const float* __restrict__ mean) {
  const uint32_t per_row = static_cast<uint32_t>(cols_pad) / 8;
  const uint64_t total = rows_pad * per_row, stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const bool vec4 = ld_src % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15u) == 0;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride) {
    const uint64_t r = total >> 32 ? t / per_row : static_cast<uint32_t>(t) / per_row;
    const int c0 = static_cast<int>(t - r * per_row) * 8;
    float v[8] = {};
    if (r < n_rows) {
      const float* row = src + (rows ? static_cast<uint64_t>(rows[r]) : r) * ld_src;
      if (vec4 && c0 + 8 <= cols) {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(row + c0);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(row + c0 + 4);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (c0 + e < cols) v[e] = row[c0 + e];
      }
      if (mean)
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (c0 + e < cols) v[e] = __fsub_rn(__fdiv_rn(__fsub_rn(v[e], mn), mx), mean[c0 + e]);
    }
    uint32_t w[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      w[e] = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[2 * e]))) |
             (static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(v[2 * e + 1]))) << 16);
    reinterpret_cast<uint4*>(dst)[t] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The first dim of ld columns of the network's output, y = v * std + mean with ms (mean[dim], std[dim]; may be null).
__global__ void finish_rows_kernel(const float* __restrict__ src, int ld, uint64_t n, int dim,
                                   const float* __restrict__ ms, float* __restrict__ out) {
  const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n * dim) return;
  const uint64_t r = t / dim;
  const int c = static_cast<int>(t - r * dim);
  const float v = src[r * ld + c];
  out[t] = ms ? __fadd_rn(__fmul_rn(v, ms[dim + c]), ms[c]) : v;
}

// The flat f32 parameters into the forward pass's operands: W1b [512][dp], W2b, W3b [dp16][512] in bf16, f32 biases.
struct OperandArgs {
  __nv_bfloat16 *W1b, *W2b, *W3b;
  float *b1, *b2, *b3;
  int d, dp, dim, dp16;
};
__global__ void __launch_bounds__(256) unpack_operands_kernel(const float* __restrict__ flat, OperandArgs a) {
  const uint32_t h = MLP_H, n1 = h * a.dp, n2 = h * h, n3 = a.dp16 * h;
  uint32_t t = blockIdx.x * 256 + threadIdx.x;
  const float *b1 = flat + static_cast<size_t>(h) * a.d, *w2 = b1 + h, *b2 = w2 + n2, *w3 = b2 + h, *b3 = w3 + h * a.dim;
  if (t < n1) {
    const uint32_t j = t / a.dp, i = t - j * a.dp;
    a.W1b[t] = __float2bfloat16_rn(i < static_cast<uint32_t>(a.d) ? flat[j * a.d + i] : 0.0f);
    return;
  }
  if ((t -= n1) < n2) {
    a.W2b[t] = __float2bfloat16_rn(w2[t]);
    return;
  }
  if ((t -= n2) < n3) {
    a.W3b[t] = __float2bfloat16_rn(t < h * a.dim ? w3[t] : 0.0f);
    return;
  }
  if ((t -= n3) < h) {
    a.b1[t] = b1[t];
  } else if ((t -= h) < h) {
    a.b2[t] = b2[t];
  } else if ((t -= h) < static_cast<uint32_t>(a.dp16)) {
    a.b3[t] = t < static_cast<uint32_t>(a.dim) ? b3[t] : 0.0f;
  }
}

// bf16 [R][C] -> bf16 [C][R] (32 x 32 tiles through shared memory).
__global__ void transpose_bf16_kernel(const __nv_bfloat16* __restrict__ src, int R, int C,
                                      __nv_bfloat16* __restrict__ dst) {
  __shared__ __nv_bfloat16 tile[32][33];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    tile[i][threadIdx.x] = (r < R && c < C) ? src[static_cast<size_t>(r) * C + c] : __float2bfloat16_rn(0.0f);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (c < C && r < R) dst[static_cast<size_t>(c) * R + r] = tile[threadIdx.x][i];
  }
}

// MSE: out [B][ld_out] (first `dim` columns), target [B][dim] -> dZ = 2 (out - t) / (B dim) as bf16
// [B][ld_dz] (zero padded) and per-block partial sums of squared errors.
__global__ void mse_grad_kernel(const float* __restrict__ out, int ld_out, const float* __restrict__ target, int B,
                                int dim, int ld_dz, __nv_bfloat16* __restrict__ dz, double* __restrict__ partial) {
  __shared__ double red[256];
  double s = 0.0;
  const float scale = 2.0f / static_cast<float>(B * dim);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < B * ld_dz; t += gridDim.x * blockDim.x) {
    const int r = t / ld_dz, c = t % ld_dz;
    float g = 0.0f;
    if (c < dim) {
      const float e = out[static_cast<size_t>(r) * ld_out + c] - target[static_cast<size_t>(r) * dim + c];
      s += static_cast<double>(e) * e;
      g = scale * e;
    }
    dz[t] = __float2bfloat16_rn(g);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}

// Bias gradients: column sums of a layer's dZ (bf16 [R][ld], its first C columns), each column one serial sum
// in row order. The three layers run side by side in one launch (grid y = layer), a block per 32 columns: the rows
// go through shared memory in double-buffered slices of CS_ROWS (16-byte asynchronous copies, 64 bytes per row) and
// one warp adds them, a column per lane. Bound by the chain of R additions: about 10 us for 4096 rows, where one
// thread per column reading global memory itself took 244 us a layer (80 % of a training step).
constexpr int CS_ROWS = 256, CS_COLS = 32, CS_THREADS = 256;
struct ColsumArgs {
  const __nv_bfloat16* src[3];
  float* out[3];
  int cols[3], ld[3];  // ld a multiple of 8 and at least the columns rounded up to 32
};

__global__ void __launch_bounds__(CS_THREADS) colsum_bf16_kernel(ColsumArgs a, int R) {
  __shared__ __align__(16) __nv_bfloat16 buf[2][CS_ROWS][CS_COLS];
  const int q = blockIdx.y, c0 = blockIdx.x * CS_COLS;
  if (c0 >= a.cols[q]) return;
  const __nv_bfloat16* src = a.src[q] + c0;
  const size_t ld = a.ld[q];
  auto stage = [&](int r0, int b) {
    for (int e = threadIdx.x; e < CS_ROWS * 4; e += CS_THREADS) {
      const int r = e >> 2, part = (e & 3) * 8;
      if (r0 + r < R) cp_async16(&buf[b][r][part], src + (r0 + r) * ld + part);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float s = 0.0f;
  stage(0, 0);
  for (int r0 = 0, b = 0; r0 < R; r0 += CS_ROWS, b ^= 1) {
    if (r0 + CS_ROWS < R) {
      stage(r0 + CS_ROWS, b ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x < CS_COLS) {
      const int m = min(CS_ROWS, R - r0);
#pragma unroll 16
      for (int r = 0; r < m; ++r) s += __bfloat162float(buf[b][r][threadIdx.x]);
    }
    __syncthreads();
  }
  const int c = c0 + threadIdx.x;
  if (threadIdx.x < CS_COLS && c < a.cols[q]) a.out[q][c] = s;
}

// dst[r][c] = src[rows[r]][c] (f32, dim columns).
__global__ void gather_rows_kernel(const float* __restrict__ src, const uint32_t* __restrict__ rows, uint64_t n_rows,
                                   int dim, float* __restrict__ dst) {
  const uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= n_rows * dim) return;
  const uint64_t r = t / dim;
  dst[t] = src[static_cast<uint64_t>(rows[r]) * dim + (t % dim)];
}

// One AdamW step (decoupled weight decay on the weights, not on the biases) of all six tensors in one launch, each
// thread writing its parameter's bf16 copies in the operand layouts too: W1b, W2b and W2^T, W3 and its padded
// transpose (the padding columns stay the zeros that MlpNet::refresh wrote). A step's 330,000 parameters are a few
// microseconds of traffic, so what counts is the launches: this one replaces 12.
struct AdamArgs {
  float *p[6], *m[6], *v[6];
  const float* g[6];
  uint32_t end[6];  // running ends of the tensors in the flat index
  __nv_bfloat16 *W1b, *W2b, *W2Tb, *W3b, *W3Tb;
  int dp16, dp64;
};

__global__ void __launch_bounds__(256) adamw_kernel(AdamArgs a, float lr, float wd, float b1c, float b2c) {
  const uint32_t i = blockIdx.x * 256 + threadIdx.x;
  if (i >= a.end[5]) return;
  int q = 0;
  while (i >= a.end[q]) ++q;
  const uint32_t t = i - (q ? a.end[q - 1] : 0u);
  const float decay = (q % 2 == 0) ? wd : 0.0f;
  const float gg = a.g[q][t];
  float mm = 0.9f * a.m[q][t] + 0.1f * gg;
  float vv = 0.999f * a.v[q][t] + 0.001f * gg * gg;
  a.m[q][t] = mm;
  a.v[q][t] = vv;
  float w = a.p[q][t] * (1.0f - lr * decay);
  w -= lr * (mm / b1c) / (sqrtf(vv / b2c) + 1e-8f);
  a.p[q][t] = w;
  const __nv_bfloat16 wb = __float2bfloat16_rn(w);
  if (q == 0) {
    a.W1b[t] = wb;
  } else if (q == 2) {
    a.W2b[t] = wb;
    a.W2Tb[(t % MLP_H) * MLP_H + t / MLP_H] = wb;
  } else if (q == 4) {  // W3T [512][dp16]
    const uint32_t r = t / a.dp16, c = t % a.dp16;
    a.W3b[c * MLP_H + r] = wb;
    a.W3Tb[r * a.dp64 + c] = wb;
  }
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, uint64_t count, __nv_bfloat16* __restrict__ dst) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < count; t += stride)
    dst[t] = __float2bfloat16_rn(src[t]);
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
inline int pad_to(int v, int m) { return (v + m - 1) / m * m; }

template <int BN, int EPI, int STAGES>
void gemm_launch(Ctx& c, const CUtensorMap& am, const CUtensorMap& bm, dim3 grid, int K, const GemmOut& o) {
  const size_t smem = 1024 + STAGES * (A_STAGE + BN * 128) + sizeof(GemmShared);
  PM_CUDA(cudaFuncSetAttribute(gemm_tn_kernel<BN, EPI, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem)));
  gemm_tn_kernel<BN, EPI, STAGES><<<grid, GEMM_THREADS, smem, c.stream>>>(am, bm, K, o, c.d_err);
  PM_LAUNCHED();
}

template <int BN, int EPI>
void gemm(Ctx& c, const __nv_bfloat16* A, int M_rows_alloc, const __nv_bfloat16* Bm, int N_rows_alloc, int K,
          const GemmOut& o) {
  // 32 columns a block where that still gives at most one block per SM: a block's K loop is bound by its operand copies
  // (160 rows of 128 bytes a step instead of 256), and more of them run. 512 x 512 and 512 x 128 of K = 4,096: 27 us each
  // against 33 with 128 columns; twice the stages changed nothing.
  if constexpr (BN >= 64) {
    if (M_rows_alloc / 128 * ((N_rows_alloc + 31) / 32) <= c.sm_count)
      return gemm<32, EPI>(c, A, M_rows_alloc, Bm, N_rows_alloc, K, o);
  }
  const CUtensorMap am = make_tmap_2d_16b(A, M_rows_alloc, K, 128, true);
  const CUtensorMap bm = make_tmap_2d_16b(Bm, N_rows_alloc, K, BN, true);
  const dim3 grid(static_cast<unsigned>(M_rows_alloc / 128), static_cast<unsigned>((N_rows_alloc + BN - 1) / BN));
  if (grid.x * grid.y <= static_cast<unsigned>(c.sm_count)) gemm_launch<BN, EPI, GEMM_STAGES_FEW>(c, am, bm, grid, K, o);
  else gemm_launch<BN, EPI, GEMM_STAGES_MANY>(c, am, bm, grid, K, o);
}

void transpose(Ctx& c, const __nv_bfloat16* src, int R, int C, __nv_bfloat16* dst) {
  transpose_bf16_kernel<<<dim3(ceil_div(C, 32), ceil_div(R, 32)), dim3(32, 8), 0, c.stream>>>(src, R, C, dst);
  PM_LAUNCHED();
}

void cast_pad(Ctx& c, const float* src, const uint32_t* rows, uint64_t n_rows, int cols, int ld_src,
              uint64_t rows_pad, int cols_pad, __nv_bfloat16* dst, float mn = 0.0f, float mx = 1.0f,
              const float* mean = nullptr) {
  const uint64_t total = rows_pad * (cols_pad / 8);
  cast_pad_kernel<<<static_cast<unsigned>(std::min<uint64_t>(ceil_div(total, 256), c.sm_count * 16ull)), 256, 0,
                    c.stream>>>(src, rows, n_rows, cols, ld_src, rows_pad, cols_pad, dst, mn, mx, mean);
  PM_LAUNCHED();
}

}  // namespace

// Network state on the device: f32 masters in GEMM-friendly layouts, their bf16 copies and moments.
struct MlpNet {
  int d = 0, dp = 0, dim = 0, dp16 = 16, dp64 = 64;
  DevBuf<float> W1, b1, W2, b2, W3T, b3;            // W1 [512][dp], W2 [512][512], W3T [512][dp16], b3 [dp16]
  DevBuf<__nv_bfloat16> W1b, W2b, W3b, W2Tb, W3Tb;   // W3b [dp16][512], W2Tb [512][512], W3Tb [512][dp64]
  void alloc(Ctx& c, int d_, int dim_) {
    d = d_;
    dim = dim_;
    dp = pad_to(d, 64);
    dp16 = pad_to(dim, 16);
    dp64 = pad_to(dim, 64);
    W1.alloc(c, static_cast<size_t>(MLP_H) * dp);
    b1.alloc(c, MLP_H);
    W2.alloc(c, static_cast<size_t>(MLP_H) * MLP_H);
    b2.alloc(c, MLP_H);
    W3T.alloc(c, static_cast<size_t>(MLP_H) * dp16);
    b3.alloc(c, dp16);
    W1b.alloc(c, W1.count);
    W2b.alloc(c, W2.count);
    W3b.alloc(c, static_cast<size_t>(dp16) * MLP_H);
    W2Tb.alloc(c, W2.count);
    W3Tb.alloc(c, static_cast<size_t>(MLP_H) * dp64);
  }
  // What the forward pass alone needs, from the flat host layout: one copy and one launch.
  void upload_operands(Ctx& c, const float* flat, int d_, int dim_) {
    d = d_;
    dim = dim_;
    dp = pad_to(d, 64);
    dp16 = pad_to(dim, 16);
    W1b.alloc(c, static_cast<size_t>(MLP_H) * dp);
    W2b.alloc(c, static_cast<size_t>(MLP_H) * MLP_H);
    W3b.alloc(c, static_cast<size_t>(dp16) * MLP_H);
    b1.alloc(c, MLP_H);
    b2.alloc(c, MLP_H);
    b3.alloc(c, dp16);
    DevBuf<float> df;
    pacmap::upload(c, df, flat, mlp_param_count(d, dim));
    const OperandArgs a{W1b.get(), W2b.get(), W3b.get(), b1.get(), b2.get(), b3.get(), d, dp, dim, dp16};
    unpack_operands_kernel<<<ceil_div(W1b.count + W2b.count + W3b.count + 2 * MLP_H + dp16, 256), 256, 0, c.stream>>>(
        df.get(), a);
    PM_LAUNCHED();
  }
  // flat host layout [W1 (512 x d), b1, W2 (512 x 512), b2, W3 (dim x 512), b3] <-> device layouts
  void upload(Ctx& c, const float* flat) {
    std::vector<float> w1(W1.count, 0.0f), w3t(W3T.count, 0.0f), bb3(dp16, 0.0f);
    const float* p = flat;
    for (int j = 0; j < MLP_H; ++j)
      for (int i = 0; i < d; ++i) w1[static_cast<size_t>(j) * dp + i] = p[static_cast<size_t>(j) * d + i];
    p += static_cast<size_t>(MLP_H) * d;
    PM_CUDA(cudaMemcpyAsync(W1.get(), w1.data(), W1.bytes(), cudaMemcpyHostToDevice, c.stream));
    PM_CUDA(cudaMemcpyAsync(b1.get(), p, MLP_H * 4, cudaMemcpyHostToDevice, c.stream));
    p += MLP_H;
    PM_CUDA(cudaMemcpyAsync(W2.get(), p, W2.bytes(), cudaMemcpyHostToDevice, c.stream));
    p += static_cast<size_t>(MLP_H) * MLP_H;
    PM_CUDA(cudaMemcpyAsync(b2.get(), p, MLP_H * 4, cudaMemcpyHostToDevice, c.stream));
    p += MLP_H;
    for (int k = 0; k < dim; ++k)
      for (int i = 0; i < MLP_H; ++i) w3t[static_cast<size_t>(i) * dp16 + k] = p[static_cast<size_t>(k) * MLP_H + i];
    p += static_cast<size_t>(dim) * MLP_H;
    for (int k = 0; k < dim; ++k) bb3[k] = p[k];
    PM_CUDA(cudaMemcpyAsync(W3T.get(), w3t.data(), W3T.bytes(), cudaMemcpyHostToDevice, c.stream));
    PM_CUDA(cudaMemcpyAsync(b3.get(), bb3.data(), b3.bytes(), cudaMemcpyHostToDevice, c.stream));
    PM_CUDA(cudaStreamSynchronize(c.stream));
    refresh(c);
  }
  void download(Ctx& c, float* flat) {
    std::vector<float> w1(W1.count), w3t(W3T.count), bb3(dp16);
    PM_CUDA(cudaMemcpyAsync(w1.data(), W1.get(), W1.bytes(), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaMemcpyAsync(w3t.data(), W3T.get(), W3T.bytes(), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaMemcpyAsync(bb3.data(), b3.get(), b3.bytes(), cudaMemcpyDeviceToHost, c.stream));
    float* p = flat;
    float* pb1 = p + static_cast<size_t>(MLP_H) * d;
    float* pW2 = pb1 + MLP_H;
    float* pb2 = pW2 + static_cast<size_t>(MLP_H) * MLP_H;
    float* pW3 = pb2 + MLP_H;
    float* pb3 = pW3 + static_cast<size_t>(dim) * MLP_H;
    PM_CUDA(cudaMemcpyAsync(pb1, b1.get(), MLP_H * 4, cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaMemcpyAsync(pW2, W2.get(), W2.bytes(), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaMemcpyAsync(pb2, b2.get(), MLP_H * 4, cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaStreamSynchronize(c.stream));
    for (int j = 0; j < MLP_H; ++j)
      for (int i = 0; i < d; ++i) p[static_cast<size_t>(j) * d + i] = w1[static_cast<size_t>(j) * dp + i];
    for (int k = 0; k < dim; ++k)
      for (int i = 0; i < MLP_H; ++i) pW3[static_cast<size_t>(k) * MLP_H + i] = w3t[static_cast<size_t>(i) * dp16 + k];
    for (int k = 0; k < dim; ++k) pb3[k] = bb3[k];
  }
  // bf16 copies in the operand layouts: W1b = W1, W2b = W2, W2Tb = W2^T, W3b = W3 [dp16][512] (=W3T^T),
  // W3Tb = W3T padded to dp64 columns.
  void refresh(Ctx& c) {
    f32_to_bf16_kernel<<<256, 256, 0, c.stream>>>(W1.get(), W1.count, W1b.get());
    PM_LAUNCHED();
    f32_to_bf16_kernel<<<256, 256, 0, c.stream>>>(W2.get(), W2.count, W2b.get());
    PM_LAUNCHED();
    transpose(c, W2b.get(), MLP_H, MLP_H, W2Tb.get());
    DevBuf<__nv_bfloat16> w3tb(c, W3T.count);
    f32_to_bf16_kernel<<<64, 256, 0, c.stream>>>(W3T.get(), W3T.count, w3tb.get());
    PM_LAUNCHED();
    transpose(c, w3tb.get(), MLP_H, dp16, W3b.get());
    cast_pad(c, W3T.get(), nullptr, MLP_H, dp16, dp16, MLP_H, dp64, W3Tb.get());
  }
};

namespace {

// Forward through the network: X bf16 [rows][dp] (rows a multiple of 128) -> H1, H2 bf16 [rows][512],
// out f32 [rows][dp16].
void mlp_forward(Ctx& c, MlpNet& net, const __nv_bfloat16* X, int rows, __nv_bfloat16* H1, __nv_bfloat16* H2,
                 float* out, int m_valid) {
  GemmOut o{};
  o.bias = net.b1.get();
  o.out_bf16 = H1;
  o.ld_out = MLP_H;
  o.m_valid = m_valid;
  o.n_valid = MLP_H;
  gemm<128, EPI_BIAS_RELU>(c, X, rows, net.W1b.get(), MLP_H, net.dp, o);
  o.bias = net.b2.get();
  o.out_bf16 = H2;
  gemm<128, EPI_BIAS_RELU>(c, H1, rows, net.W2b.get(), MLP_H, MLP_H, o);
  GemmOut f{};
  f.bias = net.b3.get();
  f.out_f32 = out;
  f.ld_out = net.dp16;
  f.m_valid = m_valid;
  f.n_valid = net.dp16;
  gemm<16, EPI_F32>(c, H2, rows, net.W3b.get(), net.dp16, MLP_H, f);
}

constexpr int LOSS_PARTS = 64;  // blocks of mse_grad_kernel

// Scratch for one batch of B rows.
struct MlpBatch {
  int B = 0;
  DevBuf<__nv_bfloat16> X, XT, H1, H1T, H2, H2T, dZ3, dZ3T, dZ2, dZ2T, dZ1, dZ1T;
  DevBuf<float> out, tgt, gW1, gb1, gW2, gb2, gW3T, gb3;
  DevBuf<double> partial;  // LOSS_PARTS partial losses per step, of `steps` steps
  void alloc(Ctx& c, const MlpNet& net, int B_, uint64_t steps = 1) {
    B = B_;
    X.alloc(c, static_cast<size_t>(B) * net.dp);
    XT.alloc(c, static_cast<size_t>(B) * net.dp);
    H1.alloc(c, static_cast<size_t>(B) * MLP_H);
    H1T.alloc(c, static_cast<size_t>(B) * MLP_H);
    H2.alloc(c, static_cast<size_t>(B) * MLP_H);
    H2T.alloc(c, static_cast<size_t>(B) * MLP_H);
    dZ3.alloc(c, static_cast<size_t>(B) * net.dp64);
    dZ3T.alloc(c, static_cast<size_t>(B) * net.dp16);
    dZ2.alloc(c, static_cast<size_t>(B) * MLP_H);
    dZ2T.alloc(c, static_cast<size_t>(B) * MLP_H);
    dZ1.alloc(c, static_cast<size_t>(B) * MLP_H);
    dZ1T.alloc(c, static_cast<size_t>(B) * MLP_H);
    out.alloc(c, static_cast<size_t>(B) * net.dp16);
    tgt.alloc(c, static_cast<size_t>(B) * net.dim);
    gW1.alloc(c, net.W1.count);
    gb1.alloc(c, MLP_H);
    gW2.alloc(c, net.W2.count);
    gb2.alloc(c, MLP_H);
    gW3T.alloc(c, net.W3T.count);
    gb3.alloc(c, net.dp16);
    partial.alloc(c, LOSS_PARTS * steps);
  }
};

// Forward + backward of one batch (X and tgt already filled); gradients into bt.g*, returns nothing
// (the loss partials go to bt.partial, slot `step`).
void mlp_forward_backward(Ctx& c, MlpNet& net, MlpBatch& bt, uint64_t step = 0) {
  const int B = bt.B;
  mlp_forward(c, net, bt.X.get(), B, bt.H1.get(), bt.H2.get(), bt.out.get(), B);
  mse_grad_kernel<<<LOSS_PARTS, 256, 0, c.stream>>>(bt.out.get(), net.dp16, bt.tgt.get(), B, net.dim, net.dp64,
                                                   bt.dZ3.get(), bt.partial.get() + step * LOSS_PARTS);
  PM_LAUNCHED();
  // dW3^T [512][dp16] = H2^T . dZ3  (A = H2^T [512][B], B = dZ3^T [dp16][B], K = B)
  transpose(c, bt.H2.get(), B, MLP_H, bt.H2T.get());
  // dZ3^T [dp16][B]: transpose [B][dp64] into scratch [dp64][B] (dZ1T has room), keep its first dp16 rows
  transpose(c, bt.dZ3.get(), B, net.dp64, bt.dZ1T.get());
  PM_CUDA(cudaMemcpyAsync(bt.dZ3T.get(), bt.dZ1T.get(), static_cast<size_t>(net.dp16) * B * 2, cudaMemcpyDeviceToDevice,
                          c.stream));
  GemmOut g3{};
  g3.out_f32 = bt.gW3T.get();
  g3.ld_out = net.dp16;
  g3.m_valid = MLP_H;
  g3.n_valid = net.dp16;
  gemm<16, EPI_F32>(c, bt.H2T.get(), MLP_H, bt.dZ3T.get(), net.dp16, B, g3);
  // dZ2 = (dZ3 . W3) * relu'(H2): A = dZ3 [B][dp64], B = W3Tb [512][dp64], K = dp64
  GemmOut g2{};
  g2.out_bf16 = bt.dZ2.get();
  g2.aux = bt.H2.get();
  g2.ld_out = MLP_H;
  g2.ld_aux = MLP_H;
  g2.m_valid = B;
  g2.n_valid = MLP_H;
  gemm<128, EPI_DRELU>(c, bt.dZ3.get(), B, net.W3Tb.get(), MLP_H, net.dp64, g2);
  // dW2 [512][512] = dZ2^T . H1 (A = dZ2^T [512][B], B = H1^T [512][B], K = B)
  transpose(c, bt.dZ2.get(), B, MLP_H, bt.dZ2T.get());
  transpose(c, bt.H1.get(), B, MLP_H, bt.H1T.get());
  GemmOut w2{};
  w2.out_f32 = bt.gW2.get();
  w2.ld_out = MLP_H;
  w2.m_valid = MLP_H;
  w2.n_valid = MLP_H;
  gemm<128, EPI_F32>(c, bt.dZ2T.get(), MLP_H, bt.H1T.get(), MLP_H, B, w2);
  // dZ1 = (dZ2 . W2) * relu'(H1): A = dZ2 [B][512], B = W2^T [512][512], K = 512
  GemmOut g1{};
  g1.out_bf16 = bt.dZ1.get();
  g1.aux = bt.H1.get();
  g1.ld_out = MLP_H;
  g1.ld_aux = MLP_H;
  g1.m_valid = B;
  g1.n_valid = MLP_H;
  gemm<128, EPI_DRELU>(c, bt.dZ2.get(), B, net.W2Tb.get(), MLP_H, MLP_H, g1);
  // dW1 [512][dp] = dZ1^T . X (A = dZ1^T [512][B], B = X^T [dp][B], K = B)
  transpose(c, bt.dZ1.get(), B, MLP_H, bt.dZ1T.get());
  transpose(c, bt.X.get(), B, net.dp, bt.XT.get());
  GemmOut w1{};
  w1.out_f32 = bt.gW1.get();
  w1.ld_out = net.dp;
  w1.m_valid = MLP_H;
  w1.n_valid = net.dp;
  if (net.dp % 128 == 0)
    gemm<128, EPI_F32>(c, bt.dZ1T.get(), MLP_H, bt.XT.get(), net.dp, B, w1);
  else
    gemm<64, EPI_F32>(c, bt.dZ1T.get(), MLP_H, bt.XT.get(), net.dp, B, w1);
  const ColsumArgs cs{{bt.dZ1.get(), bt.dZ2.get(), bt.dZ3.get()},
                      {bt.gb1.get(), bt.gb2.get(), bt.gb3.get()},
                      {MLP_H, MLP_H, net.dp16},
                      {MLP_H, MLP_H, net.dp64}};
  colsum_bf16_kernel<<<dim3(MLP_H / CS_COLS, 3), CS_THREADS, 0, c.stream>>>(cs, B);
  PM_LAUNCHED();
}

void adamw_step(Ctx& c, MlpNet& net, MlpBatch& bt, std::vector<DevBuf<float>>& mom, float lr, float wd, int t) {
  const float b1c = 1.0f - std::pow(0.9f, static_cast<float>(t));
  const float b2c = 1.0f - std::pow(0.999f, static_cast<float>(t));
  float* P[6] = {net.W1.get(), net.b1.get(), net.W2.get(), net.b2.get(), net.W3T.get(), net.b3.get()};
  const float* G[6] = {bt.gW1.get(), bt.gb1.get(), bt.gW2.get(), bt.gb2.get(), bt.gW3T.get(), bt.gb3.get()};
  const size_t N[6] = {net.W1.count, net.b1.count, net.W2.count, net.b2.count, net.W3T.count, net.b3.count};
  AdamArgs a{};
  uint32_t end = 0;  // d <= 4096: below 2^22 parameters
  for (int q = 0; q < 6; ++q) {
    a.p[q] = P[q];
    a.g[q] = G[q];
    a.m[q] = mom[2 * q].get();
    a.v[q] = mom[2 * q + 1].get();
    a.end[q] = end += static_cast<uint32_t>(N[q]);
  }
  a.W1b = net.W1b.get();
  a.W2b = net.W2b.get();
  a.W2Tb = net.W2Tb.get();
  a.W3b = net.W3b.get();
  a.W3Tb = net.W3Tb.get();
  a.dp16 = net.dp16;
  a.dp64 = net.dp64;
  adamw_kernel<<<ceil_div(end, 256), 256, 0, c.stream>>>(a, lr, wd, b1c, b2c);
  PM_LAUNCHED();
}

}  // namespace

uint64_t mlp_param_count(uint64_t d, uint64_t dim) {
  return static_cast<uint64_t>(MLP_H) * d + MLP_H + static_cast<uint64_t>(MLP_H) * MLP_H + MLP_H + dim * MLP_H + dim;
}

void mlp_init_params(uint64_t d, uint64_t dim, uint64_t seed, float* flat) {
  // PyTorch-style default: U(-1/sqrt(fan_in), 1/sqrt(fan_in)) for weights and biases, seeded.
  std::mt19937_64 rng(seed);
  auto fill = [&](float* p, uint64_t cnt, double fan_in) {
    std::uniform_real_distribution<double> u(-1.0 / std::sqrt(fan_in), 1.0 / std::sqrt(fan_in));
    for (uint64_t i = 0; i < cnt; ++i) p[i] = static_cast<float>(u(rng));
  };
  float* p = flat;
  fill(p, MLP_H * d, static_cast<double>(d));
  p += MLP_H * d;
  fill(p, MLP_H, static_cast<double>(d));
  p += MLP_H;
  fill(p, static_cast<uint64_t>(MLP_H) * MLP_H, MLP_H);
  p += static_cast<uint64_t>(MLP_H) * MLP_H;
  fill(p, MLP_H, MLP_H);
  p += MLP_H;
  fill(p, dim * MLP_H, MLP_H);
  p += dim * MLP_H;
  fill(p, dim, MLP_H);
}

void mlp_apply_device(Ctx& c, const float* params, uint64_t d, uint64_t dim, const float* d_x, uint64_t n,
                      float* d_out, const MlpAffine& around) {
  PM_REQUIRE(d >= 1 && d <= 4096 && dim >= 1 && dim <= 16, PACMAP_ERR_UNSUPPORTED, "MLP supports d <= 4096, dim <= 16");
  MlpNet net;
  net.upload_operands(c, params, static_cast<int>(d), static_cast<int>(dim));
  DevBuf<float> consts;  // mean [d], then t_mean and t_std [dim each]
  std::vector<float> hc(d + 2 * dim, 0.0f);
  if (around.pre_mean) std::copy(around.pre_mean, around.pre_mean + d, hc.begin());
  if (around.t_mean) {
    std::copy(around.t_mean, around.t_mean + dim, hc.begin() + d);
    std::copy(around.t_std, around.t_std + dim, hc.begin() + d + dim);
  }
  if (around.pre_mean || around.t_mean) upload(c, consts, hc.data(), hc.size());
  const uint64_t chunk = std::min<uint64_t>((n + 127) / 128 * 128, 1ull << 20);  // rows per pass (bounded scratch)
  DevBuf<__nv_bfloat16> X(c, chunk * net.dp), H1(c, chunk * MLP_H), H2(c, chunk * MLP_H);
  DevBuf<float> out(c, chunk * net.dp16);
  for (uint64_t r0 = 0; r0 < n; r0 += chunk) {
    const uint64_t rows = std::min<uint64_t>(chunk, n - r0);
    const int rows_pad = pad_to(static_cast<int>(rows), 128);
    cast_pad(c, d_x + r0 * d, nullptr, rows, static_cast<int>(d), static_cast<int>(d), rows_pad, net.dp, X.get(),
             around.pre_min, around.pre_max, around.pre_mean ? consts.get() : nullptr);
    mlp_forward(c, net, X.get(), rows_pad, H1.get(), H2.get(), out.get(), static_cast<int>(rows));
    finish_rows_kernel<<<ceil_div(rows * dim, 256), 256, 0, c.stream>>>(
        out.get(), net.dp16, rows, static_cast<int>(dim), around.t_mean ? consts.get() + d : nullptr, d_out + r0 * dim);
    PM_LAUNCHED();
  }
  c.check_errors("MLP inference");
}

void mlp_grad_device(Ctx& c, const float* params, uint64_t d, uint64_t dim, const float* d_x, const float* d_t,
                     uint64_t B, float* grads_flat, float* loss) {
  PM_REQUIRE(B % 128 == 0 && B > 0, PACMAP_ERR_UNSUPPORTED, "MLP batch must be a positive multiple of 128");
  MlpNet net;
  net.alloc(c, static_cast<int>(d), static_cast<int>(dim));
  net.upload(c, params);
  MlpBatch bt;
  bt.alloc(c, net, static_cast<int>(B));
  cast_pad(c, d_x, nullptr, B, static_cast<int>(d), static_cast<int>(d), B, net.dp, bt.X.get());
  PM_CUDA(cudaMemcpyAsync(bt.tgt.get(), d_t, B * dim * 4, cudaMemcpyDeviceToDevice, c.stream));
  mlp_forward_backward(c, net, bt);
  // gradients into the flat layout (reuse the download path through a scratch network)
  MlpNet g;
  g.alloc(c, static_cast<int>(d), static_cast<int>(dim));
  PM_CUDA(cudaMemcpyAsync(g.W1.get(), bt.gW1.get(), bt.gW1.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaMemcpyAsync(g.b1.get(), bt.gb1.get(), bt.gb1.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaMemcpyAsync(g.W2.get(), bt.gW2.get(), bt.gW2.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaMemcpyAsync(g.b2.get(), bt.gb2.get(), bt.gb2.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaMemcpyAsync(g.W3T.get(), bt.gW3T.get(), bt.gW3T.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  PM_CUDA(cudaMemcpyAsync(g.b3.get(), bt.gb3.get(), bt.gb3.bytes(), cudaMemcpyDeviceToDevice, c.stream));
  g.download(c, grads_flat);
  std::vector<double> part(LOSS_PARTS);
  PM_CUDA(cudaMemcpyAsync(part.data(), bt.partial.get(), bt.partial.bytes(), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  double s = 0.0;
  for (double v : part) s += v;
  *loss = static_cast<float>(s / static_cast<double>(B * dim));
  c.check_errors("MLP gradient");
}

void mlp_train_device(Ctx& c, float* params, uint64_t d, uint64_t dim, const float* d_x, const float* d_t,
                      uint64_t n, uint64_t epochs, uint64_t batch, float lr, float wd, uint64_t seed,
                      float* epoch_loss) {
  PM_REQUIRE(batch % 128 == 0 && batch > 0 && batch <= n, PACMAP_ERR_UNSUPPORTED,
             "MLP batch must be a positive multiple of 128 and at most n");
  MlpNet net;
  net.alloc(c, static_cast<int>(d), static_cast<int>(dim));
  net.upload(c, params);
  MlpBatch bt;
  const uint64_t steps = n / batch;
  bt.alloc(c, net, static_cast<int>(batch), steps);
  std::vector<DevBuf<float>> mom(12);
  const uint64_t cnt[6] = {net.W1.count, net.b1.count, net.W2.count, net.b2.count, net.W3T.count, net.b3.count};
  for (int q = 0; q < 6; ++q) {
    mom[2 * q].alloc(c, cnt[q]);
    mom[2 * q + 1].alloc(c, cnt[q]);
    PM_CUDA(cudaMemsetAsync(mom[2 * q].get(), 0, cnt[q] * 4, c.stream));
    PM_CUDA(cudaMemsetAsync(mom[2 * q + 1].get(), 0, cnt[q] * 4, c.stream));
  }
  std::vector<uint32_t> perm(n);
  DevBuf<uint32_t> dperm(c, n);
  std::mt19937_64 rng(seed);
  std::vector<double> part(LOSS_PARTS * steps);
  int t = 0;
  for (uint64_t ep = 0; ep < epochs; ++ep) {
    for (uint64_t i = 0; i < n; ++i) perm[i] = static_cast<uint32_t>(i);
    std::shuffle(perm.begin(), perm.end(), rng);
    PM_CUDA(cudaMemcpyAsync(dperm.get(), perm.data(), n * 4, cudaMemcpyHostToDevice, c.stream));
    double ep_loss = 0.0;
    for (uint64_t st = 0; st < steps; ++st) {
      const uint32_t* rows = dperm.get() + st * batch;
      cast_pad(c, d_x, rows, batch, static_cast<int>(d), static_cast<int>(d), batch, net.dp, bt.X.get());
      // targets gathered through the same rows
      gather_rows_kernel<<<ceil_div(batch * dim, 256), 256, 0, c.stream>>>(d_t, rows, batch, static_cast<int>(dim),
                                                                          bt.tgt.get());
      PM_LAUNCHED();
      mlp_forward_backward(c, net, bt, st);
      adamw_step(c, net, bt, mom, lr, wd, ++t);
    }
    // the epoch's losses in one read: a step does not wait for the host
    PM_CUDA(cudaMemcpyAsync(part.data(), bt.partial.get(), bt.partial.bytes(), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaStreamSynchronize(c.stream));
    for (uint64_t st = 0; st < steps; ++st) {
      double s = 0.0;
      for (int e = 0; e < LOSS_PARTS; ++e) s += part[st * LOSS_PARTS + e];
      ep_loss += s / static_cast<double>(batch * dim);
    }
    if (epoch_loss) epoch_loss[ep] = static_cast<float>(ep_loss / std::max<uint64_t>(steps, 1));
  }
  c.check_errors("MLP training");
  net.download(c, params);
}

}  // namespace pacmap
