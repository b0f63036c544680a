// Initialization::Pca (src/lib.rs:442-522, 753-768): principal axes of the data on the GPU.
//
// The reference calls petal-decomposition 0.8 (an exact SVD through LAPACK when d <= 100, a seeded
// randomized SVD otherwise); neither is in the reference tree. This file computes the exact principal
// axes -- the limit the randomized method approximates -- as eigenvectors of the covariance matrix:
//
//   1. column means (f64, fixed-order two-level sums);
//   2. the d x d covariance of the centred rows in f64: at most 64 row chunks (of at least 16,384 rows)
//      write partial tiles, reduced over the chunks in order (deterministic, no atomics);
//   3. the top-k axes (f64): for d <= 160 Jacobi of the whole matrix, in one block for k <= 8 well separated axes
//      (jacobi_kernel) and cyclic on the host otherwise; above that subspace iteration on k + 24 vectors with a
//      Rayleigh-Ritz step (the power iteration the reference's randomized SVD uses), on the GPU when the data
//      is there (top_axes_device) and on the host for pacmap_pca_axes, with the same operations in the same
//      order: the axes are the same bits;
//      axes by descending variance, each axis's largest-magnitude loading made positive (the reference's
//      SVD sign is LAPACK's and unpinned);
//   4. the projection (x - mean) V_k by a tiled f32 kernel with f64 accumulation.
#include <algorithm>
#include <cmath>
#include <numeric>
#include <vector>

#include <cooperative_groups.h>

#include "engine.cuh"

namespace pacmap {
namespace {

constexpr uint64_t PCA_MAX_CHUNKS = 64;  // partial covariances (row chunks of at least 16,384 rows)
constexpr int MEAN_BLOCKS = 256, MEAN_AHEAD = 16;  // row ranges of the mean; loads in flight per thread

__global__ void __launch_bounds__(256) col_sum_partial_kernel(const float* __restrict__ x, uint64_t n, uint64_t d,
                                                              double* __restrict__ partial) {
  // block b sums rows [b * rpb, ...) of every column, each thread a strided set of columns
  const uint64_t rpb = (n + gridDim.x - 1) / gridDim.x;
  const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * rpb, r1 = r0 + rpb < n ? r0 + rpb : n;
  for (uint64_t c = threadIdx.x; c < d; c += blockDim.x) {
    double s = 0.0;
    uint64_t r = r0;
    for (; r + MEAN_AHEAD <= r1; r += MEAN_AHEAD) {
      float v[MEAN_AHEAD];
#pragma unroll
      for (int q = 0; q < MEAN_AHEAD; ++q) v[q] = x[(r + q) * d + c];
#pragma unroll
      for (int q = 0; q < MEAN_AHEAD; ++q) s += v[q];
    }
    for (; r < r1; ++r) s += x[r * d + c];
    partial[static_cast<uint64_t>(blockIdx.x) * d + c] = s;
  }
}

__global__ void col_mean_final_kernel(const double* __restrict__ partial, int parts, uint64_t n, uint64_t d,
                                      double* __restrict__ mean) {
  const uint64_t c = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (c >= d) return;
  double s = 0.0;
#pragma unroll 16
  for (int b = 0; b < parts; ++b) s += partial[static_cast<uint64_t>(b) * d + c];
  mean[c] = s / static_cast<double>(n);
}

// Partial covariance of one row chunk (blockIdx.y) for one pair of column tiles ti <= tj (blockIdx.x): E x E threads
// of R x R outputs, slabs of centred rows in two buffers, the next slab's values in registers meanwhile. Each output
// is one chain of fused multiply-adds over the chunk's rows in order, whatever the tile; the products commute, so the
// tiles below the diagonal would hold the same bits and are not computed. Bound by the operands' way out of shared
// memory: 32 R cycles a row of a 16 R wide tile, against 4 R^2 in the f64 units (64 fused multiply-adds per clock and
// SM). 60,000 x 784: 11.1 ms with 32 x 32 tiles over the whole square, one output of a row by four columns a thread
// and nothing in flight; 2.9 ms so.
template <int R, int E>
__global__ void __launch_bounds__(E * E) cov_partial_kernel(const float* __restrict__ x, uint64_t n, uint64_t d,
                                                          uint64_t rows_per_chunk, const double* __restrict__ mean,
                                                          double* __restrict__ partial) {
  constexpr int T = E * R, S = R == 4 ? 16 : 32, PASS = E * E / T, LOADS = S / PASS;
  __shared__ __align__(16) double a[2][S][T], b[2][S][T];  // [buffer][row][column]
  int ti = 0, rest = blockIdx.x;
  for (const int tiles = static_cast<int>((d + T - 1) / T); rest >= tiles - ti;) rest -= tiles - ti++;
  const int tj = ti + rest;
  const uint64_t chunk = blockIdx.y;
  const uint64_t r0 = chunk * rows_per_chunk, r1 = r0 + rows_per_chunk < n ? r0 + rows_per_chunk : n;
  const int lc = threadIdx.x % T, lr = threadIdx.x / T;  // this thread's staged column and first row
  const uint64_t ci = static_cast<uint64_t>(ti) * T + lc, cj = static_cast<uint64_t>(tj) * T + lc;
  const double mi = ci < d ? mean[ci] : 0.0, mj = cj < d ? mean[cj] : 0.0;
  float fa[LOADS], fb[LOADS];
  auto load = [&](uint64_t rb) {
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const uint64_t r = rb + lr + q * PASS;
      fa[q] = r < r1 && ci < d ? x[r * d + ci] : 0.0f;
      fb[q] = r < r1 && cj < d ? x[r * d + cj] : 0.0f;
    }
  };
  auto store = [&](uint64_t rb, int buf) {
#pragma unroll
    for (int q = 0; q < LOADS; ++q) {
      const int rr = lr + q * PASS;
      a[buf][rr][lc] = rb + rr < r1 && ci < d ? static_cast<double>(fa[q]) - mi : 0.0;
      b[buf][rr][lc] = rb + rr < r1 && cj < d ? static_cast<double>(fb[q]) - mj : 0.0;
    }
  };
  const int tx = threadIdx.x % E, ty = threadIdx.x / E;
  double acc[R][R] = {};
  load(r0);
  store(r0, 0);
  __syncthreads();
  int buf = 0;
  for (uint64_t rb = r0; rb < r1; rb += S, buf ^= 1) {
    const bool more = rb + S < r1;
    if (more) load(rb + S);
#pragma unroll 8
    for (int rr = 0; rr < S; ++rr) {
      double av[R], bv[R];
#pragma unroll
      for (int h = 0; h < R / 2; ++h) {
        const double2 u = *reinterpret_cast<const double2*>(&a[buf][rr][2 * ty + 2 * E * h]);
        const double2 v = *reinterpret_cast<const double2*>(&b[buf][rr][2 * tx + 2 * E * h]);
        av[2 * h] = u.x, av[2 * h + 1] = u.y;
        bv[2 * h] = v.x, bv[2 * h + 1] = v.y;
      }
#pragma unroll
      for (int p = 0; p < R; ++p)
#pragma unroll
        for (int q = 0; q < R; ++q) acc[p][q] = fma(av[p], bv[q], acc[p][q]);
    }
    if (more) store(rb + S, buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < R; ++p) {
    const uint64_t i = static_cast<uint64_t>(ti) * T + 2 * ty + (p & 1) + 2 * E * (p >> 1);
#pragma unroll
    for (int q = 0; q < R; ++q) {
      const uint64_t j = static_cast<uint64_t>(tj) * T + 2 * tx + (q & 1) + 2 * E * (q >> 1);
      if (i < d && j < d) partial[(chunk * d + i) * d + j] = acc[p][q];
    }
  }
}

__global__ void cov_reduce_kernel(const double* __restrict__ partial, uint64_t chunks, uint64_t d,
                                  double* __restrict__ cov) {
  const uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= d * d) return;
  const uint64_t i = e / d, j = e % d, src = i <= j ? e : j * d + i;
  double s = 0.0;
  for (uint64_t c = 0; c < chunks; ++c) s += partial[c * d * d + src];
  cov[e] = s;
}

// out (n x k, f32) = scale * (x - mean) V for V (d x k, f32, row-major), k <= 8 NQ: 64 rows per block, thread (tr, tc)
// rows tr and tr + 32, columns tc + 8 q; d in slices staged in shared memory as f64, f64 accumulation over the columns
// in order. Bound by the operands' way out of shared memory. 60,000 x 784 -> 100: 1.76 ms when every form was 128
// columns wide and converted V at each product, 1.09 so.
constexpr int PJ_ROWS = 64, PJ_K = 104;  // the widest form's columns
template <int NQ>
__global__ void __launch_bounds__(256) project_kernel(const float* __restrict__ x, uint64_t n, uint64_t d,
                                                      const double* __restrict__ mean, const float* __restrict__ V,
                                                      int k, float scale, float* __restrict__ out) {
  constexpr int D = NQ > 8 ? 16 : 32, K = 8 * NQ;
  __shared__ double xs[PJ_ROWS][D + 1];
  __shared__ double vs[D][K];
  const uint64_t row0 = static_cast<uint64_t>(blockIdx.x) * PJ_ROWS;
  const int tr = threadIdx.x >> 3, tc = threadIdx.x & 7;
  double acc[2][NQ] = {};
  for (uint64_t c0 = 0; c0 < d; c0 += D) {
    __syncthreads();
#pragma unroll
    for (int e = threadIdx.x; e < PJ_ROWS * D; e += 256) {
      const int rr = e / D, cc = e % D;
      const uint64_t r = row0 + rr, c = c0 + cc;
      xs[rr][cc] =
          (r < n && c < d) ? static_cast<double>(static_cast<float>(static_cast<double>(x[r * d + c]) - mean[c])) : 0.0;
    }
    for (int e = threadIdx.x; e < D * K; e += 256) {
      const int rr = e / K, cc = e % K;
      const uint64_t c = c0 + rr;
      vs[rr][cc] = (c < d && cc < k) ? static_cast<double>(V[c * k + cc]) : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int cc = 0; cc < D; ++cc) {
      const double x0 = xs[tr][cc], x1 = xs[tr + 32][cc];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const double v = vs[cc][tc + 8 * q];
        acc[0][q] = fma(x0, v, acc[0][q]);
        acc[1][q] = fma(x1, v, acc[1][q]);
      }
    }
  }
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const uint64_t r = row0 + tr + 32 * p;
    if (r >= n) continue;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int c = tc + 8 * q;
      if (c < k) out[r * k + c] = static_cast<float>(acc[p][q] * scale);
    }
  }
}

// Cyclic Jacobi eigen-decomposition of a symmetric d x d matrix (row-major, f64): eigenvalues into w,
// eigenvectors as the columns of v.
void jacobi_eigen(std::vector<double>& a, int d, std::vector<double>& w, std::vector<double>& v) {
  v.assign(static_cast<size_t>(d) * d, 0.0);
  for (int i = 0; i < d; ++i) v[static_cast<size_t>(i) * d + i] = 1.0;
  auto A = [&](int i, int j) -> double& { return a[static_cast<size_t>(i) * d + j]; };
  double total = 0.0;
  for (double e : a) total += e * e;
  for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0.0;
    for (int i = 0; i < d; ++i)
      for (int j = i + 1; j < d; ++j) off += A(i, j) * A(i, j);
    if (off <= 1e-30 * total || off == 0.0) break;
    for (int p = 0; p < d - 1; ++p) {
      for (int q = p + 1; q < d; ++q) {
        const double apq = A(p, q);
        if (std::fabs(apq) < 1e-300) continue;
        const double theta = (A(q, q) - A(p, p)) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < d; ++k) {  // columns p, q
          const double akp = A(k, p), akq = A(k, q);
          A(k, p) = c * akp - s * akq;
          A(k, q) = s * akp + c * akq;
        }
        for (int k = 0; k < d; ++k) {  // rows p, q
          const double apk = A(p, k), aqk = A(q, k);
          A(p, k) = c * apk - s * aqk;
          A(q, k) = s * apk + c * aqk;
        }
        for (int k = 0; k < d; ++k) {
          double* vk = &v[static_cast<size_t>(k) * d];
          const double vkp = vk[p], vkq = vk[q];
          vk[p] = c * vkp - s * vkq;
          vk[q] = s * vkp + c * vkq;
        }
      }
    }
  }
  w.resize(d);
  for (int i = 0; i < d; ++i) w[i] = A(i, i);
}

// Orthonormal columns (modified Gram-Schmidt) of a d x m matrix (row-major).
void orthonormalise(std::vector<double>& q, int d, int m) {
  for (int j = 0; j < m; ++j) {
    for (int i = 0; i < j; ++i) {
      double dot = 0.0;
      for (int r = 0; r < d; ++r) dot += q[static_cast<size_t>(r) * m + i] * q[static_cast<size_t>(r) * m + j];
      for (int r = 0; r < d; ++r) q[static_cast<size_t>(r) * m + j] -= dot * q[static_cast<size_t>(r) * m + i];
    }
    double nrm = 0.0;
    for (int r = 0; r < d; ++r) nrm += q[static_cast<size_t>(r) * m + j] * q[static_cast<size_t>(r) * m + j];
    nrm = std::sqrt(nrm);
    for (int r = 0; r < d; ++r) q[static_cast<size_t>(r) * m + j] = nrm > 0 ? q[static_cast<size_t>(r) * m + j] / nrm : 0.0;
  }
}

constexpr int JACOBI_MAX_D = 160;    // whole-matrix Jacobi up to here, subspace iteration above
constexpr int SUBSPACE_MAX_K = 128;  // axes the device's form takes (columns in mgs_kernel's shared memory)
constexpr int SUBSPACE_EXTRA = 24;   // vectors iterated beyond the k wanted
constexpr int SUBSPACE_ITERS = 20;

// The subspace iteration's fixed start, element e (row-major) of the d x m block: the e-th value of a
// splitmix64 stream (Steele, Lea, Flood 2014) in [-1, 1).
__host__ __device__ __forceinline__ uint64_t start_bits(uint64_t e) {
  uint64_t z = 0x9E3779B97F4A7C15ull * (e + 2);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return z >> 11;
}

// Eigenvectors of the m x m Rayleigh-Ritz projection (its rounding symmetrised first) into z, values into w.
void ritz_eigen(std::vector<double>& proj, int m, std::vector<double>& w, std::vector<double>& z) {
  for (int i = 0; i < m; ++i)
    for (int j = i + 1; j < m; ++j) {
      const double s = 0.5 * (proj[static_cast<size_t>(i) * m + j] + proj[static_cast<size_t>(j) * m + i]);
      proj[static_cast<size_t>(i) * m + j] = proj[static_cast<size_t>(j) * m + i] = s;
    }
  jacobi_eigen(proj, m, w, z);
}

// The k columns of the d x m block vecs with the largest eigenvalues w, in descending order, each with its
// largest-magnitude entry positive (d x k, row-major).
std::vector<double> leading_axes(const std::vector<double>& vecs, const std::vector<double>& w, int d, int m, int k) {
  std::vector<int> order(m);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int p, int q) { return w[p] > w[q]; });
  std::vector<double> V(static_cast<size_t>(d) * k);
  for (int j = 0; j < k; ++j) {
    const int col = order[j];
    int arg = 0;
    for (int r = 1; r < d; ++r)
      if (std::fabs(vecs[static_cast<size_t>(r) * m + col]) > std::fabs(vecs[static_cast<size_t>(arg) * m + col])) arg = r;
    const double sign = vecs[static_cast<size_t>(arg) * m + col] < 0 ? -1.0 : 1.0;
    for (int r = 0; r < d; ++r) V[static_cast<size_t>(r) * k + j] = sign * vecs[static_cast<size_t>(r) * m + col];
  }
  return V;
}

// The k leading eigenvectors of the symmetric d x d matrix a (columns of the returned d x k matrix,
// by descending eigenvalue, largest-magnitude entry positive), on the host.
std::vector<double> top_axes(std::vector<double>& a, int d, int k) {
  std::vector<double> vecs, w;  // d x m eigenvector block and its eigenvalues
  int m;
  if (d <= JACOBI_MAX_D) {
    jacobi_eigen(a, d, w, vecs);
    m = d;
  } else {
    m = std::min(d, k + SUBSPACE_EXTRA);
    std::vector<double> q(static_cast<size_t>(d) * m), t(static_cast<size_t>(d) * m);
    for (size_t e = 0; e < q.size(); ++e)
      q[e] = static_cast<double>(start_bits(e)) * (2.0 / 9007199254740992.0) - 1.0;
    orthonormalise(q, d, m);
    for (int it = 0; it < SUBSPACE_ITERS; ++it) {
      std::fill(t.begin(), t.end(), 0.0);
      for (int r = 0; r < d; ++r)
        for (int l = 0; l < d; ++l) {
          const double arl = a[static_cast<size_t>(r) * d + l];
          const double* ql = &q[static_cast<size_t>(l) * m];
          double* tr = &t[static_cast<size_t>(r) * m];
          for (int j = 0; j < m; ++j) tr[j] += arl * ql[j];
        }
      q.swap(t);
      orthonormalise(q, d, m);
    }
    // Rayleigh-Ritz: the m x m projection q^T a q, its eigenvectors rotate q
    std::vector<double> aq(static_cast<size_t>(d) * m, 0.0), proj(static_cast<size_t>(m) * m, 0.0), z;
    for (int r = 0; r < d; ++r)
      for (int l = 0; l < d; ++l) {
        const double arl = a[static_cast<size_t>(r) * d + l];
        for (int j = 0; j < m; ++j) aq[static_cast<size_t>(r) * m + j] += arl * q[static_cast<size_t>(l) * m + j];
      }
    for (int i = 0; i < m; ++i)
      for (int j = 0; j < m; ++j) {
        double s = 0.0;
        for (int r = 0; r < d; ++r) s += q[static_cast<size_t>(r) * m + i] * aq[static_cast<size_t>(r) * m + j];
        proj[static_cast<size_t>(i) * m + j] = s;
      }
    ritz_eigen(proj, m, w, z);
    vecs.assign(static_cast<size_t>(d) * m, 0.0);
    for (int r = 0; r < d; ++r)
      for (int j = 0; j < m; ++j) {
        double s = 0.0;
        for (int l = 0; l < m; ++l) s += q[static_cast<size_t>(r) * m + l] * z[static_cast<size_t>(l) * m + j];
        vecs[static_cast<size_t>(r) * m + j] = s;
      }
  }
  return leading_axes(vecs, w, d, m, k);
}

// ------------------------------------------------------------------------------------------------
// The subspace iteration on the GPU. Every sum runs over its index in ascending order with separately rounded
// multiplications and additions, as the host's loops do, so each element is the host's bit for bit: the
// parallelism is over elements only, and what bounds it is the serial chain of d additions per element.
// 784 columns, 100 axes: 620-720 ms on a host core; here 21 orthonormalisations of 1.36 ms, 22 products of 35 us,
// and the host's Ritz problem.
// ------------------------------------------------------------------------------------------------
__global__ void subspace_start_kernel(double* __restrict__ q, uint64_t count) {
  const uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e < count)
    q[e] = __dsub_rn(__dmul_rn(static_cast<double>(start_bits(e)), 2.0 / 9007199254740992.0), 1.0);
}

// out (rows x m) = A B for B (inner x m) and A rows x inner, or its transpose (inner x rows) when TRANS; all row-major.
// 32 x 32 outputs a block, 2 x 2 a thread, slabs of 32 inner indices in two shared-memory buffers with the next slab's
// values in registers meanwhile. 784 x 784 times 784 x 124 (100 blocks): 229 us when each thread read B's rows from
// L2 one after another, 35 so; q^T (A q) of that size 119 -> 33 us.
constexpr int AP_T = 32;
template <bool TRANS>
__global__ void __launch_bounds__(256) block_apply_kernel(const double* __restrict__ A, int rows, int inner,
                                                          const double* __restrict__ B, int m,
                                                          double* __restrict__ out) {
  __shared__ __align__(16) double as[2][AP_T][AP_T + 2], bs[2][AP_T][AP_T];  // [buffer][inner][row or column]
  const int r0 = blockIdx.x * AP_T, j0 = blockIdx.y * AP_T;
  const int lo = threadIdx.x & 31, hi = threadIdx.x >> 5;  // staging: 8 values of 32 per pass
  double fa[4], fb[4];
  auto load = [&](int l0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int h = hi + 8 * q;
      if (TRANS) fa[q] = l0 + h < inner && r0 + lo < rows ? A[static_cast<size_t>(l0 + h) * rows + r0 + lo] : 0.0;
      else fa[q] = r0 + h < rows && l0 + lo < inner ? A[static_cast<size_t>(r0 + h) * inner + l0 + lo] : 0.0;
      fb[q] = l0 + h < inner && j0 + lo < m ? B[static_cast<size_t>(l0 + h) * m + j0 + lo] : 0.0;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int h = hi + 8 * q;
      as[buf][TRANS ? h : lo][TRANS ? lo : h] = fa[q];
      bs[buf][h][lo] = fb[q];
    }
  };
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  double acc[2][2] = {};
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int l0 = 0; l0 < inner; l0 += AP_T, buf ^= 1) {
    const bool more = l0 + AP_T < inner;
    if (more) load(l0 + AP_T);
    auto term = [&](int l) {
      const double2 u = *reinterpret_cast<const double2*>(&as[buf][l][2 * ty]);
      const double2 v = *reinterpret_cast<const double2*>(&bs[buf][l][2 * tx]);
      acc[0][0] = __dadd_rn(acc[0][0], __dmul_rn(u.x, v.x));
      acc[0][1] = __dadd_rn(acc[0][1], __dmul_rn(u.x, v.y));
      acc[1][0] = __dadd_rn(acc[1][0], __dmul_rn(u.y, v.x));
      acc[1][1] = __dadd_rn(acc[1][1], __dmul_rn(u.y, v.y));
    };
    if (l0 + AP_T <= inner) {
#pragma unroll 16
      for (int l = 0; l < AP_T; ++l) term(l);
    } else {
      for (int l = 0; l < inner - l0; ++l) term(l);
    }
    if (more) store(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int r = r0 + 2 * ty + p, j = j0 + 2 * tx + q;
      if (r < rows && j < m) out[static_cast<size_t>(r) * m + j] = acc[p][q];
    }
}

// Modified Gram-Schmidt of the columns of a d x m matrix (row-major in and out; in == out allowed) by one cluster of
// eight blocks, column c in the shared memory of block c % 8. Column by column: its owner normalises it, every block
// copies it over distributed shared memory, and takes its part out of the later columns it owns. For each column
// the projections onto the earlier ones are removed in ascending order, as in the host's column-by-column loop.
// Bound by two serial chains of d additions per column (the norm, then the dot products: those of a block's columns
// run side by side in the lanes of one warp): 10 of the 11 us per column of 784 rows, 11.8 cycles an addition where its
// latency alone is 8.3. 124 columns: 1.36 ms with the products formed 16 rows ahead of the additions, 1.83 with the
// loop only unrolled (8). The columns lie an odd number of doubles apart, so that the lanes' reads fall in different
// banks. At most 152 columns of 1024 rows: 19 columns per block, 164 KB.
constexpr int MGS_BLOCKS = 8, MGS_THREADS = 512, CHAIN_AHEAD = 16;
__host__ __device__ __forceinline__ int mgs_ld(int d) { return d | 1; }
size_t mgs_smem(int d, int m) {
  return (static_cast<size_t>((m + MGS_BLOCKS - 1) / MGS_BLOCKS) * mgs_ld(d) + d) * sizeof(double);
}

// The products of the next CHAIN_AHEAD rows are formed while this batch's are added up.
__device__ __forceinline__ double chain_dot(const double* a, const double* b, int d) {
  double s = 0.0, p[CHAIN_AHEAD];
  int r = 0;
  if (d >= CHAIN_AHEAD) {
#pragma unroll
    for (int q = 0; q < CHAIN_AHEAD; ++q) p[q] = __dmul_rn(a[q], b[q]);
    for (r = CHAIN_AHEAD; r + CHAIN_AHEAD <= d; r += CHAIN_AHEAD) {
      double t[CHAIN_AHEAD];
#pragma unroll
      for (int q = 0; q < CHAIN_AHEAD; ++q) t[q] = __dmul_rn(a[r + q], b[r + q]);
#pragma unroll
      for (int q = 0; q < CHAIN_AHEAD; ++q) s = __dadd_rn(s, p[q]);
#pragma unroll
      for (int q = 0; q < CHAIN_AHEAD; ++q) p[q] = t[q];
    }
#pragma unroll
    for (int q = 0; q < CHAIN_AHEAD; ++q) s = __dadd_rn(s, p[q]);
  }
  for (; r < d; ++r) s = __dadd_rn(s, __dmul_rn(a[r], b[r]));
  return s;
}

__global__ void __cluster_dims__(MGS_BLOCKS, 1, 1) __launch_bounds__(MGS_THREADS)
    mgs_kernel(const double* __restrict__ in, int d, int m, double* __restrict__ out) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double cols[];  // own columns [ncol][ld], then the current column [d]
  __shared__ double dots[32], norm;
  const int rank = static_cast<int>(cluster.block_rank()), tid = threadIdx.x, ld = mgs_ld(d);
  const int ncol = (m - rank + MGS_BLOCKS - 1) / MGS_BLOCKS;  // columns rank, rank + 8, ... < m
  double* cur = cols + static_cast<size_t>((m + MGS_BLOCKS - 1) / MGS_BLOCKS) * ld;
  for (int e = tid; e < ncol * d; e += MGS_THREADS) {
    const int r = e / ncol, q = e % ncol;
    cols[q * ld + r] = in[static_cast<size_t>(r) * m + rank + q * MGS_BLOCKS];
  }
  __syncthreads();
  for (int i = 0; i < m; ++i) {
    const int owner = i % MGS_BLOCKS, slot = i / MGS_BLOCKS;
    if (rank == owner) {
      double* v = cols + slot * ld;
      if (tid == 0) norm = __dsqrt_rn(chain_dot(v, v, d));
      __syncthreads();
      const double nrm = norm;
      for (int r = tid; r < d; r += MGS_THREADS) v[r] = nrm > 0 ? __ddiv_rn(v[r], nrm) : 0.0;
    }
    cluster.sync();  // column i is final (nothing writes it again) and may be read by every block
    const int first = rank > owner ? slot : slot + 1;  // own columns after i
    if (first >= ncol) continue;
    const double* src = cluster.map_shared_rank(cols, owner) + slot * ld;
    for (int r = tid; r < d; r += MGS_THREADS) cur[r] = src[r];
    __syncthreads();
    if (tid < ncol - first) dots[tid] = chain_dot(cur, cols + (first + tid) * ld, d);
    __syncthreads();
    for (int r = tid; r < d; r += MGS_THREADS) {
      const double c = cur[r];
      for (int q = first; q < ncol; ++q) cols[q * ld + r] = __dsub_rn(cols[q * ld + r], __dmul_rn(dots[q - first], c));
    }
    __syncthreads();
  }
  for (int e = tid; e < ncol * d; e += MGS_THREADS) {
    const int r = e / ncol, q = e % ncol;
    out[static_cast<size_t>(r) * m + rank + q * MGS_BLOCKS] = cols[q * ld + r];
  }
  cluster.sync();  // no block leaves while another may still read its columns
}

// top_axes for d > JACOBI_MAX_D with the covariance on the device. The m x m Ritz problem (m <= 152, nearly
// diagonal by then) stays on the host.
std::vector<double> top_axes_device(Ctx& c, const double* d_cov, int d, int k) {
  const int m = std::min(d, k + SUBSPACE_EXTRA);
  PM_REQUIRE(k <= SUBSPACE_MAX_K, PACMAP_ERR_UNSUPPORTED, "PCA supports at most 128 components");
  const uint64_t dm = static_cast<uint64_t>(d) * m;
  DevBuf<double> q(c, dm), t(c, dm), proj(c, static_cast<uint64_t>(m) * m), z(c, static_cast<uint64_t>(m) * m);
  const size_t ms = mgs_smem(d, m);
  PM_CUDA(cudaFuncSetAttribute(mgs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(ms)));
  auto mgs = [&](const double* in, double* out) {
    mgs_kernel<<<MGS_BLOCKS, MGS_THREADS, ms, c.stream>>>(in, d, m, out);
    PM_LAUNCHED();
  };
  auto apply = [&](const double* A, int inner, const double* B, double* out) {
    block_apply_kernel<false><<<dim3(ceil_div(d, AP_T), ceil_div(m, AP_T)), 256, 0, c.stream>>>(A, d, inner, B, m, out);
    PM_LAUNCHED();
  };
  subspace_start_kernel<<<ceil_div(dm, 256), 256, 0, c.stream>>>(q.get(), dm);
  PM_LAUNCHED();
  mgs(q.get(), q.get());
  for (int it = 0; it < SUBSPACE_ITERS; ++it) {
    apply(d_cov, d, q.get(), t.get());
    mgs(t.get(), q.get());
  }
  apply(d_cov, d, q.get(), t.get());
  // q^T (A q)
  block_apply_kernel<true><<<dim3(ceil_div(m, AP_T), ceil_div(m, AP_T)), 256, 0, c.stream>>>(q.get(), m, d, t.get(), m,
                                                                                           proj.get());
  PM_LAUNCHED();
  std::vector<double> hp(proj.count), w, hz, vecs(dm);
  PM_CUDA(cudaMemcpyAsync(hp.data(), proj.get(), proj.bytes(), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  ritz_eigen(hp, m, w, hz);
  PM_CUDA(cudaMemcpyAsync(z.get(), hz.data(), z.bytes(), cudaMemcpyHostToDevice, c.stream));
  apply(q.get(), m, z.get(), t.get());
  PM_CUDA(cudaMemcpyAsync(vecs.data(), t.get(), dm * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  return leading_axes(vecs, w, d, m, k);
}

// Jacobi's method for a symmetric d x d matrix, 2 <= d <= 160, and up to eight leading eigenvectors: one block, the
// matrix in shared memory (zero-padded to an even order n, row length ld odd so that a column's elements fall in
// different banks; only the upper triangle is kept up to date). A sweep is n - 1 steps of n / 2 rotations on disjoint
// index pairs (the round-robin order of Brent and Luk, SIAM J. Sci. Stat. Comput. 6, 1985): a thread per pair finds
// the rotation, then a thread per two pairs turns their 2 x 2 block of the matrix. The rotations go to rot; the
// wanted eigenvectors are unit vectors taken back through them, so that the full eigenvector matrix is never formed.
// out: status (1: converged and the leading k + 1 eigenvalues lie JACOBI_GAP of the largest apart), the k leading
// eigenvalues, the eigenvectors (d x k, row-major). Bound by the blocks' way through shared memory (1,490 of a step's
// 2,130 cycles at d = 100, 8 sweeps) and by the rotation's two reciprocal square roots and their chain (640; 850 with
// the tangent from two divisions and two roots). Vectors: 240 cycles a step with a barrier for their warps only, 430
// with the whole block's. Finding the next step's rotations beside the blocks (one barrier a step) was no faster. A
// 2,000 x 100 fit from the principal axes: 12.1 ms with the host's sweeps, 4.1 ms so.
constexpr int JACOBI_THREADS = 1024, JACOBI_MAX_K = 8, JACOBI_SWEEPS = 20, JACOBI_AHEAD = 8;
constexpr int JACOBI_BLOCKS = ((JACOBI_MAX_D / 2) * (JACOBI_MAX_D / 2 - 1) / 2 + JACOBI_THREADS - 1) / JACOBI_THREADS;
// The device from 32 columns on: 173 us against the host's 259 at 32 (copies in and out included), 135 against 127
// at 24, 0.97 ms against 7.2 at 100, 2.7 against 64 at 160. Its residuals are the smaller (7e-15 of the largest
// eigenvalue against 1.2e-14 at 100), and of 1,590 covariances of five kinds one had an f32 axis entry that came out
// another way than the host's (uniform data, whose eigenvalues lie close together).
// JACOBI_GAP: axes whose eigenvalues lie closer than this (of the largest) depend on the order of the rotations in
// digits that f32 keeps, and equal eigenvalues leave the choice of basis to it, so the host's cyclic order stays
// for those; above it the two methods' axes differ by at most 10 * 2.2e-16 divided by the gap (6e-13 seen), which
// shows in f32 only where an entry lies that close to the middle between two numbers. Eight axes: the start's dim; the
// 100 axes of the wide data's reduction have closer pairs among them as a rule.
constexpr int JACOBI_MIN_D = 32;
constexpr double JACOBI_GAP = 1e-3;
static_assert(JACOBI_MAX_K * JACOBI_MAX_D / 2 <= JACOBI_THREADS, "a thread per vector and pair");
size_t jacobi_smem(int d) {
  const int n = d + (d & 1);
  return (static_cast<size_t>(n) * (n | 1) + n) * sizeof(double) + static_cast<size_t>(n) * sizeof(int) +
         static_cast<size_t>(n / 2) * sizeof(double2);
}

// Pair number i of step s, 0 <= i < n / 2, 0 <= s < n - 1 = m: (s, m) for i = 0, else s + i and s - i modulo m.
__device__ __forceinline__ void jacobi_pair(int i, int s, int m, int& p, int& q) {
  p = s + i < m ? s + i : s + i - m;
  q = i == 0 ? m : (s - i >= 0 ? s - i : s - i + m);
}

__global__ void __launch_bounds__(JACOBI_THREADS)
    jacobi_kernel(const double* __restrict__ cov, int d, int k, double2* __restrict__ rot, double* __restrict__ out) {
  extern __shared__ __align__(16) char jacobi_shared[];
  __shared__ double part[JACOBI_THREADS / 32];
  __shared__ double sum;
  __shared__ int ok;
  const int tid = threadIdx.x, n = d + (d & 1), m = n - 1, h = n / 2, ld = n | 1;
  double2* cs = reinterpret_cast<double2*>(jacobi_shared);  // [h] this step's cosines and sines
  double* a = reinterpret_cast<double*>(cs + h);            // [n][ld]
  double* w = a + static_cast<size_t>(n) * ld;              // [n] eigenvalues
  int* order = reinterpret_cast<int*>(w + n);               // [n] columns by descending eigenvalue
  auto at = [&](int i, int j) -> double& { return i < j ? a[i * ld + j] : a[j * ld + i]; };
  // the sum of v over the block's threads, in a fixed order
  auto block_sum = [&](double v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((tid & 31) == 0) part[tid >> 5] = v;
    __syncthreads();
    if (tid < 32) {
      double t = part[tid];
#pragma unroll
      for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (tid == 0) sum = t;
    }
    __syncthreads();
    return sum;
  };
  double sq = 0.0;
  for (int e = tid; e < n * n; e += JACOBI_THREADS) {
    const int i = e / n, j = e % n;
    const double v = i < d && j < d ? cov[i * d + j] : 0.0;
    a[i * ld + j] = v;
    sq += v * v;
  }
  if (tid < n) order[tid] = tid;  // every entry a column, whatever the comparisons below make of a NaN
  const double total = block_sum(sq);
  // this thread's two pairs of pairs I < J (the same numbers in every step)
  int bi[JACOBI_BLOCKS], bj[JACOBI_BLOCKS];
#pragma unroll
  for (int b = 0; b < JACOBI_BLOCKS; ++b) {
    int e = tid + b * JACOBI_THREADS, i = 0;
    bi[b] = -1;
    bj[b] = 0;
    if (e < h * (h - 1) / 2) {
      while (e >= h - 1 - i) e -= h - 1 - i++;
      bi[b] = i;
      bj[b] = i + 1 + e;
    }
  }
  int sweep = 0;
  bool done = false;
  for (;; ++sweep) {
    double off = 0.0;
    for (int e = tid; e < n * n; e += JACOBI_THREADS) {
      const int i = e / n, j = e % n;
      if (i < j) off += a[i * ld + j] * a[i * ld + j];
    }
    off = block_sum(off);
    done = off <= 1e-30 * total && total <= 1e300;  // false for NaN
    if (done || sweep == JACOBI_SWEEPS) break;
    for (int s = 0; s < m; ++s) {
      if (tid < h) {
        int p, q;
        jacobi_pair(tid, s, m, p, q);
        double& apq = at(p, q);
        // tan 2 theta = b / delta with |theta| <= pi / 4: cos^2 = (1 + |delta| / r) / 2, sin = b / (2 r cos)
        double2 r = make_double2(1.0, 0.0);
        double &app = a[p * ld + p], &aqq = a[q * ld + q];
        const double delta = aqq - app, b = 2.0 * apq, r2 = delta * delta + b * b;
        if (fabs(apq) >= 1e-300 && r2 >= 1e-280 && r2 <= 1e280) {
          const double ir = rsqrt(r2), c2 = 0.5 + 0.5 * fabs(delta) * ir, ic = rsqrt(c2);
          r = make_double2(c2 * ic, (delta >= 0 ? 0.5 : -0.5) * b * ir * ic);
          const double shift = r.y * ic * apq;
          app -= shift;
          aqq += shift;
          apq = 0.0;
        }
        cs[tid] = r;
        rot[(static_cast<size_t>(sweep) * m + s) * h + tid] = cs[tid];
      }
      __syncthreads();
#pragma unroll
      for (int b = 0; b < JACOBI_BLOCKS; ++b) {
        if (bi[b] < 0) continue;
        int p, q, r, u;
        jacobi_pair(bi[b], s, m, p, q);
        jacobi_pair(bj[b], s, m, r, u);
        const double2 x = cs[bi[b]], y = cs[bj[b]];
        double &e00 = at(p, r), &e01 = at(p, u), &e10 = at(q, r), &e11 = at(q, u);
        const double f00 = x.x * e00 - x.y * e10, f01 = x.x * e01 - x.y * e11;
        const double f10 = x.y * e00 + x.x * e10, f11 = x.y * e01 + x.x * e11;
        e00 = y.x * f00 - y.y * f01;
        e01 = y.y * f00 + y.x * f01;
        e10 = y.x * f10 - y.y * f11;
        e11 = y.y * f10 + y.x * f11;
      }
      __syncthreads();
    }
  }
  // the order of the eigenvalues, descending, equal ones by column
  if (tid < d) w[tid] = a[tid * ld + tid];
  if (tid == 0) ok = done;
  __syncthreads();
  if (!ok) {
    if (tid == 0) out[0] = 0.0;
    return;
  }
  if (tid < d) {
    int rank = 0;
    for (int j = 0; j < d; ++j) rank += w[j] > w[tid] || (w[j] == w[tid] && j < tid);
    order[rank] = tid;
  }
  __syncthreads();
  if (tid < k && tid + 1 < d && !(w[order[tid]] - w[order[tid + 1]] > JACOBI_GAP * w[order[0]])) ok = 0;
  __syncthreads();
  if (!ok) {
    if (tid == 0) out[0] = 0.0;
    return;
  }
  if (tid == 0) out[0] = 1.0;
  if (tid < k) out[1 + tid] = w[order[tid]];
  // eigenvector v is J_1 J_2 ... e_{order[v]}: vector v's pair i belongs to thread v * h + i; a is reused, [k][n]
  const int v = tid / h, i = tid % h;
  __syncthreads();
  for (int e = tid; e < k * n; e += JACOBI_THREADS) a[e] = e % n == order[e / n] ? 1.0 : 0.0;
  __syncthreads();
  const int threads = (k * h + 31) / 32 * 32;  // whole warps, with a barrier of their own
  if (tid < threads) {
    int s = m - 1;
    for (int step = sweep * m - 1; step >= 0;) {
      const int batch = min(JACOBI_AHEAD, step + 1);
      double2 r[JACOBI_AHEAD];
#pragma unroll
      for (int b = 0; b < JACOBI_AHEAD; ++b)
        if (b < batch && v < k) r[b] = rot[static_cast<size_t>(step - b) * h + i];
#pragma unroll
      for (int b = 0; b < JACOBI_AHEAD; ++b) {
        if (b < batch && v < k) {
          int p, q;
          jacobi_pair(i, s, m, p, q);
          const double xp = a[v * n + p], xq = a[v * n + q];
          a[v * n + p] = r[b].x * xp + r[b].y * xq;
          a[v * n + q] = r[b].x * xq - r[b].y * xp;
        }
        if (b < batch) s = s ? s - 1 : m - 1;
        asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
      }
      step -= batch;
    }
  }
  __syncthreads();
  for (int e = tid; e < d * k; e += JACOBI_THREADS) out[1 + k + e] = a[(e % k) * n + e / k];
}

// top_axes for d <= JACOBI_MAX_D and k <= JACOBI_MAX_K with the covariance on the device; empty when the host's
// sequence of rotations has to decide (see JACOBI_GAP) or the sweeps ran out (a NaN or an infinity in the matrix).
std::vector<double> small_axes_device(Ctx& c, const double* d_cov, int d, int k) {
  PM_REQUIRE(d >= 2 && d <= JACOBI_MAX_D && k >= 1 && k <= std::min(d, JACOBI_MAX_K), PACMAP_ERR_UNSUPPORTED,
             "the one-block Jacobi takes 2 <= d <= 160 and k <= 8");
  const int n = d + (d & 1);
  DevBuf<double2> rot(c, static_cast<uint64_t>(JACOBI_SWEEPS) * (n - 1) * (n / 2));
  DevBuf<double> out(c, 1 + static_cast<uint64_t>(k) + static_cast<uint64_t>(d) * k);
  const size_t smem = jacobi_smem(d);
  PM_CUDA(cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  jacobi_kernel<<<1, JACOBI_THREADS, smem, c.stream>>>(d_cov, d, k, rot.get(), out.get());
  PM_LAUNCHED();
  std::vector<double> h(out.count);
  PM_CUDA(cudaMemcpyAsync(h.data(), out.get(), out.bytes(), cudaMemcpyDeviceToHost, c.stream));
  PM_CUDA(cudaStreamSynchronize(c.stream));
  if (h[0] != 1.0) return {};
  const std::vector<double> w(h.begin() + 1, h.begin() + 1 + k), vecs(h.begin() + 1 + k, h.end());
  return leading_axes(vecs, w, d, k, k);
}

// out (n x k) = scale * x[:, :k] for x (n x w).
__global__ void leading_columns_kernel(const float* __restrict__ x, uint64_t n, uint64_t w, uint64_t k, float scale,
                                       float* __restrict__ out) {
  const uint64_t total = n * k;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < total; t += stride) {
    const uint64_t r = t / k, c = t - r * k;
    out[t] = __fmul_rn(x[r * w + c], scale);
  }
}

}  // namespace

void pca_top_axes(const double* cov, uint64_t d, uint64_t k, double* axes) {
  PM_REQUIRE(k >= 1 && k <= d && d <= 1024, PACMAP_ERR_UNSUPPORTED, "axes need 1 <= k <= d <= 1024");
  std::vector<double> a(cov, cov + d * d);
  const std::vector<double> V = top_axes(a, static_cast<int>(d), static_cast<int>(k));
  std::copy(V.begin(), V.end(), axes);
}

void pca_top_axes_device(Ctx& c, const double* cov, uint64_t d, uint64_t k, double* axes) {
  PM_REQUIRE(k >= 1 && k <= static_cast<uint64_t>(SUBSPACE_MAX_K) && k <= d && d <= 1024 &&
                 d > static_cast<uint64_t>(JACOBI_MAX_D),
             PACMAP_ERR_UNSUPPORTED, "axes on the device need 1 <= k <= 128 and 160 < d <= 1024");
  DevBuf<double> dc;
  upload(c, dc, cov, d * d);
  const std::vector<double> V = top_axes_device(c, dc.get(), static_cast<int>(d), static_cast<int>(k));
  std::copy(V.begin(), V.end(), axes);
}

bool pca_small_axes_device(Ctx& c, const double* cov, uint64_t d, uint64_t k, double* axes) {
  PM_REQUIRE(d <= static_cast<uint64_t>(JACOBI_MAX_D) && k <= static_cast<uint64_t>(JACOBI_MAX_K),
             PACMAP_ERR_UNSUPPORTED, "the one-block Jacobi takes 2 <= d <= 160 and k <= 8");
  DevBuf<double> dc;
  upload(c, dc, cov, d * d);
  const std::vector<double> V = small_axes_device(c, dc.get(), static_cast<int>(d), static_cast<int>(k));
  std::copy(V.begin(), V.end(), axes);
  return !V.empty();
}

void leading_columns(Ctx& c, const float* d_x, uint64_t n, uint64_t w, uint64_t k, float scale, float* d_out) {
  if (!n || !k) return;
  leading_columns_kernel<<<static_cast<unsigned>(std::min<uint64_t>(ceil_div(n * k, 256), c.sm_count * 16ull)), 256, 0,
                           c.stream>>>(d_x, n, w, k, scale, d_out);
  PM_LAUNCHED();
}

void pca_project_device(Ctx& c, const float* d_x, uint64_t n, uint64_t d, uint64_t k, float scale, float* d_out,
                        std::vector<float>* axes_out) {
  PM_REQUIRE(n > 0, PACMAP_ERR_EMPTY_ARRAY_MEAN, "Failed to calculate mean axis: the array is empty");
  PM_REQUIRE(k >= 1 && k <= static_cast<uint64_t>(PJ_K) && k <= d, PACMAP_ERR_UNSUPPORTED,
             "PCA supports at most 104 components and no more than the columns");
  PM_REQUIRE(d <= 1024, PACMAP_ERR_UNSUPPORTED, "PCA supports d <= 1024");
  // 1. means
  DevBuf<double> mpart(c, static_cast<uint64_t>(MEAN_BLOCKS) * d), mean(c, d);
  col_sum_partial_kernel<<<MEAN_BLOCKS, 256, 0, c.stream>>>(d_x, n, d, mpart.get());
  PM_LAUNCHED();
  col_mean_final_kernel<<<ceil_div(d, 256), 256, 0, c.stream>>>(mpart.get(), MEAN_BLOCKS, n, d, mean.get());
  PM_LAUNCHED();
  // 2. covariance (unnormalised: the axes do not depend on the scale)
  const uint64_t rpc = std::max<uint64_t>(16384, (n + PCA_MAX_CHUNKS - 1) / PCA_MAX_CHUNKS);
  const uint64_t chunks = (n + rpc - 1) / rpc;
  auto pairs = [&](uint64_t tile) { return (d + tile - 1) / tile * ((d + tile - 1) / tile + 1) / 2; };
  DevBuf<double> part(c, chunks * d * d), cov(c, d * d);
  auto partials = [&](auto kernel, uint64_t tile, int threads) {
    kernel<<<dim3(static_cast<unsigned>(pairs(tile)), static_cast<unsigned>(chunks)), threads, 0, c.stream>>>(
        d_x, n, d, rpc, mean.get(), part.get());
    PM_LAUNCHED();
  };
  // 64-column tiles once they give every SM a block, else 16-column ones: 2.9 against 4.1 ms at 60,000 x 784 (364
  // blocks of the wide tiles), 2.0 / 2.2 at 30,000 x 784 (182), 2.25 / 2.29 at 1,000,000 x 128 (186), 0.88 / 1.31 the
  // other way at 60,000 x 300 (60), 0.058 / 0.164 at 2,000 x 100 (3), equal at 16,000 x 784 (91)
  if (pairs(64) * chunks >= static_cast<uint64_t>(c.sm_count)) partials(cov_partial_kernel<4, 16>, 64, 256);
  else partials(cov_partial_kernel<2, 8>, 16, 64);
  cov_reduce_kernel<<<ceil_div(d * d, 256), 256, 0, c.stream>>>(part.get(), chunks, d, cov.get());
  PM_LAUNCHED();
  // 3. axes
  std::vector<double> V64;
  if (d > static_cast<uint64_t>(JACOBI_MAX_D)) {
    V64 = top_axes_device(c, cov.get(), static_cast<int>(d), static_cast<int>(k));
  } else if (d >= static_cast<uint64_t>(JACOBI_MIN_D) && k <= static_cast<uint64_t>(JACOBI_MAX_K)) {
    V64 = small_axes_device(c, cov.get(), static_cast<int>(d), static_cast<int>(k));
  }
  if (V64.empty()) {
    std::vector<double> a(d * d);
    PM_CUDA(cudaMemcpyAsync(a.data(), cov.get(), d * d * sizeof(double), cudaMemcpyDeviceToHost, c.stream));
    PM_CUDA(cudaStreamSynchronize(c.stream));
    V64 = top_axes(a, static_cast<int>(d), static_cast<int>(k));
  }
  std::vector<float> V(d * k);
  for (uint64_t e = 0; e < d * k; ++e) V[e] = static_cast<float>(V64[e]);
  if (axes_out) *axes_out = V;
  // 4. projection
  DevBuf<float> dV;
  upload(c, dV, V.data(), d * k);
  auto project = [&](auto kernel) {
    kernel<<<ceil_div(n, PJ_ROWS), 256, 0, c.stream>>>(d_x, n, d, mean.get(), dV.get(), static_cast<int>(k), scale,
                                                       d_out);
  };
  // The narrowest form that holds the k columns, since the padding is computed too; 13: the 100 axes of the wide
  // data's reduction. 60,000 x 784: 0.28 ms for 2 columns, 1.09 for 100.
  if (k <= 8) project(project_kernel<1>);
  else if (k <= 32) project(project_kernel<4>);
  else if (k <= 64) project(project_kernel<8>);
  else project(project_kernel<13>);
  PM_LAUNCHED();
}

}  // namespace pacmap
