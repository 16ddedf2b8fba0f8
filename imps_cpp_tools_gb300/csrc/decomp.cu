// Per-sector dense decompositions of block-sparse MPS tensors on the device (FP64 always).
//
// The reference stacks, per charge sector, the blocks of A_s into one dense matrix
// (MPSBlockMat::GetDenseMat, MPSBlockMat.hpp:468-526 with GetSingleSecData :636-719) and
// runs LAPACK on it: qr_econ + sign fix (qr_pos, helpers.hpp:181-195) or svd_econ
// (MPSBlockUtilities.hpp:78-244, BlockObj.hpp:2422-2541).  Here a sector is the work of a cluster of
// eight CTAs (QR, SVD; one CTA where a sector of the call does not fit a cluster) or of one CTA (null space):
//  * gather: blocks -> packed column-major dense matrices (transposed for dir = r, so that
//    every matrix is handled as "tall": M = stacked dimension, N = sector dimension);
//  * Householder QR with explicit Q and diag(R) >= 0;
//  * one-sided (Hestenes) Jacobi SVD, singular values sorted descending;
//  * scatter back to the block layout.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "imps_decomp.h"
#include "imps_status.h"

namespace {

constexpr int DT = 256;  // threads per CTA (8 warps)

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide sum, result broadcast to all threads
__device__ double bsum(double v, double* sh) {
  v = wsum(v);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i];
  return t;
}

// One CTA column (blockIdx.x) per block, blockIdx.y shares its columns; lanes along the block's rows.
__global__ void gather_kernel(const imps::GatherEntry* __restrict__ ent, const double* __restrict__ src,
                              double* __restrict__ dst) {
  const imps::GatherEntry e = ent[blockIdx.x];
  const int lane = threadIdx.x & 31;
  for (int j = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5); j < e.cols; j += gridDim.y * (blockDim.x >> 5))
    for (int i = lane; i < e.rows; i += 32) {  // element (i,j) of the block
      const double v = src[e.src_off + (int64_t)j * e.rows + i];
      const int64_t di = e.transpose ? e.c0 + j : e.r0 + i, dj = e.transpose ? e.r0 + i : e.c0 + j;
      dst[e.dst_off + di + dj * e.dst_ld] = v;
    }
}

__global__ void scatter_kernel(const imps::GatherEntry* __restrict__ ent, const double* __restrict__ dense,
                               double* __restrict__ dst) {
  const imps::GatherEntry e = ent[blockIdx.x];
  const int lane = threadIdx.x & 31;
  for (int j = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5); j < e.cols; j += gridDim.y * (blockDim.x >> 5))
    for (int i = lane; i < e.rows; i += 32) {
      const int64_t di = e.transpose ? e.c0 + j : e.r0 + i, dj = e.transpose ? e.r0 + i : e.c0 + j;
      dst[e.src_off + (int64_t)j * e.rows + i] = dense[e.dst_off + di + dj * e.dst_ld];
    }
}

// Step k of the Householder QR of the M x N matrix a (column-major, ld = M): the reflector
// of column k below the diagonal (v[k] = 1 implicit), tau_s[k] its scalar, R's row k on and
// right of the diagonal.
__device__ void householder_step(double* a, int M, int N, int k, double* tau_s, double* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double p = 0.0;
  for (int i = k + threadIdx.x; i < M; i += blockDim.x) p += a[i + (int64_t)k * M] * a[i + (int64_t)k * M];
  const double nrm2 = bsum(p, sh);
  const double x0 = a[k + (int64_t)k * M];
  const double normx = sqrt(nrm2);
  double tau = 0.0, beta = x0, scal = 0.0;
  const double tail2 = nrm2 - x0 * x0;
  if (normx > 0.0 && tail2 > 0.0) {
    beta = -copysign(normx, x0);
    tau = (beta - x0) / beta;
    scal = 1.0 / (x0 - beta);
  }
  __syncthreads();
  if (tau != 0.0)
    for (int i = k + 1 + threadIdx.x; i < M; i += blockDim.x) a[i + (int64_t)k * M] *= scal;
  if (threadIdx.x == 0) { a[k + (int64_t)k * M] = beta; tau_s[k] = tau; }
  __syncthreads();
  if (tau != 0.0) {
    for (int j = k + 1 + warp; j < N; j += nw) {
      double* cj = a + (int64_t)j * M;
      const double* v = a + (int64_t)k * M;
      double w = 0.0;
      for (int i = k + 1 + lane; i < M; i += 32) w += v[i] * cj[i];
      w = wsum(w) + cj[k];
      const double tw = tau * w;
      if (lane == 0) cj[k] -= tw;
      for (int i = k + 1 + lane; i < M; i += 32) cj[i] -= tw * v[i];
    }
  }
  __syncthreads();
}

// Householder QR of the M x N matrix a (in place, column-major, ld = M), K = min(M, N):
// reflectors below the diagonal, R on and above it, tau_s[k] their scalars.
__device__ void householder(double* a, int M, int N, double* tau_s, double* sh) {
  const int K = min(M, N);
  for (int k = 0; k < K; ++k) householder_step(a, M, N, k, tau_s, sh);
}

// Householder QR with column pivoting (A P = Q R, M >= N): before step k the column of largest
// remaining norm (rows k..M-1; the first on ties) is swapped into place; piv[k] = the original
// index of column k.  cn: N doubles of scratch; sel: one shared int.
__device__ void householder_pivoted(double* a, int M, int N, double* tau_s, int* piv, double* cn, double* sh,
                                    int* sel) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j = threadIdx.x; j < N; j += blockDim.x) piv[j] = j;
  __syncthreads();
  for (int k = 0; k < N; ++k) {
    for (int j = k + warp; j < N; j += nw) {
      const double* cj = a + (int64_t)j * M;
      double t = 0.0;
      for (int i = k + lane; i < M; i += 32) t = fma(cj[i], cj[i], t);
      t = wsum(t);
      if (lane == 0) cn[j] = t;
    }
    __syncthreads();
    if (warp == 0) {
      double best = -1.0;
      int bi = k;
      for (int j = k + lane; j < N; j += 32)
        if (cn[j] > best) { best = cn[j]; bi = j; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
      }
      if (lane == 0) *sel = bi;
    }
    __syncthreads();
    const int jm = *sel;
    if (jm != k) {
      double* ck = a + (int64_t)k * M;
      double* cm = a + (int64_t)jm * M;
      for (int i = threadIdx.x; i < M; i += blockDim.x) {
        const double t = ck[i];
        ck[i] = cm[i];
        cm[i] = t;
      }
      if (threadIdx.x == 0) {
        const int t = piv[k];
        piv[k] = piv[jm];
        piv[jm] = t;
      }
    }
    __syncthreads();
    householder_step(a, M, N, k, tau_s, sh);
  }
}

// Apply H_0 ... H_{K-1} (reflectors of `a`) to the M x P matrix c (ld M), backwards.
__device__ void apply_reflectors(const double* a, int M, int K, const double* tau_s, double* c, int P) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = K - 1; k >= 0; --k) {
    const double tau = tau_s[k];
    if (tau != 0.0) {
      const double* v = a + (int64_t)k * M;
      for (int j = warp; j < P; j += nw) {
        double* cj = c + (int64_t)j * M;
        double w = 0.0;
        for (int i = k + 1 + lane; i < M; i += 32) w += v[i] * cj[i];
        w = wsum(w) + cj[k];
        const double tw = tau * w;
        if (lane == 0) cj[k] -= tw;
        for (int i = k + 1 + lane; i < M; i += 32) cj[i] -= tw * v[i];
      }
    }
    __syncthreads();
  }
}

// ---- Householder QR of a sector on a cluster of QC CTAs ----------------------------------------
// CTA r of the cluster holds the columns r, r + QC, .. of the matrix in shared memory.  Step k: every
// CTA copies reflector k from its owner's shared memory and applies it to its columns; the owner of
// column k + 1 takes that column first (its warps 0-3) and makes reflector k + 1 of it, so that the
// cluster barrier of the next step, at which everybody else has arrived long before, completes while
// the other columns are still being updated.  Q = H_0 .. H_{N-1} [I; 0] then needs no exchange but the
// reflectors: each CTA accumulates its own columns.
// What bounds it: one SM does 2 FP64 multiply-adds per clock, so a 300 x 82 sector's 4 million take 1.1
// ms on one SM (1.7 measured with the matrix in global memory); on 8 SMs they take 0.14, and the chain
// of each column is the longer part: some 6,000 cycles for dot product, update, norm, square root and
// division, 1,300 to read the reflector from another SM, 600 to arrive at the barrier.  The norm is
// taken from the updated column: from the old one's sums it costs a reduction less, but cancels (2.9e-13
// off for 1.2e-15) and was no faster.  The maker's other warps wait until it is done: sharing the FP64 pipe
// they delayed the reflector that every CTA needs next (875 us; 818 so), and their CTA has the next seven steps to
// catch up.  QR of A_C and C at Hubbard D = 1024: 3,420 -> 818 us.
constexpr int QC = 8;      // CTAs per cluster (the portable maximum)
constexpr int QT = 256;    // threads per CTA
constexpr int QR_SMEM = 200 * 1024;

// An .aligned barrier wants the whole warp at it together, and what comes before may leave its lanes apart (a
// loop over rows ends for some lanes before others, lane 0 stores alone): __syncwarp() brings them back.
__device__ __forceinline__ void cluster_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same for warps 0-3 alone (bar.sync is the aligned form)
__device__ __forceinline__ void sync128() {
  __syncwarp();
  asm volatile("bar.sync 1, 128;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// a double of CTA `rank`'s shared memory, at the place of this CTA's p
__device__ __forceinline__ double ld_cluster(const double* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), b;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(b) : "memory");
  return v;
}

// sum over the 128 threads of warps 0-3 (named barrier 1), in every one of them; sh: 8 doubles,
// `half` alternates between calls
__device__ __forceinline__ double sum128(double v, double* sh, int half) {
  v = wsum(v);
  double* s = sh + 4 * half;
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  sync128();
  return (s[0] + s[1]) + (s[2] + s[3]);
}

// Reflector of the column x (rows k..M-1) by warps 0-3: x <- v with v[k] = 1, *tau, *beta = R(k, k);
// tail: this thread's share of the sum of squares below row k
__device__ void make_reflector(double* x, int M, int k, double tail, double* tau, double* beta, double* sh) {
  const double tail2 = sum128(tail, sh, 1);
  const double x0 = x[k];
  double t = 0.0, b = x0, scal = 0.0;
  if (tail2 > 0.0) {
    b = -copysign(sqrt(fma(x0, x0, tail2)), x0);
    // both quotients in one division: tau in even lanes, the scale in odd ones
    const bool odd = threadIdx.x & 1;
    const double q = (odd ? 1.0 : b - x0) / (odd ? x0 - b : b);
    t = __shfl_sync(0xffffffffu, q, 0);
    scal = __shfl_sync(0xffffffffu, q, 1);
  }
  sync128();  // x[k] has been read
  if (t != 0.0)
    for (int i = k + 1 + (int)threadIdx.x; i < M; i += 128) x[i] *= scal;
  if (threadIdx.x == 0) {
    x[k] = 1.0;
    *tau = t;
    *beta = b;
  }
}

// c[k..M-1] <- H c for the reflector v, tau by one warp
__device__ __forceinline__ void reflect(double* c, const double* v, double tau, int M, int k, int lane) {
  double w = 0.0;
  for (int i = k + lane; i < M; i += 32) w = fma(v[i], c[i], w);
  w = -tau * wsum(w);
  for (int i = k + lane; i < M; i += 32) c[i] = fma(w, v[i], c[i]);
}

// shared memory of the cluster kernel for an M x N sector (doubles): own columns of A and, if
// q_shared, of Q, and two reflectors
__host__ __device__ constexpr size_t qr_cluster_doubles(int M, int N, bool q_shared) {
  return ((q_shared ? 2 : 1) * (size_t)((N + QC - 1) / QC) + 2) * M;
}

__global__ void __cluster_dims__(QC, 1, 1) __launch_bounds__(QT, 1)
qr_cluster_kernel(const imps::DenseMat* __restrict__ mats, const double* __restrict__ A, double* __restrict__ Q,
                  double* __restrict__ R, int transpose_out, int q_shared) {
  extern __shared__ double qsm[];
  __shared__ double sh[8];
  __shared__ double tau_s[512], beta_s[512];  // of every column; a column's owner writes its own first
  const imps::DenseMat mt = mats[blockIdx.x / QC];
  const int M = mt.M, N = mt.N, rank = (int)cluster_rank();
  if (N <= 0) return;  // the whole cluster
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mine = N > rank ? (N - rank + QC - 1) / QC : 0;  // own columns: rank + QC * jl
  double* cols = qsm;                                        // mine x M
  double* vbuf = qsm + (size_t)((N + QC - 1) / QC) * M;      // 2 x M
  const double* a = A + mt.a_off;
  for (int jl = warp; jl < mine; jl += QT / 32)
    for (int i = lane; i < M; i += 32) cols[(size_t)jl * M + i] = a[i + (int64_t)(rank + QC * jl) * M];
  __syncthreads();
  if (rank == 0 && warp < 4) {
    double tail = 0.0;
    for (int i = 1 + (int)threadIdx.x; i < M; i += 128) tail = fma(cols[i], cols[i], tail);
    make_reflector(cols, M, 0, tail, tau_s, beta_s, sh);
  }
  cluster_arrive();
  for (int k = 0; k < N; ++k) {
    cluster_wait();  // reflector k is made
    const int ow = k % QC;
    double* v = vbuf + (size_t)(k & 1) * M;
    const double* src = cols + (size_t)(k / QC) * M;
    for (int i = k + threadIdx.x; i < M; i += QT) v[i] = ld_cluster(src + i, ow);
    if (warp >= QT / 32 - 2 && lane == 0 && ow != rank) {  // one scalar per warp: their latencies overlap
      double* f = warp == QT / 32 - 1 ? tau_s + k : beta_s + k;
      *f = ld_cluster(f, ow);
    }
    __syncthreads();
    const double tau = tau_s[k];
    const bool next = k + 1 < N && (k + 1) % QC == rank;  // this CTA makes reflector k + 1
    const bool maker = next && warp < 4;
    const int first = (k + 1 - rank + QC - 1) / QC;       // first own column past k
    if (maker) {
      double* c = cols + (size_t)first * M;
      double w = 0.0, tail = 0.0;
      if (tau != 0.0) {
        for (int i = k + (int)threadIdx.x; i < M; i += 128) w = fma(v[i], c[i], w);
        w = -tau * sum128(w, sh, 0);
      }
      for (int i = k + (int)threadIdx.x; i < M; i += 128) {
        const double y = tau != 0.0 ? fma(w, v[i], c[i]) : c[i];
        c[i] = y;
        if (i > k + 1) tail = fma(y, y, tail);
      }
      make_reflector(c, M, k + 1, tail, tau_s + k + 1, beta_s + k + 1, sh);
    }
    if (k + 1 < N) cluster_arrive();
    if (next) __syncthreads();  // the FP64 pipe is the maker's until reflector k + 1 is made
    if (tau != 0.0)
      for (int jl = first + (next ? 1 : 0) + warp; jl < mine; jl += QT / 32)
        reflect(cols + (size_t)jl * M, v, tau, M, k, lane);
  }
  __syncthreads();
  // R (N x N) with a non-negative diagonal: row i times sgn_i
  double* q = Q + mt.q_off;
  double* r = R + mt.r_off;
  for (int jl = warp; jl < mine; jl += QT / 32) {
    const int j = rank + QC * jl;
    for (int i = lane; i < N; i += 32) {
      const double x = i < j ? cols[(size_t)jl * M + i] : i == j ? beta_s[j] : 0.0;
      const double y = i <= j && beta_s[i] < 0.0 ? -x : x;
      if (transpose_out) r[j + (int64_t)i * N] = y;
      else r[i + (int64_t)j * N] = y;
    }
  }
  // Q: own columns q_j = H_0 .. H_j e_j times sgn_j
  double* qc = q_shared ? vbuf + 2 * (size_t)M : q + (int64_t)rank * M;  // column jl at qc + jl * ldq
  const int64_t ldq = q_shared ? M : (int64_t)QC * M;
  for (int jl = warp; jl < mine; jl += QT / 32) {
    const int j = rank + QC * jl;
    for (int i = lane; i < M; i += 32) qc[jl * ldq + i] = i == j ? (beta_s[j] < 0.0 ? -1.0 : 1.0) : 0.0;
  }
  for (int k = N - 1; k >= 0; --k) {
    const double tau = tau_s[k];
    double* v = vbuf + (size_t)(k & 1) * M;
    const double* src = cols + (size_t)(k / QC) * M;
    for (int i = k + threadIdx.x; i < M; i += QT) v[i] = ld_cluster(src + i, k % QC);
    __syncthreads();
    if (tau != 0.0)
      for (int jl = (k - rank + QC - 1) / QC + warp; jl < mine; jl += QT / 32)
        reflect(qc + jl * ldq, v, tau, M, k, lane);
  }
  cluster_arrive();
  if (q_shared) {
    __syncthreads();
    for (int jl = warp; jl < mine; jl += QT / 32)
      for (int i = lane; i < M; i += 32) q[i + (int64_t)(rank + QC * jl) * M] = qc[jl * ldq + i];
  }
  cluster_wait();  // no CTA leaves while another may still read its columns
}

// The same where a sector of the call does not fit a cluster's shared memory, (ceil(N / 8) + 2) M over 25,600
// (M = N: 441 columns fit): one CTA, the matrix in global memory.
// Householder QR of the M x N matrix A (in place, column-major, ld = M), K = min(M,N).
// Outputs Q (M x K, ld M) and R (K x N, ld K) with diag(R) >= 0.
__global__ void __launch_bounds__(DT) qr_kernel(const imps::DenseMat* __restrict__ mats,
                                                double* __restrict__ A, double* __restrict__ Q,
                                                double* __restrict__ R, int transpose_out) {
  __shared__ double sh[32];
  __shared__ double tau_s[512];
  const imps::DenseMat mt = mats[blockIdx.x];
  const int M = mt.M, N = mt.N, K = min(M, N);
  double* a = A + mt.a_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  householder(a, M, N, tau_s, sh);
  // R (K x N) and the sign of its diagonal
  double* q = Q + mt.q_off;
  double* r = R + mt.r_off;
  __shared__ double sgn[512];
  for (int i = threadIdx.x; i < K; i += blockDim.x) sgn[i] = a[i + (int64_t)i * M] < 0.0 ? -1.0 : 1.0;
  __syncthreads();
  for (int64_t t = threadIdx.x; t < (int64_t)K * N; t += blockDim.x) {
    const int i = (int)(t % K), j = (int)(t / K);
    const double v = (j >= i) ? a[i + (int64_t)j * M] * sgn[i] : 0.0;
    if (transpose_out) r[j + (int64_t)i * N] = v;  // R^T (N x K)
    else r[i + (int64_t)j * K] = v;
  }
  // Q = H_0 ... H_{K-1} [I; 0]   (backward accumulation)
  for (int64_t t = threadIdx.x; t < (int64_t)M * K; t += blockDim.x) {
    const int i = (int)(t % M), j = (int)(t / M);
    q[t] = (i == j) ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int k = K - 1; k >= 0; --k) {
    const double tau = tau_s[k];
    if (tau != 0.0) {
      const double* v = a + (int64_t)k * M;
      for (int j = k + warp; j < K; j += nw) {
        double* cj = q + (int64_t)j * M;
        double w = 0.0;
        for (int i = k + 1 + lane; i < M; i += 32) w += v[i] * cj[i];
        w = wsum(w) + cj[k];
        const double tw = tau * w;
        if (lane == 0) cj[k] -= tw;
        for (int i = k + 1 + lane; i < M; i += 32) cj[i] -= tw * v[i];
      }
    }
    __syncthreads();
  }
  for (int64_t t = threadIdx.x; t < (int64_t)M * K; t += blockDim.x) {
    const int j = (int)(t / M);
    q[t] *= sgn[j];
  }
}

// Left null space of the M x N matrix A (M > N, full column rank; dir l of Nullspace,
// MPSBlockUtilities.hpp:247-300): the last M - N columns of the full Householder Q,
// NS = H_0 ... H_{N-1} [0; I_{M-N}] (M x (M - N), orthonormal, orthogonal to A's columns).
__global__ void __launch_bounds__(DT) nullspace_kernel(const imps::DenseMat* __restrict__ mats,
                                                       double* __restrict__ A, double* __restrict__ NS) {
  __shared__ double sh[32];
  __shared__ double tau_s[512];
  const imps::DenseMat mt = mats[blockIdx.x];
  const int M = mt.M, N = mt.N, P = M - N;
  if (P <= 0) return;
  double* a = A + mt.a_off;
  double* ns = NS + mt.ns_off;
  householder(a, M, N, tau_s, sh);
  for (int64_t t = threadIdx.x; t < (int64_t)M * P; t += blockDim.x) {
    const int i = (int)(t % M), j = (int)(t / M);
    ns[t] = (i == N + j) ? 1.0 : 0.0;
  }
  __syncthreads();
  apply_reflectors(a, M, min(M, N), tau_s, ns, P);
}

// One-sided Jacobi SVD of the M x N matrix held in U (in place, M >= N), in global memory (the
// fallback where neither a cluster's nor one CTA's shared memory holds a sector): on exit U holds the
// left singular vectors (M x N), S the singular values (descending), V the right singular vectors
// (N x N).  Round-robin pair ordering; every warp rotates disjoint column pairs.
__global__ void __launch_bounds__(DT) svd_kernel(const imps::DenseMat* __restrict__ mats,
                                                 double* __restrict__ U, double* __restrict__ S,
                                                 double* __restrict__ V, double* __restrict__ Wk,
                                                 int max_sweeps, int* __restrict__ status) {
  __shared__ int rotated;
  __shared__ int perm[512];
  const imps::DenseMat mt = mats[blockIdx.x];
  const int M = mt.M, N = mt.N;
  double* u = U + mt.q_off;
  double* v = V + mt.r_off;
  double* s = S + mt.s_off;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int64_t t = threadIdx.x; t < (int64_t)N * N; t += blockDim.x)
    v[t] = ((t % N) == (t / N)) ? 1.0 : 0.0;
  const int P = N + (N & 1);  // players (padded to even)
  for (int i = threadIdx.x; i < P; i += blockDim.x) perm[i] = i;
  __syncthreads();
  int sweep = 0;
  for (; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) rotated = 0;
    __syncthreads();
    for (int round = 0; round < P - 1; ++round) {
      for (int pr = warp; pr < P / 2; pr += nw) {
        int p = perm[pr], q = perm[P - 1 - pr];
        if (p >= N || q >= N) continue;
        if (p > q) { const int t = p; p = q; q = t; }
        double* cp = u + (int64_t)p * M;
        double* cq = u + (int64_t)q * M;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int i = lane; i < M; i += 32) {
          const double x = cp[i], y = cq[i];
          al += x * x; be += y * y; ga += x * y;
        }
        al = wsum(al); be = wsum(be); ga = wsum(ga);
        if (fabs(ga) > (double)M * 2.220446049250313e-16 * sqrt(al * be) && ga != 0.0) {
          const double zeta = (be - al) / (2.0 * ga);
          const double t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
          const double c = 1.0 / sqrt(1.0 + t * t), sn = c * t;
          for (int i = lane; i < M; i += 32) {
            const double x = cp[i], y = cq[i];
            cp[i] = c * x - sn * y;
            cq[i] = sn * x + c * y;
          }
          double* vp = v + (int64_t)p * N;
          double* vq = v + (int64_t)q * N;
          for (int i = lane; i < N; i += 32) {
            const double x = vp[i], y = vq[i];
            vp[i] = c * x - sn * y;
            vq[i] = sn * x + c * y;
          }
          if (lane == 0) rotated = 1;
        }
      }
      __syncthreads();
      // rotate players 1..P-1 (player 0 fixed)
      if (threadIdx.x == 0) {
        const int last = perm[P - 1];
        for (int i = P - 1; i > 1; --i) perm[i] = perm[i - 1];
        perm[1] = last;
      }
      __syncthreads();
    }
    const int any = rotated;
    __syncthreads();  // every thread has read the flag before thread 0 resets it
    if (!any) break;
  }
  if (threadIdx.x == 0 && sweep >= max_sweeps && status) atomicExch(status, 1);
  // singular values and normalisation
  double* sv = Wk + mt.w_off;  // N scratch values
  for (int j = warp; j < N; j += nw) {
    const double* c = u + (int64_t)j * M;
    double a2 = 0.0;
    for (int i = lane; i < M; i += 32) a2 += c[i] * c[i];
    a2 = wsum(a2);
    if (lane == 0) sv[j] = sqrt(a2);
  }
  __syncthreads();
  for (int j = warp; j < N; j += nw) {
    double* c = u + (int64_t)j * M;
    const double inv = sv[j] > 0.0 ? 1.0 / sv[j] : 0.0;
    for (int i = lane; i < M; i += 32) c[i] *= inv;
  }
  __syncthreads();
  // order descending (stable selection of ranks), applied by permuting into S and via the
  // rank table; U and V columns are permuted through the scratch area
  if (threadIdx.x == 0) {
    for (int j = 0; j < N; ++j) perm[j] = j;
    for (int a = 1; a < N; ++a) {  // insertion sort on indices by sv descending
      const int key = perm[a];
      int b = a - 1;
      while (b >= 0 && sv[perm[b]] < sv[key]) { perm[b + 1] = perm[b]; --b; }
      perm[b + 1] = key;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < N; j += blockDim.x) s[j] = sv[perm[j]];
  // permute columns of U (M x N) and V (N x N) using Wk as a staging copy
  double* stage = Wk + mt.w_off + N;
  for (int64_t t = threadIdx.x; t < (int64_t)M * N; t += blockDim.x) stage[t] = u[t];
  __syncthreads();
  for (int64_t t = threadIdx.x; t < (int64_t)M * N; t += blockDim.x) {
    const int i = (int)(t % M), j = (int)(t / M);
    u[t] = stage[i + (int64_t)perm[j] * M];
  }
  __syncthreads();
  for (int64_t t = threadIdx.x; t < (int64_t)N * N; t += blockDim.x) stage[t] = v[t];
  __syncthreads();
  for (int64_t t = threadIdx.x; t < (int64_t)N * N; t += blockDim.x) {
    const int i = (int)(t % N), j = (int)(t / N);
    v[t] = stage[i + (int64_t)perm[j] * N];
  }
}

constexpr int JT = 1024;  // threads of the shared-memory SVD kernels
constexpr size_t kPjacSmem = 226 * 1024;  // dynamic part; the static flags and sums take < 1 KB
// every column pair of a round has its own lane group (no loop over pairs in jacobi_sweeps)
static_assert((imps::kJacobiMaxN + 1) / 2 <= JT / 2, "FP64 sweeps: one 2-lane group per pair");
static_assert((imps::kMixedMaxN + 1) / 2 <= JT / 16, "FP32 sweeps: one 16-lane group per pair");

// One-sided (Hestenes) Jacobi sweeps on the N columns of B (column-major, ld, shared memory),
// the rotations accumulated into V.  G lanes per column pair split the rows (G = 1: a lane
// owns a pair, so the rotation parameters are computed once per pair, which matters on a GPU
// whose FP64 rate is a few operations per clock per SM); pairs follow the circle round-robin
// schedule in closed form; a pair is rotated while |<b_p, b_q>| > tol |b_p| |b_q|.  Returns the
// number of sweeps run (the last one without rotations), or max_sweeps + 1 if still rotating.
template <typename T, int G>
__device__ int jacobi_sweeps(T* B, T* V, int N, int ld, double tol, int max_sweeps, int* flag) {
  const int P = N + (N & 1);  // players, padded to even; player P-1 stays fixed
  const int k = threadIdx.x / G, gl = threadIdx.x % G;
  const T tl = (T)tol;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x == 0) *flag = 0;
    __syncthreads();
    for (int r = 0; r < P - 1; ++r) {
      int p = 0, q = N;
      if (k < P / 2) {
        p = k == 0 ? r : (r + k) % (P - 1);
        q = k == 0 ? P - 1 : (r - k + (P - 1)) % (P - 1);
        if (p > q) { const int t = p; p = q; q = t; }
      }
      const bool valid = k < P / 2 && q < N;  // p < q, so q < N implies p < N
      T al = 0, be = 0, ga = 0;
      if (valid) {
        const T* bp = B + (int64_t)p * ld;
        const T* bq = B + (int64_t)q * ld;
        for (int i = gl; i < N; i += G) {
          const T x = bp[i], y = bq[i];
          al = fma(x, x, al);
          be = fma(y, y, be);
          ga = fma(x, y, ga);
        }
      }
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) {  // every lane of the warp takes part
        al += __shfl_xor_sync(0xffffffffu, al, o);
        be += __shfl_xor_sync(0xffffffffu, be, o);
        ga += __shfl_xor_sync(0xffffffffu, ga, o);
      }
      if (valid && ga != (T)0 && fabs(ga) > tl * sqrt(al * be)) {
        const T zeta = (be - al) / ((T)2 * ga);
        const T t = copysign((T)1, zeta) / (fabs(zeta) + sqrt((T)1 + zeta * zeta));
        const T c = (T)1 / sqrt((T)1 + t * t), sn = c * t;
        T* bp = B + (int64_t)p * ld;
        T* bq = B + (int64_t)q * ld;
        T* vp = V + (int64_t)p * ld;
        T* vq = V + (int64_t)q * ld;
        for (int i = gl; i < N; i += G) {
          const T x = bp[i], y = bq[i];
          bp[i] = c * x - sn * y;
          bq[i] = sn * x + c * y;
          const T xv = vp[i], yv = vq[i];
          vp[i] = c * xv - sn * yv;
          vq[i] = sn * xv + c * yv;
        }
        if (gl == 0) *flag = 1;
      }
      __syncthreads();
    }
    const int any = *flag;
    __syncthreads();  // every thread has read the flag before thread 0 resets it
    if (!any) return sweep + 1;
  }
  return max_sweeps + 1;
}

// SVD of the M x N sector matrix held in U (M >= N, N <= kJacobiMaxN) by one CTA, for sectors whose columns
// do not fit a cluster's shared memory (N = 96: M > 1,470), with the preconditioning of Drmac and Veselic
// (SIAM J. Matrix Anal. Appl. 29 (2008) 1322): Householder QR with column pivoting A P = Q R, then one-sided
// Jacobi on the columns of X = R^T, which is
// strongly graded and converges in a few sweeps (the unpivoted form needs 15-30 sweeps on
// sectors whose singular values span many decades).  X Vx = Ux S gives R = Vx S Ux^T, so
// U = Q [Vx; 0] and V = P Ux.  MIXED: the first sweeps run in FP32 (many times the FP64 rate
// on this GPU) on a copy of X; their rotations V0 are made orthonormal in FP64 by one
// Cholesky-QR step (V0^T V0 = L L^T, V0 <- V0 L^-T), and FP64 sweeps on B = X V0, accumulating
// into V0, converge quadratically from there.  Either way the last sweep passes the FP64 test
// |<b_p, b_q>| <= N eps |b_p| |b_q| for all pairs.  Outputs as svd_kernel: U (M x N) left
// singular vectors, S descending, V (N x N) right singular vectors.
template <bool MIXED>
__global__ void __launch_bounds__(JT) svd_pjac_kernel(const imps::SvdSets sets, int a_smem, int max_sweeps,
                                                      int* __restrict__ status) {
  extern __shared__ double smem[];
  __shared__ double sh[32];
  __shared__ int flag, sel;
  int bi = blockIdx.x, ks = 0;
  while (ks + 1 < sets.nsets && bi >= sets.s[ks].n) {
    bi -= sets.s[ks].n;
    ++ks;
  }
  const imps::DenseMat mt = sets.s[ks].mats[bi];
  double* __restrict__ U = sets.s[ks].U;
  double* __restrict__ S = sets.s[ks].S;
  double* __restrict__ V = sets.s[ks].V;
  double* __restrict__ Wk = sets.s[ks].W;
  const int M = mt.M, N = mt.N;
  if (N <= 0 || M < N) return;
  const int ld = N | 1;  // odd: lanes owning different columns hit different banks
  const int64_t sq = (int64_t)ld * N;
  double* tau = Wk + mt.w_off;
  double* xs = smem;                       // X = R^T (FP64), rotated into B (FP64-only form)
  double* vs = xs + sq;                    // Vx
  double* tmp = MIXED ? vs + sq : nullptr; // FP32 X and V, then L, then B
  double* sig = (MIXED ? tmp : vs) + sq;
  double* cn = sig + N;
  int* perm = (int*)(cn + N);
  int* piv = perm + N;
  double* a = a_smem ? (double*)(piv + N) : Wk + mt.w_off + N;
  double* u = U + mt.q_off;
  for (int64_t t = threadIdx.x; t < (int64_t)M * N; t += blockDim.x) a[t] = u[t];
  __syncthreads();
  householder_pivoted(a, M, N, tau, piv, cn, sh, &sel);
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
    const int i = t % N, j = t / N;
    xs[i + j * ld] = i >= j ? a[j + (int64_t)i * M] : 0.0;  // X = R^T, lower triangular
    vs[i + j * ld] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  const double tol = (double)N * 2.220446049250313e-16;
  double* B = xs;
  if (MIXED) {
    float* xf = (float*)tmp;
    float* vf = xf + sq;
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int i = t % N, j = t / N;
      xf[i + j * ld] = (float)xs[i + j * ld];
      vf[i + j * ld] = i == j ? 1.0f : 0.0f;
    }
    __syncthreads();
    jacobi_sweeps<float, 16>(xf, vf, N, ld, 1e-5, 8, &flag);
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int i = t % N, j = t / N;
      vs[i + j * ld] = (double)vf[i + j * ld];
    }
    __syncthreads();
    // Cholesky-QR: lower triangle of G = V0^T V0 into tmp, G = L L^T in place, V0 <- V0 L^-T
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int i = t % N, j = t / N;
      if (i < j) continue;
      const double* ci = vs + (int64_t)i * ld;
      const double* cj = vs + (int64_t)j * ld;
      double g = 0.0;
      for (int r = 0; r < N; ++r) g = fma(ci[r], cj[r], g);
      tmp[i + j * ld] = g;
    }
    __syncthreads();
    for (int kk = 0; kk < N; ++kk) {
      if (threadIdx.x == 0) tmp[kk + kk * ld] = sqrt(fmax(tmp[kk + kk * ld], 1e-300));
      __syncthreads();
      const double dk = tmp[kk + kk * ld];
      for (int i = kk + 1 + threadIdx.x; i < N; i += blockDim.x) tmp[i + kk * ld] /= dk;
      __syncthreads();
      const int rem = N - kk - 1;
      for (int t = threadIdx.x; t < rem * rem; t += blockDim.x) {
        const int i = kk + 1 + t % rem, j = kk + 1 + t / rem;
        if (i >= j) tmp[i + j * ld] -= tmp[i + kk * ld] * tmp[j + kk * ld];
      }
      __syncthreads();
    }
    for (int r = threadIdx.x; r < N; r += blockDim.x) {  // row r of V0: x L^T = V0[r, :]
      for (int j = 0; j < N; ++j) {
        double x = vs[r + j * ld];
        for (int kk = 0; kk < j; ++kk) x = fma(-vs[r + kk * ld], tmp[j + kk * ld], x);
        vs[r + j * ld] = x / tmp[j + j * ld];
      }
    }
    __syncthreads();
    // B = X V0 (X lower triangular) into tmp
    for (int t = threadIdx.x; t < N * N; t += blockDim.x) {
      const int i = t % N, j = t / N;
      const double* vj = vs + (int64_t)j * ld;
      double b = 0.0;
      for (int kk = 0; kk <= i; ++kk) b = fma(xs[i + kk * ld], vj[kk], b);
      tmp[i + j * ld] = b;
    }
    __syncthreads();
    B = tmp;
  }
  const int sw = jacobi_sweeps<double, 2>(B, vs, N, ld, tol, max_sweeps, &flag);
  if (threadIdx.x == 0 && sw > max_sweeps && status) atomicExch(status, 1);
  // singular values, descending (ties by index)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int j = warp; j < N; j += nw) {
    const double* c = B + (int64_t)j * ld;
    double a2 = 0.0;
    for (int i = lane; i < N; i += 32) a2 = fma(c[i], c[i], a2);
    a2 = wsum(a2);
    if (lane == 0) sig[j] = sqrt(a2);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < N; j += blockDim.x) {
    int rk = 0;
    for (int i = 0; i < N; ++i) rk += (sig[i] > sig[j] || (sig[i] == sig[j] && i < j)) ? 1 : 0;
    perm[rk] = j;
  }
  __syncthreads();
  double* s_out = S + mt.s_off;
  double* v_out = V + mt.r_off;
  for (int j = threadIdx.x; j < N; j += blockDim.x) s_out[j] = sig[perm[j]];
  for (int t = threadIdx.x; t < N * N; t += blockDim.x) {  // V = P Ux: row piv[i] of V = row i of Ux
    const int i = t % N, j = t / N;
    const int pj = perm[j];
    v_out[piv[i] + (int64_t)j * N] = sig[pj] > 0.0 ? B[i + (int64_t)pj * ld] / sig[pj] : 0.0;
  }
  for (int64_t t = threadIdx.x; t < (int64_t)M * N; t += blockDim.x) {  // U = Q [Vx; 0]
    const int i = (int)(t % M), j = (int)(t / M);
    u[t] = i < N ? vs[i + (int64_t)perm[j] * ld] : 0.0;
  }
  __syncthreads();
  apply_reflectors(a, M, N, tau, u, N);
}

// ---- sector SVD on a cluster of QC CTAs ---------------------------------------------------------
// The steps of svd_pjac_kernel (pivoted QR, FP32 then FP64 one-sided Jacobi on the columns of X = R^T) with
// the work of a sector spread over eight SMs:
//   * Pivoted QR as in qr_cluster_kernel, columns staying in place: every CTA proposes the longest of its own
//     remaining columns (its norm summed anew in each update) and the cluster takes the longest of the
//     eight, so that a step needs one cluster barrier (and two of the CTA's own).
//   * Jacobi by blocks: the columns of B and V are 16 blocks in global memory (L2).  In each of 15 rounds a
//     CTA loads two blocks, rotates the pairs between them (in the first round also those inside them) in
//     shared memory, and stores them.  The tangent of a rotation is taken in FP32: it only decides how small
//     the pair's product becomes.  Cosine and sine are FP64 with c^2 + s^2 = 1 to rounding.
//   * V of the FP32 sweeps is made orthonormal by two Newton-Schulz steps V <- V (3 - V^T V) / 2 (error
//     1e-6, 1e-12, rounding; at most 6e-4, 3e-7, 6e-14 if every rounding of eight sweeps of 95 rounds, 8e-7
//     each, pulled the same way); the Cholesky factorisation of the one-CTA form is a serial chain.
// What bounds it, for a 136 x 68 sector over four decades (one CTA -> cluster, us): the QR, 2,123 -> 345, a
// chain of a cluster barrier, a remote read, square root and division a step; the FP32 sweeps, 635 -> 433, the
// latency of a turn (920 cycles: 280 to load and multiply, 210 parameters, 130 to store); the FP64 sweeps,
// 3,060 -> 458, FP64 instructions at 64 cycles a warp; the products, 300 -> 77; U, 795 -> 157.  The polar
// step of XXZ D = 512 (both directions, 42 sectors): 6,690 -> 1,610 us.  20 equal sectors of N columns:
// N = 1 27 -> 27 us, 4 131 -> 81, 16 707 -> 377, 64 5,806 -> 1,259, 118 34,322 -> 4,231, so every sector that
// fits comes here.
constexpr int JB = 2 * QC;  // column blocks
constexpr int SVD_MAXN = 256;
constexpr int SVD_SMEM = 216 * 1024;
constexpr int SVD_SMEM2 = 102 * 1024;  // with two CTAs on an SM

// shared memory (doubles) of an M x N sector: the columns of A with two reflectors and two candidates, and
// then in turn the Jacobi blocks; own columns of two N x N matrices and kc columns of a third; own columns of U
__host__ __device__ constexpr size_t svd_base_doubles(int M, int N) { return ((size_t)(N + QC - 1) / QC + 4) * M; }
__host__ __device__ constexpr size_t svd_work_doubles(int M, int N, int kc, bool u_shared) {
  const size_t own = (N + QC - 1) / QC, bs = (N + JB - 1) / JB;
  size_t w = 4 * bs * N;
  const size_t prod = 2 * own * N + (size_t)kc * (N | 1), u = u_shared ? own * M : 0;
  if (prod > w) w = prod;
  return u > w ? u : w;
}

__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
__device__ __forceinline__ int ld_cluster(const int* p, uint32_t rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), b;
  int v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(b) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(double* p, uint32_t rank, double v) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), b;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(b), "d"(v) : "memory");
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// tan of the rotation for zeta = (be - al) / (2 ga), to FP32 rounding (0 for zeta beyond 1e19)
__device__ __forceinline__ float tangent(float zeta) {
  return __fdividef(copysignf(1.f, zeta), fabsf(zeta) + sqrt_approx(fmaf(zeta, zeta, 1.f)));
}
// x 2^-(e - 1023) as a float, truncated; 0 if that is below the normal floats (e: at least x's exponent field)
__device__ __forceinline__ float scaled_float(double x, int e) {
  const int hi = __double2hiint(x), ex = ((hi >> 20) & 0x7ff) - e + 127;
  const int m = (hi & 0xfffff) << 3 | (unsigned)__double2loint(x) >> 29;
  return ex > 0 ? __int_as_float((hi & 0x80000000) | ex << 23 | m) : 0.f;
}

// The rotation that makes two columns with squared norms al, be and product ga orthogonal, and the new
// squared norms; false if |ga| <= tol sqrt(al be) already.  mr, mt: the largest |ga| / sqrt(al be) and
// |tangent| so far.
__device__ __forceinline__ bool rotation(float& al, float& be, float ga, float tol, float& c, float& s, float& mr,
                                         float& mt) {
  const float ratio = fabsf(ga) * rsqrtf(al) * rsqrtf(be);
  if (!(ratio > tol)) return false;
  const float t = tangent(__fdividef(be - al, 2.f * ga));
  mr = fmaxf(mr, ratio);
  mt = fmaxf(mt, fabsf(t));
  c = rsqrtf(fmaf(t, t, 1.f));
  s = c * t;
  al = fmaf(-t, ga, al);
  be = fmaf(t, ga, be);
  return true;
}
__device__ __forceinline__ bool rotation(double& al, double& be, double ga, double tol, double& c, double& s, float& mr,
                                         float& mt) {
  const int ea = (__double2hiint(al) >> 20) & 0x7ff, eb = (__double2hiint(be) >> 20) & 0x7ff;
  const int e = max(ea, eb);
  double t;
  if (e - min(ea, eb) < 100 && e > 200 && e < 1900) {
    const float gf = scaled_float(ga, e), ratio = fabsf(gf) * rsqrtf(scaled_float(al, e) * scaled_float(be, e));
    if (!(ratio > (float)tol)) return false;
    mr = fmaxf(mr, ratio);
    const float zeta = __fdividef(scaled_float(be - al, e), 2.f * gf);
    t = fabsf(zeta) > 1e9f ? __fdividef(0.5f, zeta) : tangent(zeta);
  } else {
    if (!(ga != 0.0 && fabs(ga) > tol * sqrt(al) * sqrt(be))) return false;
    const double zeta = (be - al) / (2.0 * ga);
    t = copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
    mr = 1.f;
  }
  mt = fmaxf(mt, fabsf((float)t));
  const double u = t * t;
  if (u < 0x1p-14) {  // (1 + u)^-1/2 by its series; the next term is below 2^-57
    c = fma(u, fma(u, fma(u, -0.3125, 0.375), -0.5), 1.0);
  } else {
    double y = rsqrtf((float)(1.0 + u));
#pragma unroll
    for (int i = 0; i < 2; ++i) y = fma(0.5 * y, fma(-(1.0 + u) * y, y, 1.0), y);  // Newton: 2^-22, 2^-43, rounding
    c = y;
  }
  s = c * t;
  al = fma(-t, ga, al);
  be = fma(t, ga, be);
  return true;
}

// One-sided Jacobi sweeps on the columns of B (N x N, global memory), the rotations into V, until every pair
// has |<b_i, b_j>| <= tol |b_i| |b_j|: the sweep rotated nothing, or so little that it left no more.  (A pair
// that the sweep has made orthogonal gets products back from later rotations of either column with a third:
// at most N of the size mr max(mr, mt), for the largest ratio |<b_i, b_j>| / |b_i| |b_j| and tangent that
// the sweep met; so `rest` = tol / N does.  And the FP32 tangent, within 2^-21 of the right one, leaves
// a pair up to 2^-21 of its ratio, more than tol for narrow sectors.)  nrm_g: squared column norms
// (scratch).  An FP64 instruction takes 64 cycles of its scheduler however many lanes it serves and a round
// of N = 68 has 5 pairs, so a pair has 16 lanes: warps 0-3 take products, parameters and B, the others V,
// one turn behind.
// G lanes per pair with R rows each (N <= G R; loops of fixed length: a branch per step cost 20 cycles each).
// Returns the sweeps run, max_sweeps + 1 if the last one still rotated.
struct SweepShared {
  double nrm[2 * SVD_MAXN / JB], rc[2][SVD_MAXN / JB], rs[2][SVD_MAXN / JB];
  int rij[2][SVD_MAXN / JB];  // rotations of this turn and the one before: columns i, j or -1
  int flag[2];
};
template <typename T, int G, int R>
__device__ int cluster_sweeps(T* B, T* V, T* nrm_g, int N, T tol, float rest, int max_sweeps, T* sm, SweepShared& sh,
                              int rank) {
  constexpr int PAIRS = 128 / G, RV = (R * G + 31) / 32;
  T* nrm = (T*)sh.nrm;
  T(*rc)[SVD_MAXN / JB] = (T(*)[SVD_MAXN / JB])sh.rc;
  T(*rs)[SVD_MAXN / JB] = (T(*)[SVD_MAXN / JB])sh.rs;
  int(*rij)[SVD_MAXN / JB] = sh.rij;
  int* flag = sh.flag;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gl = threadIdx.x & (G - 1);
  const int nblk = min(JB, max(2, N + (N & 1)));  // fewer columns than blocks: a column each
  auto start = [&](int b) { return b * N / nblk; };
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    if (threadIdx.x < 2) flag[threadIdx.x] = 0;
    float mr = 0.f, mt = 0.f;
    for (int r = 0; r < nblk - 1; ++r) {
      const int p = rank == 0 ? nblk - 1 : (r + rank) % (nblk - 1);
      const int q = rank == 0 ? r : (r - rank + QC * (nblk - 1)) % (nblk - 1);
      const bool on = rank < nblk / 2;  // else no blocks
      const int sp = start(p), np = on ? start(p + 1) - sp : 0, sq = start(q), nq = on ? start(q + 1) - sq : 0;
      const int n2 = np + nq;
      T *b = sm, *v = sm + (size_t)n2 * N;
      auto global_of = [&](int e) { return e < np * N ? sp * N + e : (sq - np) * N + e; };
#pragma unroll 4
      for (int e = threadIdx.x; e < n2 * N; e += QT) {
        const int g = global_of(e);
        const T x = __ldcg(B + g), y = __ldcg(V + g);
        b[e] = x;
        v[e] = y;
      }
      if (r == 0) {
        __syncthreads();
        for (int i = warp; i < n2; i += QT / 32) {
          T a2 = 0;
          for (int e = lane; e < N; e += 32) a2 = fma(b[(size_t)i * N + e], b[(size_t)i * N + e], a2);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) a2 += __shfl_xor_sync(0xffffffffu, a2, o);
          if (lane == 0) nrm[i] = a2;
        }
      } else if (threadIdx.x < n2) {
        nrm[threadIdx.x] = __ldcg(nrm_g + ((int)threadIdx.x < np ? sp + threadIdx.x : sq - np + threadIdx.x));
      }
      __syncthreads();
      // r = 0: all pairs of both blocks, by the circle schedule; else those between the blocks
      const int P = n2 + (n2 & 1), m = max(np, nq), turns = r == 0 ? P - 1 : m, pairs = r == 0 ? P / 2 : np;
      const int nb = min(4, (pairs * G + 31) / 32);  // warps with pairs; V: the others, idle schedulers first
      const int vw = warp < nb ? -1 : (warp & 3) >= nb ? (warp >> 2) * (4 - nb) + (warp & 3) - nb : warp + 4 - 2 * nb;
      for (int t = 0; t <= turns; ++t) {
        if (warp < nb && t < turns) {
          for (int k0 = 0; k0 < pairs; k0 += PAIRS) {
            const int k = k0 + threadIdx.x / G;
            int i = 0, j = n2;
            if (k < pairs) {
              if (r > 0) {
                i = k;
                j = k + t < m ? k + t : k + t - m;
                j = j < nq ? np + j : n2;
              } else {
                i = k == 0 ? t : (t + k) % (P - 1);
                j = k == 0 ? P - 1 : (t - k + P - 1) % (P - 1);
                if (i > j) { const int z = i; i = j; j = z; }
              }
            }
            const bool valid = j < n2;
            if (!valid) j = 0;  // loads without branches: of any column, past the end of the last element
            T *bp = b + (size_t)i * N, *bq = b + (size_t)j * N;
            T x[R], y[R], ga = 0, al, be, c = 1, s = 0;
#pragma unroll
            for (int u = 0; u < R; ++u) {
              const int e = min(gl + u * G, N - 1);
              x[u] = bp[e];
              y[u] = bq[e];
            }
            al = nrm[i];
            be = nrm[j];
#pragma unroll
            for (int u = 0; u < R; ++u) {
              ga = fma(gl + u * G < N ? x[u] : (T)0, y[u], ga);
            }
            if (G == 32) ga += __shfl_xor_sync(0xffffffffu, ga, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) ga += __shfl_xor_sync(0xffffffffu, ga, o);
            const bool turn = valid && rotation(al, be, ga, tol, c, s, mr, mt);
            if (gl == 0 && k < pairs) {
              rij[t & 1][k] = turn ? i << 16 | j : -1;
              if (turn) {
                rc[t & 1][k] = c;
                rs[t & 1][k] = s;
                nrm[i] = al;
                nrm[j] = be;
              }
            }
            if (turn) {
#pragma unroll
              for (int u = 0; u < R; ++u) {
                const int e = gl + u * G;
                const T xn = c * x[u] - s * y[u], yn = s * x[u] + c * y[u];
                if (e < N) {
                  bp[e] = xn;
                  bq[e] = yn;
                }
              }
            }
          }
        }
        if (vw >= 0 && t > 0) {
          const int h = (t - 1) & 1;
          for (int k = vw; k < pairs; k += 8 - nb) {
            const int ij = rij[h][k];
            if (ij < 0) continue;
            T *vp = v + (size_t)(ij >> 16) * N, *vq = v + (size_t)(ij & 0xffff) * N;
            const T c = rc[h][k], s = rs[h][k];
            T x[RV], y[RV];
#pragma unroll
            for (int u = 0; u < RV; ++u) {
              const int e = min(lane + u * 32, N - 1);
              x[u] = vp[e];
              y[u] = vq[e];
            }
#pragma unroll
            for (int u = 0; u < RV; ++u) {
              const int e = lane + u * 32;
              const T xn = c * x[u] - s * y[u], yn = s * x[u] + c * y[u];
              if (e < N) {
                vp[e] = xn;
                vq[e] = yn;
              }
            }
          }
        }
        __syncthreads();
      }
#pragma unroll 4
      for (int e = threadIdx.x; e < n2 * N; e += QT) {
        const int g = global_of(e);
        __stcg(B + g, b[e]);
        __stcg(V + g, v[e]);
      }
      if (threadIdx.x < n2)
        __stcg(nrm_g + ((int)threadIdx.x < np ? sp + threadIdx.x : sq - np + threadIdx.x), nrm[threadIdx.x]);
      if (r == nblk - 2 && gl == 0 && mr > 0.f) {  // non-negative floats compare as integers
        atomicMax(flag, __float_as_int(mr));
        atomicMax(flag + 1, __float_as_int(mt));
      }
      if (r == nblk - 2) __syncthreads();
      cluster_sync();
    }
    int ir = 0, it = 0;
    for (int c = 0; c < QC; ++c) {
      ir = max(ir, ld_cluster(flag, c));
      it = max(it, ld_cluster(flag + 1, c));
    }
    cluster_sync();  // every flag has been read before it is reset
    mr = __int_as_float(ir);
    if (mr * fmaxf(mr, __int_as_float(it)) <= rest && mr * 0x1p-21f <= (float)tol) return sweep + 1;
  }
  return max_sweeps + 1;
}

// ... for N up to SVD_MAXN
template <typename T>
__device__ int cluster_sweeps(T* B, T* V, T* nrm_g, int N, T tol, float rest, int max_sweeps, T* sm, SweepShared& sh,
                              int rank) {
#define IMPS_SWEEPS(G, R) return cluster_sweeps<T, G, R>(B, V, nrm_g, N, tol, rest, max_sweeps, sm, sh, rank)
  switch ((N + 15) / 16) {
    case 0: case 1: case 2: IMPS_SWEEPS(16, 2);
    case 3: IMPS_SWEEPS(16, 3);
    case 4: IMPS_SWEEPS(16, 4);
    case 5: IMPS_SWEEPS(16, 5);
    case 6: IMPS_SWEEPS(16, 6);
    case 7: case 8: IMPS_SWEEPS(16, 8);
    default: IMPS_SWEEPS(32, 8);
  }
#undef IMPS_SWEEPS
}

__global__ void __cluster_dims__(QC, 1, 1) __launch_bounds__(QT, 2)
svd_cluster_kernel(const imps::SvdSets sets, int smem_doubles, int max_sweeps, int* __restrict__ status) {
  extern __shared__ double qsm[];
  __shared__ double tau_s[SVD_MAXN], beta_s[SVD_MAXN], sig[SVD_MAXN];
  __shared__ int piv[SVD_MAXN], perm[SVD_MAXN];
  __shared__ double tail_s[32], cand[2][QC][5];  // candidates of all CTAs: norm^2, column, beta, tau, scale
  __shared__ int done_s[32];
  __shared__ SweepShared sweep_s;
  // the widest sectors first: they get SMs of their own, and the narrow ones fill up
  int bi = blockIdx.x / QC, ks = 0;
  const int total = gridDim.x / QC;
  const auto locate = [&](int g, int& k) {
    for (k = 0; k + 1 < sets.nsets && g >= sets.s[k].n; ++k) g -= sets.s[k].n;
    return g;
  };
  if (total <= SVD_MAXN) {
    for (int g = threadIdx.x; g < total; g += QT) {
      const int l = locate(g, ks);
      perm[g] = sets.s[ks].mats[l].N;
    }
    __syncthreads();
    for (int g = threadIdx.x; g < total; g += QT) {
      int rk = 0;
      for (int h = 0; h < total; ++h) rk += (perm[h] > perm[g] || (perm[h] == perm[g] && h < g)) ? 1 : 0;
      piv[rk] = g;
    }
    __syncthreads();
    bi = piv[bi];
    __syncthreads();
  }
  bi = locate(bi, ks);
  const imps::DenseMat mt = sets.s[ks].mats[bi];
  const int M = mt.M, N = mt.N, rank = (int)cluster_rank();
  if (N <= 0 || M < N) return;  // the whole cluster
  double* U = sets.s[ks].U + mt.q_off;
  double* S = sets.s[ks].S + mt.s_off;
  double* Vo = sets.s[ks].V + mt.r_off;
  double* W = sets.s[ks].W + mt.w_off + N;  // M * N doubles of scratch
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = QT / 32;
  const int own = (N + QC - 1) / QC, mine = N > rank ? (N - rank + QC - 1) / QC : 0;
  double* cols = qsm;                     // own columns rank + QC * jl of A
  double* vcand = cols + (size_t)own * M; // 2 x M: this CTA's candidate column
  double* vbuf = vcand + 2 * (size_t)M;   // 2 x M: the step's reflector
  double* buf = vbuf + 2 * (size_t)M;
  const int room = smem_doubles - (int)svd_base_doubles(M, N);

  // ---- A P = Q R
  for (int jl = warp; jl < mine; jl += nw) {
    double t = 0.0;
    for (int i = lane; i < M; i += 32) {
      const double x = U[i + (int64_t)(rank + QC * jl) * M];
      cols[(size_t)jl * M + i] = x;
      if (i > 0) t = fma(x, x, t);
    }
    t = wsum(t);
    if (lane == 0) {
      tail_s[jl] = t;
      done_s[jl] = 0;
    }
  }
  cluster_sync();  // every CTA of the cluster has started
  for (int k = 0; k < N; ++k) {
    const int par = k & 1;
    // the longest own column that is left, in every warp; squared norms compare as integers (one that is
    // not a number counts as 0, so that every step finds a column)
    double n2 = 0.0;
    long long key = -1;
    int bj = lane;
    if (lane < mine && !done_s[lane]) {
      const double x = cols[(size_t)lane * M + k];
      n2 = fma(x, x, tail_s[lane]);
      key = n2 >= 0.0 ? __double_as_longlong(n2) : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long ok = __shfl_xor_sync(0xffffffffu, key, o);
      const int oj = __shfl_xor_sync(0xffffffffu, bj, o);
      if (ok > key || (ok == key && oj < bj)) { key = ok; bj = oj; }
    }
    if (key >= 0) {
      const double* c = cols + (size_t)bj * M;
      for (int i = k + threadIdx.x; i < M; i += QT) vcand[(size_t)par * M + i] = c[i];
    }
    if (warp == 0) {
      double beta = 0.0, tau = 0.0, scal = 0.0;
      n2 = __shfl_sync(0xffffffffu, n2, bj);
      if (key >= 0) {
        const double x0 = cols[(size_t)bj * M + k];
        beta = x0;
        if (tail_s[bj] > 0.0) {
          beta = -copysign(sqrt(n2), x0);
          // both quotients in one division: tau in even lanes, the scale in odd ones
          const double q = (lane & 1 ? 1.0 : beta - x0) / (lane & 1 ? x0 - beta : beta);
          tau = __shfl_sync(0xffffffffu, q, 0);
          scal = __shfl_sync(0xffffffffu, q, 1);
        }
      }
      if (lane < QC) {
        double* d = cand[par][rank];
        st_cluster(d, lane, key >= 0 ? __longlong_as_double(key) : -1.0);
        st_cluster(d + 1, lane, (double)(rank + QC * bj));
        st_cluster(d + 2, lane, beta);
        st_cluster(d + 3, lane, tau);
        st_cluster(d + 4, lane, scal);
      }
    }
    cluster_sync();
    int cr = 0, ci = 0;  // the longest of the eight (ties: the smallest index)
    key = -1;
    for (int r = 0; r < QC; ++r) {
      const double cn = cand[par][r][0];
      const long long ok = __double_as_longlong(cn);
      const int oi = (int)cand[par][r][1];
      if (ok >= 0 && (ok > key || (ok == key && oi < ci))) { key = ok; ci = oi; cr = r; }
    }
    const double tau = cand[par][cr][3], scal = cand[par][cr][4];
    double* v = vbuf + (size_t)par * M;
    for (int i = k + threadIdx.x; i < M; i += QT) {
      const double x = ld_cluster(vcand + (size_t)par * M + i, cr);
      v[i] = i == k ? 1.0 : scal * x;
    }
    if (threadIdx.x == 0) {
      piv[k] = ci;
      tau_s[k] = tau;
      beta_s[k] = cand[par][cr][2];
      if (cr == rank) done_s[ci / QC] = 1;
    }
    __syncthreads();
    for (int jl = warp; jl < mine; jl += nw) {
      double* c = cols + (size_t)jl * M;
      if (cr == rank && jl == ci / QC) {
        for (int i = k + lane; i < M; i += 32) c[i] = v[i];
      } else if (!done_s[jl]) {
        double w = 0.0, t = 0.0;
        if (tau != 0.0) {
          for (int i = k + lane; i < M; i += 32) w = fma(v[i], c[i], w);
          w = -tau * wsum(w);
        }
        for (int i = k + lane; i < M; i += 32) {
          const double y = tau != 0.0 ? fma(w, v[i], c[i]) : c[i];
          c[i] = y;
          if (i > k + 1) t = fma(y, y, t);
        }
        t = wsum(t);
        if (lane == 0) tail_s[jl] = t;
      }
    }
    __syncthreads();
  }

  // ---- X = R^T (lower triangular) in U's place, its FP32 copy scaled to about 1, and V = 1
  float* Xf = (float*)Vo;
  float* Vf = Xf + (size_t)N * N;
  const int eb = (__double2hiint(beta_s[0]) >> 20) & 0x7ff;
  const double xs = eb > 0 && eb < 2046 ? __hiloint2double((2046 - eb) << 20, 0) : 1.0;
  for (int i = warp; i < N; i += nw) {  // column i of R is column piv[i] of A
    if (piv[i] % QC != rank) continue;
    const double* c = cols + (size_t)(piv[i] / QC) * M;
    for (int j = lane; j < N; j += 32) {
      const double x = j < i ? c[j] : j == i ? beta_s[i] : 0.0;
      __stcg(U + i + (int64_t)j * N, x);
      __stcg(Xf + i + (size_t)j * N, (float)(x * xs));
      __stcg(Vf + i + (size_t)j * N, i == j ? 1.f : 0.f);
    }
  }
  cluster_sync();
  cluster_sweeps<float>(Xf, Vf, (float*)S, N, 1e-5f, 1e-5f, 8, (float*)buf, sweep_s, rank);

  // ---- V orthonormal in FP64, every CTA its own columns rank + QC * jl (N x own in shared memory)
  const int ld = N | 1;
  double* vc = buf;
  double* yc = vc + (size_t)own * N;
  double* part = yc + (size_t)own * N;  // kc columns of an N x N matrix
  const int kc = min(N, (room - 2 * own * N) / ld);
  // out = a0 out + a1 F in, or out = F^T in; F: N x N in global memory; `held`: it is in `part` already
  auto product = [&](const double* F, bool trans, const double* in, double* out, double a0, double a1, bool held) {
    for (int k0 = 0; k0 < N; k0 += kc) {
      const int nk = min(kc, N - k0);
      __syncthreads();
      if (!held || kc < N) {
        for (int k = warp; k < nk; k += nw)
          for (int i = lane; i < N; i += 32) part[i + (size_t)k * ld] = __ldcg(F + i + (int64_t)(k0 + k) * N);
        __syncthreads();
      }
      const int nr = trans ? nk : N;
      for (int e = threadIdx.x; e < nr * mine; e += QT) {
        const int jl = e / nr, i = e - jl * nr;
        double a = 0.0;
        if (trans) {
          const double *f = part + (size_t)i * ld, *x = in + (size_t)jl * N;
#pragma unroll 4
          for (int r = 0; r < N; ++r) a = fma(f[r], x[r], a);
          out[k0 + i + (size_t)jl * N] = a;
        } else {
          const double *f = part + i, *x = in + (size_t)jl * N + k0;
#pragma unroll 4
          for (int k = 0; k < nk; ++k) a = fma(f[(size_t)k * ld], x[k], a);
          double* o = out + i + (size_t)jl * N;
          *o = fma(a1, a, k0 > 0 ? *o : a0 == 0.0 ? 0.0 : a0 * *o);
        }
      }
    }
    __syncthreads();
  };
  auto publish = [&](double* g, const double* c) {
    for (int jl = warp; jl < mine; jl += nw)
      for (int i = lane; i < N; i += 32) __stcg(g + i + (int64_t)(rank + QC * jl) * N, c[i + (size_t)jl * N]);
    cluster_sync();
  };
  for (int jl = warp; jl < mine; jl += nw)
    for (int i = lane; i < N; i += 32) vc[i + (size_t)jl * N] = (double)__ldcg(Vf + i + (size_t)(rank + QC * jl) * N);
  __syncthreads();
  publish(W, vc);
  for (int pass = 0; pass < 2; ++pass) {
    const double* F = pass == 0 ? W : Vo;
    product(F, true, vc, yc, 0.0, 1.0, false);
    product(F, false, yc, vc, 1.5, -0.5, true);
    publish(pass == 0 ? Vo : W, vc);
  }
  // ---- B = X V in V's place, and the FP64 sweeps
  product(U, false, vc, yc, 0.0, 1.0, false);
  publish(Vo, yc);
  // N eps a pair up to N = 16, as the one-CTA form; wider sectors 16 eps, above the rounding of a rotation and a
  // product of 16 lanes (12 eps at most), so that V is as orthogonal as after one-CTA sweeps that end only when
  // they find nothing to rotate: |V^T V - 1| at N = 100 4e-13 with N eps, 6e-14 so, in the same time
  const double tol = fmin((double)N, fmax(16.0, 0.125 * N)) * 2.220446049250313e-16;
  const int sw = cluster_sweeps<double>(Vo, W, S, N, tol, (float)(tol / N), max_sweeps, buf, sweep_s, rank);
  if (threadIdx.x == 0 && rank == 0 && sw > max_sweeps && status) atomicExch(status, 1);

  // ---- singular values, descending (ties by index; what is not a number last), in every CTA
  for (int j = warp; j < N; j += nw) {
    double a2 = 0.0;
    for (int i = lane; i < N; i += 32) {
      const double x = __ldcg(Vo + i + (int64_t)j * N);
      a2 = fma(x, x, a2);
    }
    a2 = wsum(a2);
    if (lane == 0) sig[j] = sqrt(a2);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < N; j += QT) {
    const double sj = sig[j] >= 0.0 ? sig[j] : -1.0;
    int rk = 0;
    for (int i = 0; i < N; ++i) {
      const double si = sig[i] >= 0.0 ? sig[i] : -1.0;
      rk += (si > sj || (si == sj && i < j)) ? 1 : 0;
    }
    perm[rk] = j;
  }
  __syncthreads();
  // V = P Ux: row piv[i] of V = row i of B / sigma; through shared memory, as B is in V's place
  for (int jl = warp; jl < mine; jl += nw) {
    const int pj = perm[rank + QC * jl];
    const double sj = sig[pj];
    for (int i = lane; i < N; i += 32) {
      const double x = __ldcg(Vo + i + (int64_t)pj * N);
      buf[piv[i] + (size_t)jl * N] = sj > 0.0 ? x / sj : 0.0;
    }
  }
  cluster_sync();
  for (int jl = warp; jl < mine; jl += nw) {
    const int j = rank + QC * jl;
    for (int i = lane; i < N; i += 32) Vo[i + (int64_t)j * N] = buf[i + (size_t)jl * N];
    if (lane == 0) S[j] = sig[perm[j]];
  }
  __syncthreads();
  // U = Q [Vx; 0], own columns; reflector k - 1 is on its way while k is applied
  const bool u_shared = own * M <= room;
  double* uc = u_shared ? buf : U + (int64_t)rank * M;  // column jl at uc + jl * ldu
  const int64_t ldu = u_shared ? M : (int64_t)QC * M;
  for (int jl = warp; jl < mine; jl += nw) {
    const int pj = perm[rank + QC * jl];
    for (int i = lane; i < M; i += 32) uc[i + jl * ldu] = i < N ? __ldcg(W + i + (int64_t)pj * N) : 0.0;
  }
  auto fetch = [&](int k) {
    const double* src = cols + (size_t)(piv[k] / QC) * M;
    for (int i = k + threadIdx.x; i < M; i += QT) vbuf[(size_t)(k & 1) * M + i] = ld_cluster(src + i, piv[k] % QC);
  };
  fetch(N - 1);
  __syncthreads();
  for (int k = N - 1; k >= 0; --k) {
    if (k > 0) fetch(k - 1);
    if (tau_s[k] != 0.0)
      for (int jl = warp; jl < mine; jl += nw) reflect(uc + jl * ldu, vbuf + (size_t)(k & 1) * M, tau_s[k], M, k, lane);
    __syncthreads();
  }
  cluster_arrive();
  if (u_shared)
    for (int jl = warp; jl < mine; jl += nw)
      for (int i = lane; i < M; i += 32) U[i + (int64_t)(rank + QC * jl) * M] = buf[i + (size_t)jl * M];
  cluster_wait();  // no CTA leaves while another may still read its columns
}

// Y = X (M x N) transposed into (N x M), per matrix (used for V^T outputs)
__global__ void transpose_kernel(const imps::DenseMat* __restrict__ mats, const double* __restrict__ X,
                                 double* __restrict__ Y, int use_r) {
  const imps::DenseMat mt = mats[blockIdx.x];
  const int n = mt.N;
  const double* x = X + mt.r_off;
  double* y = Y + mt.r_off;
  for (int64_t t = threadIdx.x; t < (int64_t)n * n; t += blockDim.x) {
    const int i = (int)(t % n), j = (int)(t / n);
    y[j + (int64_t)i * n] = x[t];
  }
  (void)use_r;
}

// X_q[:, j] *= S_q[j]^power for square sector blocks (BlockDiagMat << BlockLam,
// BlockObj.hpp:2316 with lam = S^power)
__global__ void colscale_kernel(const imps::DenseMat* __restrict__ mats, double* __restrict__ X,
                                const double* __restrict__ S, double power) {
  const imps::DenseMat mt = mats[blockIdx.x];
  const int n = mt.N;
  double* x = X + mt.r_off;
  const double* s = S + mt.s_off;
  for (int64_t t = threadIdx.x; t < (int64_t)n * n; t += blockDim.x) {
    const int j = (int)(t / n);
    x[t] *= pow(s[j], power);
  }
}

}  // namespace

namespace imps {

int dc_colscale(const DenseMat* d_mats, int nmat, double* X, const double* S, double power, cudaStream_t st) {
  if (nmat > 0) imps::count_launch();
  if (nmat > 0) colscale_kernel<<<nmat, 256, 0, st>>>(d_mats, X, S, power);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_gather(const GatherEntry* d_ent, int nent, const double* src, double* dense, cudaStream_t st) {
  if (nent > 0) imps::count_launch();
  if (nent > 0) gather_kernel<<<dim3(nent, 4), 256, 0, st>>>(d_ent, src, dense);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_scatter(const GatherEntry* d_ent, int nent, const double* dense, double* dst, cudaStream_t st) {
  if (nent > 0) imps::count_launch();
  if (nent > 0) scatter_kernel<<<dim3(nent, 4), 256, 0, st>>>(d_ent, dense, dst);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_setup() {
  const auto smem = [](const void* kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
  };
  return smem((const void*)qr_cluster_kernel, QR_SMEM) && smem((const void*)svd_cluster_kernel, SVD_SMEM) &&
                 smem((const void*)svd_pjac_kernel<false>, kPjacSmem) &&
                 smem((const void*)svd_pjac_kernel<true>, kPjacSmem)
             ? IMPS_OK
             : IMPS_ERR_CUDA;
}

int dc_qr(const std::vector<DenseMat>& mats, const DenseMat* d_mats, double* A, double* Q, double* R, int transpose_r,
          cudaStream_t st) {
  const int nmat = (int)mats.size();
  if (nmat <= 0) return IMPS_OK;
  imps::count_launch();
  size_t need[2] = {0, 0};  // shared memory without and with Q in it
  for (const DenseMat& m : mats)
    for (int s = 0; s < 2; ++s) need[s] = std::max(need[s], qr_cluster_doubles(m.M, m.N, s) * sizeof(double));
  if (need[0] <= QR_SMEM) {
    const int s = need[1] <= QR_SMEM;
    qr_cluster_kernel<<<nmat * QC, QT, need[s], st>>>(d_mats, A, Q, R, transpose_r, s);
  } else {
    qr_kernel<<<nmat, DT, 0, st>>>(d_mats, A, Q, R, transpose_r);
  }
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_nullspace(const DenseMat* d_mats, int nmat, double* A, double* NS, cudaStream_t st) {
  if (nmat <= 0) return IMPS_OK;
  imps::count_launch();
  nullspace_kernel<<<nmat, DT, 0, st>>>(d_mats, A, NS);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_svd(const std::vector<DenseMat>& mats, const DenseMat* d_mats, double* U, double* S, double* V, double* W,
           int* status, cudaStream_t st) {
  SvdSets sets{};
  sets.nsets = 1;
  sets.s[0] = SvdSet{d_mats, U, S, V, W, (int)mats.size()};
  const std::vector<DenseMat>* m = &mats;
  return dc_svd_sets(sets, &m, status, st);
}

int dc_svd_sets(const SvdSets& sets, const std::vector<DenseMat>* const* mats, int* status, cudaStream_t st) {
  if (sets.nsets < 1 || sets.nsets > kSvdSets) return IMPS_ERR_BAD_ARG;
  int nmat = 0, maxN = 0;
  int64_t maxMN = 0;
  size_t least = 0, good = 0, want = 0;  // shared memory (doubles) of the cluster kernel
  for (int k = 0; k < sets.nsets; ++k) {
    nmat += sets.s[k].n;
    for (const DenseMat& m : *mats[k]) {
      maxN = std::max(maxN, (int)m.N);
      maxMN = std::max(maxMN, (int64_t)m.M * m.N);
      const size_t base = svd_base_doubles(m.M, m.N);
      least = std::max(least, base + svd_work_doubles(m.M, m.N, std::min(m.N, 16), false));
      good = std::max(good, base + svd_work_doubles(m.M, m.N, std::min(m.N, 16), true));
      want = std::max(want, base + svd_work_doubles(m.M, m.N, m.N, true));
    }
  }
  if (nmat <= 0) return IMPS_OK;
  if (maxN <= SVD_MAXN && least * sizeof(double) <= (size_t)SVD_SMEM) {
    imps::count_launch();
    // two CTAs per SM if U still fits, with the products in pieces
    const size_t most = good * sizeof(double) <= SVD_SMEM2 ? SVD_SMEM2 : SVD_SMEM;
    const size_t doubles = std::min(want, most / sizeof(double));
    svd_cluster_kernel<<<nmat * QC, QT, doubles * sizeof(double), st>>>(sets, (int)doubles, 30, status);
    return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
  }
  if (maxN > kJacobiMaxN) {  // global-memory fallback, one launch per set
    for (int k = 0; k < sets.nsets; ++k) {
      if (sets.s[k].n <= 0) continue;
      imps::count_launch();
      svd_kernel<<<sets.s[k].n, DT, 0, st>>>(sets.s[k].mats, sets.s[k].U, sets.s[k].S, sets.s[k].V, sets.s[k].W,
                                             40, status);
    }
    return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
  }
  imps::count_launch();
  const bool mixed = maxN <= kMixedMaxN;
  const int64_t ld = maxN | 1;
  const size_t base = ((size_t)(mixed ? 3 : 2) * ld * maxN + 2 * (size_t)maxN) * 8 + (size_t)2 * maxN * 4 + 16;
  const int a_smem = base + (size_t)maxMN * 8 <= kPjacSmem ? 1 : 0;
  const size_t bytes = base + (a_smem ? (size_t)maxMN * 8 : 0);
  if (bytes > kPjacSmem) return IMPS_ERR_TOO_LARGE;
  if (mixed) svd_pjac_kernel<true><<<nmat, JT, bytes, st>>>(sets, a_smem, 20, status);
  else svd_pjac_kernel<false><<<nmat, JT, bytes, st>>>(sets, a_smem, 30, status);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

int dc_transpose_sq(const DenseMat* d_mats, int nmat, const double* X, double* Y, cudaStream_t st) {
  if (nmat > 0) imps::count_launch();
  if (nmat > 0) transpose_kernel<<<nmat, 256, 0, st>>>(d_mats, X, Y, 1);
  return cudaGetLastError() == cudaSuccess ? IMPS_OK : IMPS_ERR_CUDA;
}

}  // namespace imps
