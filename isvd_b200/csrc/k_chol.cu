// Small dense FP64 kernels of the QR-based stages and of Wen-Yin integration: batched Cholesky
// with an in-place triangular inverse, the Householder sign rule of a QR factor, batched dot
// products and small linear combinations.  One CTA per l x l matrix, the matrix in shared memory.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "runtime.h"

namespace isvdb {
namespace {

constexpr int kCholThreads = 512;
// row stride 4 (mod 16) doubles, so that four threads on each of eight rows hit distinct bank pairs, up to
// the size whose padding still fits the shared memory
__host__ __device__ constexpr int chol_ld(int n) { return n <= 160 ? (n + 15) / 16 * 16 + 4 : n + 1; }

// Sum over the block; every thread returns the same value (same summation order).
__device__ double block_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double s = 0.0;
  for (int i = 0; i < nw; ++i) s += red[i];
  return s;
}

// A = alpha W + (shift_abs + shift_rel trace(alpha W)) I from the upper triangle of W (n x n,
// row-major, batch stride n^2).  Cholesky A = R' R (R upper; right-looking, four rows at a time: the 4 x 4
// pivot block is factored by every thread alike, thread j takes column j of the four rows, one rank-4
// update follows), then X = R^-1 by back substitution, four threads per column and no barrier between
// the steps: column j of X goes below the diagonal, into row j.  Bound by the latency of the pivot
// block's chain of reciprocal roots (n / 4 of them) and of a column's n dot products.  With a barrier per
// column in both phases (one column at a time, the inverse in place) n = 48 took 66 us, n = 96 200 us and
// n = 128 380 us, now 50, 117 and 186.
// A pivot that is not above piv_rel times its starting diagonal value (or is not finite) stops
// the CTA and sets *status = kStatusNotPD.  Output: X with zeros below the diagonal (kCholFactor)
// or out_scale X X' = out_scale A^-1 (kCholInverse).
// null_mask (kCholFactor only; n ints per matrix): a finite pivot at or below the threshold marks
// its column as numerically dependent on the ones before it instead of failing -- the column's row
// of R becomes e_k' (its Schur complement row is zero to rounding) and column k of X is zeroed, so
// Y X has an exact zero column there and the later columns are orthogonalized against the others
// only.  Each newly marked column adds 1 to *null_count.
// perm (n ints per matrix): factor P A P' instead (row / column i of the factored matrix is
// row / column perm[i] of A) and store X at the original positions, out[perm[i], perm[j]] = X[i, j].
// desc (optional): matrix blockIdx.x is desc[blockIdx.x] (its own n, W and out) instead of the
// batch entry of the uniform-size arguments.
__global__ void __launch_bounds__(kCholThreads)
    chol_inv_kernel(int n, const double *__restrict__ W, double alpha, double shift_abs, double shift_rel,
                    double piv_rel, double *__restrict__ out, double out_scale, int mode, int *status,
                    int *__restrict__ null_mask, int *__restrict__ null_count, const int *__restrict__ perm,
                    const CholDesc *__restrict__ desc) {
  extern __shared__ double sm[];
  __shared__ double red[kCholThreads / 32];
  if (desc) n = desc[blockIdx.x].n;
  const int ld = chol_ld(n), tid = threadIdx.x, nt = blockDim.x;
  double *R = sm;                       // n x ld
  double *aux = sm + (size_t)n * ld;    // n: starting diagonal, then the column being inverted
  const double *w = desc ? desc[blockIdx.x].W : W + (size_t)blockIdx.x * n * n;
  const int *pm = perm ? perm + (size_t)blockIdx.x * n : nullptr;
  int *mask = null_mask ? null_mask + (size_t)blockIdx.x * n : nullptr;
  double tr = 0.0;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    const int pi = pm ? pm[i] : i, pj = pm ? pm[j] : j;
    const double v = alpha * ((pi <= pj) ? w[(size_t)pi * n + pj] : w[(size_t)pj * n + pi]);
    R[i * ld + j] = v;
    if (i == j) tr += v;
  }
  const double shift = shift_abs + shift_rel * block_sum(tr, red);
  for (int i = tid; i < n; i += nt) {
    R[i * ld + i] += shift;
    aux[i] = R[i * ld + i];
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
  for (int k = 0; k < n; k += 4) {
    const int kw = min(4, n - k);
    double D[4][4], inv[4];  // pivot block (row c, columns c..3) and the reciprocals of its diagonal
    bool null[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = c; r < 4; ++r) D[c][r] = r < kw ? R[(k + c) * ld + k + r] : (r == c ? 1.0 : 0.0);
    bool fail = false;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const double d = D[c][c];
      null[c] = false;
      // the same decisions in every thread
      if (c < kw && (!(d > piv_rel * aux[k + c]) || !(d > 0.0) || !(d < INFINITY))) {
        if (mask && d == d && d < INFINITY) null[c] = true;  // a dependent column: null, not a failure
        else fail = true;
      }
      // row k of a null pivot is e_k': the Schur update it would make is zero
      inv[c] = null[c] ? 1.0 : rsqrt(d);
      D[c][c] = null[c] ? 1.0 : d * inv[c];
#pragma unroll
      for (int r = c + 1; r < 4; ++r) D[c][r] = null[c] ? 0.0 : D[c][r] * inv[c];
#pragma unroll
      for (int c2 = c + 1; c2 < 4; ++c2)
#pragma unroll
        for (int r = c2; r < 4; ++r) D[c2][r] -= D[c][c2] * D[c][r];
    }
    if (fail) {
      if (tid == 0) atomicExch(status, kStatusNotPD);
      return;
    }
    __syncthreads();  // every thread has read the pivot block
    if (tid == 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (c >= kw) break;
#pragma unroll
        for (int r = c; r < 4; ++r)
          if (r < kw) R[(k + c) * ld + k + r] = D[c][r];
        if (null[c] && !mask[k + c]) {
          mask[k + c] = 1;
          atomicAdd(null_count, 1);
        }
      }
    }
    for (int j = k + 4 + tid; j < n; j += nt) {
      double v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) v[c] = R[(k + c) * ld + j];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        v[c] = null[c] ? 0.0 : v[c] * inv[c];
#pragma unroll
        for (int c2 = c + 1; c2 < 4; ++c2) v[c2] -= D[c][c2] * v[c];
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) R[(k + c) * ld + j] = v[c];
    }
    __syncthreads();
    const double *r0 = R + k * ld, *r1 = r0 + ld, *r2 = r1 + ld, *r3 = r2 + ld;
    for (int i = k + 4 + warp; i < n; i += nwarp) {
      const double a0 = r0[i], a1 = r1[i], a2 = r2[i], a3 = r3[i];
      for (int j = i + lane; j < n; j += 32)
        R[i * ld + j] -= (a0 * r0[j] + a1 * r1[j]) + (a2 * r2[j] + a3 * r3[j]);
    }
    __syncthreads();
  }
  for (int i = tid; i < n; i += nt) aux[i] = 1.0 / R[i * ld + i];
  __syncthreads();
  // X(i, j) = -(sum_{i < k <= j} R(i, k) X(k, j)) / r_ii, X(j, j) = aux[j]; X(i, j) at R[j * ld + i], i < j
  const int quad = tid >> 2, ql = tid & 3, nq = nt >> 2;
  for (int j0 = 0; j0 < n; j0 += nq) {
    const int j = j0 + quad;
    const int jmax = min(n - 1, j0 + (quad | 7));  // the warp's last column
    double *x = R + (size_t)min(j, n - 1) * ld;
    for (int i = jmax - 1; i >= 0; --i) {
      const bool in = j < n && i < j;
      double acc = 0.0, acc2 = 0.0;
      if (in) {
        const double *r = R + i * ld;
        int kk = i + 1 + ql;
        for (; kk + 12 < j; kk += 16) {  // eight loads ahead of the chains
          const double a0 = r[kk], a1 = r[kk + 4], a2 = r[kk + 8], a3 = r[kk + 12];
          const double b0 = x[kk], b1 = x[kk + 4], b2 = x[kk + 8], b3 = x[kk + 12];
          acc += a0 * b0 + a2 * b2;
          acc2 += a1 * b1 + a3 * b3;
        }
        for (; kk < j; kk += 4) acc += r[kk] * x[kk];
        acc += acc2;
        if (ql == 0) acc += r[j] * aux[j];
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      if (in && ql == 0) x[i] = -acc * aux[i];
      __syncwarp();
    }
  }
  __syncthreads();
  auto X = [&](int i, int j) { return i == j ? aux[i] : R[j * ld + i]; };  // i <= j
  double *o = desc ? desc[blockIdx.x].out : out + (size_t)blockIdx.x * n * n;
  if (mode == kCholFactor) {
    for (int e = tid; e < n * n; e += nt) {
      const int i = e / n, j = e - i * n;
      const double v = (j >= i && !(mask && mask[j])) ? out_scale * X(i, j) : 0.0;
      if (pm) o[(size_t)pm[i] * n + pm[j]] = v;
      else o[e] = v;
    }
  } else {
    for (int e = tid; e < n * n; e += nt) {
      const int i = e / n, j = e - i * n;
      double acc = 0.0;
      for (int k = (i > j ? i : j); k < n; ++k) acc += X(i, k) * X(j, k);
      o[e] = out_scale * acc;
    }
  }
}

// out = out_scale A^-1 for A = alpha W + shift I (upper triangle of W, n x n, one CTA per matrix) by
// the sweep operator (Goodnight, "A tutorial on the SWEEP operator", Amer. Statist. 33 (1979)):
// sweeping pivot k maps a_kk -> -1/a_kk, a_ik -> a_ik/a_kk, a_ij -> a_ij - a_ik a_kj / a_kk; after
// all pivots the matrix is -A^-1.  For a symmetric positive definite A the pivots are the Cholesky
// pivots (Schur-complement diagonals), so the elimination needs no pivoting; one pivot that is not
// above piv_rel times its starting diagonal value sets *status = kStatusNotPD.  Symmetry halves the
// per-pivot reads: row k equals column k.
constexpr int kSwThreads = 1024;

__global__ void __launch_bounds__(kSwThreads)
    spd_inverse_kernel(int n, const double *__restrict__ W, double alpha, double shift, double piv_rel,
                       double *__restrict__ out, double out_scale, int *status) {
  extern __shared__ double sm[];
  const int ld = n + 1, tid = threadIdx.x;
  double *A = sm, *col = sm + (size_t)n * ld, *diag0 = col + n;
  const double *w = W + (size_t)blockIdx.x * n * n;
  const int tx = tid & 31, ty = tid >> 5;  // element (ty + 32 a, tx + 32 b)
  for (int i = ty; i < n; i += 32)
    for (int j = tx; j < n; j += 32) {
      const double v = alpha * ((i <= j) ? w[(size_t)i * n + j] : w[(size_t)j * n + i]) + (i == j ? shift : 0.0);
      A[i * ld + j] = v;
      if (i == j) diag0[i] = v;
    }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    for (int i = tid; i < n; i += kSwThreads) col[i] = A[i * ld + k];
    __syncthreads();
    const double d = col[k];
    if (!(d > piv_rel * diag0[k]) || !(d > 0.0) || !(d < INFINITY)) {  // same decision in every thread
      if (tid == 0) atomicExch(status, kStatusNotPD);
      return;
    }
    const double inv = 1.0 / d;
    for (int i = ty; i < n; i += 32) {
      const double ci = col[i];
      for (int j = tx; j < n; j += 32) {
        double v;
        if (i == k) v = (j == k) ? -inv : col[j] * inv;
        else if (j == k) v = ci * inv;
        else v = A[i * ld + j] - ci * col[j] * inv;
        A[i * ld + j] = v;
      }
    }
    __syncthreads();
  }
  double *o = out + (size_t)blockIdx.x * n * n;
  for (int i = ty; i < n; i += 32)
    for (int j = tx; j < n; j += 32) o[(size_t)i * n + j] = -out_scale * A[i * ld + j];
}

// Householder sign rule.  P = Qtop X is the top n x n block of the next Q factor (positive-
// diagonal convention).  A Householder QR (LAPACK geqrf / gelqf) of the same matrix returns
// Q diag(s) with s_j = -sign(pivot_j) of the LU factorization of P - diag(s) carried out with
// exactly that choice of s (Ballard, Demmel, Grigori, Jacquelin, Knight, Nguyen, "Reconstructing
// Householder vectors from tall-skinny QR", J. Parallel Distrib. Comput. 85 (2015)).  X's
// columns are multiplied by s, so that Q X is the Householder factor.
template <class T>
__global__ void __launch_bounds__(kCholThreads)
    hh_sign_kernel(int n, const T *__restrict__ Q, long long q_ld, long long q_bs, double *__restrict__ X) {
  extern __shared__ double sm[];
  const int ld = n + 1, tid = threadIdx.x, nt = blockDim.x;
  double *P = sm, *sg = sm + (size_t)n * ld;
  const T *q = Q + blockIdx.x * q_bs;
  double *x = X + (size_t)blockIdx.x * n * n;
  for (int e = tid; e < n * n; e += nt) {
    const int i = e / n, j = e - i * n;
    double acc = 0.0;
    for (int k = 0; k <= j; ++k) acc += (double)q[i * q_ld + k] * x[(size_t)k * n + j];
    P[i * ld + j] = acc;
  }
  __syncthreads();
  for (int j = 0; j < n; ++j) {
    const double piv = P[j * ld + j];
    const double s = (piv >= 0.0) ? -1.0 : 1.0;
    const double u = piv - s;  // |u| >= 1
    __syncthreads();
    if (tid == 0) sg[j] = s;
    for (int i = j + 1 + tid; i < n; i += nt) P[i * ld + j] /= u;
    __syncthreads();
    const int mm = n - j - 1;
    for (int e = tid; e < mm * mm; e += nt) {
      const int i = j + 1 + e / mm, c = j + 1 + e % mm;
      P[i * ld + c] -= P[i * ld + j] * P[j * ld + c];
    }
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += nt) x[e] *= sg[e % n];
}

constexpr int kDotThreads = 256;
constexpr int kDotBlocks = 64;  // CTAs per job; partial sums combined in a fixed order

// Partial sums: CTA (x, job) sums the entries x, x + kDotBlocks, ... (in units of its thread count).
__global__ void __launch_bounds__(kDotThreads) dots_kernel(DotJobs jobs, double *__restrict__ partial) {
  __shared__ double red[kDotThreads / 32];
  const DotJob jb = jobs.job[blockIdx.y];
  const long long stride = (long long)gridDim.x * blockDim.x;
  double v = 0.0;
  if (jb.trace) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < jb.n; i += stride) v += jb.a[i * jb.n + i];
  } else {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < jb.n; i += stride) {
      const double x = jb.a[i] - (jb.b ? jb.b[i] : 0.0);
      const double y = jb.c[i] - (jb.d ? jb.d[i] : 0.0);
      v += x * y;
    }
  }
  v = block_sum(v, red);
  if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = v;
}

__global__ void dots_final_kernel(const double *__restrict__ partial, int nblocks, int count, double *__restrict__ out) {
  const int j = threadIdx.x;
  if (j < count) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += partial[j * nblocks + b];
    out[j] = s;
  }
}

// (out may alias x or y: each entry is read and written by the same thread)
__global__ void lincomb_kernel(double *out, const double *x, double a, const double *y, double b, double c,
                               long long rows, long long cols) {
  const long long total = rows * cols;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long i = e / cols, j = e - i * cols;
    double v = (i == j) ? c : 0.0;
    if (x) v += a * x[e];
    if (y) v += b * y[e];
    out[e] = v;
  }
}

__global__ void copy_diag_blocks_kernel(const double *__restrict__ G, int Nl, int l, int N, double *__restrict__ out) {
  const long long total = (long long)N * l * l;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long b = e / ((long long)l * l), r = e - b * l * l;
    const long long i = r / l, j = r - i * l;
    out[e] = G[(b * l + i) * Nl + b * l + j];
  }
}

// d_i = num / (half * max(lambda_i, 0) + add)
__global__ void recip_affine_kernel(const double *__restrict__ lam, int n, double num, double half, double add,
                                    double *__restrict__ d) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = num / (half * fmax(lam[i], 0.0) + add);
}

size_t chol_smem(int n) { return ((size_t)n * chol_ld(n) + n) * sizeof(double); }

}  // namespace

void chol_inv_batched(int n, int batch, const double *W, double alpha, double shift_abs, double shift_rel,
                      double piv_rel, double *out, double out_scale, int mode, int *status, cudaStream_t st,
                      int *null_mask, int *null_count, const int *perm) {
  if (n <= 0 || batch <= 0) return;
  if ((null_mask || perm) && mode != kCholFactor) fail(kErrArgument, "Cholesky: null columns / permutation need kCholFactor");
  if (null_mask && !null_count) fail(kErrArgument, "Cholesky: a null-column mask needs its counter");
  if (mode == kCholInverse && shift_rel == 0.0) {  // the full inverse: sweep operator, fewer dependent steps
    const size_t smem = ((size_t)n * (n + 1) + 2 * n) * sizeof(double);
    if (smem > Runtime::get().smem_optin) fail(kErrUnsupported, "SPD inverse: l = %d exceeds on-chip capacity", n);
    CK(cudaFuncSetAttribute(spd_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    spd_inverse_kernel<<<batch, kSwThreads, smem, st>>>(n, W, alpha, shift_abs, piv_rel, out, out_scale, status);
    KLAUNCHED();
    return;
  }
  const size_t smem = chol_smem(n);
  if (smem > Runtime::get().smem_optin) fail(kErrUnsupported, "Cholesky: l = %d exceeds on-chip capacity", n);
  CK(cudaFuncSetAttribute(chol_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  chol_inv_kernel<<<batch, kCholThreads, smem, st>>>(n, W, alpha, shift_abs, shift_rel, piv_rel, out, out_scale,
                                                     mode, status, null_mask, null_count, perm, nullptr);
  KLAUNCHED();
}

void chol_inv_grouped(const CholDesc *desc, int count, int max_n, int *status, cudaStream_t st) {
  if (count <= 0 || max_n <= 0) return;
  const size_t smem = chol_smem(max_n);
  if (smem > Runtime::get().smem_optin) fail(kErrUnsupported, "Cholesky: l = %d exceeds on-chip capacity", max_n);
  CK(cudaFuncSetAttribute(chol_inv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  chol_inv_kernel<<<count, kCholThreads, smem, st>>>(0, nullptr, 1.0, 0.0, 0.0, 0.0, nullptr, 1.0, kCholFactor, status,
                                                     nullptr, nullptr, nullptr, desc);
  KLAUNCHED();
}

template <class T>
void hh_sign_batched(int n, int batch, const T *Q, long long q_ld, long long q_bs, double *X, cudaStream_t st) {
  if (n <= 0 || batch <= 0) return;
  const size_t smem = chol_smem(n);
  if (smem > Runtime::get().smem_optin) fail(kErrUnsupported, "QR sign rule: l = %d exceeds on-chip capacity", n);
  CK(cudaFuncSetAttribute(hh_sign_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  hh_sign_kernel<T><<<batch, kCholThreads, smem, st>>>(n, Q, q_ld, q_bs, X);
  KLAUNCHED();
}

void dots(const DotJobs &jobs, double *out, cudaStream_t st) {
  if (jobs.count <= 0) return;
  if (jobs.count > kMaxDotJobs) fail(kErrArgument, "dots: %d jobs > %d", jobs.count, kMaxDotJobs);
  DBuf<double> partial((size_t)kDotBlocks * jobs.count);
  dots_kernel<<<dim3(kDotBlocks, jobs.count), kDotThreads, 0, st>>>(jobs, partial.p);
  KLAUNCHED();
  dots_final_kernel<<<1, 32, 0, st>>>(partial.p, kDotBlocks, jobs.count, out);
  KLAUNCHED();
}

void lincomb(double *out, const double *x, double a, const double *y, double b, double c, long long rows,
             long long cols, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return;
  const long long total = rows * cols;
  const int grid = (int)std::min<long long>((total + 255) / 256, 8LL * Runtime::get().num_sms);
  lincomb_kernel<<<grid, 256, 0, st>>>(out, x, a, y, b, c, rows, cols);
  KLAUNCHED();
}

void copy_diag_blocks(const double *G, int Nl, int l, int N, double *out, cudaStream_t st) {
  const long long total = (long long)N * l * l;
  if (total <= 0) return;
  const int grid = (int)std::min<long long>((total + 255) / 256, 8LL * Runtime::get().num_sms);
  copy_diag_blocks_kernel<<<grid, 256, 0, st>>>(G, Nl, l, N, out);
  KLAUNCHED();
}

void recip_affine(const double *lam, int n, double num, double half, double add, double *d, cudaStream_t st) {
  if (n <= 0) return;
  recip_affine_kernel<<<1, 256, 0, st>>>(lam, n, num, half, add, d);
  KLAUNCHED();
}

template void hh_sign_batched<double>(int, int, const double *, long long, long long, double *, cudaStream_t);
template void hh_sign_batched<float>(int, int, const float *, long long, long long, double *, cudaStream_t);

}  // namespace isvdb
