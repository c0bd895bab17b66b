// Symmetric eigendecomposition of l x l FP64 matrices, l <= 128: a single-precision one-sided Jacobi
// for a first set of eigenvectors, then FP64 refinement by matrix products.
//
//   W + c I = L L'  (Cholesky, FP64; c = 0 for a Gram matrix, c > ||W|| for an indefinite one),
//   L J = U Sigma   (one-sided Jacobi on the columns of L in FP32; J orthogonal, never formed): the
//                   normalized columns U are the eigenvectors of L L', to single precision,
//   X <- X + X E    (FP64; Ogita & Aishima, "Iterative refinement for symmetric eigenvalue
//                   decomposition", Japan J. Indust. Appl. Math. 35 (2018)): with R = I - X'X,
//                   S = X'WX and lambda_i = s_ii / (1 - r_ii),
//                   e_ij = (s_ij + lambda_j r_ij) / (lambda_j - lambda_i), e_ii = r_ii / 2.
// The error is squared by every refinement, which also restores orthonormality: two or three take it from single
// precision to FP64 rounding.  A matrix that they do not settle (clusters that FP32
// cannot separate, a Cholesky breakdown, non-finite entries) sets its `need` word and is solved by
// the FP64 two-sided Jacobi of k_small.cu instead; so is a graded one, whose row norms differ by more than
// kGraded: the refinement's eigenvalues are good to rounding of ||W||, Jacobi's to rounding of their own rows
// (singular values from Gram matrices D H D, l = 64, relative to themselves: D down to 1e-3 8e-15 by either,
// 1e-4 1e-14 by Jacobi and 7e-14 refined, 1e-6 9e-15 and 1e-10).
//
// Why: the two-sided Jacobi in FP64 is bound by the latency of its n - 1 rounds a sweep, nine to ten
// sweeps (about 2.5 us a round: FP64 root and division chains, 2 n^2 doubles through shared memory,
// the barriers).  The one-sided rounds in FP32 need no eigenvector matrix; the refinement is four
// products of a cluster (rows.cuh), 10 to 20 us a step, two or three steps.  Measured for the Gram of a
// solve, two-sided -> this: l = 11 84 -> 37 us, l = 32 273 -> 73, l = 65 987 -> 224, l = 96 2098 -> 364,
// l = 128 3492 (on a 16-CTA cluster) -> 608, plus 2 to 9 us for the row norms of the test for grading.  What is left is the FP32 Jacobi on one SM: six to eight
// sweeps of n rounds of n / 2 rotations, 0.2 us a round at l = 32 (latency of the reduction and the
// rotation), 0.5 us at l = 128 (FP32 pipe and shuffles of the SM).
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "kernels.h"
#include "rows.cuh"
#include "runtime.h"

namespace isvdb {
namespace {

namespace cg = cooperative_groups;

constexpr double kEps = 2.220446049250313e-16;
constexpr int kMaxN = kKrMaxL;
constexpr int kOsjSweeps = 16;
constexpr int kRefine = 8;
constexpr int kEigBlocks = 4;  // X, T = X W, R (then E'), S
// (row norms of D H D differ by about the range of D; those of a solve's Gram matrices, whose bases mix the
// singular directions, by factors of 2 to 6)
constexpr double kGraded = 500.0;

// work of one matrix (doubles): X0 | X1 | W (symmetrised) | S | lambda | slots[64], scalars
struct EigWork {
  double *X0, *X1, *W, *S, *lam, *slots, *fro;
  int *need;
  __device__ EigWork(double *p, int n) {
    const size_t nn = (size_t)n * n;
    X0 = p; X1 = p + nn; W = X1 + nn; S = W + nn; lam = S + nn; slots = lam + n; fro = slots + 48;
    need = (int *)(p + eig_need_at(n));
  }
};

__device__ __forceinline__ size_t pl(int i, int j) { return (size_t)i * (i + 1) / 2 + j; }  // lower, packed by rows

// Columns in blocks of four, an even number of blocks (the columns beyond n are zero); column stride nx.
__host__ __device__ constexpr int osj_blocks(int n) { return ((n + 3) / 4 + 1) / 2 * 2; }
__host__ __device__ constexpr int osj_nx(int n) { return (n + 31) / 32 * 32; }
size_t osj_smem(int n) {
  const size_t npk = ((size_t)n * (n + 1) / 2 + 1) & ~(size_t)1;
  return npk * 8 + (size_t)osj_blocks(n) * 4 * (osj_nx(n) + 1) * 4;
}
int osj_threads(int n) { return std::max(128, (osj_blocks(n) / 2 * 16 + 31) / 32 * 32); }

typedef unsigned long long f2;  // two floats, for the packed FP32 instructions
__device__ __forceinline__ f2 f2_dup(float x) {
  f2 r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float f2_sum(f2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
  return x + y;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

__device__ __forceinline__ float rsqrt_a(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_a(float x, float y) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}

// Sums over 16 lanes of four values per lane: lane l gets the sum of value l & 3.
__device__ __forceinline__ float osj_sum4(const float (&v)[4]) {
  const unsigned full = 0xffffffffu;
  const bool b0 = threadIdx.x & 1, b1 = threadIdx.x & 2;
  const float s0 = (b0 ? v[1] : v[0]) + __shfl_xor_sync(full, b0 ? v[0] : v[1], 1);
  const float s1 = (b0 ? v[3] : v[2]) + __shfl_xor_sync(full, b0 ? v[2] : v[3], 1);
  float s = (b1 ? s1 : s0) + __shfl_xor_sync(full, b1 ? s0 : s1, 2);
  s += __shfl_xor_sync(full, s, 4);
  return s + __shfl_xor_sync(full, s, 8);
}

template <int EPL>
__device__ __forceinline__ float osj_dot(const f2 (&a)[EPL], const f2 (&b)[EPL]) {
  f2 acc = f2_mul(a[0], b[0]);
#pragma unroll
  for (int u = 1; u < EPL; ++u) acc = f2_fma(a[u], b[u], acc);
  return f2_sum(acc);
}

// Four disjoint rotations of the eight columns that 16 lanes hold (EPL float pairs each): pair i
// rotates columns pq(i).x and pq(i).y.  Lane l computes the rotation of pair l & 3 from its squared
// column norms al, be (updated) and hands it to the others.
template <int EPL, class PQ>
__device__ __forceinline__ void osj_rotate(f2 (&x)[8][EPL], float &al, float &be, int &big, PQ pq) {
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = osj_dot<EPL>(x[pq(i).x], x[pq(i).y]);
  const float ga = osj_sum4(v);
  const float g2 = ga * ga, ab = al * be;
  // t = sign(d) 2 ga / (|d| + sqrt(d^2 + 4 ga^2)), d = be - al (the smaller rotation)
  const float d = be - al, e = 2.f * ga, h2 = fmaf(d, d, e * e);
  float t = div_a(d >= 0.f ? e : -e, fmaf(h2, rsqrt_a(h2), fabsf(d)));
  t = (g2 > 1e-14f * ab && h2 > 1e-37f) ? t : 0.f;
  if (g2 > 1e-6f * ab) big = 1;
  const float c = rsqrt_a(fmaf(t, t, 1.f)), s = t * c;
  al = fmaxf(fmaf(-t, ga, al), 0.f);
  be = fmaf(t, ga, be);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int p = pq(i).x, q = pq(i).y;
    const float ci = __shfl_sync(0xffffffffu, c, i, 4), si = __shfl_sync(0xffffffffu, s, i, 4);
    const f2 c2 = f2_dup(ci), s2 = f2_dup(si), m2 = f2_dup(-si);
#pragma unroll
    for (int u = 0; u < EPL; ++u) {
      const f2 y = f2_fma(c2, x[p][u], f2_mul(m2, x[q][u]));
      x[q][u] = f2_fma(c2, x[q][u], f2_mul(s2, x[p][u]));
      x[p][u] = y;
    }
  }
}

// One CTA per matrix: symmetrised copy of W, Cholesky factor, FP32 one-sided Jacobi.  Sixteen lanes
// take two blocks of four columns into registers and make the sixteen rotations between them before
// they go back to shared memory (a round of single pairs is bound by shared-memory bandwidth: 2 n^2
// floats each way; blocks of four move a quarter of that), in FP32 pairs.
template <int EPL>
__global__ void __launch_bounds__(256) osj_kernel(int n_uniform, const double *__restrict__ Ag, double *workg,
                                                  size_t work_stride, int psd, bool loose, const EigDesc *desc) {
  extern __shared__ double sm[];
  const int b = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarp = nt >> 5;
  const int n = desc ? desc[b].n : n_uniform;
  const double *A0 = desc ? desc[b].A : Ag + (size_t)b * n * n;
  EigWork w(desc ? desc[b].work : workg + (size_t)b * work_stride, n);
  const int nb = osj_blocks(n), nx = osj_nx(n);
  const size_t npk = ((size_t)n * (n + 1) / 2 + 1) & ~(size_t)1;
  double *L = sm;
  float *X = (float *)(sm + npk), *nrms = X + (size_t)nb * 4 * nx;
  double *cols = (double *)X;  // 4 n doubles, before X is filled
  __shared__ double red[16], scal[2];
  __shared__ int ok;

  // symmetrised W, ||W||_F, largest diagonal entry
  double fr = 0.0, dm = 0.0;
  for (int i = warp; i < n; i += nwarp)
    for (int j = lane; j <= i; j += 32) {
      const double v = 0.5 * (A0[(size_t)i * n + j] + A0[(size_t)j * n + i]);
      w.W[(size_t)i * n + j] = v;
      w.W[(size_t)j * n + i] = v;
      L[pl(i, j)] = v;
      fr += (i == j ? 1.0 : 2.0) * v * v;
      if (i == j) dm = fmax(dm, fabs(v));
    }
  for (int o = 16; o > 0; o >>= 1) {
    fr += __shfl_xor_sync(0xffffffffu, fr, o);
    dm = fmax(dm, __shfl_xor_sync(0xffffffffu, dm, o));
  }
  if (lane == 0) red[warp] = fr;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int i = 0; i < nwarp; ++i) s += red[i];
    scal[0] = sqrt(s);
    *w.fro = scal[0];
    *w.need = 0;
  }
  __syncthreads();
  if (lane == 0) red[warp] = dm;
  __syncthreads();
  dm = 0.0;
  for (int i = 0; i < nwarp; ++i) dm = fmax(dm, red[i]);
  const double fro = scal[0];

  if (!loose) {  // graded: Jacobi's
    double lo = INFINITY, hi = 0.0;
    for (int i = warp; i < n; i += nwarp) {
      double s = 0.0;
      for (int j = lane; j < n; j += 32) {
        const double v = L[j <= i ? pl(i, j) : pl(j, i)];
        s += v * v;
      }
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      lo = fmin(lo, s);
      hi = fmax(hi, s);
    }
    __syncthreads();  // red has been read
    if (lane == 0) {
      red[warp] = lo;
      red[8 + warp] = hi;
    }
    __syncthreads();
    for (int i = 0; i < nwarp; ++i) {
      lo = fmin(lo, red[i]);
      hi = fmax(hi, red[8 + i]);
    }
    __syncthreads();
    if (hi > kGraded * kGraded * lo) {
      if (tid == 0) *w.need = 1;
      return;
    }
  }

  // Cholesky (right-looking, one column per step); a Gram matrix that is singular to rounding is
  // factored once more with a shift that leaves its eigenvectors alone
  bool done = false;
  for (int attempt = 0; attempt < 2 && !done; ++attempt) {
    const double c = (psd ? 0.0 : 1.0625 * fro) + (attempt ? 1e-8 * fro : 0.0);
    if (attempt) {
      for (int i = warp; i < n; i += nwarp)
        for (int j = lane; j <= i; j += 32) L[pl(i, j)] = w.W[(size_t)i * n + j];
      __syncthreads();
    }
    for (int i = tid; i < n; i += nt) L[pl(i, i)] += c;
    if (tid == 0) ok = 1;
    __syncthreads();
    const double floor_ = 4.0 * n * kEps * (dm + c);
    bool good = true;
    // panels of four columns: the 4 x 4 pivot block is factored by every thread alike, thread i takes
    // row i of the panel, and one rank-4 update follows
    for (int k = 0; k < n && good; k += 4) {
      const int kw = min(4, n - k);
      double D[4][4], inv[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = c; r < 4; ++r) D[r][c] = r < kw ? L[pl(k + r, k + c)] : (r == c ? 1.0 : 0.0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double d = D[c][c];
        if (c < kw && (!(d > floor_) || !(d < 1e300))) good = false;  // the same in every thread
        inv[c] = rsqrt(d);
        D[c][c] = d * inv[c];
#pragma unroll
        for (int r = c + 1; r < 4; ++r) D[r][c] *= inv[c];
#pragma unroll
        for (int c2 = c + 1; c2 < 4; ++c2)
#pragma unroll
          for (int r = c2; r < 4; ++r) D[r][c2] -= D[r][c] * D[c2][c];
      }
      __syncthreads();  // every thread has read the pivot block
      for (int i = k + tid; i < n; i += nt) {
        double v[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = (c < kw && k + c <= i) ? L[pl(i, k + c)] : 0.0;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          v[c] *= inv[c];
#pragma unroll
          for (int c2 = c + 1; c2 < 4; ++c2) v[c2] -= v[c] * D[c2][c];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const bool in = c < kw && k + c <= i;
          if (in) L[pl(i, k + c)] = v[c];
          cols[c * n + i] = in ? v[c] : 0.0;
        }
      }
      __syncthreads();
      for (int i = k + 4 + warp; i < n; i += nwarp) {
        const double a0 = cols[i], a1 = cols[n + i], a2 = cols[2 * n + i], a3 = cols[3 * n + i];
        for (int j = k + 4 + lane; j <= i; j += 32)
          L[pl(i, j)] -= (a0 * cols[j] + a1 * cols[n + j]) + (a2 * cols[2 * n + j] + a3 * cols[3 * n + j]);
      }
      __syncthreads();
    }
    done = good;
    __syncthreads();
  }
  if (!done) {
    if (tid == 0) *w.need = 1;
    return;
  }
  const double scale = rsqrt(fmax(fro, 1e-300) + (psd ? 0.0 : 1.0625 * fro));
  for (int j = warp; j < 4 * nb; j += nwarp)
    for (int i = lane; i < nx; i += 32)
      X[(size_t)j * nx + i] = (i < n && j < n && i >= j) ? (float)(L[pl(i, j)] * scale) : 0.f;
  __syncthreads();

  // round-robin tournament of the blocks: block 0 stays, the others move one place per round
  const int grp = tid >> 4, sub = tid & 15;
  const bool live = grp < nb / 2;
  int p = live ? grp : 0, q = live ? nb - 1 - grp : 0;
  for (int sweep = 0; sweep < kOsjSweeps; ++sweep) {
    int big = 0;
    for (int r = 0; r < nb - 1; ++r) {
      f2 x[8][EPL];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const f2 *src = (const f2 *)(X + (size_t)(4 * (c < 4 ? p : q) + (c & 3)) * nx) + sub;
#pragma unroll
        for (int u = 0; u < EPL; ++u) x[c][u] = 32 * u < nx && live ? src[16 * u] : 0ull;
      }
      float al, be;  // squared norms: columns sub & 3 of the first block, and of the second
      auto norms = [&](int c0) {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = osj_dot<EPL>(x[c0 + i], x[c0 + i]);
        return osj_sum4(v);
      };
      if (r == 0) {  // each block is in one group: the rotations within the blocks, and new norms
        auto within = [&](auto pq) {
          float va[4], vb[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            va[i] = osj_dot<EPL>(x[pq(i).x], x[pq(i).x]);
            vb[i] = osj_dot<EPL>(x[pq(i).y], x[pq(i).y]);
          }
          float na = osj_sum4(va), nb2 = osj_sum4(vb);
          osj_rotate<EPL>(x, na, nb2, big, pq);
        };
        within([](int i) { return make_int2(2 * i, 2 * i + 1); });
        within([](int i) { return make_int2(4 * (i >> 1) + (i & 1), 4 * (i >> 1) + 2 + (i & 1)); });
        within([](int i) { return make_int2(4 * (i >> 1) + (i & 1), 4 * (i >> 1) + 3 - (i & 1)); });
        al = norms(0);
        be = norms(4);
      } else {
        al = nrms[4 * p + (sub & 3)];
        be = nrms[4 * q + (sub & 3)];
      }
      // lane l: column l & 3 of the first block against column (l + s) & 3 of the second
      const int nxt = (sub + 1) & 3;
      osj_rotate<EPL>(x, al, be, big, [](int i) { return make_int2(i, 4 + i); });
      be = __shfl_sync(0xffffffffu, be, nxt, 4);
      osj_rotate<EPL>(x, al, be, big, [](int i) { return make_int2(i, 4 + ((i + 1) & 3)); });
      be = __shfl_sync(0xffffffffu, be, nxt, 4);
      osj_rotate<EPL>(x, al, be, big, [](int i) { return make_int2(i, 4 + ((i + 2) & 3)); });
      be = __shfl_sync(0xffffffffu, be, nxt, 4);
      osj_rotate<EPL>(x, al, be, big, [](int i) { return make_int2(i, 4 + ((i + 3) & 3)); });
      if (live) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          f2 *dst = (f2 *)(X + (size_t)(4 * (c < 4 ? p : q) + (c & 3)) * nx) + sub;
#pragma unroll
          for (int u = 0; u < EPL; ++u)
            if (32 * u < nx) dst[16 * u] = x[c][u];
        }
        if (sub < 4) {
          nrms[4 * p + sub] = al;
          nrms[4 * q + ((sub + 3) & 3)] = be;
        }
        if (p > 0) p = (p == nb - 1) ? 1 : p + 1;
        q = (q == nb - 1) ? 1 : q + 1;
      }
      __syncthreads();
    }
    // cosines of at most 1e-3 throughout a sweep: the rotations left them at about their squares
    if (!__syncthreads_or(big)) break;
  }
  // rows of X0: the normalized columns
  for (int j = warp; j < n; j += nwarp) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) {
      const double v = X[(size_t)j * nx + i];
      s += v * v;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const double inv = rsqrt(s);  // a zero column: infinite, the refinement gives up
    for (int i = lane; i < n; i += 32) w.X0[(size_t)j * n + i] = X[(size_t)j * nx + i] * inv;
  }
}

// The larger of two magnitudes; a NaN, once met, stays.
__device__ __forceinline__ double larger(double a, double b) { return isnan(a) ? a : (isnan(b) || b > a) ? b : a; }

// One cluster per matrix: the FP64 refinement on the rows of X' (row i = eigenvector i), then the
// eigenpairs in order (as sym_eig_batched).  loose: eigenvectors that are not separated stay mixed, as
// orthonormal as the others.
__global__ void __launch_bounds__(kKrThreads, 1)
    eig_refine_kernel(int n_uniform, double *workg, size_t work_stride, double *__restrict__ Vg,
                      double *__restrict__ wg, int order, bool absval, bool loose, const EigDesc *desc) {
  extern __shared__ double sm[];
  __shared__ double red[kKrWarps], lam[kMaxN];
  __shared__ int sbad;
  cg::cluster_group cluster = cg::this_cluster();
  const int b = blockIdx.x / (int)cluster.num_blocks(), tid = threadIdx.x;
  const int n = desc ? desc[b].n : n_uniform;
  EigWork g(desc ? desc[b].work : workg + (size_t)b * work_stride, n);
  double *V = desc ? desc[b].V : Vg + (size_t)b * n * n;
  double *wo = desc ? desc[b].w : wg + (size_t)b * n;
  if (__ldcg(g.need)) return;  // the same word in every CTA of the cluster
  Kr k;
  kr_init(k, n, (int)cluster.num_blocks(), (int)cluster.block_rank(), sm);
  const int ld = k.ld, r0 = k.r0, rows = 8 * k.mt;
  double *X = k.block(0), *T = k.block(1), *R = k.block(2), *S = k.block(3);
  auto each = [&](auto f) {
    for (int e = tid; e < rows * k.lr; e += kKrThreads) {
      const int i = e / k.lr, j = e - i * k.lr;
      f(i, j, r0 + i < n && j < n);
    }
  };
  const double fro = __ldcg(g.fro), thr = 8.0 * kEps * fro;
  for (int e = tid; e < k.lr * ld; e += kKrThreads) k.full[e] = 0.0;
  each([&](int i, int j, bool in) { X[(size_t)i * ld + j] = in ? __ldcg(g.X0 + (size_t)(r0 + i) * n + j) : 0.0; });
  bool settled = false;
  for (int it = 0; it < kRefine && !settled; ++it) {
    const double *Xg = (it & 1) ? g.X1 : g.X0;
    double *Xn = (it & 1) ? g.X0 : g.X1;
    __syncthreads();
    kr_load(k, g.W);
    __syncthreads();
    kr_mm(k, X, [&](int i, int j, double v) { T[(size_t)i * ld + j] = v; });
    __syncthreads();
    kr_load(k, Xg);
    __syncthreads();
    kr_mm<true>(k, X, [&](int i, int j, double v) {
      R[(size_t)i * ld + j] = ((r0 + i == j && j < n) ? 1.0 : 0.0) - v;
    });
    kr_mm<true>(k, T, [&](int i, int j, double v) {
      S[(size_t)i * ld + j] = v;
      if (r0 + i < n && j < n) g.S[(size_t)(r0 + i) * n + j] = v;
    });
    __syncthreads();
    for (int i = tid; i < rows; i += kKrThreads)
      if (r0 + i < n) g.lam[r0 + i] = S[(size_t)i * ld + r0 + i] / (1.0 - R[(size_t)i * ld + r0 + i]);
    if (tid == 0) sbad = 0;
    cluster.sync();
    for (int i = tid; i < n; i += kKrThreads) lam[i] = __ldcg(g.lam + i);
    __syncthreads();
    // E' over R: row i of E' is column i of E.  r is symmetric as computed; s is averaged with its
    // transpose, so that e_ij + e_ji = r_ij and the step keeps X orthonormal to rounding (the two
    // differ by rounding of s, which small gaps would amplify)
    double mx = 0.0;
    int bad = 0;
    each([&](int i, int j, bool in) {
      if (!in) return;
      const size_t e = (size_t)i * ld + j;
      const double r = R[e];
      double v = 0.5 * r, m = fabs(v);
      if (r0 + i != j) {
        const double sij = 0.5 * (S[e] + __ldcg(g.S + (size_t)j * n + r0 + i));
        const double num = sij + lam[r0 + i] * r, gap = lam[r0 + i] - lam[j];
        const double q = num / gap;
        if (fabs(num) <= thr) {  // coupled at rounding level: only a step whose square is below it too
          if (fabs(q) <= 1e-8) v = q;
        } else if (fabs(q) <= 0.25) {
          v = q;
          m = fabs(q);
        } else {
          bad = !loose;  // not separated, and coupled above rounding (or not a number)
        }
      }
      R[e] = v;
      mx = larger(mx, m);
    });
    if (bad) sbad = 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mx = larger(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((tid & 31) == 0) red[tid >> 5] = mx;
    __syncthreads();
    kr_mm(k, R, [&](int i, int j, double v) { X[(size_t)i * ld + j] += v; });  // X' + E' X'
    __syncthreads();
    each([&](int i, int j, bool in) {
      if (in) Xn[(size_t)(r0 + i) * n + j] = X[(size_t)i * ld + j];
    });
    if (tid == 0) {
      double m = 0.0;
      for (int i = 0; i < kKrWarps; ++i) m = larger(m, red[i]);
      g.slots[k.rank] = m;
      g.slots[16 + k.rank] = sbad;
    }
    cluster.sync();
    double m = 0.0, nbad = 0.0;
    for (int r = 0; r < k.cs; ++r) {
      m = larger(m, __ldcg(g.slots + r));
      nbad += __ldcg(g.slots + 16 + r);
    }
    settled = nbad == 0.0 && m <= 3e-9;  // what is left is of the order of m^2
    if (!(m < 1e3)) break;               // lost (or not a number)
  }
  if (!settled) {
    if (k.rank == 0 && tid == 0) *g.need = 1;
    return;
  }
  for (int i = tid >> 5; i < rows; i += kKrWarps) {
    const int x = r0 + i;
    if (x >= n) continue;
    const double kx = lam[x];
    int rank = 0;
    for (int y = tid & 31; y < n; y += 32) {
      const double ky = lam[y];
      rank += (order > 0) ? (fabs(ky) > fabs(kx) || (fabs(ky) == fabs(kx) && y < x)) : (ky < kx || (ky == kx && y < x));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
    if ((tid & 31) == 0) wo[rank] = absval ? fabs(kx) : kx;
    for (int j = tid & 31; j < n; j += 32) V[(size_t)j * n + rank] = X[(size_t)i * ld + j];
  }
}

// Cluster size of the refinement: one CTA per eight rows for one matrix; for many, as few as the
// shared memory allows.
int refine_cluster(int n, int count) {
  const size_t cap = Runtime::get().smem_optin - 4096;
  const int want = std::max(1, std::min(16, Runtime::get().num_sms / count));
  int cs = 1;
  while (2 * cs <= want && kr_rows(n, cs) > 8) cs *= 2;
  while (cs < 16 && kr_bytes(n, cs, kEigBlocks) > cap) cs *= 2;
  return kr_bytes(n, cs, kEigBlocks) <= cap ? cs : 0;
}

template <class F>
void with_epl(int n, F f) {
  if (n <= 32) f(osj_kernel<1>);
  else if (n <= 64) f(osj_kernel<2>);
  else if (n <= 96) f(osj_kernel<3>);
  else f(osj_kernel<4>);
}

}  // namespace

size_t eig_work_doubles(int n) { return (4 * (size_t)n * n + n + 64 + 3) & ~(size_t)3; }

// Whether the refinement's clusters can run on this device.
bool eig_refined_usable(int n) {
  static const bool ok = [] {
    const char *e = getenv("ISVD_GPU_EIG_REFINED");
    if (e && atoi(e) == 0) return false;
    const int cs = refine_cluster(kMaxN, 1);
    if (cs == 0) return false;
    const size_t bytes = kr_bytes(kMaxN, cs, kEigBlocks);
    CK(cudaFuncSetAttribute(eig_refine_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    CK(cudaFuncSetAttribute(eig_refine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(kKrThreads);
    cfg.dynamicSmemBytes = bytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int c = 0;
    if (cudaOccupancyMaxActiveClusters(&c, eig_refine_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return c >= 1;
  }();
  return ok && n <= kMaxN;
}

void eig_refined(int n, int count, const double *A, double *work, double *V, double *w, int order, bool absval,
                 const EigDesc *desc, cudaStream_t st, bool loose) {
  const size_t stride = eig_work_doubles(n);
  const size_t osm = osj_smem(n);
  with_epl(n, [&](auto kern) {
    CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)osm));
    kern<<<count, osj_threads(n), osm, st>>>(n, A, work, stride, absval ? 1 : 0, loose, desc);
    KLAUNCHED();
  });
  const int cs = refine_cluster(n, count);
  const int bytes = (int)kr_bytes(n, cs, kEigBlocks);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(count * cs);
  cfg.blockDim = dim3(kKrThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  CK(cudaFuncSetAttribute(eig_refine_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CK(cudaFuncSetAttribute(eig_refine_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  CK(cudaLaunchKernelEx(&cfg, eig_refine_kernel, n, work, stride, V, w, order, absval, loose, desc));
  KLAUNCHED();
}

}  // namespace isvdb
