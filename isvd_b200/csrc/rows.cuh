// Chains of l x l FP64 products on one thread-block cluster, cut by rows: CTA `rank` owns rows
// [r0, r0 + rb) of every matrix, kept as blocks of rb rows in shared memory, and `full` holds one
// whole l x l right operand.  A product of the CTA's rows with the whole operand is local; a new right
// operand is exchanged through global memory (L2) and the hardware cluster barrier.  Row stride ld =
// 4 (mod 16) doubles: the mma.sync fragment reads hit 16 distinct bank pairs.  Columns and rows
// between l and its next multiple of 8 are zero.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

namespace isvdb {
namespace {

namespace rows_cg = cooperative_groups;

constexpr int kKrThreads = 512;
constexpr int kKrWarps = kKrThreads / 32;
constexpr int kKrMaxL = 128;

__host__ __device__ constexpr int kr_ld(int l) { return (l + 15) / 16 * 16 + 4; }
__host__ __device__ constexpr int kr_rows(int l, int cs) { return 8 * (((l + 7) / 8 + cs - 1) / cs); }
__host__ __device__ constexpr size_t kr_bytes(int l, int cs, int blocks) {
  return ((size_t)((l + 7) / 8 * 8) * kr_ld(l) + (size_t)blocks * kr_rows(l, cs) * kr_ld(l)) * sizeof(double);
}

struct Kr {
  int l, lr, l4, ld, rb, r0, cs, rank, mt, nt;  // mt x nt: 8 x 8 tiles of this CTA's rows
  double *full, *blk;
  __device__ double *block(int i) const { return blk + (size_t)i * rb * ld; }
};

__device__ __forceinline__ void kr_init(Kr &k, int l, int cs, int rank, double *sm) {
  k.l = l; k.lr = (l + 7) & ~7; k.l4 = (l + 3) & ~3; k.ld = kr_ld(l);
  k.cs = cs; k.rank = rank;
  k.rb = kr_rows(l, cs); k.r0 = rank * k.rb;
  k.mt = max(0, min(k.rb, k.lr - k.r0)) / 8; k.nt = k.lr / 8;
  k.full = sm; k.blk = sm + (size_t)k.lr * k.ld;
}

// One 8 x 8 tile of rows (A) times eight columns of the whole operand (B), two accumulation chains.
// TB: times eight rows of it instead (the product with the transposed operand).
template <bool TB = false>
__device__ __forceinline__ void kr_tile(const Kr &k, const double *A, const double *B, double (&d)[2]) {
  const int lane = threadIdx.x & 31;
  const double *ap = A + (lane >> 2) * k.ld + (lane & 3);
  const double *bp = TB ? B + (lane >> 2) * k.ld + (lane & 3) : B + (lane & 3) * k.ld + (lane >> 2);
  const int sb = TB ? 4 : 4 * k.ld;
  double e[2] = {0.0, 0.0};
  d[0] = d[1] = 0.0;
  int kk = 0;
#pragma unroll 4
  for (; kk + 8 <= k.l4; kk += 8, ap += 8, bp += 2 * sb) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(ap[0]), "d"(bp[0]));
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(e[0]), "+d"(e[1])
                 : "d"(ap[4]), "d"(bp[sb]));
  }
  if (kk < k.l4)
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(ap[0]), "d"(bp[0]));
  d[0] += e[0];
  d[1] += e[1];
}

// epi(i, j, v) for the entries (local row i < 8 mt, column j < lr) of A (row block, or the rows of
// `full` at r0) times `full` (TB: times its transpose).
template <bool TB = false, class Epi>
__device__ __forceinline__ void kr_mm(const Kr &k, const double *A, Epi epi) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = warp; t < k.mt * k.nt; t += kKrWarps) {
    const int m0 = (t / k.nt) * 8, n0 = (t % k.nt) * 8;
    double d[2];
    kr_tile<TB>(k, A + (size_t)m0 * k.ld, k.full + (TB ? (size_t)n0 * k.ld : n0), d);
    epi(m0 + (lane >> 2), n0 + 2 * (lane & 3), d[0]);
    epi(m0 + (lane >> 2), n0 + 2 * (lane & 3) + 1, d[1]);
  }
}

// Whole l x l matrix (written by every CTA of the cluster, so read through L2) into `full`.
__device__ __forceinline__ void kr_load(const Kr &k, const double *src) {
  const int l = k.l;
  if ((l & 1) == 0) {
    const int l2 = l >> 1, total = l * l2;
    for (int e0 = threadIdx.x; e0 < total; e0 += 8 * kKrThreads) {
      double2 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = e0 + u * kKrThreads;
        if (e < total) v[u] = __ldcg((const double2 *)src + e);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int e = e0 + u * kKrThreads;
        if (e < total) {
          const int i = e / l2, j = 2 * (e - i * l2);
          *(double2 *)(k.full + (size_t)i * k.ld + j) = v[u];
        }
      }
    }
  } else {
    for (int e = threadIdx.x; e < l * l; e += kKrThreads) {
      const int i = e / l, j = e - i * l;
      k.full[(size_t)i * k.ld + j] = __ldcg(src + e);
    }
  }
}

// The symmetric completion of the upper triangle of src (as syev 'U' reads Z) into `full`; returns
// this thread's part of the sum of its squares.
__device__ __forceinline__ double kr_load_sym(const Kr &k, const double *src) {
  const int l = k.l, total = l * l;
  double f = 0.0;
  for (int e0 = threadIdx.x; e0 < total; e0 += 8 * kKrThreads) {
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * kKrThreads;
      v[u] = e < total ? __ldcg(src + e) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = e0 + u * kKrThreads;
      const int i = e / l, j = e - i * l;
      if (e < total && i <= j) {
        k.full[(size_t)i * k.ld + j] = v[u];
        if (i != j) k.full[(size_t)j * k.ld + i] = v[u];
        f += (i == j ? 1.0 : 2.0) * v[u] * v[u];
      }
    }
  }
  return f;
}

__device__ __forceinline__ double kr_block_sum(double v, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = red[0];
#pragma unroll
  for (int i = 1; i < kKrWarps; ++i) s += red[i];
  return s;
}

// Sum over the cluster of the CTAs' values, the same in every CTA; everything that the CTAs wrote
// to global memory before it is visible to all after it.
__device__ __forceinline__ double kr_cluster_sum(const Kr &k, rows_cg::cluster_group &cluster, double v, double *slots,
                                                 double *red) {
  v = kr_block_sum(v, red);
  if (threadIdx.x == 0) slots[k.rank] = v;
  cluster.sync();
  double s = 0.0;
  for (int r = 0; r < k.cs; ++r) s += __ldcg(slots + r);
  return s;
}

}  // namespace
}  // namespace isvdb
