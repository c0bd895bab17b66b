// FP64 matrix product on the FP64 tensor-core path (mma.sync m8n8k4 .f64: the only tensor-core
// instruction with FP64 operands on sm_100a; tcgen05 has no FP64 kind).  Same contract as the
// CUDA-core gemm<double, double> (arbitrary strides with one unit stride per operand, batch,
// split-K, alpha / beta); every product term is an IEEE FP64 fused multiply-add, so results
// differ from the CUDA-core kernel only in the order of the K summation.
//
// Tiling: BM x BN output tile per CTA of WM x WN warps, each warp a (BM / WM) x (BN / WN) block
// of 8 x 8 mma tiles held in registers.  BK = 16 deep K slices are copied global -> shared by
// cp.async (8-byte elements, zero-filled outside the matrix) in a 3-stage ring.  Each operand is
// staged in the orientation of its unit stride (K-contiguous rows of BK + 4, or MN-contiguous
// rows of BM + 4 / BN + 4 doubles), which makes both the copies and the fragment reads free of
// shared-memory bank conflicts.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>

#include "grouped_next.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "planes.cuh"
#include "runtime.h"

namespace isvdb {
namespace {

constexpr int kBK = 16, kStages = 3, kPad = 4;

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem, bool valid) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 8 : 0));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// D = A B + D for one 8 x 8 x 4 tile: a = A(lane / 4, lane % 4), b = B(lane % 4, lane / 4),
// d = D(lane / 4, 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

template <int BM, int BN, bool A_KC, bool B_NC>
struct DmmaLayout {
  static constexpr int a_elems = A_KC ? BM * (kBK + kPad) : kBK * (BM + kPad);
  static constexpr int b_elems = B_NC ? kBK * (BN + kPad) : BN * (kBK + kPad);
  static constexpr int stage = a_elems + b_elems;
  __device__ static int a_at(int m, int k) { return A_KC ? m * (kBK + kPad) + k : k * (BM + kPad) + m; }
  __device__ static int b_at(int k, int n) { return B_NC ? k * (BN + kPad) + n : n * (kBK + kPad) + k; }
};

// acc += A[m0 .. m0 + BM, kb .. ke) B[kb .. ke, n0 .. n0 + BN) for one output tile, with A(i, k) =
// A[i a_rs + k a_cs] and B(k, j) = B[k b_rs + j b_cs]; rows >= M, columns >= N read as zero.  K
// slices flow through the kStages-deep cp.async ring in smem.  On return every copy has landed,
// but warps may still read the ring: a caller that refills it must synchronise the block first.
template <int BM, int BN, int WM, int WN, bool A_KC, bool B_NC>
__device__ __forceinline__ void dmma_tile(double *smem, const double *__restrict__ A, long long a_rs, long long a_cs,
                                          const double *__restrict__ B, long long b_rs, long long b_cs, int M, int N,
                                          int kb, int ke, int m0, int n0,
                                          double (&acc)[BM / WM / 8][BN / WN / 8][2]) {
  using L = DmmaLayout<BM, BN, A_KC, B_NC>;
  constexpr int NT = WM * WN * 32;
  constexpr int TM = BM / WM / 8, TN = BN / WN / 8;  // 8 x 8 tiles per warp
  constexpr int LA = BM * kBK / NT, LB = BN * kBK / NT;
  static_assert(LA * NT == BM * kBK && LB * NT == BN * kBK, "tile / thread mismatch");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm0 = (warp / WN) * (BM / WM), wn0 = (warp % WN) * (BN / WN);
  const int nk = ke > kb ? (ke - kb + kBK - 1) / kBK : 0;

  auto issue = [&](int kt) {  // k slice kt into stage kt % kStages
    double *As = smem + (kt % kStages) * L::stage, *Bs = As + L::a_elems;
    const int k0 = kb + kt * kBK;
#pragma unroll
    for (int r = 0; r < LA; ++r) {
      const int e = tid + r * NT;
      const int mm = A_KC ? e / kBK : e % BM, kk = A_KC ? e % kBK : e / BM;
      const int gm = m0 + mm, gk = k0 + kk;
      const bool ok = gm < M && gk < ke;
      cp_async8(As + L::a_at(mm, kk), ok ? A + (long long)gm * a_rs + (long long)gk * a_cs : A, ok);
    }
#pragma unroll
    for (int r = 0; r < LB; ++r) {
      const int e = tid + r * NT;
      const int nn = B_NC ? e % BN : e / kBK, kk = B_NC ? e / BN : e % kBK;
      const int gn = n0 + nn, gk = k0 + kk;
      const bool ok = gn < N && gk < ke;
      cp_async8(Bs + L::b_at(kk, nn), ok ? B + (long long)gk * b_rs + (long long)gn * b_cs : B, ok);
    }
  };

#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < nk) issue(s);
    cp_async_commit();
  }
  const int fr = lane >> 2, fc = lane & 3;  // fragment row / column within an 8 x 4 (4 x 8) tile
  for (int kt = 0; kt < nk; ++kt) {
    cp_async_wait<kStages - 2>();
    __syncthreads();  // slice kt visible to all; slice kt - 1 no longer read (its stage is refilled)
    if (kt + kStages - 1 < nk) issue(kt + kStages - 1);
    cp_async_commit();
    const double *As = smem + (kt % kStages) * L::stage, *Bs = As + L::a_elems;
#pragma unroll
    for (int k4 = 0; k4 < kBK; k4 += 4) {
      double av[TM], bv[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = As[L::a_at(wm0 + 8 * i + fr, k4 + fc)];
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = Bs[L::b_at(k4 + fc, wn0 + 8 * j + fr)];
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) dmma884(acc[i][j], av[i], bv[j]);
    }
  }
  cp_async_wait<0>();
}

template <int BM, int BN, int WM, int WN, bool A_KC, bool B_NC>
__global__ void __launch_bounds__(WM * WN * 32)
    dmma_gemm_kernel(const Gemm<double, double> g, const int splits, const int kchunk, double *__restrict__ partial) {
  constexpr int TM = BM / WM / 8, TN = BN / WN / 8;  // 8 x 8 tiles per warp
  extern __shared__ double smem[];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm0 = (warp / WN) * (BM / WM), wn0 = (warp % WN) * (BN / WN);
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  if (g.upper && n0 + BN <= m0) return;  // tile strictly below the diagonal: mirrored by the caller
  // (128 x 128 tiles) computed on the int8 tensor cores already (k_i8.cu)
  if (g.done && g.done[(size_t)blockIdx.x * gridDim.y + blockIdx.y] >= g.done_need) return;
  const int b = blockIdx.z / splits, sp = blockIdx.z % splits;
  const int kb = sp * kchunk, ke = min(g.K, kb + kchunk);

  double acc[TM][TN][2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  dmma_tile<BM, BN, WM, WN, A_KC, B_NC>(smem, g.A + (long long)b * g.a_bs, g.a_rs, g.a_cs, g.B + (long long)b * g.b_bs,
                                        g.b_rs, g.b_cs, g.M, g.N, kb, ke, m0, n0, acc);

  const int fr = lane >> 2, fc = lane & 3;
  const bool direct = splits == 1;
  double *__restrict__ C = direct ? g.C + (long long)b * g.c_bs : partial + ((long long)blockIdx.z * g.M) * g.N;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int gm = m0 + wm0 + 8 * i + fr;
    if (gm >= g.M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int gn = n0 + wn0 + 8 * j + 2 * fc + h;
        if (gn >= g.N) continue;
        if (direct) {
          double *c = C + (long long)gm * g.c_rs + (long long)gn * g.c_cs;
          double v = g.alpha * acc[i][j][h];
          if (g.beta != 0.0) v += g.beta * *c;
          *c = v;
          acc[i][j][h] = v;  // the stored value, for the plane output below
        } else {
          C[(long long)gm * g.N + gn] = acc[i][j][h];
        }
      }
  }
  using L = DmmaLayout<BM, BN, A_KC, B_NC>;
  if constexpr (BN * (BM + 1) <= kStages * L::stage) {
    if (direct && g.pl_t && b == g.pl_batch) {
      // bf16 planes of this tile's transpose: the values go through the (now idle) cp.async ring
      // as a BN x BM tile, then each thread splits 8 consecutive rows of one output column and
      // stores 16 bytes per plane (plane row gn, columns gm .. gm + 7)
      constexpr int TLD = BM + 1;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h)
            smem[(wn0 + 8 * j + 2 * fc + h) * TLD + (wm0 + 8 * i + fr)] = acc[i][j][h];
      __syncthreads();
      constexpr int NT = WM * WN * 32;
      for (int t = tid; t < BN * (BM / 8); t += NT) {
        const int cl = t / (BM / 8), seg = t - cl * (BM / 8);
        const int gn = n0 + cl;
        if (gn >= g.N) continue;
        __nv_bfloat16 o[3][8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          __nv_bfloat16 pc[3];
          split3<double>(smem[cl * TLD + 8 * seg + e], pc, 3);
#pragma unroll
          for (int q = 0; q < 3; ++q) o[q][e] = pc[q];
        }
        const long long po = (long long)gn * g.pl_ld + m0 + 8 * seg;
#pragma unroll
        for (int q = 0; q < 3; ++q) *(uint4 *)(g.pl_t + q * g.pl_ps + po) = pack8(o[q]);
      }
    }
  }
}

// Small products: the CTAs of a cluster compute one output tile from a K chunk each, and add their partial
// tiles through distributed shared memory, CTA `rank` the rows rank, rank + splits, ... in the order of the
// ranks.  Against partial sums in global memory this saves their round trip and the reduction's launch.
template <int BM, int BN, int WM, int WN, bool A_KC, bool B_NC>
__global__ void __launch_bounds__(WM * WN * 32)
    dmma_cluster_kernel(const Gemm<double, double> g, const int splits, const int kchunk) {
  constexpr int TM = BM / WM / 8, TN = BN / WN / 8, NT = WM * WN * 32, LD = BN + 2;
  static_assert(BM * LD <= kStages * DmmaLayout<BM, BN, A_KC, B_NC>::stage, "the tile fits the ring");
  extern __shared__ double smem[];
  namespace cg = cooperative_groups;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm0 = (warp / WN) * (BM / WM), wn0 = (warp % WN) * (BN / WN);
  const int fr = lane >> 2, fc = lane & 3;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int b = blockIdx.z / splits, sp = blockIdx.z % splits;
  const int kb = min(g.K, sp * kchunk), ke = min(g.K, kb + kchunk);
  double acc[TM][TN][2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  pdl_wait();
  dmma_tile<BM, BN, WM, WN, A_KC, B_NC>(smem, g.A + (long long)b * g.a_bs, g.a_rs, g.a_cs, g.B + (long long)b * g.b_bs,
                                        g.b_rs, g.b_cs, g.M, g.N, kb, ke, m0, n0, acc);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) smem[(wm0 + 8 * i + fr) * LD + wn0 + 8 * j + 2 * fc + h] = acc[i][j][h];
  pdl_trigger();  // not earlier: CTAs of the next kernel placed around this one's would be spread unevenly
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  double *__restrict__ C = g.C + (long long)b * g.c_bs;
  const int mine = (BM - sp + splits - 1) / splits;  // rows sp, sp + splits, ...
  for (int t = tid; t < mine * BN; t += NT) {
    const int r = sp + (t / BN) * splits, c = t % BN, gm = m0 + r, gn = n0 + c;
    if (gm >= g.M || gn >= g.N) continue;
    double v = 0.0;
#pragma unroll 8
    for (int q = 0; q < splits; ++q) v += cl.map_shared_rank(smem, q)[r * LD + c];
    double *o = C + (long long)gm * g.c_rs + (long long)gn * g.c_cs;
    v *= g.alpha;
    if (g.beta != 0.0) v += g.beta * *o;
    *o = v;
  }
  if (g.pl_t && b == g.pl_batch) {  // splits == 1: planes of this tile's transpose, as dmma_gemm_kernel writes them
    for (int t = tid; t < BN * (BM / 8); t += NT) {
      const int c = t / (BM / 8), seg = t - c * (BM / 8), gn = n0 + c;
      if (gn >= g.N) continue;
      __nv_bfloat16 o[3][8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int r = 8 * seg + e;
        double v = g.alpha * smem[r * LD + c];
        __nv_bfloat16 pc[3];
        split3<double>(v, pc, 3);
#pragma unroll
        for (int q = 0; q < 3; ++q) o[q][e] = pc[q];
      }
      const long long po = (long long)gn * g.pl_ld + m0 + 8 * seg;
#pragma unroll
      for (int q = 0; q < 3; ++q) *(uint4 *)(g.pl_t + q * g.pl_ps + po) = pack8(o[q]);
    }
  }
  cl.sync();  // the peers' reads of this CTA's tile are done
}

// Grouped products (dmma_grouped): each CTA takes the work item blockIdx.x and then the next one that no CTA
// has; a work item is one BM x BN output tile of the product that owns it (binary search on tile0).
template <int BM, int BN, int WM, int WN, bool A_KC, bool B_NC>
__global__ void __launch_bounds__(WM * WN * 32)
    dmma_grouped_kernel(const GroupedProd *__restrict__ prods, int nprod, int total, int *next) {
  constexpr int TM = BM / WM / 8, TN = BN / WN / 8;
  extern __shared__ double smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm0 = (warp / WN) * (BM / WM), wn0 = (warp % WN) * (BN / WN);
  const int fr = lane >> 2, fc = lane & 3;
  __shared__ int snext;
  GroupedNext items(next, &snext);
  for (int t = blockIdx.x; t < total; t = items.take()) {
    items.fetch();
    int lo = 0, hi = nprod - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (prods[mid].tile0 <= t) lo = mid;
      else hi = mid - 1;
    }
    const GroupedProd g = prods[lo];
    const int tt = t - g.tile0, m0 = (tt / g.tn) * BM, n0 = (tt % g.tn) * BN;
    if (g.upper && n0 + BN <= m0) continue;  // strictly below the diagonal (uniform in the CTA)
    if (g.gate && *g.gate <= g.gate_tol) continue;
    double acc[TM][TN][2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    __syncthreads();  // the previous work item's reads of the ring are done before it is refilled
    dmma_tile<BM, BN, WM, WN, A_KC, B_NC>(smem, static_cast<const double *>(g.A), g.a_rs, g.a_cs,
                                          static_cast<const double *>(g.B), g.b_rs, g.b_cs, g.M, g.N, 0, g.K, m0, n0,
                                          acc);
    double *__restrict__ C = static_cast<double *>(g.C);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int gm = m0 + wm0 + 8 * i + fr;
      if (gm >= g.M) continue;
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int gn = n0 + wn0 + 8 * j + 2 * fc + h;
          if (gn >= g.N) continue;
          double *c = C + (long long)gm * g.c_rs + (long long)gn * g.c_cs;
          double v = g.alpha * acc[i][j][h];
          if (g.beta != 0.0) v += g.beta * *c;
          *c = v;
        }
    }
  }
  items.done();
}

template <int BM, int BN, int WM, int WN, bool A_KC, bool B_NC>
void dmma_grouped_launch(const GroupedProd *prods, int nprod, int total, int *next, cudaStream_t st) {
  auto *k = dmma_grouped_kernel<BM, BN, WM, WN, A_KC, B_NC>;
  constexpr int NT = WM * WN * 32;
  const int bytes = kStages * DmmaLayout<BM, BN, A_KC, B_NC>::stage * (int)sizeof(double);
  static int per_sm = 0;  // resident CTAs per SM, resolved on first use
  if (per_sm == 0) {
    CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, NT, bytes));
    per_sm = std::max(1, per_sm);
  }
  const int grid = std::max(1, std::min(total, per_sm * Runtime::get().num_sms));
  k<<<grid, NT, bytes, st>>>(prods, nprod, total, next);
  KLAUNCHED();
}

// K splits of dmma_launch, by a time model: the busiest SM runs ceil(tiles s / SMs) CTAs of BM BN (K / s)
// FMAs (about 0.23 TFLOP/s per SM on mma.sync f64) plus a fixed 2 us each, and s > 1 adds the partial
// sums' round trip (s + 1) M N 8 bytes at about 4 TB/s; the smallest s within 3 % of the best, with at
// least 64 of K per split and at most 512 MB of partials.
int dmma_splits(const Gemm<double, double> &g, int BM, int BN) {
  if (g.splits > 0) return g.splits;
  const int sms = Runtime::get().num_sms;
  const long long tiles = (long long)((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN) * g.batch;
  const double rate = 0.23e12, fixed = 2e-6, bw = 4e12;
  const long long mnb = (long long)g.M * g.N * g.batch;
  auto model = [&](long long s) {
    const long long per_sm = (tiles * s + sms - 1) / sms;
    const double kc = (double)((g.K + s - 1) / s);
    return per_sm * (2.0 * BM * BN * kc / rate + fixed) + (s > 1 ? (double)(s + 1) * mnb * 8.0 / bw : 0.0);
  };
  const long long smax = std::max<long long>(
      1, std::min<long long>({64, (long long)g.K / 64, (512LL << 20) / std::max<long long>(1, mnb * 8)}));
  double best = model(1);
  for (long long s = 2; s <= smax; ++s) best = std::min(best, model(s));
  for (long long s = 1; s <= smax; ++s)
    if (model(s) <= 1.03 * best) return (int)s;
  return 1;
}

// Sum of the K splits' partial products for the 128 x 128 tiles that are not done, 16 rows per CTA.
__global__ void __launch_bounds__(256)
    rest_reduce_kernel(const Gemm<double, double> g, const int splits, const double *__restrict__ partial) {
  const int m0 = blockIdx.x * 128, n0 = blockIdx.y * 128;
  if (g.upper && n0 + 128 <= m0) return;
  if (g.done[(size_t)blockIdx.x * gridDim.y + blockIdx.y] >= g.done_need) return;
  const long long MN = (long long)g.M * g.N;
#pragma unroll 2
  for (int t = threadIdx.x; t < 16 * 128; t += 256) {
    const int r = m0 + blockIdx.z * 16 + (t >> 7), c = n0 + (t & 127);
    if (r >= g.M || c >= g.N) continue;
    const double *p = partial + (long long)r * g.N + c;
    double v = 0.0;
#pragma unroll 8
    for (int sp = 0; sp < splits; ++sp) v += p[sp * MN];
    g.C[(long long)r * g.c_rs + (long long)c * g.c_cs] = g.alpha * v;
  }
}

template <int BM, int BN, int WM, int WN>
void dmma_launch(const Gemm<double, double> &g, bool a_kc, bool b_nc, cudaStream_t st) {
  const int gx = (g.M + BM - 1) / BM, gy = (g.N + BN - 1) / BN;
  int splits = dmma_splits(g, BM, BN);
  int kchunk = (g.K + splits - 1) / splits;
  kchunk = ((kchunk + kBK - 1) / kBK) * kBK;
  if (kchunk <= 0) kchunk = kBK;
  splits = std::max(1, (g.K + kchunk - 1) / kchunk);
  DBuf<double> part;
  if (splits > 1) part.alloc((size_t)g.batch * splits * g.M * g.N);
  const dim3 grid(gx, gy, g.batch * splits);
  constexpr int NT = WM * WN * 32;
#define ISVD_DMMA_CASE(AK, BNC)                                                                        \
  if (a_kc == AK && b_nc == BNC) {                                                                     \
    auto *k = dmma_gemm_kernel<BM, BN, WM, WN, AK, BNC>;                                               \
    const int bytes = kStages * DmmaLayout<BM, BN, AK, BNC>::stage * (int)sizeof(double);              \
    CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));                   \
    k<<<grid, NT, bytes, st>>>(g, splits, kchunk, part.p);                                             \
    KLAUNCHED();                                                                                       \
  }
  ISVD_DMMA_CASE(true, true)
  ISVD_DMMA_CASE(true, false)
  ISVD_DMMA_CASE(false, true)
  ISVD_DMMA_CASE(false, false)
#undef ISVD_DMMA_CASE
  if (splits > 1 && g.done) {
    rest_reduce_kernel<<<dim3(gx, gy, 8), 256, 0, st>>>(g, splits, part.p);
    KLAUNCHED();
  } else if (splits > 1) {
    splitk_reduce(g, splits, part.p, st);
  }
}

template <int BM, int BN, int WM, int WN>
void dmma_cluster_launch(const Gemm<double, double> &g, int splits, bool a_kc, bool b_nc, cudaStream_t st) {
  const int kchunk = ((g.K + splits - 1) / splits + 3) / 4 * 4;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((g.M + BM - 1) / BM, (g.N + BN - 1) / BN, g.batch * splits);
  cfg.blockDim = dim3(WM * WN * 32);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[1] = pdl_attribute();
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = splits;
  cfg.attrs = at;
  // CTAs that start beside those of the kernel before are spread unevenly over the SMs, so only launches
  // that leave SMs idle anyway, of the small tiles, whose time is latency (2048 x 128 x 2048, 256 CTAs of
  // 64 x 64: 52 us after the kernel before, 102 us beside its end)
  const bool pdl = BM <= 32 && (long long)cfg.gridDim.x * cfg.gridDim.y * cfg.gridDim.z <= Runtime::get().num_sms;
  cfg.numAttrs = pdl ? 2 : 1;
#define ISVD_DMMA_CASE(AK, BNC)                                                                        \
  if (a_kc == AK && b_nc == BNC) {                                                                     \
    auto *k = dmma_cluster_kernel<BM, BN, WM, WN, AK, BNC>;                                            \
    cfg.dynamicSmemBytes = kStages * DmmaLayout<BM, BN, AK, BNC>::stage * sizeof(double);              \
    CK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes)); \
    CK(cudaLaunchKernelEx(&cfg, k, g, splits, kchunk));                                                \
    KLAUNCHED();                                                                                       \
  }
  ISVD_DMMA_CASE(true, true)
  ISVD_DMMA_CASE(true, false)
  ISVD_DMMA_CASE(false, true)
  ISVD_DMMA_CASE(false, false)
#undef ISVD_DMMA_CASE
}

// Shape of a small product's clusters.  Modelled time of a launch: 5 us, and per 16-deep K slice of a CTA
// the slice's latency for a CTA alone or, when the busiest SM's CTAs together take longer, their sum
// (measured: 64 x 64 tiles 1.2 and 0.75 us, 32 x 32 tiles 0.57 and 0.265 us).  The partial tiles' sum costs
// 0.5 us and their bytes at about 3 TB/s; partials through global memory, 5 us of a second launch and their
// round trip at about 1 TB/s.  Measured, launches
// back to back, before and after: 2048 x 128 x 2048 100 -> 55 us, 1536 x 96 x 1536 57 -> 33, 1040 x 65 x
// 1040 35 -> 19, 256 x 32 x 256 14.4 -> 6.3; 2 x 65 x 65 x 1040 15.7 -> 10.4; 2 x 1536 x 96 x 192 19.6 -> 12.4.
struct ClusterPlan {
  int bm = 0, splits = 1;  // bm 0: not by clusters
};
ClusterPlan cluster_plan(const Gemm<double, double> &g) {
  ClusterPlan p;
  const int sms = Runtime::get().num_sms;
  const double mb = (double)g.M * g.N * g.batch * 8.0 / 1e6;
  auto time = [&](int bm, int s) {
    const double ctas = std::ceil(g.M / (double)bm) * std::ceil(g.N / (double)bm) * g.batch * s;
    const double slices = std::ceil(g.K / (double)s / kBK);
    return 5.0 + slices * std::max(bm == 64 ? 1.2 : 0.57, std::ceil(ctas / sms) * (bm == 64 ? 0.75 : 0.265));
  };
  const int s0 = dmma_splits(g, 64, 64);
  double best = time(64, s0) + (s0 > 1 ? 5.0 + (s0 + 1.0) * mb : 0.0);
  for (int bm = 64; bm >= 32; bm /= 2)
    for (int s = 1; s <= (g.pl_t ? 1 : 8) && (s == 1 || g.K / s >= kBK); s *= 2)
      if (const double t = time(bm, s) + (s > 1 ? 0.5 + s * mb / 3 : 0.0); t < 0.97 * best) {
        best = t;
        p.bm = bm;
        p.splits = s;
      }
  return p;
}

}  // namespace

bool dmma_enabled() {
  static const bool on = [] {
    const char *e = getenv("ISVD_GPU_DMMA");
    return !(e && atoi(e) == 0);
  }();
  return on;
}

void dmma_gemm(const Gemm<double, double> &g, bool a_kc, bool b_nc, cudaStream_t st) {
  // 128 x 128 tiles when they fill the GPU or a long K lets split-K fill it; otherwise 64 x 64
  const long long tiles128 = (long long)((g.M + 127) / 128) * ((g.N + 127) / 128) * g.batch;
  const int sms = Runtime::get().num_sms;
  const bool long_k = g.splits <= 0 && (long long)g.K >= 2048 && tiles128 * (g.K / 1024) >= 2LL * sms;
  if (g.pl_t && (g.splits != 1 || g.M % 64 || g.pl_ld % 8 || ((uintptr_t)g.pl_t & 15) || g.pl_ps % 8 ||
                 g.pl_batch < 0 || g.pl_batch >= g.batch))
    fail(kErrArgument, "dmma_gemm: plane output needs splits = 1, M %% 64 == 0 and 16-byte aligned plane rows");
  if (!g.upper && tiles128 < 2LL * sms && !long_k) {  // few output tiles and a short K: clusters of splits
    const ClusterPlan p = cluster_plan(g);
    if (p.bm == 64) return dmma_cluster_launch<64, 64, 2, 2>(g, p.splits, a_kc, b_nc, st);
    if (p.bm == 32) return dmma_cluster_launch<32, 32, 2, 2>(g, p.splits, a_kc, b_nc, st);
  }
  // plane output: 64 x 64 tiles (their epilogue stages a tile's transpose through the cp.async
  // ring; without split-K the tile shape does not change the results)
  if (g.pl_t || g.M <= 64 || g.N <= 64 || (tiles128 < 2LL * sms && !long_k))
    dmma_launch<64, 64, 2, 2>(g, a_kc, b_nc, st);
  else
    dmma_launch<128, 128, 2, 4>(g, a_kc, b_nc, st);
}

// C_b = A_b B_b over A (column blocks of a tall matrix times N x N blocks): a CTA holds its rows' whole block
// in one tile and has read all of it (the barrier of the last K slice) before it writes.  Saves the
// temporary and its copy back: 0.5 ms of 0.98 GB for the 16 blocks of 40000 x 96.
bool dmma_apply_in_place(const Gemm<double, double> &g, cudaStream_t st) {
  if (!dmma_enabled() || g.N > 128 || g.K != g.N || g.beta != 0.0) return false;
  Gemm<double, double> f = g;
  f.C = const_cast<double *>(g.A);
  f.c_rs = g.a_rs; f.c_cs = g.a_cs; f.c_bs = g.a_bs;
  f.splits = 1;
  if (g.N <= 64) dmma_launch<64, 64, 2, 2>(f, true, true, st);
  else dmma_launch<128, 128, 2, 4>(f, true, true, st);
  return true;
}

void dmma_gemm_rest(const Gemm<double, double> &g, bool a_kc, bool b_nc, const unsigned long long *done,
                    unsigned long long need, cudaStream_t st) {
  Gemm<double, double> f = g;
  f.done = done; f.done_need = need;
  // K splits as for the whole product: a tall K with few tiles (G = Qs'Qs) is otherwise a serial tail of its own.
  // One KN iteration on 16 blocks of 40000 x 64 with ten rows a hundred times the others takes 3.0 ms in place of
  // 7.6 (all on this kernel, without digits: 2.8); without such rows 1.1 ms.
  dmma_launch<128, 128, 2, 4>(f, a_kc, b_nc, st);
}

int dmma_grouped_bm(int shape) { return shape == 2 ? 128 : shape == 4 ? 32 : 64; }
int dmma_grouped_bn(int shape) { return (shape == 0 || shape >= 3) ? 32 : 64; }

void dmma_grouped(const GroupedProd *prods, int nprod, int total, int shape, bool a_kc, bool b_nc, int *next,
                  cudaStream_t st) {
  if (nprod <= 0 || total <= 0) return;
#define ISVD_DMMA_GROUPED(BM, BN, WM, WN)                                                              \
  if (a_kc && b_nc) dmma_grouped_launch<BM, BN, WM, WN, true, true>(prods, nprod, total, next, st);          \
  else if (a_kc) dmma_grouped_launch<BM, BN, WM, WN, true, false>(prods, nprod, total, next, st);            \
  else if (b_nc) dmma_grouped_launch<BM, BN, WM, WN, false, true>(prods, nprod, total, next, st);            \
  else dmma_grouped_launch<BM, BN, WM, WN, false, false>(prods, nprod, total, next, st);
  switch (shape) {  // warp tiles of 32 x 32 outputs (4 x 4 mma tiles), or 32 x 16 (shape 3)
    case 0: ISVD_DMMA_GROUPED(64, 32, 2, 1) break;
    case 1: ISVD_DMMA_GROUPED(64, 64, 2, 2) break;
    case 2: ISVD_DMMA_GROUPED(128, 64, 4, 2) break;
    case 3: ISVD_DMMA_GROUPED(64, 32, 2, 2) break;
    default: ISVD_DMMA_GROUPED(32, 32, 1, 1) break;
  }
#undef ISVD_DMMA_GROUPED
}

}  // namespace isvdb
