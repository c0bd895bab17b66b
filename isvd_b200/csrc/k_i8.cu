// FP64 products on the int8 tensor cores (tcgen05 kind::i8), by error-free splitting into digits (Ozaki,
// Ogita, Oishi & Rump, "Error-free transformations of matrix multiplication by using fast routines of
// matrix multiplication and its applications", Numer. Algorithms 59 (2012)):
//
//   a_ik = 2^(eA_i - 55) X_ik,  X_ik = sum_{p < 7} d_p 2^(8 (6 - p)),  d_p in [-128, 127]  (b_kj alike),
//   c_ij = 2^(eA_i + eB_j - 110) sum_{s < 7} 2^(8 (12 - s)) sum_{p + q = s} sum_k d_p(i, k) d_q(k, j).
//
// eA_i is the exponent of the row's (eB_j: the column's) largest entry, so an entry keeps 55 bits below
// it; the inner sums are exact in int32 (at most 16384 terms at a time), and what is left out, the digit
// pairs with p + q >= 7 and the bits below 2^-55, is a random error of about 2^-56.3 sqrt(K) 2^eA 2^eB,
// where a chain of K FP64 multiply-adds makes about 2^-54 sum_k |a_ik| |b_kj| (Gaussian: 2^-54.5 K rms(a_i)
// rms(b_j)).  A tile is computed here when the one is below the other for each of its entries.  First by rows
// and columns, from their splits,
//   max_i (2^eA_i / rms a_i) max_j (2^eB_j / rms b_j) <= 2.5 sqrt(K)                       (*)
// (Gaussian rows: 8 x 8 against 2.5 sqrt(K), so from K = 655 on): rows with outliers, zeros for most entries,
// exponents beyond 2^400, infinities or NaN fail it.  Then by entries, from the product of the leading bits
// m = floor(|x| 2^(7 - e)), an eighth plane that takes the fourth accumulator of the second pass,
//   2^-14 sum_k m(a_ik) m(b_kj) >= 0.2 sqrt(K)      (then the error is below 2^-54 sum |a_ik| |b_kj|)   (**)
// which operands graded against each other fail (large entries of a row meeting small ones of a column:
// all terms are small, and so is the chain's error).  The tiles that fail are computed by the FP64 tensor-core
// kernel (k_dmma.cu), which is launched behind and skips the others: both go by the tile's sum over the
// splits of the smallest sum in (**), zero where (*) failed; the host does not wait.
//
// One CTA per 128 x 128 tile (and K split, where the tiles alone leave SMs idle): warp 0 moves 64-byte deep
// blocks of the digit planes by TMA (two stages of 14 planes), warp 1 issues the MMAs, warps 2..9 drain.
// The seven sums s need 7 x 128 TMEM columns of 512, so a K chunk runs in two passes: s = 3..6 (22 products
// of the 28, all 14 planes), then s = 0..2 (6 products, the three leading planes of either side) and (**).  The
// drained int32 sums of a pass combine exactly in int64 and join the FP64 running sums in registers.
//
// Measured, mma.sync f64 -> here with the digits: 40000 x 1536 x 6000 26.6 -> 8.2 ms (7.2 ms of products at
// 2.9e15 int8 op/s of the 28 pairs, the tensor cores' rate with (**)'s 29th product); 20011 x 1024 x 1501
// 2.35 -> 0.85 ms; Gram 1536 x 1536 x 40000 7.0 -> 1.4 ms; 777 x 1000 x 9001 0.71 -> 0.31 ms.  (**) costs 4 to 5 %
// of that.  Errors against exact sums, rms relative to sum |a_ik| |b_kj|: 1.1e-17 (mma.sync f64: 3.7e-17) at K = 1501,
// 8.9e-18 (5.3e-17) at 6000, with positive entries 3.7e-17 (4.9e-16) at 1501.  Operands of which every tile fails (*)
// cost 4 to 10 % more than mma.sync alone, those of which every tile fails only (**) 30 to 36 %.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "kernels.h"
#include "runtime.h"
#include "umma.h"
#include "umma_ptx.cuh"

extern "C" size_t isvd_gpu_memory_limit;  // include/isvd/gpu/env.h

namespace isvdb {
namespace {

constexpr int kSlices = 7;
constexpr int kPlanes = kSlices + 1;                // and the leading bits of the magnitudes
constexpr int kLead = 4;                            // planes per side of the second pass
constexpr int kZeroRow = 1 << 20;                   // in place of a zero row's exponent
constexpr int kTile = 128, kBk = 64;
constexpr int kPlane = kTile * kBk;                 // bytes of one plane's tile
constexpr int kStage = 2 * kSlices * kPlane;        // 112 KB
constexpr int kStages = 2;
constexpr int kChunkBlocks = 16384 / kBk;           // int32 stays exact: 7 * 128 * 128 * 16384 < 2^31
constexpr int kI8Threads = 320;
constexpr size_t kI8Smem = (size_t)kStages * kStage + 1024 + 256;

struct I8Params {
  int M, N, nkb;
  int per;                     // K blocks of a split
  double *C;                   // the product, or split z's partial product at C + z c_zs
  long long c_rs, c_cs, c_zs;
  double alpha;
  int upper;
  const int *ea, *eb;          // exponents of the rows and columns
  const float *ra, *rb;        // 128-row (128-column) maxima of 2^e / rms
  float lim;
  unsigned long long *sum;     // per tile (N tiles fastest): the left side of (**) over the splits, in units of 2^-14
  unsigned long long need;     // its right side
  int *status;
};

__device__ __forceinline__ void umma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::
          "r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(acc));
}
// kind::i8: S32 accumulator, signed A and B, both K-major
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) |
                            ((uint32_t)(kTile >> 4) << 24);

__device__ __forceinline__ void tmem_ld8i(uint32_t taddr, int *r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

// 2^e of a row's exponent (anything for a zero row)
__device__ __forceinline__ double pow2(int e) {
  if (e == kZeroRow) e = 0;
  return __longlong_as_double((long long)(e + 1023) << 52);
}

// The products of one pass: LO <= p + q <= HI, accumulator p + q - LO; MAG: the last planes' product too, in
// the accumulator behind.
template <int NS, int LO, int HI, bool MAG>
__device__ __forceinline__ void issue_pass(uint32_t tmem, uint64_t base, uint32_t more) {
  constexpr int ND = MAG ? NS - 1 : NS;
#pragma unroll
  for (int p = 0; p < NS; ++p)
#pragma unroll
    for (int q = 0; q < NS; ++q) {
      const bool mag = MAG && p == ND && q == ND;
      if (!mag && (p >= ND || q >= ND || p + q < LO || p + q > HI)) continue;
      const uint32_t d = tmem + (uint32_t)((mag ? HI + 1 - LO : p + q - LO) * kTile);
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
        umma_i8(d, base + (uint32_t)(p * kPlane >> 4) + kk * 2, base + (uint32_t)((NS + q) * kPlane >> 4) + kk * 2, kIdesc,
                kk > 0 || (p > 0 && !mag) ? 1u : more);
    }
}

__global__ void __launch_bounds__(kI8Threads, 1)
    i8_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const I8Params p) {
  const int nt = blockIdx.x, mt = blockIdx.y;
  const int m0 = mt * kTile, n0 = nt * kTile;
  if (p.upper && n0 + kTile <= m0) return;            // tile strictly below the diagonal: mirrored later
  if (!(p.ra[mt] * p.rb[nt] <= p.lim)) return;        // (*) fails (the tile's sum stays zero)
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ unsigned least[8];  // of each epilogue warp, the smallest sum of (**)
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(smem + (size_t)kStages * kStage);
  uint64_t *empty = full + kStages;
  uint64_t *tfull = empty + kStages;  // the pass's sums are complete
  uint64_t *tempty = tfull + 1;       // ... and drained
  uint64_t *mdone = tempty + 1;       // an aborted CTA's last MMAs have finished
  uint32_t *tslot = (uint32_t *)(mdone + 1);
  volatile int *abort_flag = (volatile int *)(tslot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, 8);
    mbar_init(mdone, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  const int kfirst = blockIdx.z * p.per, nkb = min(p.per, p.nkb - kfirst);
  const int nchunks = (nkb + kChunkBlocks - 1) / kChunkBlocks;

  if (warp == 0 && lane == 0) {
    // ---------------------------------------------------------------- TMA producer
    int issued = 0, s = 0;
    uint32_t ph = 1;
    for (int c = 0; c < nchunks && !*abort_flag; ++c)
      for (int pass = 0; pass < 2 && !*abort_flag; ++pass) {
        const int ns = pass == 0 ? kSlices : kLead;
        const int kb1 = min(nkb, (c + 1) * kChunkBlocks);
        for (int kb = c * kChunkBlocks; kb < kb1; ++kb) {
          if (issued >= kStages && !mbar_try(&empty[s], ph) && !mbar_wait(&empty[s], ph, abort_flag)) {
            *abort_flag = 1;
            break;
          }
          uint8_t *st = smem + (size_t)s * kStage;
          mbar_expect_tx(&full[s], (uint32_t)(2 * ns * kPlane));
          auto plane = [&](int q) { return q == kLead - 1 && pass ? kSlices : q; };
          for (int q = 0; q < ns; ++q) tma_load_3d(st + q * kPlane, &mapA, &full[s], (kfirst + kb) * kBk, m0, plane(q));
          for (int q = 0; q < ns; ++q)
            tma_load_3d(st + (ns + q) * kPlane, &mapB, &full[s], (kfirst + kb) * kBk, n0, plane(q));
          ++issued;
          if (++s == kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    // Drain: every issued load has landed before the CTA can exit (bounded).
    for (int i = max(0, issued - kStages); i < issued; ++i) {
      long long w = 0;
      while (!mbar_try(&full[i % kStages], (i / kStages) & 1) && ++w < kWaitLimit) {
      }
    }
  } else if (warp == 1 && lane == 0) {
    // ---------------------------------------------------------------- MMA issuer
    const uint64_t d0 = sdesc(0, 16, 512, 4u);  // 64-byte rows, SWIZZLE_64B
    const uint32_t smem16 = su32(smem) >> 4;
    int s = 0, t = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int c = 0; c < nchunks && ok; ++c)
      for (int pass = 0; pass < 2 && ok; ++pass, ++t) {
        if (t > 0 && !mbar_wait(tempty, (t - 1) & 1, abort_flag)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const int kb0 = c * kChunkBlocks, kb1 = min(nkb, kb0 + kChunkBlocks);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_try(&full[s], ph) && !mbar_wait(&full[s], ph, abort_flag)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t base = d0 + (uint64_t)(smem16 + (uint32_t)s * (kStage >> 4));
          if (pass == 0) issue_pass<kSlices, 3, 6, false>(tmem, base, kb > kb0);
          else issue_pass<kLead, 0, 2, true>(tmem, base, kb > kb0);
          umma_commit(&empty[s]);
          if (++s == kStages) {
            s = 0;
            ph ^= 1u;
          }
        }
        umma_commit(tfull);
      }
    if (!ok) *abort_flag = 1;
  } else if (warp >= 2) {
    // ---------------------------------------------------------------- epilogue
    const int q = warp & 3, h = (warp - 2) >> 2;  // TMEM lane quarter, column half
    double acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.0;
    // the entries that (**) is asked of: not the padding, and not zero rows or columns, whose products are exact
    const int row = m0 + q * 32 + lane, col = n0 + h * 64 + lane;
    const bool ask = row < p.M && p.ea[row] != kZeroRow;
    const unsigned cols0 = __ballot_sync(0xffffffffu, col < p.N && p.eb[col] != kZeroRow);
    const unsigned cols1 = __ballot_sync(0xffffffffu, col + 32 < p.N && p.eb[col + 32] != kZeroRow);
    unsigned long long sum = 0;  // over the chunks, of the smallest of this thread's entries
    bool ok = true;
    for (int t = 0; t < 2 * nchunks; ++t) {
      int okw = 0;
      if (lane == 0) okw = mbar_wait(tfull, t & 1, abort_flag) ? 1 : 0;
      ok = __shfl_sync(0xffffffffu, okw, 0) != 0;
      if (!ok) {
        if (lane == 0) *abort_flag = 1;
        break;
      }
      tc_fence_after();
      const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * 64);
      if ((t & 1) == 0) {
#pragma unroll
        for (int j = 0; j < 64; j += 8) {
          int a3[8], a4[8], a5[8], a6[8];
          tmem_ld8i(tb + j, a3);
          tmem_ld8i(tb + kTile + j, a4);
          tmem_ld8i(tb + 2 * kTile + j, a5);
          tmem_ld8i(tb + 3 * kTile + j, a6);
          tmem_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i)
            acc[j + i] += (double)(((long long)a3[i] << 24) + ((long long)a4[i] << 16) + ((long long)a5[i] << 8) +
                                   (long long)a6[i]);
        }
      } else {
        int low = 0x7fffffff;
#pragma unroll
        for (int j = 0; j < 64; j += 8) {
          int a0[8], a1[8], a2[8], mm[8];
          tmem_ld8i(tb + j, a0);
          tmem_ld8i(tb + kTile + j, a1);
          tmem_ld8i(tb + 2 * kTile + j, a2);
          tmem_ld8i(tb + 3 * kTile + j, mm);
          tmem_wait();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            acc[j + i] = fma((double)(((long long)a0[i] << 16) + ((long long)a1[i] << 8) + (long long)a2[i]), 0x1p32,
                             acc[j + i]);
            if (((j < 32 ? cols0 : cols1) >> ((j + i) & 31)) & 1u) low = min(low, mm[i]);
          }
        }
        sum += (unsigned)low;
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(tempty)) : "memory");
    }
    const unsigned small = __reduce_min_sync(0xffffffffu, ask ? (unsigned)min(sum, 0xffffffffull) : 0xffffffffu);
    if (lane == 0) least[warp - 2] = small;
    if (ok) {
      // every MMA has completed, so the pipeline buffers are free: whole rows through them
      constexpr int SROW = 65;
      double *stg = (double *)smem + (size_t)(warp - 2) * 32 * SROW;
      // the sums count units of 2^(48 - 110)
      const double sa = row < p.M ? p.alpha * 0x1p-62 * pow2(p.ea[row]) : 0.0;
#pragma unroll
      for (int j = 0; j < 64; ++j) stg[lane * SROW + j] = acc[j] * sa;
      __syncwarp();
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int gn = n0 + h * 64 + u * 32 + lane;
        if (gn >= p.N) continue;
        const double sb = pow2(p.eb[gn]);
        for (int r = 0; r < 32; ++r) {
          const int gr = m0 + q * 32 + r;
          if (gr >= p.M) break;
          if (p.upper && gn < gr) continue;
          p.C[blockIdx.z * p.c_zs + (long long)gr * p.c_rs + (long long)gn * p.c_cs] = stg[r * SROW + u * 32 + lane] * sb;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x == 0 && !*abort_flag) {
    unsigned low = least[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) low = min(low, least[i]);
    atomicAdd(p.sum + (size_t)mt * gridDim.x + nt, (unsigned long long)low);
  }
  if (warp == 1) {
    if (*abort_flag && lane == 0) {
      atomicExch(p.status, kErrTimeout);
      umma_commit(mdone);  // MMAs still in flight finish before the TMEM is freed (bounded)
      long long w = 0;
      while (!mbar_try(mdone, 0) && ++w < kWaitLimit) {
      }
    }
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  }
}

// Sum of the splits' partial products (in their order) for the tiles that were computed here.
__global__ void __launch_bounds__(256) i8_reduce_kernel(const I8Params p, int splits, double *C, long long c_rs, long long c_cs) {
  const long long total = (long long)p.M * p.N;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
    const int r = (int)(i / p.N), c = (int)(i - (long long)r * p.N);
    if ((p.upper && c < r) || p.sum[(size_t)(r >> 7) * ((p.N + 127) >> 7) + (c >> 7)] < p.need) continue;
    double v = 0.0;
    for (int z = 0; z < splits; ++z) v += p.C[z * p.c_zs + i];
    C[r * c_rs + c * c_cs] = v;
  }
}

// ------------------------------------------------------------------------------ digits

// Exponent for a largest magnitude mx: |x| 2^-e <= 0.98 (the leading digit stays within int8), and whether
// the row can be split at all.
__device__ __forceinline__ bool digit_exponent(double mx, int &e) {
  e = 0;
  if (!(mx < 1e300)) return false;
  if (mx == 0.0) return true;
  int ex;
  const double f = frexp(mx, &ex);
  e = f > 0.98 ? ex + 1 : ex;
  if (e > 400 || e < -400) {
    e = 0;
    return false;
  }
  return true;
}

// Digits of four entries, plane p's four bytes in w[p]; scale = 2^(55 - e).  With 128 added to each of the
// six lower digits' places, the digits are the bytes less 128.  The leading bits of the magnitudes go to w[7].
__device__ __forceinline__ void digits4(const double *x, double scale, uint32_t *w) {
  uint32_t lo[4], hi[4];
  w[7] = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long z = __double2ll_rn(x[i] * scale), y = z + 0x808080808080LL;
    w[7] |= (uint32_t)((unsigned long long)(z < 0 ? -z : z) >> 48) << (8 * i);
    lo[i] = (uint32_t)y;
    hi[i] = (uint32_t)((unsigned long long)y >> 32);
  }
  const uint32_t a = __byte_perm(lo[0], lo[1], 0x5140), b = __byte_perm(lo[2], lo[3], 0x5140);
  const uint32_t c = __byte_perm(lo[0], lo[1], 0x7362), d = __byte_perm(lo[2], lo[3], 0x7362);
  w[6] = __byte_perm(a, b, 0x5410) ^ 0x80808080u;
  w[5] = __byte_perm(a, b, 0x7632) ^ 0x80808080u;
  w[4] = __byte_perm(c, d, 0x5410) ^ 0x80808080u;
  w[3] = __byte_perm(c, d, 0x7632) ^ 0x80808080u;
  const uint32_t f = __byte_perm(hi[0], hi[1], 0x5140), g = __byte_perm(hi[2], hi[3], 0x5140);
  w[2] = __byte_perm(f, g, 0x5410) ^ 0x80808080u;
  w[1] = __byte_perm(f, g, 0x7632) ^ 0x80808080u;
  w[0] = __byte_perm(__byte_perm(hi[0], hi[1], 0x0062), __byte_perm(hi[2], hi[3], 0x0062), 0x5410);
}

// Digits of eight consecutive entries, stored to the planes at dst (8-byte aligned).
__device__ __forceinline__ void store_digits8(const double *x, double scale, int8_t *dst, long long ps) {
  uint32_t u[kPlanes], v[kPlanes];
  digits4(x, scale, u);
  digits4(x + 4, scale, v);
#pragma unroll
  for (int p = 0; p < kPlanes; ++p) *(uint2 *)(dst + p * ps) = make_uint2(u[p], v[p]);
}

__device__ __forceinline__ void max_ratio(float *slot, float r) {  // r >= 0: ordered as integers
  atomicMax((int *)slot, __float_as_int(r));
}

// Rows with K contiguous: one CTA per row.  The first read gives the largest entry and the row's rms, so a
// row that fails (*) by itself (the other side's ratio is at least 1) costs no more than that read.  Rows
// of up to kRowKeep entries stay in shared memory for the digits; longer ones are read again, from L2.
constexpr int kRowKeep = 6144;
__device__ __forceinline__ int row_slot(long long k) { return (int)(k + (k >> 3)); }  // 8 apart: distinct banks
__global__ void __launch_bounds__(256)
    i8_split_rows_kernel(const double *__restrict__ src, long long ld, long long rows, long long K, float lim,
                         int8_t *__restrict__ dst, long long pld, long long ps, int *__restrict__ ex, float *ratio) {
  __shared__ double red[16];
  extern __shared__ double keep[];
  const bool resident = pld <= kRowKeep;
  const long long r = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double *row = src + r * ld;
  double mx = 0.0, sq = 0.0;
  bool nan = false;
  if (r < rows) {
#pragma unroll 8
    for (long long k = tid; k < K; k += 256) {
      const double x = row[k], v = fabs(x);
      if (resident) keep[row_slot(k)] = x;
      nan |= v != v;
      mx = fmax(mx, v);
      sq += v * v;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    sq += __shfl_xor_sync(0xffffffffu, sq, o);
  }
  if (lane == 0) {
    red[warp] = mx;
    red[8 + warp] = sq;
  }
  const bool any_nan = __syncthreads_or(nan);
  mx = red[0];
  sq = red[8];
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    mx = fmax(mx, red[i]);
    sq += red[8 + i];
  }
  int e;
  const bool ok = digit_exponent(mx, e) && !any_nan;  // |e| <= 400: the squares stay in range
  const float rr = !ok ? INFINITY : mx == 0.0 ? 0.f : (float)(ldexp(1.0, e) / sqrt(sq / (double)K));
  if (r < rows && tid == 0) {
    ex[r] = mx == 0.0 ? kZeroRow : e;
    max_ratio(ratio + (r >> 7), rr);
  }
  if (!(rr <= lim)) return;
  const double scale = ldexp(1.0, 55 - e);
  int8_t *out = dst + r * pld;
  for (long long k0 = 8LL * tid; k0 < pld; k0 += 8 * 256) {
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      x[i] = (r < rows && k0 + i < K) ? (resident ? keep[row_slot(k0 + i)] : row[k0 + i]) : 0.0;
    store_digits8(x, scale, out + k0, ps);
  }
}

// Columns of a K x cols matrix (cols contiguous), `per` of the K rows per blockIdx.y: largest magnitudes as
// bit patterns (a NaN orders above infinity), and partial sums of the squares.
__global__ void __launch_bounds__(256)
    i8_colmax_kernel(const double *__restrict__ src, long long ld, long long K, long long cols, long long per,
                     unsigned long long *mx, double *__restrict__ sq) {
  __shared__ unsigned long long red[8][33];
  __shared__ double sum[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const long long c = blockIdx.x * 32LL + tx, k0 = blockIdx.y * per, k1 = min(K, k0 + per);
  unsigned long long m = 0;
  double s = 0.0;
  if (c < cols) {
#pragma unroll 8
    for (long long k = k0 + ty; k < k1; k += 8) {
      const double v = fabs(src[k * ld + c]);
      m = max(m, (unsigned long long)__double_as_longlong(v));
      s += v * v;
    }
  }
  red[ty][tx] = m;
  sum[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c < cols) {
#pragma unroll
    for (int i = 1; i < 8; ++i) {
      m = max(m, red[i][tx]);
      s += sum[i][tx];
    }
    atomicMax(mx + c, m);
    sq[blockIdx.y * cols + c] = s;
  }
}

// Exponents and ratios; the sums in a fixed order, so that the same input always takes the same path.
__global__ void i8_colexp_kernel(const unsigned long long *__restrict__ mx, const double *__restrict__ sqp, int nb,
                                 long long cols, double K, int *__restrict__ ex, float *ratio) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= cols) return;
  double sq = 0.0;
  for (int b = 0; b < nb; ++b) sq += sqp[b * cols + c];
  int e;
  const bool ok = digit_exponent(__longlong_as_double((long long)mx[c]), e);
  ex[c] = mx[c] == 0 ? kZeroRow : e;
  max_ratio(ratio + (c >> 7), !ok ? INFINITY : mx[c] == 0 ? 0.f : (float)(ldexp(1.0, e) / sqrt(sq / K)));
}

// Digits of the columns, K contiguous: 64 (k) x 32 (column) tiles; nothing for columns whose 128 fail (*).
__global__ void __launch_bounds__(256)
    i8_split_cols_kernel(const double *__restrict__ src, long long ld, long long K, long long cols,
                         const int *__restrict__ ex, const float *__restrict__ ratio, float lim,
                         int8_t *__restrict__ dst, long long pld, long long ps) {
  __shared__ double tile[64][33];
  const long long k0 = blockIdx.x * 64LL, c0 = blockIdx.y * 32LL;
  if (!(ratio[c0 >> 7] <= lim)) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int j = ty; j < 64; j += 8) {
    const long long k = k0 + j, c = c0 + tx;
    tile[j][tx] = (k < K && c < cols) ? src[k * ld + c] : 0.0;
  }
  __syncthreads();
  const int cl = threadIdx.x >> 3, seg = threadIdx.x & 7;
  const long long c = c0 + cl;
  const int e = c < cols ? ex[c] : 0;
  const double scale = ldexp(1.0, 55 - (e == kZeroRow ? 0 : e));
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = tile[8 * seg + i][cl];
  store_digits8(x, scale, dst + c * pld + k0 + 8 * seg, ps);  // rows padded to 128
}

// ------------------------------------------------------------------------------ host side
struct Digits {
  DBuf<int8_t> buf;
  DBuf<int> ex;
  DBuf<float> ratio;  // per 128 rows
  long long ld = 0, ps = 0, rows = 0;
};

long long pad128(long long x) { return (x + 127) / 128 * 128; }

// Digits of `rows` vectors of length K: row r at src + r ld (kc) or column r of a K x rows matrix.
void make_digits(Digits &d, const double *src, long long ld, long long rows, long long K, bool kc, float lim, cudaStream_t st) {
  const long long rp = pad128(rows);
  d.rows = rows;
  d.ld = (K + 63) / 64 * 64;
  d.ps = rp * d.ld;
  d.buf.ensure((size_t)kPlanes * d.ps);
  d.ex.ensure(rp);
  d.ratio.ensure(rp / 128);
  CK(cudaMemsetAsync(d.ratio.p, 0, rp / 128 * sizeof(float), st));
  if (kc) {
    const size_t keep = d.ld <= kRowKeep ? (size_t)(d.ld + d.ld / 8) * sizeof(double) : 0;
    CK(cudaFuncSetAttribute(i8_split_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            kRowKeep / 8 * 9 * (int)sizeof(double)));
    i8_split_rows_kernel<<<(unsigned)rp, 256, keep, st>>>(src, ld, rows, K, lim, d.buf.p, d.ld, d.ps, d.ex.p,
                                                         d.ratio.p);
    KLAUNCHED();
    return;
  }
  const long long cx = (rows + 31) / 32, want = 8LL * Runtime::get().num_sms;
  const long long cy = std::max<long long>(1, std::min<long long>((K + 63) / 64, want / cx + 1)), per = (K + cy - 1) / cy;
  DBuf<unsigned long long> mx(rows);
  DBuf<double> sq((size_t)cy * rows);
  CK(cudaMemsetAsync(mx.p, 0, rows * sizeof(unsigned long long), st));
  i8_colmax_kernel<<<dim3((unsigned)cx, (unsigned)cy), 256, 0, st>>>(src, ld, K, rows, per, mx.p, sq.p);
  KLAUNCHED();
  i8_colexp_kernel<<<(unsigned)((rows + 63) / 64), 64, 0, st>>>(mx.p, sq.p, (int)cy, rows, (double)K, d.ex.p, d.ratio.p);
  KLAUNCHED();
  i8_split_cols_kernel<<<dim3((unsigned)(d.ld / 64), (unsigned)(rp / 32)), 256, 0, st>>>(
      src, ld, K, rows, d.ex.p, d.ratio.p, lim, d.buf.p, d.ld, d.ps);
  KLAUNCHED();
}

CUtensorMap digit_map(const Digits &d) {
  typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                               const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static EncodeFn fn = [] {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q));
    if (!ptr || q != cudaDriverEntryPointSuccess) fail(kErrCuda, "cuTensorMapEncodeTiled unavailable");
    return (EncodeFn)ptr;
  }();
  CUtensorMap m;
  memset(&m, 0, sizeof(m));
  // the padding rows and columns are stored (zero digits), so every box lies inside
  cuuint64_t dims[3] = {(cuuint64_t)d.ld, (cuuint64_t)pad128(d.rows), (cuuint64_t)kPlanes};
  cuuint64_t strides[2] = {(cuuint64_t)d.ld, (cuuint64_t)d.ps};
  cuuint32_t box[3] = {kBk, kTile, 1}, es[3] = {1, 1, 1};
  const CUresult r = fn(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void *)d.buf.p, dims, strides, box, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(kErrCuda, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return m;
}

bool i8_off() {
  const char *e = getenv("ISVD_GPU_FP64_INT8");
  return e && atoi(e) == 0;
}

// Seconds of the int8 products with K in `splits` parts: 28 of whole tiles, one CTA per SM (14 bf16
// equivalents at about 1.4 PFLOP/s over 148 CTAs), and the partial products' traffic.
double i8_gemm_time(double M, double N, double K, bool upper, int splits) {
  const double waves = std::ceil(std::ceil(M / 128) * std::ceil(N / 128) * (upper ? 0.55 : 1.0) * splits / 148);
  return waves * 148 * 2.0 * 128 * 128 * (K / splits) * 14.0 / 1.4e15 +
         (splits > 1 ? (splits + 1) * M * N * 8.0 / 4e12 + 5e-6 : 0.0);
}
int i8_splits(double M, double N, double K, bool upper) {
  int best = 1;
  for (int s = 2; s <= 8 && K / s >= 1024; ++s)
    if (i8_gemm_time(M, N, K, upper, s) < 0.95 * i8_gemm_time(M, N, K, upper, best)) best = s;
  return best;
}

// Either path's time: 26 TFLOP/s on mma.sync f64; here also 24 bytes per split element at about 4 TB/s, and
// 60 us of launches.
bool i8_pays(double M, double N, double K, bool same, bool upper) {
  const double dmma = (upper ? 0.55 : 1.0) * 2.0 * M * N * K / 26e12;
  const double i8 = i8_gemm_time(M, N, K, upper, i8_splits(M, N, K, upper)) + (same ? M : M + N) * K * 24.0 / 4e12 + 60e-6;
  return i8 < 0.8 * dmma;
}

}  // namespace

bool f64_int8_pays(double M, double N, double K, bool gram) {
  return !i8_off() && Runtime::get().cc_major == 10 && K >= 640 && M >= 64 && N >= 64 && i8_pays(M, N, K, gram, gram);
}

bool gemm_f64_int8(const Gemm<double, double> &g, bool a_kc, bool b_nc, cudaStream_t st) {
  if (g.batch != 1 || g.beta != 0.0 || g.pl_t || g.splits > 1 || i8_off() || Runtime::get().cc_major != 10) return false;
  if (g.K < 640 || g.M < 64 || g.N < 64 || g.N > (1 << 20)) return false;
  const bool same = g.A == g.B && !a_kc && b_nc && g.a_cs == g.b_rs && g.M == g.N;
  if (g.upper && !same) return false;
  if (!i8_pays(g.M, g.N, g.K, same, g.upper)) return false;
  cudaStreamCaptureStatus cap_st;
  CK(cudaStreamIsCapturing(st, &cap_st));
  if (cap_st != cudaStreamCaptureStatusNone) return false;  // the digits' buffers live for this call only
  long long cap = 4LL << 30;
  if (isvd_gpu_memory_limit > 0)
    cap = std::max<long long>(32LL << 20, std::min<long long>(cap, (long long)(isvd_gpu_memory_limit / 16)));
  const long long ld = (g.K + 63) / 64 * 64, per = kPlanes * ld;
  // rows of A at a time (a multiple of 128); the digits of B (or of A = B') are held whole
  const long long step = same ? g.M : std::min<long long>(g.M, std::max<long long>(128, cap / per / 128 * 128));
  if (per * pad128(g.N) > 3 * cap) return false;
  const float lim = (float)(2.5 * std::sqrt((double)g.K));
  Digits da, db;
  DBuf<unsigned long long> sum;
  try {
    make_digits(db, g.B, b_nc ? g.b_rs : g.b_cs, g.N, g.K, !b_nc, lim, st);
    CK(cudaFuncSetAttribute(i8_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kI8Smem));
    const CUtensorMap mb = digit_map(db);
    for (long long r0 = 0; r0 < g.M; r0 += step) {
      const int rows = (int)std::min<long long>(step, g.M - r0);
      Digits &d = same ? db : da;
      if (!same) make_digits(da, g.A + r0 * (a_kc ? g.a_rs : 1), a_kc ? g.a_rs : g.a_cs, rows, g.K, a_kc, lim, st);
      I8Params p;
      const int splits = i8_splits(rows, g.N, g.K, g.upper);
      double *const C = g.C + r0 * g.c_rs;
      DBuf<double> part;
      p.M = rows; p.N = g.N; p.nkb = (int)(ld / kBk);
      p.per = (p.nkb + splits - 1) / splits;
      p.C = C; p.c_rs = g.c_rs; p.c_cs = g.c_cs; p.c_zs = 0;
      const int nz = (p.nkb + p.per - 1) / p.per;  // no empty split
      if (nz > 1) {
        part.alloc((size_t)nz * rows * g.N);
        p.C = part.p; p.c_rs = g.N; p.c_cs = 1; p.c_zs = (long long)rows * g.N;
      }
      p.alpha = g.alpha;
      p.upper = g.upper ? 1 : 0;
      p.ea = d.ex.p; p.eb = db.ex.p; p.ra = d.ratio.p; p.rb = db.ratio.p;
      p.lim = lim;
      const dim3 grid((g.N + kTile - 1) / kTile, (rows + kTile - 1) / kTile, nz);
      const size_t tiles = (size_t)grid.x * grid.y;
      sum.ensure(tiles);
      CK(cudaMemsetAsync(sum.p, 0, tiles * sizeof(unsigned long long), st));
      p.sum = sum.p;
      p.need = (unsigned long long)std::ceil(0.2 * std::sqrt((double)g.K) * 16384.0);
      p.status = g.status ? g.status : reinterpret_cast<int *>(Runtime::get().ctl + 16);  // the stages' status word
      i8_gemm_kernel<<<grid, kI8Threads, kI8Smem, st>>>(digit_map(d), mb, p);
      KLAUNCHED();
      inject_timeout("int8", p.status, st);
      if (nz > 1) {
        const int blocks = (int)std::min<long long>(((long long)rows * g.N + 255) / 256, 16LL * Runtime::get().num_sms);
        i8_reduce_kernel<<<blocks, 256, 0, st>>>(p, nz, C, g.c_rs, g.c_cs);
        KLAUNCHED();
      }
      Gemm<double, double> f = g;  // the tiles that fail (*) or (**)
      f.M = rows;
      f.A = g.A + r0 * (a_kc ? g.a_rs : 1);
      f.C = C;
      dmma_gemm_rest(f, a_kc, b_nc, sum.p, p.need, st);
    }
    return true;
  } catch (const Error &e) {
    if (e.code != kErrMemory) throw;
    return false;  // no room for the digits: the caller computes all of C
  }
}

}  // namespace isvdb
