// Kolmogorov-Nagumo l x l step (reference @x@_integrate_kolmogorov_nagumo.c:184-226) on one
// thread-block cluster.
//
// With g(z) = 1/2 + (1/4 - z)^(1/2) = 1 - sum_{n>=1} Cat(n-1) z^n (Cat: Catalan numbers), the step
// needs C = g(Z)^(1/2) and C^-1 = g(Z)^(-1/2) for Z = Dgc - Dc Dc.  Both are power series in Z with
// radius of convergence 1/4 (coefficients from J. C. P. Miller's recurrence for powers of a
// series).  When rho >= ||4 Z||_2 is small, as in all but the first iterations, a series of degree
// d evaluated by the Paterson-Stockmeyer scheme (powers Z^2..Z^s by doubling, then Horner in Z^s)
// needs ceil(log2 s) + d / s dependent products, against about twenty for two coupled
// Newton-Schulz square roots; d is the smallest degree whose tail bound
// sum_{n>d} max(|c_n|, |d_n|) (rho / 4)^n is below the target.  When no degree up to the table
// size reaches it (rho close to 1), the step runs the Newton-Schulz iteration instead.
//
// The cost of the step is the chain of dependent l x l products and the barriers between them, not
// their flops (2 l^3 = 4 MFLOP at l = 128).  Every matrix of the chain is a polynomial in the
// symmetric Z, so the chain is cut by rows (kn_rows_kernel, l <= 128): a CTA of the cluster owns
// eight (or more) rows of every matrix in shared memory and holds one whole right operand (Z, then
// Z^4 or Z^8, then Dc) beside them.  A product of its rows with the whole operand is then local to
// the CTA, a __syncthreads() apart from the next one; only a new right operand is exchanged (rows
// written to L2, one hardware cluster barrier, read back whole).  A step near convergence makes two
// such exchanges where the tile-split form below made one per product.  l in (128, 160] keeps that
// form (kn_cluster_kernel): the whole operand and the rows do not fit in shared memory together.
// Every CTA follows the same control flow (decisions come from values that all CTAs compute alike),
// and there is no software spin-wait.
//
// What bounds a step: at l = 128 a CTA's product of eight rows, 2000 cycles of the SM's FP64 pipe (66
// FMA per cycle); at l <= 32 the latency of a product (about 0.3 us) and of the two exchanges (2 us
// each).  Measured per step, the first step of a loop / one near convergence, tile-split form ->
// rows: l = 11 107 / 29 -> 24 / 11 us, l = 32 341 / 34 -> 28 / 12, l = 65 548 / 42 -> 59 / 17,
// l = 96 593 / 45 -> 80 / 21, l = 128 649 / 48 -> 141 / 28 (the first steps took Newton-Schulz for
// want of the sharper bound on ||4 Z||_2 below and of a table of 128 coefficients).  Clusters of
// fewer, longer row blocks are slower: l = 96 near convergence 27 us on 8 CTAs, 34 on 4.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "kn_common.cuh"
#include "pdl.cuh"
#include "rows.cuh"
#include "runtime.h"

namespace cg = cooperative_groups;

namespace isvdb {
namespace {

constexpr int kKsThreads = 1024;  // one output of a 32 x 32 tile per thread
constexpr int kKsMaxL = 160;
// shared-memory row strides of the A tile (32 x l) and the B tile (l x 32), both 4 (mod 16) doubles:
// the mma.sync fragment reads (8 rows x 4 inner indices, or 4 x 8) hit 16 distinct bank pairs
constexpr int kAld = kKsMaxL + 4;
constexpr int kBld = 36;
constexpr int kKsPer = (32 * kKsMaxL + kKsThreads - 1) / kKsThreads;

struct Ks {
  int l, nr, cs, rank;
  double *As, *Bs, *part;
};

// C = alpha A B + beta Cin + diag I on the 32 x 32 output tiles [tile_begin, tile_end) of a phase
// (tiles numbered across the products of the phase); CTA r takes the tiles t = r mod cs.
// Row-major l x l operands; every load goes through L2 (__ldcg), as they are written by other CTAs.
// Tile product on the FP64 tensor-core path (mma.sync m8n8k4 f64): 16 tiles of 8 x 8, two warps
// per tile (halves of the inner dimension, zero-padded to a multiple of 4); the halves' partial
// sums meet in shared memory and are added in a fixed order.
// C2, C3 (optional) receive copies of C.
__device__ void ks_mm(const Ks &k, int tile_begin, int tile_end, double alpha, const double *A, const double *B,
                      double beta, const double *Cin, double diag, double *C, double *C2 = nullptr,
                      double *C3 = nullptr) {
  const int l = k.l, tid = threadIdx.x;
  const int ty = tid >> 5, tx = tid & 31;  // output (ty, tx) of the tile in the epilogue
  const int lane = tid & 31, half = ty >> 4, mt = ty & 15, ti = mt >> 2, tj = mt & 3;  // warp: 8 x 8 tile, half
  const int l4 = (l + 3) & ~3, kh = ((l4 >> 1) + 3) & ~3;
  const int kb = half * kh, ke = min(l4, kb + kh);
  const int first = tile_begin + (((k.rank - tile_begin) % k.cs) + k.cs) % k.cs;
  for (int t = first; t < tile_end; t += k.cs) {
    const int tt = t - tile_begin;
    const int i0 = (tt / k.nr) * 32, j0 = (tt % k.nr) * 32;
    const int i = i0 + ty, j = j0 + tx;
    const double cin = (beta != 0.0 && i < l && j < l) ? __ldcg(Cin + (size_t)i * l + j) : 0.0;
    double ra[kKsPer], rb[kKsPer];
#pragma unroll
    for (int u = 0; u < kKsPer; ++u) {
      const int e = tid + u * kKsThreads;
      const int r = e / l, kk = e - r * l;  // A tile: 32 rows x l
      ra[u] = (e < 32 * l && i0 + r < l) ? __ldcg(A + (size_t)(i0 + r) * l + kk) : 0.0;
      const int kr = e >> 5, cb = e & 31;   // B tile: l rows x 32
      rb[u] = (e < 32 * l && j0 + cb < l) ? __ldcg(B + (size_t)kr * l + j0 + cb) : 0.0;
    }
    __syncthreads();  // the previous tile's shared memory reads are done
#pragma unroll
    for (int u = 0; u < kKsPer; ++u) {
      const int e = tid + u * kKsThreads;
      if (e < 32 * l) {
        const int r = e / l, kk = e - r * l;
        k.As[r * kAld + kk] = ra[u];
        k.Bs[(e >> 5) * kBld + (e & 31)] = rb[u];
      }
    }
    for (int e = tid; e < 32 * 4; e += kKsThreads) {  // zero the inner-dimension padding [l, l4)
      const int r = e >> 2, kk = l + (e & 3);
      if (kk < l4) {
        k.As[r * kAld + kk] = 0.0;
        k.Bs[kk * kBld + r] = 0.0;
      }
    }
    __syncthreads();
    double d[2] = {0.0, 0.0};
    const double *ap = k.As + (ti * 8 + (lane >> 2)) * kAld + (lane & 3);
    const double *bq = k.Bs + (lane & 3) * kBld + tj * 8 + (lane >> 2);
    for (int kk = kb; kk < ke; kk += 4)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                   : "+d"(d[0]), "+d"(d[1])
                   : "d"(ap[kk]), "d"(bq[kk * kBld]));
    double *part = k.part + half * 1024;  // 32 x 32 partial sums of this half
    const int orow = ti * 8 + (lane >> 2), ocol = tj * 8 + 2 * (lane & 3);
    part[orow * 32 + ocol] = d[0];
    part[orow * 32 + ocol + 1] = d[1];
    __syncthreads();
    const int o = ty * 32 + tx;
    const double acc = k.part[o] + k.part[1024 + o];
    if (i < l && j < l) {
      const double v = alpha * acc + beta * cin + (i == j ? diag : 0.0);
      C[(size_t)i * l + j] = v;
      if (C2) C2[(size_t)i * l + j] = v;
      if (C3) C3[(size_t)i * l + j] = v;
    }
  }
}

// Block-wide sum or max; every thread gets the result.
__device__ double ks_block_reduce(double v, bool is_max, double *red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, w) : v + w;
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = red[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) s = is_max ? fmax(s, red[i]) : s + red[i];
  return s;
}

// Cluster-wide sum: every CTA adds its value into partial slot base + rank, the cluster
// synchronises, and each CTA sums the slots in rank order (the same value in every CTA).
__device__ double ks_cluster_sum(const Ks &k, cg::cluster_group &cluster, double v, double *slots, double *red) {
  v = ks_block_reduce(v, false, red);
  if (threadIdx.x == 0) slots[k.rank] = v;
  cluster.sync();
  double s = 0.0;
  for (int r = 0; r < k.cs; ++r) s += __ldcg(slots + r);
  return s;
}

// Series degree for rho >= ||4 Z||_2: the smallest d whose tail bound
//   tail(d) = sum_{d < n < 32 PER} max(|c_n|, |d_n|) (rho / 4)^n + (table remainder)
// is below the target, or -1 (the remainder beyond the table is bounded by the last term times
// rho / (1 - rho)).  Evaluated by one warp: lane j holds the terms PER j .. PER j + PER - 1, suffix
// sums by shuffles, and tail is decreasing in d, so the degree is the first d whose bound passes.
template <int PER>
__device__ int ks_degree_warp(const KnSeries &ser, double rho, double target) {
  if (!(rho < 0.9)) return -1;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, n0 = PER * lane;
  const double x = 0.25 * rho;
  double xn = 1.0, b = x;  // x^(PER lane) by repeated squaring
  for (int e = n0; e; e >>= 1, b *= b)
    if (e & 1) xn *= b;
  double t[PER], sum = 0.0;
#pragma unroll
  for (int u = 0; u < PER; ++u, xn *= x) {
    t[u] = fmax(fabs(ser.c[n0 + u]), fabs(ser.d[n0 + u])) * xn;
    sum += t[u];
  }
  const double rem = __shfl_sync(full, t[PER - 1], 31) * rho / (1.0 - rho);
  if (rem > target) return -1;
  double suf = sum;  // sum of the terms of lanes lane..31
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_down_sync(full, suf, o);
    if (lane + o < 32) suf += v;
  }
  const double after = __shfl_down_sync(full, suf, 1);  // terms of lanes lane+1..31
  double tail = rem + (lane < 31 ? after : 0.0);        // d = n0 + PER - 1
  int d = PER * 32;
#pragma unroll
  for (int u = PER - 1; u >= 0; --u) {
    const unsigned ok = __ballot_sync(full, tail <= target);
    if (ok) d = min(d, PER * (__ffs(ok) - 1) + u);
    tail += t[u];
  }
  return min(d, PER * 32 - 1);
}

// Block size s of the Paterson-Stockmeyer scheme: fewest dependent products, then the smallest.
__device__ int ks_block_size(int deg) {
  if (deg < 1) return 1;
  int sb = 1, best = 1 << 30;
  for (int cand = 1; cand <= 8; ++cand) {
    int lg = 0;
    while ((1 << lg) < cand) ++lg;
    const int cost = lg + deg / cand;
    if (cost < best) { best = cost; sb = cand; }
  }
  if (deg / sb > 7) sb = 8;  // at most 8 blocks B_0..B_7
  return sb;
}

__global__ void __launch_bounds__(kKsThreads, 1) kn_cluster_kernel(KnStep a, KnSeries ser) {
  extern __shared__ double sm[];
  __shared__ double red[kKsThreads / 32];
  __shared__ int plan[3];  // degree (-1: Newton-Schulz), block size, Newton-Schulz steps
  cg::cluster_group cluster = cg::this_cluster();
  const int l = a.l;
  const size_t ll = (size_t)l * l;
  Ks k{l, (l + 31) / 32, (int)cluster.num_blocks(), (int)cluster.block_rank(), sm, sm + 32 * kAld,
         sm + 32 * kAld + (kKsMaxL + 4) * kBld};
  const int nt = k.nr * k.nr;
  const int gtid = k.rank * kKsThreads + threadIdx.x, gstride = k.cs * kKsThreads;
  // work: Z | P_1..P_8 | accC x2 | accCi x2 | BC_0..BC_7 | BI_0..BI_7 (Newton-Schulz: P_1..P_5), then
  // partial sums of the cluster reductions (3 x 16 slots)
  double *Zm = a.work, *P = Zm + ll, *AC = P + 8 * ll, *AI = AC + 2 * ll, *BC = AI + 2 * ll, *BI = BC + 8 * ll;
  double *slots = a.work + (size_t)kKnWorkMatrices * ll;

  ks_mm(k, 0, nt, -1.0, a.Dc, a.Dc, 1.0, a.Dgc, 0.0, Zm);  // Z = Dgc - Dc Dc (:184-190)
  cluster.sync();
  // P_1 = Zsym from the upper triangle (as syev 'U' reads Z); rho = ||4 Zsym||_F >= ||4 Z||_2
  double f = 0.0;
  for (int e = gtid; e < (int)ll; e += gstride) {
    const int i = e / l, j = e - i * l;
    const double z = __ldcg(Zm + (size_t)min(i, j) * l + max(i, j));
    P[e] = z;
    f += 16.0 * z * z;
  }
  const double rho = sqrt(ks_cluster_sum(k, cluster, f, slots, red));
  if (threadIdx.x < 32) {
    const int d = ks_degree_warp<2>(ser, rho, a.ns_target);  // blocks B_0..B_7: degree < 64
    if (threadIdx.x == 0) {
      plan[0] = d;
      plan[1] = ks_block_size(d);
      plan[2] = d < 0 ? kn_ns_steps(rho, a.ns_target) : 0;
    }
  }
  __syncthreads();
  const int deg = plan[0];
  const double *C, *Ci;
  if (deg >= 0) {
    const int sb = plan[1];
    for (int h = 1; h < sb; h *= 2) {  // P_j = P_h P_(j-h), h < j <= min(2h, sb)
      const int hi = min(2 * h, sb);
      for (int j = h + 1; j <= hi; ++j) {
        const int slot = j - h - 1;
        ks_mm(k, slot * nt, (slot + 1) * nt, 1.0, P + (h - 1) * ll, P + (j - h - 1) * ll, 0.0, nullptr, 0.0,
              P + (j - 1) * ll);
      }
      cluster.sync();
    }
    // Paterson-Stockmeyer: B_b = sum_{t<sb} coef[b sb + t] Z^t (b = 0..q); acc = B_q; acc = acc Z^sb + B_b
    const int q = deg / sb;
    for (int e = gtid; e < (int)ll; e += gstride) {
      const int i = e / l, j = e - i * l;
      for (int b = 0; b <= q; ++b) {
        double vc = (i == j) ? ser.c[b * sb] : 0.0, vd = (i == j) ? ser.d[b * sb] : 0.0;
        for (int t = 1; t < sb && b * sb + t <= deg; ++t) {
          const double p = __ldcg(P + (t - 1) * ll + e);
          vc += ser.c[b * sb + t] * p;
          vd += ser.d[b * sb + t] * p;
        }
        BC[b * ll + e] = vc;
        BI[b * ll + e] = vd;
      }
    }
    cluster.sync();
    const double *accC = BC + q * ll, *accI = BI + q * ll;
    int cur = 0;
    for (int b = q - 1; b >= 0; --b) {
      ks_mm(k, 0, nt, 1.0, accC, P + (sb - 1) * ll, 1.0, BC + b * ll, 0.0, AC + cur * ll);
      ks_mm(k, nt, 2 * nt, 1.0, accI, P + (sb - 1) * ll, 1.0, BI + b * ll, 0.0, AI + cur * ll);
      cluster.sync();
      accC = AC + cur * ll;
      accI = AI + cur * ll;
      cur = 1 - cur;
    }
    C = accC;
    Ci = accI;
  } else {
    // Two coupled Newton-Schulz square roots (Higham, Functions of Matrices, eq. 6.35):
    //   T = Q Y;  Y <- Y (3I - T)/2;  Q <- (3I - T) Q / 2   ->  Y -> X^(1/2), Q -> X^(-1/2),
    // first of X = I - 4 Zsym (sqrt(I/4 - Z) = Y/2), then of P = I/2 + Y/2.
    double *Y = P, *Yn = P + ll, *Q = P + 2 * ll, *Qn = P + 3 * ll, *T = P + 4 * ll;
    for (int e = gtid; e < (int)ll; e += gstride) {
      const int i = e / l, j = e - i * l;
      Y[e] = (i == j ? 1.0 : 0.0) - 4.0 * __ldcg(P + e);  // Y is P_1: each entry read, then written
      Q[e] = (i == j ? 1.0 : 0.0);
    }
    cluster.sync();
    int steps = plan[2];
    for (int stage = 0; stage < 2; ++stage) {
      for (int it = 0; it < steps; ++it) {
        ks_mm(k, 0, nt, 1.0, Q, Y, 0.0, nullptr, 0.0, T);
        cluster.sync();
        ks_mm(k, 0, nt, -0.5, Y, T, 1.5, Y, 0.0, Yn);
        ks_mm(k, nt, 2 * nt, -0.5, T, Q, 1.5, Q, 0.0, Qn);
        cluster.sync();
        double *t1 = Y; Y = Yn; Yn = t1;
        double *t2 = Q; Q = Qn; Qn = t2;
      }
      if (stage == 0) {
        double d2 = 0.0;
        for (int e = gtid; e < (int)ll; e += gstride) {
          const int i = e / l, j = e - i * l;
          const double pv = 0.5 * __ldcg(Y + e) + (i == j ? 0.5 : 0.0);
          Yn[e] = pv;
          Qn[e] = (i == j ? 1.0 : 0.0);
          const double d = (i == j ? 1.0 : 0.0) - pv;
          d2 += d * d;
        }
        steps = kn_ns_steps(fmin(sqrt(ks_cluster_sum(k, cluster, d2, slots + 16, red)), 0.5), a.ns_target);
        double *t1 = Y; Y = Yn; Yn = t1;
        double *t2 = Q; Q = Qn; Qn = t2;
      }
    }
    C = Y;
    Ci = Q;
  }
  // C, C^-1, F = C - Dc C^-1 (:218), the stacked copies, err = ||C - I||_F (:230-234)
  double e2 = 0.0;
  for (int e = gtid; e < (int)ll; e += gstride) {
    const int i = e / l, j = e - i * l;
    const double cv = __ldcg(C + e), ci = __ldcg(Ci + e);
    a.C[e] = cv;
    a.Cinv[e] = ci;
    if (a.fstack) {
      a.fstack[ll + e] = a.fstack_scale * ci;
      a.fstack[3 * ll + e] = ci;
    }
    const double d = cv - (i == j ? 1.0 : 0.0);
    e2 += d * d;
  }
  // F once, written to F and to both F slots of the stack
  ks_mm(k, 0, nt, -1.0, a.Dc, Ci, 1.0, C, 0.0, a.F, a.fstack, a.fstack ? a.fstack + 2 * ll : nullptr);
  const double err = sqrt(ks_cluster_sum(k, cluster, e2, slots + 32, red));
  if (k.rank == 0 && threadIdx.x == 0) {
    *a.err = err;
    if (!(err == err)) atomicExch(a.status, kErrNumerical);
  }
}

// ------------------------------------------------------------------------------------------
// The step cut by rows (rows.cuh).
constexpr int kKrBlocks = 8;       // Z, Z^2, Z^3, scratch, accumulators of C and C^-1 (two each)
constexpr int kKrBlocksWide = 12;  // Z .. Z^7, scratch and the accumulators: Horner steps of Z^8

// Degree of the series: at most kKrChain by the chain of powers Z^t = Z^(t-1) Z, each added to both
// sums as it comes (one product per degree, no exchange); above it by Horner steps in Z^4 (two
// products per four degrees after one exchange), above kKrSb8 in Z^8 where the blocks fit.  With
// rho >= ||4 Z||_2 from the Frobenius norm of Z above kKrRefine degrees, the norm of Z^4 gives the
// sharper rho = 4 ||Z^4||_F^(1/4) (Z is positive semidefinite), which cuts most degrees in half.
constexpr int kKrRefine = 7, kKrChain = 11, kKrSb8 = 31;

__device__ __forceinline__ void kn_rows_body(const KnStep &a, const KnSeries &ser, int blocks) {
  extern __shared__ double sm[];
  __shared__ double red[kKrWarps];
  __shared__ int plan[2];  // degree (-1: Newton-Schulz), Newton-Schulz steps
  cg::cluster_group cluster = cg::this_cluster();
  const int l = a.l, tid = threadIdx.x;
  const size_t ll = (size_t)l * l;
  Kr k;
  kr_init(k, l, (int)cluster.num_blocks(), (int)cluster.block_rank(), sm);
  const int ld = k.ld, r0 = k.r0, rows = 8 * k.mt;
  const bool wide = blocks >= kKrBlocksWide;
  // block 0: scratch; blocks 1 .. 3 (wide: 1 .. 7): powers of Z
  double *acc = k.block(blocks - 4), *acc2 = k.block(blocks - 2);  // C rows, then C^-1 rows
  const size_t accn = (size_t)k.rb * ld;
  // global: Z | Z^4 | Z^8 | Newton-Schulz Y, Q (two each); partial sums of the cluster reductions
  double *Zg = a.work, *P4g = Zg + ll, *P8g = P4g + ll, *NSg = P8g + ll;
  double *slots = a.work + (size_t)kKnWorkMatrices * ll;

  // entries of this CTA's rows: f(local row, column, row, column valid)
  auto each = [&](auto f) {
    for (int e = tid; e < rows * k.lr; e += kKrThreads) {
      const int i = e / k.lr, j = e - i * k.lr;
      f(i, j, r0 + i < l && j < l);
    }
  };
  auto publish = [&](const double *blkp, double *dst) {
    each([&](int i, int j, bool in) {
      if (in) dst[(size_t)(r0 + i) * l + j] = blkp[(size_t)i * ld + j];
    });
  };

  for (int e = tid; e < k.lr * ld; e += kKrThreads) k.full[e] = 0.0;
  __syncthreads();
  kr_load(k, a.Dc);
  __syncthreads();
  // Z = Dgc - Dc Dc (:184-190)
  kr_mm(k, k.full + (size_t)r0 * ld, [&](int i, int j, double v) {
    if (r0 + i < l && j < l) {
      const size_t e = (size_t)(r0 + i) * l + j;
      Zg[e] = __ldcg(a.Dgc + e) - v;
    }
  });
  cluster.sync();
  const double f1 = kr_load_sym(k, Zg);
  double rho = 4.0 * sqrt(kr_block_sum(f1, red));  // ||4 Z||_F >= ||4 Z||_2; also: `full` is complete
  auto decide = [&](double r) {
    __syncthreads();
    if (tid < 32) {
      const int d = ks_degree_warp<kSeriesLen / 32>(ser, r, a.ns_target);
      if (tid == 0) {
        plan[0] = d;
        plan[1] = d < 0 ? kn_ns_steps(r, a.ns_target) : 0;
      }
    }
    __syncthreads();
    return plan[0];
  };
  int deg = decide(rho);
  double *P1 = k.block(1);
  each([&](int i, int j, bool) { P1[(size_t)i * ld + j] = k.full[(size_t)(r0 + i) * ld + j]; });
  __syncthreads();
  int have = 1;  // powers of Z in blocks
  if (deg < 0 || deg > kKrRefine) {
    // Z^2, Z^3 in blocks 2 and 3, Z^4 in the scratch block
    double n4 = 0.0;
    for (int t = 2; t <= 4; ++t) {
      double *dst = k.block(t & 3);
      kr_mm(k, k.block(t - 1), [&](int i, int j, double v) {
        dst[(size_t)i * ld + j] = v;
        if (t == 4) {
          n4 += v * v;
          if (r0 + i < l && j < l) P4g[(size_t)(r0 + i) * l + j] = v;
        }
      });
      __syncthreads();
    }
    const double s4 = kr_cluster_sum(k, cluster, n4, slots, red);
    rho = fmin(rho, 4.0 * sqrt(sqrt(sqrt(s4))));
    deg = decide(rho);
    have = 4;
  }
  const double *C, *Ci;
  if (deg >= 0 && deg <= kKrChain) {
    const int h = min(have, deg);
    each([&](int i, int j, bool in) {
      const double dg = (in && r0 + i == j) ? 1.0 : 0.0;
      double vc = ser.c[0] * dg, vd = ser.d[0] * dg;
      for (int t = 1; t <= h; ++t) {
        const double p = k.block(t & 3)[(size_t)i * ld + j];
        vc += ser.c[t] * p;
        vd += ser.d[t] * p;
      }
      acc[(size_t)i * ld + j] = vc;
      acc[accn + (size_t)i * ld + j] = vd;
    });
    __syncthreads();
    for (int t = have + 1; t <= deg; ++t) {  // each thread adds to the entries of its own tiles
      double *dst = k.block(t & 3);
      const double ct = ser.c[t], dt = ser.d[t];
      kr_mm(k, k.block((t - 1) & 3), [&](int i, int j, double v) {
        const size_t e = (size_t)i * ld + j;
        dst[e] = v;
        acc[e] += ct * v;
        acc[accn + e] += dt * v;
      });
      __syncthreads();
    }
    C = acc;
    Ci = acc + accn;
  } else if (deg >= 0) {
    // Paterson-Stockmeyer: B_b = sum_{t<sb} coef[b sb + t] Z^t (b = 0..q); acc = B_q; acc = acc Z^sb + B_b
    kr_load(k, P4g);
    __syncthreads();
    int sb = 4;
    if (wide && deg > kKrSb8) {
      // Z^5, Z^6, Z^7 in their blocks (Z^4 moves to block 4 first), Z^8 published
      double *P4 = k.block(4);
      each([&](int i, int j, bool) { P4[(size_t)i * ld + j] = k.block(0)[(size_t)i * ld + j]; });
      __syncthreads();
      for (int t = 5; t <= 8; ++t) {
        double *dst = k.block(t & 7);
        kr_mm(k, k.block(t - 4), [&](int i, int j, double v) {
          dst[(size_t)i * ld + j] = v;
          if (t == 8 && r0 + i < l && j < l) P8g[(size_t)(r0 + i) * l + j] = v;
        });
      }
      cluster.sync();
      kr_load(k, P8g);
      __syncthreads();
      sb = 8;
    }
    const int q = deg / sb;
    auto coef_block = [&](int b, int i, int j, double &vc, double &vd) {
      const double dg = (r0 + i == j && j < l) ? 1.0 : 0.0;
      vc = ser.c[b * sb] * dg;
      vd = ser.d[b * sb] * dg;
      for (int t = 1; t < sb && b * sb + t <= deg; ++t) {
        const double p = k.block(t)[(size_t)i * ld + j];
        vc += ser.c[b * sb + t] * p;
        vd += ser.d[b * sb + t] * p;
      }
    };
    each([&](int i, int j, bool) {
      double vc, vd;
      coef_block(q, i, j, vc, vd);
      acc[(size_t)i * ld + j] = vc;
      acc[accn + (size_t)i * ld + j] = vd;
    });
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
    for (int b = q - 1; b >= 0; --b) {
      // both sums at once: tiles of the C rows, then of the C^-1 rows
      for (int t = warp; t < 2 * k.mt * k.nt; t += kKrWarps) {
        const int inv = t >= k.mt * k.nt, tt = t - inv * k.mt * k.nt;
        const int m0 = (tt / k.nt) * 8, n0 = (tt % k.nt) * 8;
        double d[2];
        kr_tile(k, acc + inv * accn + (size_t)m0 * ld, k.full + n0, d);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int i = m0 + (lane >> 2), j = n0 + 2 * (lane & 3) + u;
          double vc, vd;
          coef_block(b, i, j, vc, vd);
          acc2[inv * accn + (size_t)i * ld + j] = d[u] + (inv ? vd : vc);
        }
      }
      __syncthreads();
      double *t1 = acc; acc = acc2; acc2 = t1;
    }
    C = acc;
    Ci = acc + accn;
  } else {
    // Two coupled Newton-Schulz square roots (Higham, Functions of Matrices, eq. 6.35):
    //   Y <- (3 I - Y Q) Y / 2,  Q <- (3 I - Q Y) Q / 2   ->  Y -> X^(1/2), Q -> X^(-1/2),
    // first of X = I - 4 Z (sqrt(I/4 - Z) = Y/2), then of P = I/2 + Y/2.  Both iterates are exchanged
    // once per step (two global buffers in turn); S = Y Q and T = Q Y are local rows.
    double *Y = acc, *Q = acc + accn, *S = k.block(2), *T = k.block(3);
    each([&](int i, int j, bool in) {
      const double dg = (in && r0 + i == j) ? 1.0 : 0.0;
      Y[(size_t)i * ld + j] = dg - 4.0 * P1[(size_t)i * ld + j];
      Q[(size_t)i * ld + j] = dg;
    });
    __syncthreads();
    int steps = plan[1], par = 0;
    for (int stage = 0; stage < 2; ++stage) {
      for (int it = 0; it < steps; ++it, par ^= 1) {
        double *Yg = NSg + 2 * par * ll, *Qg = Yg + ll;
        publish(Y, Yg);
        publish(Q, Qg);
        cluster.sync();
        kr_load(k, Qg);
        __syncthreads();
        kr_mm(k, Y, [&](int i, int j, double v) { S[(size_t)i * ld + j] = v; });
        __syncthreads();
        kr_load(k, Yg);
        __syncthreads();
        kr_mm(k, Q, [&](int i, int j, double v) { T[(size_t)i * ld + j] = v; });
        kr_mm(k, S, [&](int i, int j, double v) {
          const size_t e = (size_t)i * ld + j;
          Y[e] = 1.5 * Y[e] - 0.5 * v;
        });
        __syncthreads();
        kr_load(k, Qg);
        __syncthreads();
        kr_mm(k, T, [&](int i, int j, double v) {
          const size_t e = (size_t)i * ld + j;
          Q[e] = 1.5 * Q[e] - 0.5 * v;
        });
        __syncthreads();
      }
      if (stage == 0) {
        double d2 = 0.0;
        each([&](int i, int j, bool in) {
          const size_t e = (size_t)i * ld + j;
          const double dg = (in && r0 + i == j) ? 1.0 : 0.0;
          const double pv = 0.5 * Y[e] + 0.5 * dg;
          Y[e] = pv;
          Q[e] = dg;
          d2 += (dg - pv) * (dg - pv);
        });
        steps = kn_ns_steps(fmin(sqrt(kr_cluster_sum(k, cluster, d2, slots + 16, red)), 0.5), a.ns_target);
      }
    }
    C = Y;
    Ci = Q;
  }
  // C, C^-1, F = C - Dc C^-1 (:218) and the stacked copies, err = ||C - I||_F (:230-234).  C, C^-1 and
  // Dc are symmetric: the rows of F' = C - C^-1 Dc are the columns of F.
  kr_load(k, a.Dc);
  double e2 = 0.0;
  each([&](int i, int j, bool in) {
    if (!in) return;
    const size_t e = (size_t)(r0 + i) * l + j;
    const double cv = C[(size_t)i * ld + j], ci = Ci[(size_t)i * ld + j];
    a.C[e] = cv;
    a.Cinv[e] = ci;
    if (a.fstack) {
      a.fstack[ll + e] = a.fstack_scale * ci;
      a.fstack[3 * ll + e] = ci;
    }
    const double d = cv - (r0 + i == j ? 1.0 : 0.0);
    e2 += d * d;
  });
  __syncthreads();
  kr_mm(k, Ci, [&](int i, int j, double v) {
    if (r0 + i < l && j < l) {
      const size_t e = (size_t)j * l + r0 + i;
      const double fv = C[(size_t)i * ld + j] - v;
      a.F[e] = fv;
      if (a.fstack) {
        a.fstack[e] = fv;
        a.fstack[2 * ll + e] = fv;
      }
    }
  });
  pdl_trigger();  // the next product is placed on the SMs now
  const double err = sqrt(kr_cluster_sum(k, cluster, e2, slots + 32, red));
  if (k.rank == 0 && tid == 0) {
    *a.err = err;
    if (!(err == err)) atomicExch(a.status, kErrNumerical);
  }
}

__global__ void __launch_bounds__(kKrThreads, 1) kn_rows_kernel(KnStep a, KnSeries ser, int blocks) {
  pdl_wait();
  kn_rows_body(a, ser, blocks);
}

// One cluster per step of steps[] (grid = count x cluster size): many independent problems.
__global__ void __launch_bounds__(kKrThreads, 1) kn_rows_grouped_kernel(const KnStep *steps, KnSeries ser, int blocks) {
  const KnStep a = steps[blockIdx.x / cg::this_cluster().num_blocks()];
  if (a.gate && *a.gate <= a.gate_tol) return;  // alike in every CTA of the cluster
  kn_rows_body(a, ser, blocks);
}

// Coefficients of g(z)^(1/2) and g(z)^(-1/2), g(z) = 1 - sum_{n>=1} Cat(n-1) z^n: for h = f^alpha
// with f_0 = 1, h_0 = 1 and h_n = (1/n) sum_{k=1..n} (alpha k - (n - k)) f_k h_(n-k).
KnSeries make_series() {
  KnSeries s;
  double f[kSeriesLen], cat = 1.0;  // Cat(0) = 1, Cat(n) = Cat(n-1) 2 (2n - 1) / (n + 1)
  f[0] = 1.0;
  for (int n = 1; n < kSeriesLen; ++n) {
    f[n] = -cat;
    cat = cat * 2.0 * (2.0 * n - 1.0) / (n + 1.0);
  }
  const double alpha[2] = {0.5, -0.5};
  double *out[2] = {s.c, s.d};
  for (int w = 0; w < 2; ++w) {
    double *h = out[w];
    h[0] = 1.0;
    for (int n = 1; n < kSeriesLen; ++n) {
      double acc = 0.0;
      for (int kk = 1; kk <= n; ++kk) acc += (alpha[w] * kk - (n - kk)) * f[kk] * h[n - kk];
      h[n] = acc / n;
    }
  }
  return s;
}

constexpr size_t kKsSmem = (size_t)(32 * kAld + (kKsMaxL + 4) * kBld + 4 * 1024) * sizeof(double);
int g_cluster_size = -1;  // -1: not decided yet; 0: no cluster launch possible

int choose_cluster_size(const KnStep &a, cudaStream_t st) {
  if (g_cluster_size >= 0) return g_cluster_size;
  CK(cudaFuncSetAttribute(kn_cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CK(cudaFuncSetAttribute(kn_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKsSmem));
  g_cluster_size = 0;
  for (int cs = 16; cs >= 2; cs /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cs);
    cfg.blockDim = dim3(kKsThreads);
    cfg.dynamicSmemBytes = kKsSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kn_cluster_kernel, &cfg);
    if (e != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (n >= 1) {
      g_cluster_size = cs;
      break;
    }
  }
  (void)a;
  return g_cluster_size;
}

}  // namespace

namespace {

int kr_blocks(int l, int cs) {
  const size_t cap = Runtime::get().smem_optin - 1024;
  if (kr_bytes(l, cs, kKrBlocksWide) <= cap) return kKrBlocksWide;
  return kr_bytes(l, cs, kKrBlocks) <= cap ? kKrBlocks : 0;
}

// Cluster size of a row-cut step: one CTA per eight rows (a power of two, at most `want`, at least
// what the shared memory needs), or 0 when there is none.
int kr_cluster(int l, int want) {
  if (l > kKrMaxL) return 0;
  int cs = 1;
  while (cs < want && kr_rows(l, cs) > 8) cs *= 2;
  while (cs < 16 && kr_blocks(l, cs) == 0) cs *= 2;
  return kr_blocks(l, cs) ? cs : 0;
}

template <class Kern, class Arg>
void kr_launch(Kern kern, int cs, int grid, int l, bool pdl, cudaStream_t st, Arg a, const KnSeries &series) {
  const int blocks = kr_blocks(l, cs);
  const int bytes = (int)kr_bytes(l, cs, blocks);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kKrThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[1] = pdl_attribute();
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 2 : 1;  // pdl: the kernel calls pdl_wait()
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  CK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  CK(cudaLaunchKernelEx(&cfg, kern, a, series, blocks));
  KLAUNCHED();
}

// Whether the device can run a 16-CTA cluster of the row-cut step at its largest shared memory.
bool kr_usable() {
  static const bool ok = [] {
    const size_t bytes = kr_bytes(kKrMaxL, 16, kr_blocks(kKrMaxL, 16));
    CK(cudaFuncSetAttribute(kn_rows_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    CK(cudaFuncSetAttribute(kn_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kKrThreads);
    cfg.dynamicSmemBytes = bytes;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 16;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kn_rows_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    return n >= 1;
  }();
  return ok;
}

}  // namespace

void kn_step_grouped(const KnStep *steps, int count, int max_l, int cluster, cudaStream_t st) {
  if (count <= 0) return;
  if (max_l > kKrMaxL) fail(kErrUnsupported, "grouped Kolmogorov-Nagumo step: l = %d > %d", max_l, kKrMaxL);
  const int cs = kr_usable() ? kr_cluster(max_l, cluster > 0 ? cluster : 8) : 0;
  if (cs == 0) fail(kErrUnsupported, "grouped Kolmogorov-Nagumo step: no thread-block cluster launch on this device");
  static const KnSeries series = make_series();
  kr_launch(kn_rows_grouped_kernel, cs, count * cs, max_l, false, st, steps, series);
}

void kn_step(const KnStep &a, cudaStream_t st) {
  if (a.l > kKsMaxL) fail(kErrUnsupported, "Kolmogorov-Nagumo step: l = %d > %d", a.l, kKsMaxL);
  static const KnSeries series = make_series();
  if (const int rc = kr_usable() ? kr_cluster(a.l, 16) : 0) {
    kr_launch(kn_rows_kernel, rc, rc, a.l, true, st, a, series);
    return;
  }
  const int cs = choose_cluster_size(a, st);
  if (cs == 0) {  // no cluster launch on this device: the grid-barrier kernel (work 8 l^2 + 64 fits)
    CK(cudaMemsetAsync(a.bar, 0, 8, st));  // its barrier counters
    kn_step_fixed(a, Runtime::get().num_sms, st);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cs);
  cfg.blockDim = dim3(kKsThreads);
  cfg.dynamicSmemBytes = kKsSmem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  CK(cudaLaunchKernelEx(&cfg, kn_cluster_kernel, a, series));
  KLAUNCHED();
}

}  // namespace isvdb
