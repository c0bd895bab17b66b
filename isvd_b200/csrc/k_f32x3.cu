// FP32 products on the bf16 tensor cores: an FP32 operand is the sum of three bf16 planes to its last
// bit (8 + 8 + 8 significant bits; below 2^-110 the last plane runs out of bf16's exponents), and the six
// plane pairs (p, q) with p + q < 3 leave out terms below 2^-24 of a term, under the rounding of one FP32
// multiply-add.  The tcgen05 engine (umma.h) adds them in FP32 in chunks of one k-block (32 or 64 terms, by
// the tile shape), and the chunks round-to-nearest in FP32, so that long sums carry less rounding than the
// single FP32 chain per output of the CUDA-core kernel (k_gemm.cu).  A NaN or an infinity in an operand makes
// its outputs non-finite (an infinity meets the other operand's zero planes as NaN; a sketch with a drawn
// Omega, one plane, keeps it infinite).
//
// gemm<float, .> comes here for products that are large enough to pay for the splits (plane_product_pays).
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "kernels.h"
#include "mixed.h"
#include "panels.h"
#include "planes.cuh"
#include "runtime.h"
#include "umma.h"

extern "C" size_t isvd_gpu_memory_limit;  // include/isvd/gpu/env.h

namespace isvdb {
namespace {

bool planes_off() {
  const char *e = getenv("ISVD_GPU_FP32_PLANES");
  return e && atoi(e) == 0;
}

// Planes of nblk column blocks (w columns each, block b from column b bs of src, row stride s_ld) with
// every block starting at a multiple of lp (a multiple of 8) columns and the columns between zero: as
// MN-major operands or operands with per-batch K offsets, TMA boxes start on 16-byte boundaries
// whatever w is.  Eight columns per thread, one 16-byte store per plane.
__global__ void split_blocks_kernel(const float *__restrict__ src, long long s_ld, long long rows, int nblk, long long bs,
                                    int w, int lp, long long rows_pad, __nv_bfloat16 *__restrict__ dst, long long ld,
                                    long long ps) {
  const long long c0 = 8LL * (blockIdx.x * blockDim.x + threadIdx.x);
  if (c0 >= ld) return;
  const int b = (int)(c0 / lp), j0 = (int)(c0 - (long long)b * lp);
  for (long long r = blockIdx.y; r < rows_pad; r += gridDim.y) {
    const float *row = src + r * s_ld + (long long)b * bs + j0;
    __nv_bfloat16 o[3][8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float x = (r < rows && b < nblk && j0 + i < w) ? row[i] : 0.f;
      __nv_bfloat16 t[3];
      split3f(x, t);
      o[0][i] = t[0]; o[1][i] = t[1]; o[2][i] = t[2];
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) *(uint4 *)(dst + q * ps + r * ld + c0) = pack8(o[q]);
  }
}

// Planes of the transposes of nblk small blocks side by side: dst(n, b kp + k) = src[b bs + k s_ld + n]
// for k < K, n < N, zero elsewhere in rows_pad x ld.
__global__ void split_t_blocks_kernel(const float *__restrict__ src, long long s_ld, int K, int N, int nblk, long long bs,
                                      int kp, long long rows_pad, __nv_bfloat16 *__restrict__ dst, long long ld,
                                      long long ps) {
  const long long total = rows_pad * ld;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const long long n = e / ld, c = e - n * ld;
    const int b = (int)(c / kp), k = (int)(c - (long long)b * kp);
    __nv_bfloat16 t[3];
    split3f(n < N && b < nblk && k < K ? src[b * bs + k * s_ld + n] : 0.f, t);
#pragma unroll
    for (int q = 0; q < 3; ++q) dst[q * ps + e] = t[q];
  }
}

int grid_y(long long rows) { return (int)std::min<long long>(rows, 65535); }

void block_planes(PlaneBuf &pb, const float *src, long long s_ld, long long rows, int nblk, long long bs, int w, int lp,
                  cudaStream_t st) {
  const long long cols = (long long)nblk * lp, ld = plane_ld(cols), rp = plane_rows(rows), ps = rp * ld;
  pb.buf.ensure((size_t)3 * ps);
  const dim3 grid((unsigned)((ld / 8 + 255) / 256), grid_y(rp));
  split_blocks_kernel<<<grid, 256, 0, st>>>(src, s_ld, rows, nblk, bs, w, lp, rp, pb.buf.p, ld, ps);
  KLAUNCHED();
  pb.P.ptr = pb.buf.p; pb.P.np = 3; pb.P.rows = rows; pb.P.cols = cols; pb.P.ld = ld; pb.P.plane_stride = ps;
  pb.P.mn_major = false;
}

void block_planes_t(PlaneBuf &pb, const float *src, long long s_ld, int K, int N, int nblk, long long bs, int kp,
                    cudaStream_t st) {
  const long long cols = (long long)nblk * kp, ld = plane_ld(cols), rp = plane_rows(N), ps = rp * ld;
  pb.buf.ensure((size_t)3 * ps);
  const int blocks = (int)std::min<long long>((ps + 255) / 256, 16LL * Runtime::get().num_sms);
  split_t_blocks_kernel<<<blocks, 256, 0, st>>>(src, s_ld, K, N, nblk, bs, kp, rp, pb.buf.p, ld, ps);
  KLAUNCHED();
  pb.P.ptr = pb.buf.p; pb.P.np = 3; pb.P.rows = N; pb.P.cols = cols; pb.P.ld = ld; pb.P.plane_stride = ps;
  pb.P.mn_major = false;
}

void six_products(UmmaGemm &g) {
  g.nprod = 0;
  for (int s = 2; s >= 0; --s)
    for (int p = 0; p <= s; ++p) { g.pa[g.nprod] = p; g.pb[g.nprod] = s - p; ++g.nprod; }
  g.unbias = true;
  g.chunk_k = 1;  // one k-block
}

int *engine_status() { return reinterpret_cast<int *>(Runtime::get().ctl + 16); }  // the stages' status word

// Bytes of planes held for one operand at a time; larger operands run in chunks of their output rows
// or columns.
long long plane_cap() {
  long long cap = 4LL << 30;
  if (isvd_gpu_memory_limit > 0) cap = std::min<long long>(cap, (long long)(isvd_gpu_memory_limit / 16));
  return std::max<long long>(cap, 32LL << 20);
}

}  // namespace

// Depth of an accumulation chunk: one k-block, except in long sketches.  The tensor core truncates at every
// 16-deep step of a chunk, the chunks are added in round-to-nearest.  The plane pairs run smallest first, so that
// in a chunk of one k-block only the last steps truncate at the full magnitude.  Relative error of A Omega against 64 bits
// at n = 150 / 300 / 1000 / 10000: CUDA-core FP32 2.2e-7 / 3.1e-7 / 4.0e-7 / 1.8e-6; chunks of 128 3.5e-7 /
// 3.6e-7 / 3.8e-7 / 4.1e-7, of 64 1.7e-7 / 1.8e-7 / 1.8e-7 / 2.9e-7, of 32 0.7e-7 / 0.9e-7 / 0.8e-7 / 3.2e-7.
// Long sketches, which are bound by the tensor pipe, take 64 (32 costs 9 % at n = 10000).
static int f32_sketch_chunk(int n) { return n <= 1024 ? 32 : 64; }

// Time of the product by either path.  CUDA cores: 30 TFLOP/s on whole tiles (64 x 64 when either side
// is at most 64, else 128 x 128).  Planes: a split reads 4 and writes 6 bytes per element and the product
// reads 6 at about 5 TB/s, six bf16 products of 128 x 128 tiles at about 1.1 PFLOP/s, and 20 us of
// launches, tensor-memory set-up and pipeline fill.  The line is where the second wins by a quarter.
static bool plane_product_pays(double M, double N, double K, double batch, double elems_a, double elems_b) {
  auto padded = [&](double t) { return std::ceil(M / t) * t * std::ceil(N / t) * t; };
  const double cuda = 2.0 * padded(M <= 64 || N <= 64 ? 64 : 128) * K * batch / 30e12;
  const double planes = (elems_a + elems_b) * 16.0 / 5e12 + 6.0 * 2.0 * padded(128) * K * batch / 1.1e15 + 20e-6;
  return planes < 0.8 * cuda;
}

bool f32_planes_pay(double M, double N, double K, bool gram) {
  return !planes_off() && Runtime::get().cc_major == 10 && plane_product_pays(M, N, K, 1, M * K, gram ? 0.0 : N * K);
}

template <class Tout>
bool gemm_f32_planes(const Gemm<float, Tout> &g, bool a_kc, bool b_nc, cudaStream_t st) {
  if (planes_off() || Runtime::get().cc_major != 10 || g.beta != 0.0 || g.pl_t) return false;
  const int M = g.M, N = g.N, K = g.K, nb = g.batch;
  const bool same = (const void *)g.A == (const void *)g.B && !a_kc && b_nc && g.a_cs == g.b_rs && M == N &&
                    (nb == 1 || g.a_bs == g.b_bs);
  if (!plane_product_pays(M, N, K, nb, (double)M * K * nb, same ? 0.0 : (double)N * K * nb)) return false;
  UmmaGemm u;
  u.M = M; u.N = N; u.K = K;
  u.C = g.C; u.c_double = sizeof(Tout) == 8; u.c_rs = g.c_rs; u.c_cs = g.c_cs;
  u.alpha = g.alpha;
  u.upper = g.upper;
  u.status = g.status ? g.status : engine_status();
  u.tag = "fp32";
  six_products(u);
  u.unbias = g.unbias;
  PlaneBuf pa, pb;
  try {
    if (nb > 1) {
      u.batch = nb;
      u.c_step = g.c_bs;
      const int lp = (std::max(M, N) + 7) & ~7;
      if (!a_kc && b_nc && g.a_bs > 0 && g.a_bs < g.a_cs && g.b_bs > 0 && g.b_bs < g.b_rs) {
        // C_b = A_b' B_b of column blocks of tall matrices (Grams, products Q(i)' Q(i+h))
        block_planes(pa, g.A, g.a_cs, K, nb, g.a_bs, M, lp, st);
        if (!same) block_planes(pb, g.B, g.b_rs, K, nb, g.b_bs, N, lp, st);
        u.A = pa.P; u.B = same ? pa.P : pb.P;
        u.A.mn_major = u.B.mn_major = true;
        u.a_mn_step = u.b_mn_step = lp;
      } else if (a_kc && b_nc && g.a_bs == K && g.a_rs >= (long long)nb * K && g.b_bs == (long long)K * g.b_rs) {
        // C_b = A_b B_b, A's column blocks times small blocks: K runs to the next multiple of 64, over
        // columns of the next block that meet zeros
        const int ap = (K + 7) & ~7, kp = (K + 63) / 64 * 64;
        block_planes(pa, g.A, g.a_rs, M, nb, g.a_bs, K, ap, st);
        block_planes_t(pb, g.B, g.b_rs, K, N, nb, g.b_bs, kp, st);
        u.A = pa.P; u.B = pb.P;
        u.K = kp;
        u.a_k_step = ap; u.b_k_step = kp;
      } else {
        return false;
      }
      umma_gemm(u, st);
      return true;
    }
    if (same) {  // C = A' A of a tall matrix
      make_planes<float>(pa, g.A, g.a_cs, K, M, 3, false, st);
      u.A = pa.P; u.B = pa.P;
      u.A.mn_major = u.B.mn_major = true;
      umma_gemm(u, st);
      return true;
    }
    if (g.upper) return false;
    // The engine takes (A, B) as (K-major, K-major), (K-major, MN-major) or (MN-major, MN-major).  The
    // smaller operand is split with K contiguous, transposed where it is stored otherwise; the larger
    // one as it is stored, as the B operand when that is MN-major (C' = B' A').
    const bool big_a = (long long)M >= (long long)N;
    struct Side {
      const float *p;
      long long ld;
      int mn;
      bool kc;  // K contiguous
    } a{g.A, a_kc ? g.a_rs : g.a_cs, M, a_kc}, b{g.B, b_nc ? g.b_rs : g.b_cs, N, !b_nc};
    const Side big = big_a ? a : b, sm = big_a ? b : a;
    if (sm.kc) make_planes<float>(pb, sm.p, sm.ld, sm.mn, K, 3, false, st);
    else make_planes<float>(pb, sm.p, sm.ld, K, sm.mn, 3, true, st);
    const long long per = 6LL * K;  // plane bytes per row / column of the output along the larger operand
    const long long step = std::max<long long>(256, plane_cap() / per / 256 * 256);
    for (long long x0 = 0; x0 < big.mn; x0 += step) {
      const int cnt = (int)std::min<long long>(step, big.mn - x0);
      UmmaGemm v = u;
      if (big.kc) make_planes<float>(pa, big.p + x0 * big.ld, big.ld, cnt, K, 3, false, st);
      else make_planes<float>(pa, big.p + x0, big.ld, K, cnt, 3, false, st);
      Planes P = pa.P;
      P.mn_major = !big.kc;
      Tout *C = g.C + x0 * (big_a ? g.c_rs : g.c_cs);
      v.C = C;
      const bool big_is_b = !big.kc || !big_a;
      v.A = big_is_b ? pb.P : P;
      v.B = big_is_b ? P : pb.P;
      v.M = big_is_b ? sm.mn : cnt;
      v.N = big_is_b ? cnt : sm.mn;
      // rows of the engine's C: the small operand's index when the large one is B
      const bool rows_are_m = big_is_b ? !big_a : big_a;
      v.c_rs = rows_are_m ? g.c_rs : g.c_cs;
      v.c_cs = rows_are_m ? g.c_cs : g.c_rs;
      umma_gemm(v, st);
    }
  } catch (const Error &e) {
    if (e.code != kErrMemory) throw;
    return false;  // no room for the planes: the CUDA-core kernel needs none
  }
  return true;
}
template bool gemm_f32_planes<float>(const Gemm<float, float> &, bool, bool, cudaStream_t);
template bool gemm_f32_planes<double>(const Gemm<float, double> &, bool, bool, cudaStream_t);

// ------------------------------------------------------------------------- stages (mixed.h)
bool f32_block_planes(PlaneBuf &pb, const float *y, long long ldy, long long rows, int l, int N, cudaStream_t st) {
  if (planes_off() || Runtime::get().cc_major != 10) return false;
  // the Grams and the applies from one split
  if (!plane_product_pays((double)rows, l, l, N, 0.5 * rows * l * N, 0.0)) return false;
  return fits_memory([&] { block_planes(pb, y, ldy, rows, N, l, l, (l + 7) & ~7, st); });
}

bool f32_block_gram(const PlaneBuf &yp, int rows, int l, int N, double *W, cudaStream_t st) {
  UmmaGemm u;
  u.M = l; u.N = l; u.K = rows;
  u.A = u.B = yp.P;
  u.A.mn_major = u.B.mn_major = true;
  u.batch = N; u.a_mn_step = u.b_mn_step = (l + 7) & ~7; u.c_step = (long long)l * l;
  u.C = W; u.c_double = true; u.c_rs = l; u.c_cs = 1;
  u.status = engine_status();
  u.tag = "block_gram";
  six_products(u);
  return fits_memory([&] { umma_gemm(u, st); });
}

bool f32_block_apply(const PlaneBuf &yp, int rows, int l, int N, const float *Wp, float *out, long long ldo,
                     cudaStream_t st) {
  // K runs to the next multiple of 64, over columns of the next block that meet zeros of Wp's planes
  const int kp = (l + 63) / 64 * 64;
  PlaneBuf wt;
  if (!fits_memory([&] { block_planes_t(wt, Wp, l, l, l, N, (long long)l * l, kp, st); })) return false;
  UmmaGemm u;
  u.M = rows; u.N = l; u.K = kp;
  u.A = yp.P; u.B = wt.P;
  u.batch = N; u.a_k_step = (l + 7) & ~7; u.b_k_step = kp; u.c_step = l;
  u.C = out; u.c_rs = ldo; u.c_cs = 1;
  u.status = engine_status();
  u.tag = "block_apply";
  six_products(u);
  return fits_memory([&] { umma_gemm(u, st); });
}

bool f32_operator_pays(long long m, long long n, int k) {
  // A is split once for all the products of the iterations: each reads its planes
  if (planes_off() || Runtime::get().cc_major != 10) return false;
  if (isvd_gpu_memory_limit > 0 && 6.0 * m * n > isvd_gpu_memory_limit / 2.0) return false;
  const double kp = std::ceil(k / 64.0) * 64;
  return (double)m * n * 6.0 / 5e12 + 6.0 * 2.0 * m * n * kp / 1.1e15 + 20e-6 < 0.7 * 2.0 * m * n * kp / 30e12;
}

bool f32_tall_planes(PlaneBuf &pb, const float *qs, long long ldq, long long rows, int Nl, cudaStream_t st) {
  if (planes_off() || Runtime::get().cc_major != 10) return false;
  if (!plane_product_pays(Nl, Nl, (double)rows, 1, (double)rows * Nl, 0.0)) return false;
  return fits_memory([&] { make_planes<float>(pb, qs, ldq, rows, Nl, 3, false, st); });
}

bool f32_tall_gram(const PlaneBuf &qp, int rows, int Nl, double *G, cudaStream_t st) {
  UmmaGemm u;
  u.M = Nl; u.N = Nl; u.K = rows;
  u.A = u.B = qp.P;
  u.A.mn_major = u.B.mn_major = true;
  u.C = G; u.c_double = true; u.c_rs = Nl; u.c_cs = 1;
  u.upper = true;
  u.status = engine_status();
  u.tag = "gram_full";
  six_products(u);
  if (!fits_memory([&] { umma_gemm(u, st); })) return false;
  mirror_upper(G, Nl, Nl, st);
  return true;
}

bool f32_tall_apply(const PlaneBuf &qp, int rows, int Nl, int l, const float *M, long long ldm, float *out, long long ldo,
                    cudaStream_t st) {
  PlaneBuf mt;
  if (!fits_memory([&] { make_planes<float>(mt, M, ldm, Nl, l, 3, true, st); })) return false;  // M' planes (l x Nl)
  UmmaGemm u;
  u.M = rows; u.N = l; u.K = Nl;
  u.A = qp.P; u.B = mt.P;
  u.C = out; u.c_rs = ldo; u.c_cs = 1;
  u.status = engine_status();
  u.tag = "coeff_apply";
  six_products(u);
  return fits_memory([&] { umma_gemm(u, st); });
}

// Rows of A per panel of the plane sketch: about plane_cap() of planes.
long long f32_sketch_panel(long long m, long long n) {
  return std::min<long long>(m, std::max<long long>(256, plane_cap() / (6LL * plane_ld(n)) / 256 * 256));
}

bool f32_sketch_pays(long long m, long long n, long long Nl, long long offset) {
  if (planes_off() || Runtime::get().cc_major != 10 || offset % 2) return false;
  const double flops = 2.0 * m * n * Nl;
  return (double)m * n * 16.0 / 5e12 + 3.0 * flops / 1.1e15 + 25e-6 < 0.8 * flops / 30e12;
}

void f32_sketch_rows(const Planes &omega_t, long long rows, int n, int Nl, char ordera, const float *a, long long ld,
                     float *y, long long ldy, MixedCache *keep, cudaStream_t st) {
  const long long pld = plane_ld(n);
  // the planes of all rows when they can stay for the projection, else panel by panel
  if (keep) {
    const long long bytes = 6LL * plane_rows(rows) * pld;
    bool fits = bytes <= (1LL << 30) && isvd_gpu_memory_limit == 0;
    if (!fits) fits = bytes <= (long long)(device_budget() / 3);
    try {
      if (fits) keep->buf.alloc((size_t)bytes / 2);
    } catch (const Error &e) {
      if (e.code != kErrMemory) throw;
      fits = false;
    }
    if (!fits) keep = nullptr;
  }
  long long P = f32_sketch_panel(rows, n), rp = plane_rows(keep ? rows : P), ps = rp * pld;
  PlaneBuf pa;
  while (!keep && !pa.buf.p) try {
    pa.buf.alloc((size_t)3 * ps);
  } catch (const Error &e) {
    if (e.code != kErrMemory || P <= 256) throw;
    P = std::max<long long>(256, P / 2 / 256 * 256);  // smaller panels
    rp = plane_rows(P);
    ps = rp * pld;
  }
  __nv_bfloat16 *base = keep ? keep->buf.p : pa.buf.p;
  auto split = [&](long long r0, long long cnt, __nv_bfloat16 *dst) {
    if (ordera == 'R') split_rows<float>(a + r0 * ld, ld, 1, cnt, n, 3, false, dst, pld, ps, st);
    else split_rows<float>(a + r0, ld, 1, n, cnt, 3, true, dst, pld, ps, st);
  };
  auto zero_rows = [&](long long r0, long long r1) {  // TMA boxes of the last tile read them
    for (int q = 0; q < 3; ++q)
      if (r1 > r0)
        CK(cudaMemsetAsync(base + (size_t)q * ps + (size_t)r0 * pld, 0, (size_t)(r1 - r0) * pld * 2, st));
  };
  UmmaGemm g;
  g.N = Nl; g.K = n;
  g.B = omega_t;
  g.nprod = 3;  // Omega is exact in one plane
  for (int p = 0; p < 3; ++p) { g.pa[p] = 2 - p; g.pb[p] = 0; }
  g.c_rs = ldy; g.c_cs = 1;
  g.status = engine_status();
  g.tag = "sketch";
  g.chunk_k = f32_sketch_chunk(n);
  sketch_tile_order(g, n, Nl, Nl > 128 ? 256 : 128);
  Planes all;
  all.ptr = base; all.np = 3; all.cols = n; all.ld = pld; all.plane_stride = ps;
  const long long step = keep ? rows : P;  // rows per launch
  for (long long r0 = 0; r0 < rows; r0 += step) {
    const long long cnt = std::min(step, rows - r0);
    for (long long q0 = 0; q0 < cnt; q0 += P) split(r0 + q0, std::min(P, cnt - q0), base + (size_t)q0 * pld);
    zero_rows(cnt, plane_rows(cnt));
    g.M = (int)cnt;
    all.rows = cnt;
    g.A = all;
    g.C = y + r0 * ldy;
    umma_gemm(g, st);
  }
  if (keep) {
    keep->src = a; keep->m = rows; keep->n = n; keep->ordera = ordera;
    keep->A = all;
    keep->spare(true);
  }
}

bool f32_project(MixedCache *mc, int m, int n, int l, char ordera, const float *a, const float *qt, long long ldqt,
                 float *z, cudaStream_t st) {
  if (!mc || mc->src != a || mc->m != m || mc->n != n || mc->ordera != ordera || !mc->buf.p || mc->A.np != 3)
    return false;
  mc->spare(false);  // read below
  PlaneBuf qp;
  if (!fits_memory([&] { make_planes<float>(qp, qt, ldqt, m, l, 3, true, st); })) {  // Qbar' planes (l x m)
    mc->drop();
    return false;
  }
  UmmaGemm u;
  u.M = l; u.N = n; u.K = m;
  u.A = qp.P;
  u.B = mc->A;
  u.B.mn_major = true;
  u.C = z; u.c_rs = 1; u.c_cs = l;  // Z' tile written into Z (n x l)
  u.status = engine_status();
  u.tag = "project";
  six_products(u);
  if (fits_memory([&] { umma_gemm(u, st); })) return true;
  mc->drop();
  return false;
}

}  // namespace isvdb
