// gemm.cuh — CTA-level complex FP64 GEMM with general strides.
//
// C(m,n) = op(A)(m,k) * op(B)(k,n)  [+ C if accumulate]
//   A element (m,k) at A[m*am + k*ak], conjugated if conjA
//   B element (k,n) at B[k*bk + n*bn], conjugated if conjB
//   C element (m,n) at C[m*cm + n*cn]
// Every tensor contraction of the TDVP path (Algorithms.jl:199-226) is
// written as one such GEMM over the reference's column-major layouts.
//
// Tiling: 64 x GBN_EFF output tiles (64 x 64 for a 256-thread program, 64 x
// 32 for a 128-thread one), K slices of 16 staged in shared memory by cp.async
// through a ring of two (one barrier per slice, zero-filled outside the
// matrix): the work of a slice has to outweigh its barrier (L = 30, chi 64,
// FP64: 1525 ms against 1799 with a ring of four 8-deep slices; sums shorter
// than 32 take as long either way).  The 8 x 8 blocks of a tile are dealt to the
// warps in rows and columns (warp (wm, wn) owns block rows wm + 2 i and block
// columns wn + NW/2 j), so a tile that is only partly inside the matrix still
// spreads over all warps; blocks outside it issue no MMA and stage no data.
// Conjugation is applied when a slice is read from shared memory.
#pragma once
#include "common.cuh"

#define GBM 64
#define GBN 64
#define GBK 16
#define GSTAGES 2
#define GROWS (GSTAGES * GBK)  // k rows in the ring
// Output columns of one CTA tile: the warps form a 2 x NW/2 grid.
#define GBN_EFF (16 * (NW / 2))
static_assert(NW % 2 == 0 && GBN_EFF <= GBN, "the GEMM needs an even warp count of at most 8");

// Rows of a slice are padded by two values: a quarter warp reads four k rows
// at two columns each, and 66 (34) x 16 bytes puts those in eight different
// 16-byte bank groups (65 gave two-way conflicts).
struct GemmSmem {
  cplx As[GROWS][GBM + 2];
  cplx Bs[GROWS][GBN_EFF + 2];
};

static __device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(sz) : "memory");
}
static __device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
static __device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
static __device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
template <int N>
static __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

struct GemmArgs {
  int M, N, K;
  const cplx* A;
  long long am, ak;
  const cplx* B;
  long long bk, bn;
  cplx* C;
  long long cm, cn;
  bool conjA, conjB, accumulate;
};

static __device__ __forceinline__ GemmArgs gemm_args(int M, int N, int K, const cplx* A, long long am, long long ak,
                                              const cplx* B, long long bk, long long bn, cplx* C, long long cm,
                                              long long cn, bool conjA = false, bool conjB = false,
                                              bool accumulate = false) {
  GemmArgs g;
  g.M = M;
  g.N = N;
  g.K = K;
  g.A = A;
  g.am = am;
  g.ak = ak;
  g.B = B;
  g.bk = bk;
  g.bn = bn;
  g.C = C;
  g.cm = cm;
  g.cn = cn;
  g.conjA = conjA;
  g.conjB = conjB;
  g.accumulate = accumulate;
  return g;
}

// FP64 tensor-core product: D (8x8) += A (8x4, row) * B (4x8, col).
// Fragments (per lane, g = lane/4, t = lane%4): A[g][t], B[t][g],
// D[g][2t], D[g][2t+1].
static __device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

static __device__ __forceinline__ double flip_sign(double x, unsigned mask) {
  return __hiloint2double(__double2hiint(x) ^ (int)mask, __double2loint(x));
}

// CTA-collective; ends with a cta_sync() so C is visible to all.
//
// Complex products run on the FP64 tensor cores (mma.sync m8n8k4): an 8 x 8
// block accumulates re and im with four real MMAs per four k.  Bound: the
// FP64 pipe, 64 FMA per clock and SM (0.23 TFLOP/s of an SM's share); a block
// step of four MMAs takes 16 clocks of it and 8 of shared memory.  Against the
// two-stage 16-deep slices with two barriers each, which multiplied whole
// 64 x 64 tiles of mostly padding for small operands, L = 16 at chi 128 went
// from 600 to 550 ms and L = 6 at chi 16 from 528 to 446 ms, with the same
// bits.
static __device__ __noinline__ void cta_gemm_tiled(const GemmArgs g, GemmSmem& sm) {
  ProfScope prof_scope_(PF_GEMM);
  ASSUME_SHARED(&sm);
  const int tid = ltid();
  const int lane = tid & 31, wid = tid >> 5;
  const int wm = wid & 1, wn = wid >> 1;  // 2 x NW/2 warps
  const int gq = lane >> 2, tq = lane & 3;
  const unsigned sgA = g.conjA ? 0x80000000u : 0u, sgB = g.conjB ? 0x80000000u : 0u;
  const bool a_m_fast = (g.am == 1) || (g.ak != 1);
  const bool b_n_fast = (g.bn == 1) || (g.bk != 1);
  // element offsets inside one operand stay far below 2^31
  const int am = (int)g.am, ak = (int)g.ak, bk = (int)g.bk, bn = (int)g.bn;
  const int M = g.M, N = g.N, K = g.K;
  const int nslice = (K + GBK - 1) / GBK;
  for (int tm = 0; tm < M; tm += GBM) {
    for (int tn = 0; tn < N; tn += GBN_EFF) {
      const int mrem = min(GBM, M - tm), nrem = min(GBN_EFF, N - tn);
      const int mlim = (mrem + 7) & ~7, nlim = (nrem + 7) & ~7;  // staged rows and columns
      double cr[4][2][2], ci[4][2][2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          cr[i][j][0] = cr[i][j][1] = 0.0;
          ci[i][j][0] = ci[i][j][1] = 0.0;
        }
      auto issue = [&](int t, int buf) {  // slice t into stage buf; empty past the end
        const int k0 = t * GBK;
        if (t < nslice) {
#pragma unroll
          for (int e = 0; e < GBM * GBK / NT; ++e) {
            const int idx = tid + NT * e;
            const int mi = a_m_fast ? (idx & (GBM - 1)) : (idx / GBK);
            const int ki = a_m_fast ? (idx / GBM) : (idx & (GBK - 1));
            const int ka = k0 + ki;
            const bool va = mi < mrem && ka < K;
            if (mi < mlim) cp_async16(&sm.As[buf * GBK + ki][mi], g.A + (va ? (tm + mi) * am + ka * ak : 0), va);
          }
#pragma unroll
          for (int e = 0; e < GBN_EFF * GBK / NT; ++e) {
            const int idx = tid + NT * e;
            const int ni = b_n_fast ? (idx & (GBN_EFF - 1)) : (idx / GBK);
            const int kj = b_n_fast ? (idx / GBN_EFF) : (idx & (GBK - 1));
            const int kb = k0 + kj;
            const bool vb = ni < nrem && kb < K;
            if (ni < nlim) cp_async16(&sm.Bs[buf * GBK + kj][ni], g.B + (vb ? kb * bk + (tn + ni) * bn : 0), vb);
          }
        }
        cp_async_commit();
      };
      cta_sync();  // the ring's last readers (the tile before) are done
#pragma unroll 1
      for (int p = 0; p < GSTAGES - 1; ++p) issue(p, p);
      for (int t = 0; t < nslice; ++t) {
        cp_async_wait<GSTAGES - 2>();  // slice t has landed (this thread's part)
        cta_sync();                    // everybody's part; slice t - 1 is consumed
        issue(t + GSTAGES - 1, (t + GSTAGES - 1) % GSTAGES);
        const int buf = t % GSTAGES;
#pragma unroll
        for (int k4 = 0; k4 < GBK; k4 += 4) {
          if (t * GBK + k4 >= K) break;
          double ar[4], ai[4], br[2], bi[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int n0 = (wn + (NW / 2) * j) * 8;
            if (n0 < nrem) {
              const cplx b = sm.Bs[buf * GBK + k4 + tq][n0 + gq];
              br[j] = b.x;
              bi[j] = flip_sign(b.y, sgB);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int m0 = (wm + 2 * i) * 8;
            if (m0 >= mrem) break;
            const cplx a = sm.As[buf * GBK + k4 + tq][m0 + gq];
            ar[i] = a.x;
            ai[i] = flip_sign(a.y, sgA);
            // first products of both blocks before the second ones, which wait
            // for the same accumulators
            const bool one = wn * 8 < nrem, two = (wn + NW / 2) * 8 < nrem;
            if (one) {
              dmma884(cr[i][0][0], cr[i][0][1], ar[i], br[0]);
              dmma884(ci[i][0][0], ci[i][0][1], ar[i], bi[0]);
            }
            if (two) {
              dmma884(cr[i][1][0], cr[i][1][1], ar[i], br[1]);
              dmma884(ci[i][1][0], ci[i][1][1], ar[i], bi[1]);
            }
            if (one) {
              dmma884(cr[i][0][0], cr[i][0][1], -ai[i], bi[0]);
              dmma884(ci[i][0][0], ci[i][0][1], ai[i], br[0]);
            }
            if (two) {
              dmma884(cr[i][1][0], cr[i][1][1], -ai[i], bi[1]);
              dmma884(ci[i][1][0], ci[i][1][1], ai[i], br[1]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int mm = tm + (wm + 2 * i) * 8 + gq;
        if (mm >= M) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int nn = tn + (wn + (NW / 2) * j) * 8 + 2 * tq + h;
            if (nn >= N) continue;
            cplx* c = g.C + (mm * (int)g.cm + nn * (int)g.cn);
            cplx v = make_double2(cr[i][j][h], ci[i][j][h]);
            if (g.accumulate) v = cadd(v, *c);
            *c = v;
          }
      }
    }
  }
  cta_sync();
}

// A product of a few 8 x 8 blocks and a short sum, straight from global memory:
// two blocks a warp at most, no staging and one barrier.  The tiled form's
// slices, copies and barriers cost more than such a product.  Same bits.
#define GDIRECT_K 32
static __device__ __noinline__ void cta_gemm_direct(const GemmArgs g) {
  ProfScope prof_scope_(PF_GEMM);
  const int lane = ltid() & 31, wid = ltid() >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const unsigned sgA = g.conjA ? 0x80000000u : 0u, sgB = g.conjB ? 0x80000000u : 0u;
  const int mb = (g.M + 7) >> 3, nb = (g.N + 7) >> 3;
#pragma unroll 1
  for (int q = wid; q < mb * nb; q += NW) {
    const int nq = q / mb, row = (q - nq * mb) * 8 + gq, n0 = nq * 8;
    const bool rm = row < g.M, rn = n0 + gq < g.N;
    const cplx* A = g.A + (long long)(rm ? row : 0) * g.am;
    const cplx* B = g.B + (long long)(rn ? n0 + gq : 0) * g.bn;
    double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
#pragma unroll 1
    for (int k0 = 0; k0 < g.K; k0 += 16) {
      cplx a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = k0 + 4 * u + tq;
        const bool in = k < g.K;
        a[u] = in && rm ? A[k * g.ak] : make_double2(0.0, 0.0);
        b[u] = in && rn ? B[k * g.bk] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (k0 + 4 * u >= g.K) break;
        const double ai = flip_sign(a[u].y, sgA), bi = flip_sign(b[u].y, sgB);
        dmma884(cr[0], cr[1], a[u].x, b[u].x);
        dmma884(ci[0], ci[1], a[u].x, bi);
        dmma884(cr[0], cr[1], -ai, bi);
        dmma884(ci[0], ci[1], ai, b[u].x);
      }
    }
    if (rm) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int n = n0 + 2 * tq + e;
        if (n < g.N) {
          cplx* c = g.C + (long long)row * g.cm + (long long)n * g.cn;
          cplx v = make_double2(cr[e], ci[e]);
          if (g.accumulate) v = cadd(v, *c);
          *c = v;
        }
      }
    }
  }
  cta_sync();
}

static __device__ __forceinline__ void cta_gemm(const GemmArgs g, GemmSmem& sm) {
  if (g.K <= GDIRECT_K && ((g.M + 7) >> 3) * ((g.N + 7) >> 3) <= 2 * NW)
    cta_gemm_direct(g);
  else
    cta_gemm_tiled(g, sm);
}
