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
// 32 for a 128-thread one), 8-deep K slices staged in shared memory by
// cp.async through a four-stage ring (one barrier per slice, zero-filled
// outside the matrix).  The 8 x 8 blocks of a tile are dealt to the warps in
// rows and columns (warp (wm, wn) owns block rows wm + 2 i and block columns
// wn + NW/2 j), so a tile that is only partly inside the matrix still spreads
// over all warps; blocks outside it issue no MMA and stage no data.
// Conjugation is applied when a slice is read from shared memory.
//
// A product may be a sum over segments, C = sum_s coef_s A_s B_s, that share
// one output tile in registers (the effective Hamiltonian in krylov.cuh): the
// K slices of all segments form one stream through the ring.
#pragma once
#include "common.cuh"

#define GBM 64
#define GBN 64
#define GBK 8
#define GSTAGES 4
// Output columns of one CTA tile: the warps form a 2 x NW/2 grid.
#define GBN_EFF (16 * (NW / 2))
static_assert(NW % 2 == 0 && GBN_EFF <= GBN, "the GEMM needs an even warp count of at most 8");

// Rows of a slice are padded by two values: a quarter warp reads four k rows
// at two columns each, and 66 (34) x 16 bytes puts those in eight different
// 16-byte bank groups (65 gave two-way conflicts).
struct GemmSmem {
  cplx As[GSTAGES][GBK][GBM + 2];
  cplx Bs[GSTAGES][GBK][GBN_EFF + 2];
};

static __device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int sz = valid ? 16 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(sz) : "memory");
}
static __device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
static __device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }
static __device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
static __device__ __forceinline__ void cp_async_wait_ring() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(GSTAGES - 2) : "memory");
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

// One segment of a product: A (m,k) at A[m am + k ak], B (k,n) at
// B[k bk + n bn], the product scaled by the provider's coef(s) unless unit(s).
struct GemmSeg {
  const cplx* A;
  const cplx* B;
  int am, ak, bk, bn;  // element offsets inside one operand stay far below 2^31
  int K;
};

static __device__ __forceinline__ double flip_sign(double x, unsigned mask) {
  return __hiloint2double(__double2hiint(x) ^ (int)mask, __double2loint(x));
}

// C(M x N) = sum over the provider's segments; pv.nseg segments, pv.get(s, seg)
// fills segment s, epi(mm, nn, value) stores one element.  CTA-collective;
// ends with a cta_sync() so C is visible to all.
//
// Complex products run on the FP64 tensor cores (mma.sync m8n8k4): an 8 x 8
// block accumulates re and im with four real MMAs per four k.  Bound: the
// FP64 pipe, 64 FMA per clock and SM (0.23 TFLOP/s of an SM's share); a block
// step of four MMAs takes 16 clocks of it and 8 of shared memory.  Against the
// two-stage 16-deep slices with two barriers each, which multiplied whole
// 64 x 64 tiles of mostly padding for small operands, the analog run on L = 30,
// chi 64, FP64 (260 trajectories, 2 time indices) went from 1588 to 1453 ms,
// L = 16 at chi 128 from 600 to 550 ms and L = 6 at chi 16 from 528 to 446 ms,
// with the same bits.
template <class Prov, class Epi>
static __device__ __forceinline__ void gemm_core(const Prov& pv, int M, int N, bool conjA, bool conjB, Epi epi,
                                                 GemmSmem& sm) {
  const int tid = ltid();
  const int lane = tid & 31, wid = tid >> 5;
  const int wm = wid & 1, wn = wid >> 1;  // 2 x NW/2 warps
  const int gq = lane >> 2, tq = lane & 3;
  const unsigned sgA = conjA ? 0x80000000u : 0u, sgB = conjB ? 0x80000000u : 0u;
  int nslice = 0;
  for (int s = 0; s < pv.nseg; ++s) nslice += (pv.K(s) + GBK - 1) / GBK;
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
      GemmSeg o;
      int is = 0, ik = 0;  // segment and k of the next slice to stage
      pv.get(0, o);
      auto issue = [&](int buf) {
        if (is < pv.nseg) {
          const bool a_m_fast = (o.am == 1) || (o.ak != 1);
          const bool b_n_fast = (o.bn == 1) || (o.bk != 1);
#pragma unroll
          for (int e = 0; e < GBM * GBK / NT; ++e) {
            const int idx = tid + NT * e;
            const int mi = a_m_fast ? (idx & (GBM - 1)) : (idx / GBK);
            const int ki = a_m_fast ? (idx / GBM) : (idx & (GBK - 1));
            const int ka = ik + ki;
            const bool va = mi < mrem && ka < o.K;
            if (mi < mlim)
              cp_async16(&sm.As[buf][ki][mi], o.A + (va ? (tm + mi) * o.am + ka * o.ak : 0), va);
          }
#pragma unroll
          for (int e = 0; e < GBN_EFF * GBK / NT; ++e) {
            const int idx = tid + NT * e;
            const int ni = b_n_fast ? (idx & (GBN_EFF - 1)) : (idx / GBK);
            const int kj = b_n_fast ? (idx / GBN_EFF) : (idx & (GBK - 1));
            const int kb = ik + kj;
            const bool vb = ni < nrem && kb < o.K;
            if (ni < nlim)
              cp_async16(&sm.Bs[buf][kj][ni], o.B + (vb ? kb * o.bk + (tn + ni) * o.bn : 0), vb);
          }
          ik += GBK;
          if (ik >= o.K) {
            ik = 0;
            if (++is < pv.nseg) pv.get(is, o);
          }
        }
        cp_async_commit();
      };
      cta_sync();  // the ring's last readers (the tile before) are done
#pragma unroll
      for (int p = 0; p < GSTAGES - 1; ++p) issue(p);
      int cs = 0, ck = 0, cK = pv.K(0);
      for (int t = 0; t < nslice; ++t) {
        cp_async_wait_ring();  // slice t has landed (this thread's part)
        cta_sync();            // everybody's part; slice t - 1 is consumed
        issue((t + GSTAGES - 1) % GSTAGES);
        const int buf = t % GSTAGES;
        const bool unit = pv.unit(cs);
#pragma unroll
        for (int k4 = 0; k4 < GBK; k4 += 4) {
          if (ck + k4 >= cK) break;
          double ar[4], ai[4], br[2], bi[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int n0 = (wn + (NW / 2) * j) * 8;
            if (n0 < nrem) {
              const cplx b = sm.Bs[buf][k4 + tq][n0 + gq];
              br[j] = b.x;
              bi[j] = flip_sign(b.y, sgB);
              if (!unit) {
                const cplx f = pv.coef(cs);
                const double x = br[j], y = bi[j];
                br[j] = f.x * x - f.y * y;
                bi[j] = f.x * y + f.y * x;
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int m0 = (wm + 2 * i) * 8;
            if (m0 >= mrem) break;
            const cplx a = sm.As[buf][k4 + tq][m0 + gq];
            ar[i] = a.x;
            ai[i] = flip_sign(a.y, sgA);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              if ((wn + (NW / 2) * j) * 8 >= nrem) break;
              dmma884(cr[i][j][0], cr[i][j][1], ar[i], br[j]);
              dmma884(ci[i][j][0], ci[i][j][1], ar[i], bi[j]);
              dmma884(cr[i][j][0], cr[i][j][1], -ai[i], bi[j]);
              dmma884(ci[i][j][0], ci[i][j][1], ai[i], br[j]);
            }
          }
        }
        ck += GBK;
        if (ck >= cK) {
          ck = 0;
          if (++cs < pv.nseg) cK = pv.K(cs);
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
            if (nn < N) epi(mm, nn, make_double2(cr[i][j][h], ci[i][j][h]));
          }
      }
    }
  }
  cta_sync();
}

// The plain product: one segment.
struct OneSeg {
  const GemmArgs& g;
  int nseg;
  __device__ __forceinline__ int K(int) const { return g.K; }
  __device__ __forceinline__ bool unit(int) const { return true; }
  __device__ __forceinline__ cplx coef(int) const { return make_double2(1.0, 0.0); }
  __device__ __forceinline__ void get(int, GemmSeg& o) const {
    o.A = g.A;
    o.B = g.B;
    o.am = (int)g.am;
    o.ak = (int)g.ak;
    o.bk = (int)g.bk;
    o.bn = (int)g.bn;
    o.K = g.K;
  }
};

static __device__ __noinline__ void cta_gemm(const GemmArgs g, GemmSmem& sm) {
  ProfScope prof_scope_(PF_GEMM);
  const OneSeg pv{g, 1};
  gemm_core(pv, g.M, g.N, g.conjA, g.conjB,
            [&](int mm, int nn, cplx v) {
              cplx* c = g.C + (mm * (int)g.cm + nn * (int)g.cn);
              if (g.accumulate) v = cadd(v, *c);
              *c = v;
            },
            sm);
}
