// krylov.cuh — effective-Hamiltonian product and Lanczos exponential.
//
// dev_heff restates project_site (Algorithms.jl:215-220, :330-361):
//   T1[a,m,p,c]   = sum_k L[a,m,k] x[k,p,c]                    (GEMM)
//   T2[a,p',m',c] = sum_{m,p} W[m,p',p,m'] T1[a,m,p,c]         (sparse MPO apply)
//   y[a,p',b]     = sum_{m',c} T2[a,p',m',c] R[b,m',c]         (GEMM)
// In mixed runs next to isometric sites the identity channels are taken out
// (HPlan, tsgemm.cuh).
//
// dev_expm_krylov restates expm_krylov (Algorithms.jl:144-187) / KrylovKit
// exponentiate: Lanczos with classical Gram-Schmidt against the whole basis,
// refined by a second pass when the first kept less than 1/sqrt(2) of the
// norm (DGKS), stopping at krylov_dim, at breakdown (beta <= |dt| tol), or
// once prod(beta_i |dt|)/k! <= exit_tol; the small tridiagonal exponential
// is taken on one warp by Taylor series over substeps of norm <= 1/2.  Three
// forms: the general one, dev_expm_small (at most one value a thread, in shared
// memory, the same bits), and dev_expm_predicted for mixed runs, which projects
// what the three-term recurrence leaves.
#pragma once
#include "common.cuh"
#include "gemm_tf32.cuh"
#include "tcgemm.cuh"

#define WAPPLY_IN_CPLX 2560  // staged inputs: ni x PT values, PT = 256, 128 or 64 by what fits
#define WAPPLY_MAXI 32
#define WAPPLY_MAXNNZ 512
#define WAPPLY_LB 8  // inputs a thread loads back to back
#define KRYLOV_MAX 32

// Structure of an effective Hamiltonian whose left environment holds the
// identity in MPO channel il and the right one in channel ir, as an MPO's
// running-sum form gives them next to isometric sites.  With those blocks
// taken out the product is, per output physical index p',
//   y_{p'} = sum_s coef_s A_s B_s + sum_p loc[p', p] x_p
// over terms L_m x_p (the term ends on the left), x_p R_m' (it starts there)
// and (L_m x)_p R_m' (it passes through; the products T1 = L_m x for m in
// [t1m, t1m + nt1) are formed first).  The mixed form takes it (tsgemm.cuh),
// with the terms gathered by environment block: block b multiplies channel
// m[b] with, per output index p', coef * (slice src of x, or of row block t1
// of T1 where t1 >= 0); src < 0: no term.
#define TS_MAX_BLOCKS 8
struct TsSide {
  int nb;
  int m[TS_MAX_BLOCKS];
  int src[TS_MAX_BLOCKS][4], t1[TS_MAX_BLOCKS][4];
  float2 coef[TS_MAX_BLOCKS][4];
};
struct HPlan {
  TsSide left, right;
  int il, ir;  // channels that have to be the identity
  int t1m, nt1, has_loc;
  int nleft, nright;  // terms on each side
  cplx loc[16];       // [p' + D p]
};

// Sparse MPO matrix M[o, i] in CSR form (rows are outputs).
struct WMat {
  int no, ni, nnz;
  int ident;  // identity map with a physical dimension of 1 (bond): T2 is T1
  int idc;    // environment maps: output channel that is the identity next to isometric sites, -1 for none
  const HPlan* plan;  // effective-Hamiltonian maps: the structured product, null when it does not pay
  const int* rowp;  // no+1
  const int* col;   // nnz
  const cplx* val;  // nnz
};

struct WApplyGeom {
  int n0, n1;
  long long is0, is1, ii1, ii2;
  int ni1;
  long long os0, os1, oo1, oo2;
  int no1;
};

struct WApplySmem {
  cplx in[WAPPLY_IN_CPLX];
  cplx val[WAPPLY_MAXNNZ];
  int col[WAPPLY_MAXNNZ];
  int rowp[WAPPLY_MAXI + 1];
  int in_off[WAPPLY_MAXI];
  int out_off[WAPPLY_MAXI];
};

// out[q0,q1,o] = sum_i M[o,i] in[q0,q1,i].  CTA-collective.  A tile holds PT
// pairs (the largest of 256, 128, 64 whose ni inputs fit the staging
// buffer); each thread owns pair slot tid % PT of every tile and
// input/output rows tid / PT + k NT / PT, so index arithmetic is per tile,
// not per element, and with PT = NT a thread issues all ni loads of its pair
// back to back.  T is cplx (FP64 form) or float2 (mixed form, FP32 products).
// in and out may be the same buffer when every pair's inputs and outputs
// occupy the same addresses (a tile reads all its inputs before it writes).
static __device__ __forceinline__ void wfma(cplx& acc, cplx v, cplx x) { cfma(acc, v, x); }
static __device__ __forceinline__ void wfma(float2& acc, cplx v, float2 x) {
  const float vr = (float)v.x, vi = (float)v.y;
  acc.x = fmaf(vr, x.x, fmaf(-vi, x.y, acc.x));
  acc.y = fmaf(vr, x.y, fmaf(vi, x.x, acc.y));
}
static __device__ __forceinline__ void wzero(cplx& z) { z = make_double2(0.0, 0.0); }
static __device__ __forceinline__ void wzero(float2& z) { z = make_float2(0.f, 0.f); }

template <class T>
static __device__ __noinline__ void dev_wapply(const T* in, T* out, const WMat W,
                                        const WApplyGeom g, WApplySmem& ws) {
  ProfScope prof_scope_(PF_WAPPLY);
  ASSUME_SHARED(&ws);
  T* sin = reinterpret_cast<T*>(&ws.in[0]);
  const int cap = (int)(WAPPLY_IN_CPLX * sizeof(cplx) / sizeof(T));
  const int PT = W.ni * NT <= cap ? NT : (W.ni * (NT / 2) <= cap ? NT / 2 : NT / 4);
  const int tid = ltid();
  for (int e = tid; e < W.nnz; e += NT) {
    ws.val[e] = W.val[e];
    ws.col[e] = W.col[e];
  }
  for (int e = tid; e <= W.no; e += NT) ws.rowp[e] = W.rowp[e];
  for (int i = tid; i < W.ni; i += NT) ws.in_off[i] = (int)((i % g.ni1) * g.ii1 + (i / g.ni1) * g.ii2);
  for (int o = tid; o < W.no; o += NT) ws.out_off[o] = (int)((o % g.no1) * g.oo1 + (o / g.no1) * g.oo2);
  const int npair = g.n0 * g.n1;
  const int pl = tid % PT, r0 = tid / PT;
  const int RS = NT / PT;
  T zero;
  wzero(zero);
  for (int base = 0; base < npair; base += PT) {
    const int pair = base + pl;
    const bool live = pair < npair;
    const int q0 = live ? pair % g.n0 : 0, q1 = live ? pair / g.n0 : 0;
    const long long ib = q0 * g.is0 + q1 * g.is1, ob = q0 * g.os0 + q1 * g.os1;
    cta_sync();
    // batches of WAPPLY_LB loads issued before their stores: `in` may alias
    // the staging buffer as far as the compiler knows, so a plain loop would
    // wait out one L2 latency per input
    for (int i0 = r0; i0 < W.ni; i0 += RS * WAPPLY_LB) {
      T v[WAPPLY_LB];
#pragma unroll
      for (int k = 0; k < WAPPLY_LB; ++k) {
        const int i = i0 + k * RS;
        v[k] = (live && i < W.ni) ? in[ib + ws.in_off[i]] : zero;
      }
#pragma unroll
      for (int k = 0; k < WAPPLY_LB; ++k) {
        const int i = i0 + k * RS;
        if (i < W.ni) sin[i * PT + pl] = v[k];
      }
    }
    cta_sync();
    if (live) {
      for (int o = r0; o < W.no; o += RS) {
        T acc = zero;
        for (int z = ws.rowp[o]; z < ws.rowp[o + 1]; ++z) wfma(acc, ws.val[z], sin[ws.col[z] * PT + pl]);
        out[ob + ws.out_off[o]] = acc;
      }
    }
  }
  cta_sync();
}

struct HeffOp {
  int blocked = 0;  // the run may reorder sums
  const HPlan* plan = nullptr;  // mixed form: set when both identity channels were found in the environments
  const cplx* L;  // (chil, wl, chil)
  const cplx* R;  // (chir, wr, chir)
  WMat W;         // rows p'+D m', cols m + wl p
  int chil, D, chir, wl, wr;
  cplx* T1;
  cplx* T2;
  // mixed form: FP32 copies of the environments and FP32 intermediates
  int mixed = 0;
  const cflt* Lf = nullptr;
  const cflt* Rf = nullptr;
  cflt* xf = nullptr;
  cflt* T1f = nullptr;
  cflt* T2f = nullptr;
  // mixed form on tcgen05 (tc = 1): TMA-staged operands of the two products,
  // tensor maps maps[0..3] = SL (A, MN-major), Sx (B, K-major), ST2 (A,
  // MN-major), SR (B, MN-major); pitches in complex FP32 values
  int tc = 0;
  const CUtensorMap* maps = nullptr;
  cflt* SL = nullptr;
  cflt* Sx = nullptr;
  cflt* ST2 = nullptr;
  cflt* SR = nullptr;
  int pL = 0, px = 0, pT2 = 0, pR = 0;
};

struct KrySmem {
  double alpha[KRYLOV_MAX + 1];
  double beta[KRYLOV_MAX + 1];
  cplx h[KRYLOV_MAX + 1];
  cplx y[KRYLOV_MAX + 1];
  int m;
};

// Shared memory of one CTA.  The GEMM / MPO-apply staging and the SVD block
// buffer are never live at the same time and share storage.
#define SVD_SMEM_CPLX_K 4096
union EngineSmemU {
  union {  // the GEMM and the MPO apply run one after the other, never together
    GemmSmem g;
    WApplySmem w;
  } gw;
  cplx svd[SVD_SMEM_CPLX_K];
#if YAQS_TC
  TcSmem t;  // the tensor-core pipeline (mixed form), no larger than the GEMM staging
#endif
};
struct EngineSmem {
  RedScratch r;
  KrySmem k;
  TcState tc;
#if YAQS_TC
  TsSide ts[2];  // left and right blocks of the solve's plan
  cplx loc[16];  // and its local term
#endif
  EngineSmemU u;
};
#if YAQS_TC
static_assert(sizeof(TcSmem) <= sizeof(GemmSmem), "the default pipeline must not grow the CTA's shared memory");
#endif

#if YAQS_TC
#include "tsgemm.cuh"

// Mixed form on tcgen05 (compiled only into the tensor-core kernel,
// engine_tc.cu: a kernel that contains tcgen05 code is given one CTA per
// SM).  x is staged as the K-major B operand of the first product, the MPO
// apply writes T2 straight into the MN-major A operand of the second
// product, and both products run in tc_gemm; the environments were staged
// once per Krylov solve.
static __device__ void dev_heff_tc(const HeffOp& h, const cplx* x, cplx* y, EngineSmem& sm) {
  const int chil = h.chil, D = h.D, chir = h.chir, wl = h.wl, wr = h.wr;
  if (h.plan) {
    ts_heff(h, x, y, sm.ts, sm.loc, sm.u.t, sm.tc);
    return;
  }
  const long long n = (long long)chil * D * chir;
  // Sx[nn px + k] = x[k + chil nn], 8 loads in flight per thread
  for (long long e0 = ltid(); e0 < n; e0 += 8 * NT) {
    cplx v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = e0 + u * NT < n ? x[e0 + u * NT] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const long long e = e0 + u * NT;
      if (e < n) h.Sx[(e / chil) * h.px + e % chil] = make_float2((float)v[u].x, (float)v[u].y);
    }
  }
  const TcOp A1{h.maps + 0, 1, 0}, B1{h.maps + 1, 0, 0}, A2{h.maps + 2, 1, 0}, B2{h.maps + 3, 1, 0};
  tc_gemm<cflt>(chil * wl, D * chir, chil, A1, B1, h.T1f, 1, (long long)chil * wl, false, sm.u.t, sm.tc);
  if (h.W.ident) {  // bond (D = 1, wl = wr): T2 is T1 re-laid into ST2
    const long long nt1 = (long long)chil * wl * chir;
    for (long long e0 = ltid(); e0 < nt1; e0 += 8 * NT) {
      cflt v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = e0 + u * NT < nt1 ? h.T1f[e0 + u * NT] : make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const long long e = e0 + u * NT;
        if (e >= nt1) continue;
        const long long a = e % chil, m = (e / chil) % wl, c = e / ((long long)chil * wl);
        h.ST2[(m + (long long)wr * c) * h.pT2 + a] = v[u];
      }
    }
  } else {
    WApplyGeom g;
    g.n0 = chil;
    g.n1 = chir;
    g.is0 = 1;
    g.is1 = (long long)chil * wl * D;
    g.ni1 = wl;
    g.ii1 = chil;
    g.ii2 = (long long)chil * wl;
    g.os0 = 1;                      // a
    g.os1 = (long long)h.pT2 * wr;  // c: rows m' + wr c of ST2
    g.no1 = D;
    g.oo1 = chil;   // p'
    g.oo2 = h.pT2;  // m'
    dev_wapply<cflt>(h.T1f, h.ST2, h.W, g, sm.u.gw.w);
  }
  tc_gemm<cplx>(chil * D, chir, wr * chir, A2, B2, y, 1, (long long)chil * D, false, sm.u.t, sm.tc);
}
#endif

// y = H_eff x.  CTA-collective.  In the mixed form x is rounded to FP32, the
// three contractions run in FP32 (tensor cores for the two GEMMs) and y is
// written back in FP64.
static __device__ __noinline__ void dev_heff(const HeffOp& h, const cplx* x, cplx* y, EngineSmem& sm) {
  const int chil = h.chil, D = h.D, chir = h.chir, wl = h.wl, wr = h.wr;
#if YAQS_TC
  if (h.tc) {
    dev_heff_tc(h, x, y, sm);
    return;
  }
#endif
  if (h.mixed) {
    GemmSmemF& gf = reinterpret_cast<GemmSmemF&>(sm.u.gw.g);
    cta_to_f32(h.xf, x, (long long)chil * D * chir);
    cta_gemm_tf32<cflt>(gemm_args_f(chil * wl, D * chir, chil, h.Lf, 1, (long long)chil * wl, h.xf, 1, chil, h.T1f,
                                    1, (long long)chil * wl),
                        gf);
  } else {
    cta_gemm(gemm_args(chil * wl, D * chir, chil, h.L, 1, (long long)chil * wl, x, 1, chil, h.T1, 1,
                       (long long)chil * wl),
             sm.u.gw.g);
  }
  WApplyGeom g;
  g.n0 = chil;
  g.n1 = chir;
  g.is0 = 1;
  g.is1 = (long long)chil * wl * D;
  g.ni1 = wl;
  g.ii1 = chil;
  g.ii2 = (long long)chil * wl;
  g.os0 = 1;
  g.os1 = (long long)chil * D * wr;
  g.no1 = D;
  g.oo1 = chil;
  g.oo2 = (long long)chil * D;
  // an identity W with D = 1 (the bond operator) leaves T1 in T2's layout.
  // With wl == wr the pair (a, b) holds its wl*D inputs and its wr*D outputs
  // at the same addresses (a + chil * j within the block of b), so the MPO
  // apply runs in place: T2's stores land on the lines T1 just left in L2
  // and one buffer per slot is written back instead of two.
  const bool inplace = wl == wr;
  if (h.mixed) {
    GemmSmemF& gf = reinterpret_cast<GemmSmemF&>(sm.u.gw.g);
    const cflt* T2 = h.T1f;
    if (!h.W.ident) {
      dev_wapply<cflt>(h.T1f, inplace ? h.T1f : h.T2f, h.W, g, sm.u.gw.w);
      T2 = inplace ? h.T1f : h.T2f;
    }
    cta_gemm_tf32<cplx>(gemm_args_f(chil * D, chir, wr * chir, T2, 1, (long long)chil * D, h.Rf, chir, 1, y, 1,
                                    (long long)chil * D),
                        gf);
  } else {
    const cplx* T2 = h.T1;
    if (!h.W.ident) {
      dev_wapply<cplx>(h.T1, inplace ? h.T1 : h.T2, h.W, g, sm.u.gw.w);
      T2 = inplace ? h.T1 : h.T2;
    }
    cta_gemm(gemm_args(chil * D, chir, wr * chir, T2, 1, (long long)chil * D, h.R, chir, 1, y, 1,
                       (long long)chil * D),
             sm.u.gw.g);
  }
}

static __device__ __forceinline__ double heff_flops(int chil, int wl, int D, int chir, int wr) {
  return 8.0 * ((double)chil * chil * wl * D * chir + (double)chil * chir * D * D * wl * wr +
                (double)chil * D * chir * chir * wr);
}

// Floating-point operations of one product in the form it takes.
static __device__ __forceinline__ double heff_work(const HeffOp& h) {
  if (!h.plan || !h.tc) return heff_flops(h.chil, h.wl, h.D, h.chir, h.wr);
  const double l = h.chil, r = h.chir;
  return 8.0 * (l * l * h.plan->nt1 * h.D * r + h.plan->nleft * l * l * r + h.plan->nright * l * r * r);
}

struct KrylovCfg {
  int kdim;
  double tol;
  double exit_tol;
};

// Warp 0: y = exp(-i dt T) e_1 for the m x m Lanczos matrix in ks, by Taylor
// series over substeps of norm <= 1/2, each stopped after the first term with
// |term|^2 < 1e-40.
//
// One serial chain on one warp while the others wait (12-31 % of a small
// chain's step when every term ended in a warp reduction and a division), so
// terms go in groups of four: their sizes are reduced together, the first
// small one is found by a ballot and the sum up to it is taken.  h / n comes
// from a table filled once.
static __device__ __noinline__ void dev_tridiag_expm(int m, double dt, KrySmem& ks) {
  ProfScope prof_scope_(PF_TRIDIAG);
  ASSUME_SHARED(&ks);
  if (ltid() >= 32) return;
  const int j = ltid();
  const bool on = j < m;
  const double a = on ? ks.alpha[j] : 0.0;
  const double bl = (on && j > 0) ? ks.beta[j - 1] : 0.0;
  const double br = (on && j + 1 < m) ? ks.beta[j] : 0.0;
  double rowsum = on ? fabs(a) + bl + br : 0.0;
  const double tn = warp_max(rowsum) * fabs(dt);
  int ns = (int)ceil(tn / 0.5);
  if (ns < 1) ns = 1;
  const double h = dt / ns;
  double* rcp = reinterpret_cast<double*>(ks.y);  // h / n; y is written at the end
  rcp[j] = h / j;
  rcp[32 + j] = h / (32 + j);
  __syncwarp();
  cplx v = make_double2(j == 0 ? 1.0 : 0.0, 0.0);
  for (int s = 0; s < ns; ++s) {
    cplx term = v, acc = v;
    for (int n0 = 1; n0 < 60; n0 += 4) {
      cplx at[4];
      double size[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        // term <- (-i h T) term / n
        cplx tl = make_double2(__shfl_up_sync(0xffffffffu, term.x, 1), __shfl_up_sync(0xffffffffu, term.y, 1));
        cplx tr = make_double2(__shfl_down_sync(0xffffffffu, term.x, 1), __shfl_down_sync(0xffffffffu, term.y, 1));
        cplx tt = make_double2(a * term.x + bl * tl.x + br * tr.x, a * term.y + bl * tl.y + br * tr.y);
        if (!on) tt = make_double2(0.0, 0.0);
        // multiply by -i h / n:  (x + i y) * (-i c) = c y - i c x
        const double c = rcp[n0 + u];
        term = make_double2(c * tt.y, -c * tt.x);
        acc = cadd(acc, term);
        at[u] = acc;
        size[u] = cabs2(term);
      }
      warp_sum_multi<4>(size);  // lane l holds the size of term l / 8 of the group
      const unsigned small = __ballot_sync(0xffffffffu, size[0] < 1e-40);
      if (small) {
        const int u = (__ffs(small) - 1) >> 3;
        acc = u == 0 ? at[0] : u == 1 ? at[1] : u == 2 ? at[2] : at[3];
        break;
      }
      if (n0 == 57) acc = at[2];  // 59 terms at most
    }
    v = acc;
  }
  __syncwarp();
  if (on) ks.y[j] = v;
}

// The roundings of the sums that FP64 sweeps keep (DevParams::blocked),
// spelled out: where a product meets a sum the compiler fuses one or the other
// factor as the code around it falls, and the last bit follows.
// v - c a
static __device__ __forceinline__ cplx csub_mul(cplx v, cplx c, cplx a) {
  return make_double2(__dsub_rn(v.x, __fma_rn(c.x, a.x, -__dmul_rn(c.y, a.y))),
                      __dsub_rn(v.y, __fma_rn(c.y, a.x, __dmul_rn(c.x, a.y))));
}
// conj(a) b
static __device__ __forceinline__ cplx cmulc_rn(cplx a, cplx b) {
  return make_double2(__fma_rn(a.x, b.x, __dmul_rn(a.y, b.y)), __fma_rn(a.x, b.y, -__dmul_rn(a.y, b.x)));
}
// |a|^2
static __device__ __forceinline__ double cabs2_rn(cplx a) { return __fma_rn(a.x, a.x, __dmul_rn(a.y, a.y)); }

// h_j = <q_j, w> (j < k) into ks.h and |w|^2 in the same pass over w: the
// first group takes seven vectors and the norm, later groups eight.  Each
// thread takes two elements per iteration so that up to 18 independent
// loads are in flight (the pass is bound by memory latency).  Out of line, like
// basis_combine: inlined into the solver the loads of a group spill (L = 30,
// chi 64: 1631 against 1513 ms; 2-site, L = 16, chi 64: 279 against 266).
static __device__ __noinline__ double lanczos_dots(const cplx* Q, long long qs, const cplx* w, int n, int k,
                                                   EngineSmem& sm) {
  ASSUME_SHARED(&sm);
  const int tid = ltid();
  double nw2 = 0.0;
  for (int j0 = 0, first = 1; j0 < k || first; first = 0) {
    const int G = first ? 7 : 8;
    double d[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) d[e] = 0.0;
#pragma unroll 1
    for (int i0 = tid; i0 < n; i0 += 2 * NT) {
      const bool two = i0 + NT < n;
      const int i1 = two ? i0 + NT : i0;
      const cplx w0 = w[i0];
      const cplx w1 = two ? w[i1] : make_double2(0.0, 0.0);
      cplx a0[8], a1[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const bool live = e < G && j0 + e < k;
        const cplx* q = Q + qs * (j0 + e);
        a0[e] = live ? q[i0] : make_double2(0.0, 0.0);
        a1[e] = live ? q[i1] : make_double2(0.0, 0.0);
      }
      if (first) d[15] += cabs2_rn(w0) + __fma_rn(w1.y, w1.y, __dmul_rn(w1.x, w1.x));
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (e == 7 && first) continue;
        const cplx p = cadd(cmulc_rn(a0[e], w0), cmulc_rn(a1[e], w1));
        d[2 * e] += p.x;
        d[2 * e + 1] += p.y;
      }
    }
    block_sum_n<16>(d, sm.r);
    if (tid < G && j0 + tid < k) sm.k.h[j0 + tid] = make_double2(d[2 * tid], d[2 * tid + 1]);
    if (first) nw2 = d[15];
    j0 += G;
  }
  cta_sync();
  return nw2;
}

// out_i = s (w_i - sum_{j<k} h_j q_j[i]) for i < n (w null: w_i = 0; out may
// be w), h in ks.h; returns the CTA sum of |out_i|^2 when norm.
// Basis vectors go in groups of eight, two elements per thread, so the loads
// of a group are in flight together.  CTA-collective.
static __device__ __noinline__ double basis_combine(const cplx* Q, long long qs, const cplx* w, cplx* out, int n,
                                                    int k, double s, bool norm, EngineSmem& sm) {
  ASSUME_SHARED(&sm);
  double part = 0.0;
#pragma unroll 1
  for (int i0 = ltid(); i0 < n; i0 += 2 * NT) {
    const bool two = i0 + NT < n;
    const int i1 = two ? i0 + NT : i0;
    cplx v0 = w ? w[i0] : make_double2(0.0, 0.0);
    cplx v1 = w ? w[i1] : make_double2(0.0, 0.0);
#pragma unroll 1
    for (int j0 = 0; j0 < k; j0 += 8) {
      cplx a0[8], a1[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const bool live = j0 + e < k;
        const cplx* q = Q + qs * (j0 + e);
        a0[e] = live ? q[i0] : make_double2(0.0, 0.0);
        a1[e] = live ? q[i1] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        if (j0 + e < k) {
          const cplx ce = sm.k.h[j0 + e];
          v0 = csub_mul(v0, ce, a0[e]);
          v1 = csub_mul(v1, ce, a1[e]);
        }
      }
    }
    v0 = cscale(v0, s);
    v1 = two ? cscale(v1, s) : make_double2(0.0, 0.0);
    out[i0] = v0;
    if (two) out[i1] = v1;
    part += cabs2_rn(v0) + cabs2_rn(v1);
  }
  if (!norm) {
    cta_sync();
    return 0.0;
  }
  return block_sum(part, sm.r);
}

// ---------------------------------------------------------------------------
// Small problems: the whole Krylov solve in shared memory
// ---------------------------------------------------------------------------
// A solve on n = chil D chir <= SMALL_N values is bound by latency, not by
// work: every H_eff product of the general path stages 64-wide tiles of
// operands that fill a corner of one, and its dot products read vectors that
// another thread has just written through L2.  Here the environments, the
// intermediates and as many Krylov vectors as fit live in the CTA's staging
// buffer, the products run on 8 x 8 blocks dealt to the warps straight from
// it, and a Lanczos step takes four barriers (eight with a refinement)
// instead of about thirty.  Loops are kept rolled: with most of its time spent
// in code that runs a few dozen times, a solve waits for instruction fetches
// before it waits for anything else.
// Every sum is formed in the general path's order (four-deep MMA steps from
// k = 0, the same reduction trees), so both give the same bits, which FP64
// sweeps need (DevParams::blocked).
// SMALL_N is one value per thread, up to which the general path adds a thread's
// values in this order too; wider solves fill its tiles.  Measured with the sweep on L = 6 Ising, chi 16, 200 trajectories, 51
// time indices: 445 ms with the general path alone, 180 ms with this one.
#define SMALL_N NT
#define SMALL_MIN_VECS 4  // Krylov vectors that have to fit beside the operands

struct SmallPlan {
  int oR, oT1, oVal, oIdx, oQ;  // offsets in the buffer; L at 0
  int nfit;                     // Krylov vectors held in the buffer
};

static __host__ __device__ __forceinline__ bool small_layout(int chil, int D, int chir, int wl, int wr, int ident,
                                                             int no, int nnz, SmallPlan& p) {
  const int n = chil * D * chir;
  if (n > SMALL_N) return false;
  const int cap = (int)(sizeof(EngineSmemU) / sizeof(cplx));
  int off = chil * wl * chil;
  p.oR = off;
  off += chir * wr * chir;
  p.oT1 = off;
  off += chil * wl * D * chir;
  p.oVal = off;
  off += ident ? 0 : nnz;
  p.oIdx = off;  // row pointers, then columns
  off += ident ? 0 : (no + 1 + nnz + 3) / 4;
  p.oQ = off;
  p.nfit = (cap - off) / n;
  return cap > off && p.nfit >= SMALL_MIN_VECS;
}
static __device__ __forceinline__ bool small_plan(const HeffOp& h, SmallPlan& p) {
  return small_layout(h.chil, h.D, h.chir, h.wl, h.wr, h.W.ident, h.W.no, h.W.nnz, p);
}

// C(M x N) = A B on 8 x 8 blocks dealt to the warps, C (m,n) at C[m + n M].
// fa(row, k) starts a row's walk at k; its () gives the value there and then
// moves on by four.  fb(k, col) gives B inside the matrix.
template <class FA, class FB>
static __device__ __forceinline__ void small_gemm(int M, int N, int K, FA fa, FB fb, cplx* C) {
  const int lane = ltid() & 31, wid = ltid() >> 5;
  const int gq = lane >> 2, tq = lane & 3;
  const int mb = (M + 7) >> 3, nb = (N + 7) >> 3;
#pragma unroll 1
  for (int q = wid; q < mb * nb; q += NW) {
    const int nq = q / mb, row = (q - nq * mb) * 8 + gq, n0 = nq * 8;
    const bool rm = row < M, rn = n0 + gq < N;
    auto arow = fa(row, tq);
    double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
#pragma unroll 1
    for (int k = tq; k - tq < K; k += 4) {
      cplx a = make_double2(0.0, 0.0), b = make_double2(0.0, 0.0);
      if (rm && k < K) a = arow();
      if (rn && k < K) b = fb(k, n0 + gq);
      dmma884(cr[0], cr[1], a.x, b.x);
      dmma884(ci[0], ci[1], a.x, b.y);
      dmma884(cr[0], cr[1], -a.y, b.y);
      dmma884(ci[0], ci[1], a.y, b.x);
    }
    if (rm) {
#pragma unroll
      for (int e = 0; e < 2; ++e)
        if (n0 + 2 * tq + e < N) C[row + (n0 + 2 * tq + e) * M] = make_double2(cr[e], ci[e]);
    }
  }
}

// w = H_eff x, all in shared memory (w may lie in global memory).  The MPO
// map is applied while the second product loads its left operand: every
// value is loaded by one block column only (chir <= 8) or a few, and T2 and
// its barriers go away.
static __device__ __noinline__ void small_heff(const HeffOp& h, const SmallPlan& p, cplx* buf, const cplx* x,
                                               cplx* w) {
  ASSUME_SHARED(buf);
  const int chil = h.chil, D = h.D, chir = h.chir, wl = h.wl, wr = h.wr;
  cplx* T1 = buf + p.oT1;
  const int ml = chil * wl;
  small_gemm(ml, D * chir, chil,
             [&](int row, int k) {
               const cplx* at = buf + row + k * ml;
               return [=]() mutable {
                 const cplx v = *at;
                 at += 4 * ml;
                 return v;
               };
             },
             [&](int k, int n) { return x[k + n * chil]; }, T1);
  cta_sync();
  const cplx* R = buf + p.oR;
  const cplx* val = buf + p.oVal;
  const int* rowp = reinterpret_cast<const int*>(buf + p.oIdx);
  const int* col = rowp + h.W.no + 1;
  const bool ident = h.W.ident != 0;
  small_gemm(chil * D, chir, wr * chir,
             [&](int row, int k) {
               // T2[a, p', m', c] = sum W[(p', m'), (m, p)] T1[a, m, p, c], k = m' + wr c;
               // ident: T2[a, k] = T1[a + chil k]
               const int pp = row / chil, a = row - pp * chil;
               int c = k / wr, mp = k - c * wr;
               const cplx* in = T1 + a + (ident ? k * chil : c * ml * D);
               return [=]() mutable {
                 if (ident) {
                   const cplx v = *in;
                   in += 4 * chil;
                   return v;
                 }
                 const int o = pp + D * mp;
                 cplx acc = make_double2(0.0, 0.0);
#pragma unroll 1
                 for (int z = rowp[o]; z < rowp[o + 1]; ++z) wfma(acc, val[z], in[col[z] * chil]);
                 for (mp += 4; mp >= wr; mp -= wr) in += ml * D;
                 return acc;
               };
             },
             [&](int k, int n) { return R[n + k * chir]; }, w);
  cta_sync();
}

// h_j = <q_j, w> (j < k) into ks.h; returns |w|^2.  A warp forms one sum: the
// tree over the lanes of each 32 values, then these in order, which is how
// the general path's threads, warps and block add them.
static __device__ __noinline__ double small_dots(const cplx* sQ, int nfit, const cplx* Q, long long qs, const cplx* w,
                                                 int n, int k, KrySmem& ks) {
  ASSUME_SHARED(&ks);
  const int lane = ltid() & 31, wid = ltid() >> 5;
#pragma unroll 1
  for (int j = wid; j <= k; j += NW) {  // j = k: the norm
    const cplx* q = j < nfit ? sQ + j * n : Q + qs * j;
    double sx = 0.0, sy = 0.0;
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 64) {
      double d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = i0 + 32 * u + lane;
        if (i < n) {
          const cplx w0 = w[i];
          if (j < k) {
            const cplx v = cmulc_rn(q[i], w0);
            d[2 * u] = v.x;
            d[2 * u + 1] = v.y;
          } else {
            d[2 * u] = cabs2_rn(w0);
          }
        }
      }
      warp_sum_multi<4>(d);  // lane l holds sum l / 8
      sx += __shfl_sync(0xffffffffu, d[0], 0);
      sy += __shfl_sync(0xffffffffu, d[0], 8);
      sx += __shfl_sync(0xffffffffu, d[0], 16);
      sy += __shfl_sync(0xffffffffu, d[0], 24);
    }
    if (lane == 0) ks.h[j] = make_double2(sx, sy);
  }
  cta_sync();
  return ks.h[k].x;
}

// dev_expm_krylov for a solve that fits small_plan.  Its vectors lie in the
// buffer or, past the first nfit, in global memory, so it is told nothing of
// where sm points; the routines that read the buffer alone are.
static __device__ __noinline__ int dev_expm_small(const HeffOp& h, const SmallPlan& p, cplx* x, double dt,
                                                  const KrylovCfg& kc, cplx* Q, long long qs, EngineSmem& sm) {
  cplx* buf = reinterpret_cast<cplx*>(&sm.u);
  cplx* sQ = buf + p.oQ;
  KrySmem& ks = sm.k;
  const int tid = ltid();
  const int n = h.chil * h.D * h.chir, nfit = p.nfit;
  const double beta0 = sqrt(cta_norm2(x, n, sm.r));
  if (beta0 == 0.0) return 0;
  const double tau = fabs(dt);
  for (int e = tid; e < h.chil * h.wl * h.chil; e += NT) buf[e] = h.L[e];
  for (int e = tid; e < h.chir * h.wr * h.chir; e += NT) buf[p.oR + e] = h.R[e];
  if (!h.W.ident) {
    int* idx = reinterpret_cast<int*>(buf + p.oIdx);
    for (int e = tid; e <= h.W.no; e += NT) idx[e] = h.W.rowp[e];
    for (int e = tid; e < h.W.nnz; e += NT) {
      idx[h.W.no + 1 + e] = h.W.col[e];
      buf[p.oVal + e] = h.W.val[e];
    }
  }
  for (int i = tid; i < n; i += NT) sQ[i] = cscale(x[i], 1.0 / beta0);
  cta_sync();
  auto vec = [&](int j) { return j < nfit ? sQ + j * n : Q + qs * j; };
  // out = s (w - sum_{j<k} h_j q_j); this thread's part of |out|^2
  auto combine = [&](const cplx* w, cplx* out, int k, double s) {
    double part = 0.0;
    for (int i = tid; i < n; i += NT) {
      cplx v = w ? w[i] : make_double2(0.0, 0.0);
#pragma unroll 2
      for (int j = 0; j < k; ++j) v = csub_mul(v, ks.h[j], j < nfit ? sQ[j * n + i] : Q[qs * j + i]);
      v = cscale(v, s);
      out[i] = v;
      part += cabs2_rn(v);
    }
    return part;
  };
  double bound = 1.0;
  int m = 0, mv = 0;
  for (int k = 1; k <= kc.kdim; ++k) {
    cplx* w = vec(k);
    small_heff(h, p, buf, vec(k - 1), w);
    ++mv;
    ProfScope orth_scope_(PF_ORTH);
    const double nw2 = small_dots(sQ, nfit, Q, qs, w, n, k, ks);
    double hh = 0.0;
    for (int j = 0; j < k; ++j) hh += cabs2(ks.h[j]);
    double a_k = ks.h[k - 1].x;
    const double r2 = nw2 - hh;
    const bool accept = r2 >= 0.5 * nw2;
    double b_k;
    if (accept) {
      b_k = sqrt(r2);
    } else {
      combine(w, w, k, 1.0);
      cta_sync();
      small_dots(sQ, nfit, Q, qs, w, n, k, ks);
      a_k += ks.h[k - 1].x;
      b_k = sqrt(block_sum(combine(w, w, k, 1.0), sm.r));
    }
    if (tid == 0) ks.alpha[k - 1] = a_k;
    m = k;
    if (b_k <= tau * kc.tol) break;
    if (k == kc.kdim) break;
    bound *= b_k * tau / k;
    if (kc.exit_tol > 0.0 && bound <= kc.exit_tol) break;
    if (tid == 0) ks.beta[k - 1] = b_k;
    const double inv = 1.0 / b_k;
    if (accept) {
      combine(w, w, k, inv);
    } else {
      for (int i = tid; i < n; i += NT) w[i] = cscale(w[i], inv);
    }
    cta_sync();
  }
  cta_sync();
  dev_tridiag_expm(m, dt, ks);
  cta_sync();
  if (tid < m) ks.h[tid] = make_double2(-ks.y[tid].x, -ks.y[tid].y);  // x = beta0 sum_j y_j q_j
  cta_sync();
  combine(nullptr, x, m, beta0);
  cta_sync();
  return mv;
}

// ---------------------------------------------------------------------------
// Lanczos steps of the runs that may reorder sums
// ---------------------------------------------------------------------------
// With w = H q_{k-1}, the projections of w' = w - sigma q_{k-1} - beta q_{k-2}
// on q_{k-1}, q_{k-2}, ..., q_0 into ks.h (ks.h[j] belongs to q_j) and |w'|^2.
// sigma and beta are what the recurrence predicts (the first diagonal entry
// and the last off-diagonal one), so what is left is small beside the residual
// and one pass leaves it orthogonal: without them the large diagonal entry
// sent half of the steps through a second projection, two more passes over the
// basis.  The passes are bound by memory latency and by L2: 7 vectors and two
// values a thread keep 16 loads in flight.  CTA-collective.
static __device__ __noinline__ double predicted_dots(const cplx* Q, long long qs, const cplx* w, int n, int k,
                                                     double sigma, double beta, EngineSmem& sm) {
  ASSUME_SHARED(&sm);
  const int tid = ltid(), lane = tid & 31, wid = tid >> 5;
  const cplx* q0 = Q + qs * (k - 1);
  const cplx* q1 = k > 1 ? q0 - qs : q0;
  if (k == 1) beta = 0.0;
  double nw2 = 0.0;
  for (int j0 = 0; j0 < k; j0 += 7) {  // vectors q_{k-1-j0}, q_{k-2-j0}, ...
    double d[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) d[e] = 0.0;
#pragma unroll 1
    for (int i0 = tid; i0 < n; i0 += 2 * NT) {
      const int i1 = i0 + NT < n ? i0 + NT : i0;
      const double on = i0 + NT < n ? 1.0 : 0.0;
      cplx a0[7], a1[7];
#pragma unroll
      for (int e = 0; e < 7; ++e) {
        const bool live = j0 + e < k;
        const cplx* q = q0 - qs * (j0 + e);
        a0[e] = live ? q[i0] : make_double2(0.0, 0.0);
        a1[e] = live ? q[i1] : make_double2(0.0, 0.0);
      }
      cplx w0 = w[i0], w1 = w[i1];
      const cplx s0 = j0 == 0 ? a0[0] : q0[i0], s1 = j0 == 0 ? a1[0] : q0[i1];
      const cplx t0 = j0 == 0 && k > 1 ? a0[1] : q1[i0], t1 = j0 == 0 && k > 1 ? a1[1] : q1[i1];
      w0.x = fma(-beta, t0.x, fma(-sigma, s0.x, w0.x));
      w0.y = fma(-beta, t0.y, fma(-sigma, s0.y, w0.y));
      w1.x = on * fma(-beta, t1.x, fma(-sigma, s1.x, w1.x));
      w1.y = on * fma(-beta, t1.y, fma(-sigma, s1.y, w1.y));
      d[14] += cabs2(w0) + cabs2(w1);
#pragma unroll
      for (int e = 0; e < 7; ++e) {
        cplx p = make_double2(d[2 * e], d[2 * e + 1]);
        cfmac(p, a0[e], w0);
        cfmac(p, a1[e], w1);
        d[2 * e] = p.x;
        d[2 * e + 1] = p.y;
      }
    }
    warp_sum_multi<16>(d);
    if ((lane & 1) == 0) sm.r.v[wid * 16 + (lane >> 1)] = d[0];
    cta_sync();
    if (tid < 16) {
      double v = 0.0;
      for (int u = 0; u < NW; ++u) v += sm.r.v[u * 16 + tid];
      sm.r.v[NW * 16 + tid] = v;
      const int j = k - 1 - j0 - (tid >> 1);
      if (tid < 14 && j >= 0) reinterpret_cast<double*>(sm.k.h + j)[tid & 1] = v;
    }
    cta_sync();
    if (j0 == 0) nw2 = sm.r.v[NW * 16 + 14];
  }
  cta_sync();
  return nw2;
}

// out = s (w - sum_{j<k} h_j q_j) with h in ks.h; w null: no w.  One pass,
// eight vectors and two values a thread at a time.  CTA-collective.
// With out32 the result is also stored in FP32.
static __device__ __noinline__ void combine_pass(const cplx* Q, long long qs, const cplx* w, cplx* out, int n, int k,
                                                 double s, EngineSmem& sm, cflt* out32 = nullptr) {
  ASSUME_SHARED(&sm);
  const cplx* h = sm.k.h;
#pragma unroll 1
  for (int i0 = ltid(); i0 < n; i0 += 2 * NT) {
    const int i1 = i0 + NT < n ? i0 + NT : i0;
    cplx v0 = w ? w[i0] : make_double2(0.0, 0.0), v1 = w ? w[i1] : make_double2(0.0, 0.0);
#pragma unroll 1
    for (int j0 = 0; j0 < k; j0 += 8) {
      cplx a0[8], a1[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const bool live = j0 + e < k;
        const cplx* q = Q + qs * (j0 + e);
        a0[e] = live ? q[i0] : make_double2(0.0, 0.0);
        a1[e] = live ? q[i1] : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const cplx c = h[min(j0 + e, KRYLOV_MAX)], nc = make_double2(-c.x, -c.y);
        cfma(v0, nc, a0[e]);
        cfma(v1, nc, a1[e]);
      }
    }
    v0 = cscale(v0, s);
    v1 = cscale(v1, s);
    out[i0] = v0;
    if (i1 != i0) out[i1] = v1;
    if (out32) {
      out32[i0] = make_float2((float)v0.x, (float)v0.y);
      if (i1 != i0) out32[i1] = make_float2((float)v1.x, (float)v1.y);
    }
  }
  cta_sync();
}

// dev_expm_krylov with predicted projections.
static __device__ __noinline__ int dev_expm_predicted(const HeffOp& h, cplx* x, double dt, const KrylovCfg& kc, cplx* Q,
                                                      long long qs, EngineSmem& sm) {
  const int tid = ltid();
  const int n = h.chil * h.D * h.chir;
  const double beta0 = sqrt(cta_norm2(x, n, sm.r));
  if (beta0 == 0.0) return 0;
  const double tau = fabs(dt);
  // the structured mixed product takes its vector in FP32 from here
  cflt* xf = h.tc && h.plan ? h.xf : nullptr;
  for (int i = tid; i < n; i += NT) {
    const cplx v = cscale(x[i], 1.0 / beta0);
    Q[i] = v;
    if (xf) xf[i] = make_float2((float)v.x, (float)v.y);
  }
  if (tid <= KRYLOV_MAX) sm.k.h[tid] = make_double2(0.0, 0.0);  // combine_pass reads whole groups
  cta_sync();
  double bound = 1.0, sigma = 0.0, beta = 0.0;
  int m = 0, mv = 0;
  for (int k = 1; k <= kc.kdim; ++k) {
    cplx* w = Q + qs * k;
    dev_heff(h, Q + qs * (k - 1), w, sm);
    ++mv;
    ProfScope orth_scope_(PF_ORTH);
    const double nw2 = predicted_dots(Q, qs, w, n, k, sigma, beta, sm);
    double hh = 0.0;
    for (int j = 0; j < k; ++j) hh += cabs2(sm.k.h[j]);
    double a_k = sm.k.h[k - 1].x + sigma;
    const double r2 = nw2 - hh;
    const bool accept = r2 >= 0.5 * nw2;  // DGKS, on what the prediction left
    cta_sync();
    if (tid == 0) {
      sm.k.h[k - 1].x += sigma;
      if (k > 1) sm.k.h[k - 2].x += beta;
    }
    cta_sync();
    double b_k;
    if (accept) {
      b_k = sqrt(r2);
    } else {
      combine_pass(Q, qs, w, w, n, k, 1.0, sm);
      const double n2 = predicted_dots(Q, qs, w, n, k, 0.0, 0.0, sm);
      a_k += sm.k.h[k - 1].x;
      hh = 0.0;
      for (int j = 0; j < k; ++j) hh += cabs2(sm.k.h[j]);
      b_k = sqrt(fmax(n2 - hh, 0.0));  // hh is rounding: the first projection took the rest
    }
    if (tid == 0) sm.k.alpha[k - 1] = a_k;
    m = k;
    if (b_k <= tau * kc.tol) break;
    if (k == kc.kdim) break;
    bound *= b_k * tau / k;
    if (kc.exit_tol > 0.0 && bound <= kc.exit_tol) break;
    if (tid == 0) sm.k.beta[k - 1] = b_k;
    combine_pass(Q, qs, w, w, n, k, 1.0 / b_k, sm, xf);
    if (k == 1) sigma = a_k;
    beta = b_k;
  }
  cta_sync();
  dev_tridiag_expm(m, dt, sm.k);
  cta_sync();
  if (tid < m) sm.k.h[tid] = make_double2(-sm.k.y[tid].x, -sm.k.y[tid].y);  // x = beta0 sum_j y_j q_j
  cta_sync();
  combine_pass(Q, qs, nullptr, x, n, m, beta0, sm);
  return mv;
}

// In place: x <- exp(-i dt H_eff) x.  Q holds kdim+1 vectors of stride qs.
// Returns the number of H_eff products.  CTA-collective.
static __device__ __noinline__ int dev_expm_krylov(const HeffOp& h, cplx* x, double dt, const KrylovCfg& kc, cplx* Q,
                                            long long qs, EngineSmem& sm) {
  SmallPlan sp;
  if (small_plan(h, sp)) return dev_expm_small(h, sp, x, dt, kc, Q, qs, sm);
  if (h.blocked) return dev_expm_predicted(h, x, dt, kc, Q, qs, sm);
  const int tid = ltid();
  const int n = h.chil * h.D * h.chir;
  const double beta0 = sqrt(cta_norm2(x, n, sm.r));
  if (beta0 == 0.0) return 0;
  const double tau = fabs(dt);
  for (int i = tid; i < n; i += NT) Q[i] = cscale(x[i], 1.0 / beta0);
  cta_sync();
  double bound = 1.0;
  int m = 0;
  int mv = 0;
  for (int k = 1; k <= kc.kdim; ++k) {
    cplx* w = Q + qs * k;
    dev_heff(h, Q + qs * (k - 1), w, sm);
    ++mv;
    ProfScope orth_scope_(PF_ORTH);
    // classical Gram-Schmidt.  One pass gives h_j = <q_j, w> and |w|^2; when
    // the projection keeps at least 1/sqrt(2) of the norm (DGKS criterion,
    // |w - Q h|^2 = |w|^2 - |h|^2 >= |w|^2 / 2) the residual norm follows from
    // Pythagoras and one more pass forms q_k = (w - Q h) / b_k; otherwise a
    // refinement pass projects again and the norm is taken directly.
    const double nw2 = lanczos_dots(Q, qs, w, n, k, sm);
    double hh = 0.0;
    for (int j = 0; j < k; ++j) hh += cabs2(sm.k.h[j]);
    double a_k = sm.k.h[k - 1].x;
    const double r2 = nw2 - hh;
    const bool accept = r2 >= 0.5 * nw2;
    double b_k;
    if (accept) {
      b_k = sqrt(r2);
    } else {
      basis_combine(Q, qs, w, w, n, k, 1.0, false, sm);
      lanczos_dots(Q, qs, w, n, k, sm);
      a_k += sm.k.h[k - 1].x;
      b_k = sqrt(basis_combine(Q, qs, w, w, n, k, 1.0, true, sm));
    }
    if (tid == 0) sm.k.alpha[k - 1] = a_k;
    m = k;
    if (b_k <= tau * kc.tol) break;
    if (k == kc.kdim) break;
    bound *= b_k * tau / k;
    if (kc.exit_tol > 0.0 && bound <= kc.exit_tol) break;
    if (tid == 0) sm.k.beta[k - 1] = b_k;
    const double inv = 1.0 / b_k;
    if (accept) {
      basis_combine(Q, qs, w, w, n, k, inv, false, sm);
    } else {
      for (int i = tid; i < n; i += NT) w[i] = cscale(w[i], inv);
      cta_sync();
    }
  }
  cta_sync();
  dev_tridiag_expm(m, dt, sm.k);
  cta_sync();
  if (tid < m) sm.k.h[tid] = make_double2(-sm.k.y[tid].x, -sm.k.y[tid].y);  // x = beta0 sum_j y_j q_j
  cta_sync();
  basis_combine(Q, qs, nullptr, x, n, m, beta0, false, sm);
  return mv;
}
