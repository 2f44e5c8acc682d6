// engine.cu — kernels and C-ABI of the B200 TJM trajectory engine.
//
// One persistent kernel launch per advance call, covering any number of
// recorded time indices (or circuit layers).  Each CTA (256 threads) owns a
// workspace slot and pulls (time index, trajectory) units from an atomic
// queue; for each it runs that trajectory's share of analog_tjm_2 /
// analog_tjm_1 (AnalogTJM.jl:21-176) or of run_digital_tjm entirely on the
// device, with the MPS of every trajectory resident in HBM throughout.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <map>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/yaqs_tjm.h"
#include "../../include/yaqs_tjm_components.h"
#include "digital.cuh"
#include "tcgemm.cuh"

#include "program.cuh"
#include "engine_dg.h"
#include "engine_tc.h"

__global__ void __launch_bounds__(NT, 2) tjm_step_kernel(const DevParams P, int first, int count) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CtaSmem& sm = *reinterpret_cast<CtaSmem*>(align_smem_1024(smraw));
  run_units(P, sm, first, count, [](Ctx& c, int j) { run_step(c, j); });
}

// Digital TJM: position 0 prepares every trajectory, position l >= 1 applies
// layer l-1 of the circuit (run_digital_tjm, DigitalTJM.jl:363-450).
__global__ void __launch_bounds__(NT, 2) digital_step_kernel(const DevParams P, const DigParams D, int first,
                                                             int count) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CtaSmem& sm = *reinterpret_cast<CtaSmem*>(align_smem_1024(smraw));
  run_units(P, sm, first, count, [&D](Ctx& c, int j) { run_digital_step(c, D, j); });
}

// Canonical defect of the listed trajectories' states, slot by slot.
__global__ void __launch_bounds__(NT, 1) gauge_kernel(const DevParams P, const int* list, int n, double* defect) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CtaSmem& sm = *reinterpret_cast<CtaSmem*>(align_smem_1024(smraw));
  const int slot = blockIdx.x;
  for (int k = slot; k < n; k += gridDim.x) {
    const int t = list[k];
    Ctx c{P, sm, P.ws + (long long)slot * P.lay.total, P.wsi + (long long)slot * P.lay.itotal, slot, t, nullptr, nullptr};
    const DState s{P.phi + (long long)t * P.mps_size, P.phi_chi + (long long)t * (P.L + 1), P.phi_oc + t};
    const double d = canonical_defect(c, s);
    if (ltid() == 0) defect[k] = d;
  }
}

// ---------------------------------------------------------------------------
// Component kernels (one CTA per problem) used by the parity tests
// ---------------------------------------------------------------------------
struct CompSmem {
  EngineSmem e;
  LinalgSmem la;
};

__global__ void __launch_bounds__(NT, 1) svd_kernel(int m, int n, const cplx* M, cplx* U, double* S, cplx* SVt,
                                                    cplx* work, long long wstride, int* iwork) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CompSmem& sm = *reinterpret_cast<CompSmem*>(align_smem_1024(smraw));
  const int b = blockIdx.x;
  const int k = min(m, n);
  const long long big = (long long)max(m, n) * max(m, n);
  cplx* w0 = work + wstride * b;
  SvdWork w;
  w.B = w0;
  w.X = w0 + big;
  w.Yo = w0 + 2 * big;
  w.Zo = w0 + 3 * big;
  w.y = w0 + 4 * big;
  w.sig = reinterpret_cast<double*>(w0 + 4 * big + max(m, n));
  w.ord = iwork + (long long)b * SVD_MAX_COLS;
  const cplx* Mb = M + (long long)m * n * b;
  if (ltid() == 0) sm.la.blocked = 0;
  cta_sync();
  SvdResult r = dev_svd(Mb, m, n, SVD_LEFT, w, sm.la, sm.e.r, sm.e.u.svd);
  dev_svd_vectors(r, k, w, sm.e.r);
  cplx* Ub = U + (long long)m * k * b;
  cplx* Sb = SVt + (long long)k * n * b;
  cta_copy(Ub, w.Yo, (long long)m * k);
  cta_sync();
  cta_gemm(gemm_args(k, n, m, w.Yo, m, 1, Mb, 1, m, Sb, 1, k, true, false), sm.e.u.gw.g);
  for (int e = ltid(); e < k * n; e += NT)
    if ((int)(e % k) >= r.rank) Sb[e] = make_double2(0.0, 0.0);
  for (int e = ltid(); e < k; e += NT) S[(long long)k * b + e] = w.sig[e];
}

__global__ void __launch_bounds__(NT, 1) qr_kernel(int m, int n, const cplx* M, cplx* Q, cplx* R, cplx* work) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CompSmem& sm = *reinterpret_cast<CompSmem*>(align_smem_1024(smraw));
  const int b = blockIdx.x;
  const int k = min(m, n);
  cplx* H = work + (long long)m * n * b;
  cta_copy(H, M + (long long)m * n * b, (long long)m * n);
  cta_sync();
  dev_qr_factor(H, m, n, sm.la, sm.e.r);
  dev_qr_formq(H, m, n, Q + (long long)m * k * b, sm.la);
  dev_qr_extract_r(H, m, n, R + (long long)k * n * b);
}

__global__ void __launch_bounds__(NT, 1) expm_kernel(int chil, int D, int chir, int wl, int wr, const cplx* Lb,
                                                     const cplx* Rb, const WMat W, cplx* x, double dt, KrylovCfg kc,
                                                     cplx* work, long long wstride, int* matvecs, int heff_only,
                                                     cplx* out) {
  extern __shared__ __align__(16) unsigned char smraw[];
  CompSmem& sm = *reinterpret_cast<CompSmem*>(align_smem_1024(smraw));
  const int b = blockIdx.x;
  const long long n = (long long)chil * D * chir;
  const long long tsz = (long long)chil * chir * max(wl, wr) * D;
  cplx* w0 = work + wstride * b;
  HeffOp h;
  h.L = Lb + (long long)chil * wl * chil * b;
  h.R = Rb + (long long)chir * wr * chir * b;
  h.W = W;
  h.chil = chil;
  h.D = D;
  h.chir = chir;
  h.wl = wl;
  h.wr = wr;
  h.T1 = w0;
  h.T2 = w0 + tsz;
  cplx* Q = w0 + 2 * tsz;
  cplx* xb = x + n * b;
  if (heff_only) {
    dev_heff(h, xb, out + n * b, sm.e);
    return;
  }
  int mv = dev_expm_krylov(h, xb, dt, kc, Q, n, sm.e);
  if (ltid() == 0) matvecs[b] = mv;
}

// FP64 FMA throughput probe: 8 independent chains per thread.
__global__ void fp64_probe_kernel(double* out, int iters, double a, double b) {
  double x0 = ltid(), x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b);
    x1 = fma(x1, a, b);
    x2 = fma(x2, a, b);
    x3 = fma(x3, a, b);
    x4 = fma(x4, a, b);
    x5 = fma(x5, a, b);
    x6 = fma(x6, a, b);
    x7 = fma(x7, a, b);
  }
  double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == 12345.678) out[0] = s;  // keep the chains live
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
using hcd = std::complex<double>;

struct yaqs_ctx {
  int device = 0;
  int sms = 0;
  std::string err;
  std::mutex mu;
  // Freed blocks of this context's runs, up to POOL_BLOCK_BYTES each, kept for
  // the next run up to POOL_KEEP_BYTES (the driver's pool: thread-safe, trimmed
  // under pressure) and given back with the context.  A small run takes about
  // as long on the device as its two dozen cudaMalloc / cudaFree pairs took on
  // the host; gigabyte blocks go through cudaMalloc, which maps them faster
  // (digital L = 40, 11 GB: 11 ms of set-up against 150 with the pool).
  cudaMemPool_t pool = nullptr;
  ~yaqs_ctx() {
    if (pool) cudaMemPoolDestroy(pool);
  }
};

namespace {

// a run holds two large blocks, trajectory states and slot workspaces: both fit
constexpr unsigned long long POOL_KEEP_BYTES = 1792ull << 20;
constexpr size_t POOL_BLOCK_BYTES = 768u << 20;

// A pool for device memory of `device`, or null (plain cudaMalloc is used then).
cudaMemPool_t make_pool(int device) {
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.handleTypes = cudaMemHandleTypeNone;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  cudaMemPool_t pool = nullptr;
  unsigned long long keep = POOL_KEEP_BYTES;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    cudaGetLastError();
    if (pool) cudaMemPoolDestroy(pool);
    return nullptr;
  }
  return pool;
}

// Gives back what the pool holds without using it; frees under way land first.
// The pool's device has to be current.
cudaError_t trim_pool(cudaMemPool_t pool) {
  const cudaError_t e = cudaStreamSynchronize(0);
  return e == cudaSuccess ? cudaMemPoolTrimTo(pool, 0) : e;
}

// Bytes the pool holds without using them: as good as free to this context.
size_t pool_idle(const yaqs_ctx* ctx) {
  unsigned long long held = 0, used = 0;
  if (!ctx->pool || cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
      cudaMemPoolGetAttribute(ctx->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    return 0;
  return held > used ? (size_t)(held - used) : 0;
}


thread_local std::string g_static_err;

int set_err(yaqs_ctx* ctx, int code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  else g_static_err = msg;
  return code;
}

#define CUDA_TRY(ctx, x)                                                                  \
  do {                                                                                    \
    cudaError_t e_ = (x);                                                                 \
    if (e_ != cudaSuccess) return set_err(ctx, YAQS_E_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
  } while (0)

// Device allocations owned by one call; freed on scope exit, when nothing on
// the device uses them any more (the owner synchronises first; a failed call's
// kernels ran on the legacy stream, which the frees are ordered in).
struct DevMem {
  cudaMemPool_t pool = nullptr;  // the context's pool, null for cudaMalloc
  std::vector<void*> ptrs, pooled;
  int device = 0;  // of the pooled blocks: their frees go to its legacy stream
  ~DevMem() {
    for (void* p : ptrs) cudaFree(p);
    if (pooled.empty()) return;
    int caller = 0;
    cudaGetDevice(&caller);
    if (caller != device) cudaSetDevice(device);
    for (void* p : pooled) cudaFreeAsync(p, 0);
    if (caller != device) cudaSetDevice(caller);
  }
  template <class T>
  cudaError_t alloc(T** p, size_t count) {
    void* q = nullptr;
    const size_t bytes = std::max<size_t>(count, 1) * sizeof(T);
    if (pool && bytes <= POOL_BLOCK_BYTES) {
      if (cudaMallocFromPoolAsync(&q, bytes, pool, 0) == cudaSuccess) {
        cudaGetDevice(&device);
        pooled.push_back(q);
        *p = reinterpret_cast<T*>(q);
        return cudaSuccess;
      }
      cudaGetLastError();
    }
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e == cudaErrorMemoryAllocation && pool) {  // what the pool holds idle counted as free
      cudaGetLastError();
      trim_pool(pool);
      e = cudaMalloc(&q, bytes);
    }
    if (e == cudaSuccess) {
      ptrs.push_back(q);
      *p = reinterpret_cast<T*>(q);
    }
    return e;
  }
};

// Tensor maps of staged tc_gemm operands (cuTensorMapEncodeTiled, reached
// through the runtime's driver entry point so the library links no driver
// stub).  A staged operand is a 2D FP32 array of `rows` rows of
// 2 * pitch floats (pitch complex values, even, so every row starts on a
// 16-byte boundary); the box is fixed by the operand's role (tcgemm.cuh).
enum TcRole { TC_A_MN = 0, TC_A_K = 1, TC_B_MN = 2, TC_B_K = 3 };

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// Fills *out for a staged operand at `base` (16-byte aligned).  Returns false
// when the driver refuses the map or the geometry breaks the alignment rules.
bool make_tc_map(CUtensorMap* out, const void* base, long long pitch, long long rows, int role) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn || pitch < 2 || (pitch & 1) || rows < 1 || (reinterpret_cast<uintptr_t>(base) & 15)) return false;
  const int inner_c = role == TC_A_MN ? TC_BM : role == TC_B_MN ? TC_BN : TC_BK;
  const int box_rows = role == TC_A_K ? TC_BM : role == TC_B_K ? TC_BN : TC_BK;
  cuuint64_t dims[2] = {(cuuint64_t)(2 * pitch), (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(2 * pitch * sizeof(float))};
  cuuint32_t box[2] = {(cuuint32_t)(2 * inner_c), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Sparse M[o, i] built from a dense lambda, in CSR.
struct HostWMat {
  int no = 0, ni = 0;
  int ident = 0;
  int idc = -1;
  bool planned = false;
  HPlan plan{};
  std::vector<int> rowp, col;
  std::vector<hcd> val;
};

template <class F>
HostWMat build_wmat(int no, int ni, F f) {
  HostWMat m;
  m.no = no;
  m.ni = ni;
  m.rowp.push_back(0);
  for (int o = 0; o < no; ++o) {
    for (int i = 0; i < ni; ++i) {
      hcd v = f(o, i);
      if (v != hcd(0.0)) {
        m.col.push_back(i);
        m.val.push_back(v);
      }
    }
    m.rowp.push_back((int)m.col.size());
  }
  return m;
}

// Channels of every bond in which the left (right) environment next to
// isometric sites is the identity: reached from the boundary through W = 1
// alone.  -1 where there is none.
template <class F>
void identity_channels(int L, const int* w, F Wat, std::vector<int>& left, std::vector<int>& right) {
  left.assign(L + 1, -1);
  right.assign(L + 1, -1);
  auto is = [&](int i, int m, int mr, bool one) {
    for (int po = 0; po < 2; ++po)
      for (int pi = 0; pi < 2; ++pi)
        if (Wat(i, m, po, pi, mr) != hcd(one && po == pi ? 1.0 : 0.0)) return false;
    return true;
  };
  left[0] = w[0] == 1 ? 0 : -1;
  for (int i = 0; i < L && left[i] >= 0; ++i)
    for (int mr = 0; mr < w[i + 1] && left[i + 1] < 0; ++mr) {
      bool ok = true;
      for (int m = 0; m < w[i] && ok; ++m) ok = is(i, m, mr, m == left[i]);
      if (ok) left[i + 1] = mr;
    }
  right[L] = w[L] == 1 ? 0 : -1;
  for (int i = L - 1; i >= 0 && right[i + 1] >= 0; --i)
    for (int m = 0; m < w[i] && right[i] < 0; ++m) {
      bool ok = true;
      for (int mr = 0; mr < w[i + 1] && ok; ++mr) ok = is(i, m, mr, mr == right[i + 1]);
      if (ok) right[i] = m;
    }
}

// The structured product of an effective-Hamiltonian map M[(p' + D m'),
// (m + wl p)] with identity channels il and ir, kept when every environment
// block has one term at most per p', every p' has one, and it multiplies no
// more chi^3 blocks than the general product (wl + wr a physical index).
void plan_heff(HostWMat& m, int D, int wl, int wr, int il, int ir) {
  if (il < 0 || ir < 0) return;
  struct Term {
    int side, mi, mp, po, pi;  // side 0: left block mi, 1: right block mp, 2: right block mp of L_mi x
    cplx coef;
  };
  std::vector<Term> terms;
  HPlan& pl = m.plan;
  pl = HPlan{};
  pl.il = il;
  pl.ir = ir;
  for (int pp = 0; pp < D; ++pp)
    for (int mp = 0; mp < wr; ++mp) {
      const int o = pp + D * mp;
      for (int z = m.rowp[o]; z < m.rowp[o + 1]; ++z) {
        const int mi = m.col[z] % wl, p = m.col[z] / wl;
        const cplx v = make_double2(m.val[z].real(), m.val[z].imag());
        if (mi == il && mp == ir) {
          pl.loc[pp + D * p] = v;
          pl.has_loc = 1;
        } else {
          terms.push_back({mp == ir ? 0 : mi == il ? 1 : 2, mi, mp, pp, p, v});
        }
      }
    }
  int lo = wl, hi = -1;
  std::array<bool, 4> has{};
  for (const Term& t : terms) {
    has[t.po] = true;
    ++(t.side == 0 ? pl.nleft : pl.nright);
    if (t.side == 2) {
      lo = std::min(lo, t.mi);
      hi = std::max(hi, t.mi);
    }
  }
  pl.nt1 = hi >= 0 ? hi - lo + 1 : 0;
  pl.t1m = hi >= 0 ? lo : 0;
  for (TsSide* sd : {&pl.left, &pl.right})
    for (int b = 0; b < TS_MAX_BLOCKS; ++b)
      for (int pp = 0; pp < 4; ++pp) sd->src[b][pp] = sd->t1[b][pp] = -1;
  bool ok = true;
  for (const Term& t : terms) {
    TsSide& sd = t.side == 0 ? pl.left : pl.right;
    const int ch = t.side == 0 ? t.mi : t.mp;
    int b = 0;
    while (b < sd.nb && sd.m[b] != ch) ++b;
    if (b == TS_MAX_BLOCKS || sd.src[b][t.po] >= 0) {
      ok = false;
      break;
    }
    if (b == sd.nb) {
      sd.m[b] = ch;
      ++sd.nb;
    }
    sd.src[b][t.po] = t.pi;
    sd.t1[b][t.po] = t.side == 2 ? t.mi - lo : -1;
    sd.coef[b][t.po] = make_float2((float)t.coef.x, (float)t.coef.y);
  }
  for (int pp = 0; pp < D; ++pp) ok = ok && has[pp];
  m.planned = ok && pl.left.nb > 0 && pl.right.nb > 0 && pl.nt1 * D + (int)terms.size() <= (wl + wr) * D;
}

// The sparse maps of an MPO (W(i, m, p_out, p_in, m') via Wat) in the order
// heff1[L], heff2[L-1] (merged two-site W of Algorithms.jl:639-643),
// envL[L], envR[L].
template <class F>
void append_mpo_wmats(int L, const int* w, F Wat, std::vector<HostWMat>& all) {
  std::vector<int> left, right;
  identity_channels(L, w, Wat, left, right);
  for (int i = 0; i < L; ++i) {  // heff1: M[(p' + 2 m'), (m + wl p)]
    int wl = w[i], wr = w[i + 1];
    all.push_back(build_wmat(2 * wr, wl * 2, [&](int o, int in) {
      int pp = o % 2, mp = o / 2, m = in % wl, p = in / wl;
      return Wat(i, m, pp, p, mp);
    }));
    plan_heff(all.back(), 2, wl, wr, left[i], right[i + 1]);
  }
  for (int i = 0; i + 1 < L; ++i) {  // heff2 (merged)
    int wl = w[i], wm = w[i + 1], wr = w[i + 2];
    std::vector<hcd> G((size_t)wl * 16 * wr, 0.0);
    for (int l = 0; l < wl; ++l)
      for (int r = 0; r < wr; ++r)
        for (int p1o = 0; p1o < 2; ++p1o)
          for (int p2o = 0; p2o < 2; ++p2o)
            for (int p1i = 0; p1i < 2; ++p1i)
              for (int p2i = 0; p2i < 2; ++p2i) {
                hcd s = 0;
                for (int k = 0; k < wm; ++k) s += Wat(i, l, p1o, p1i, k) * Wat(i + 1, k, p2o, p2i, r);
                G[l + (size_t)wl * ((p1o + 2 * p2o) + 4 * ((p1i + 2 * p2i) + 4 * (size_t)r))] = s;
              }
    all.push_back(build_wmat(4 * wr, wl * 4, [&](int o, int in) {
      int pp = o % 4, mp = o / 4, m = in % wl, p = in / wl;
      return G[m + (size_t)wl * (pp + 4 * (p + 4 * (size_t)mp))];
    }));
    plan_heff(all.back(), 4, wl, wr, left[i], right[i + 2]);
  }
  for (int i = 0; i < L; ++i) {  // envL: M[(po + 2 m'), (ml + wl pi)]
    int wl = w[i], wr = w[i + 1];
    all.push_back(build_wmat(2 * wr, wl * 2, [&](int o, int in) {
      int po = o % 2, mp = o / 2, ml = in % wl, pi = in / wl;
      return Wat(i, ml, po, pi, mp);
    }));
    all.back().idc = left[i + 1];
  }
  for (int i = 0; i < L; ++i) {  // envR: M[(po + 2 ml), (pi + 2 mr)]
    int wl = w[i], wr = w[i + 1];
    all.push_back(build_wmat(2 * wl, 2 * wr, [&](int o, int in) {
      int po = o % 2, ml = o / 2, pi = in % 2, mr = in / 2;
      return Wat(i, ml, po, pi, mr);
    }));
    all.back().idc = right[i];
  }
}

// exp(c * H) for a small Hermitian H (cyclic complex Jacobi).
void herm_expm(int n, const hcd* Hm, double c, hcd* out) {
  std::vector<hcd> A(Hm, Hm + n * n), V(n * n, 0.0);
  for (int i = 0; i < n; ++i) V[i + n * i] = 1.0;
  for (int sweep = 0; sweep < 60; ++sweep) {
    double off = 0;
    for (int i = 0; i < n; ++i)
      for (int j = 0; j < n; ++j)
        if (i != j) off += std::norm(A[i + n * j]);
    if (off < 1e-34) break;
    for (int p = 0; p < n - 1; ++p)
      for (int q = p + 1; q < n; ++q) {
        hcd apq = A[p + n * q];
        double ag = std::abs(apq);
        if (ag == 0.0) continue;
        double zeta = (A[q + n * q].real() - A[p + n * p].real()) / (2.0 * ag);
        double t = (zeta >= 0 ? 1.0 : -1.0) / (std::fabs(zeta) + std::sqrt(1.0 + zeta * zeta));
        double cc = 1.0 / std::sqrt(1.0 + t * t), s = cc * t;
        hcd e = apq / ag;
        for (int k = 0; k < n; ++k) {
          hcd x = A[k + n * p], y = A[k + n * q];
          A[k + n * p] = cc * x - s * std::conj(e) * y;
          A[k + n * q] = s * e * x + cc * y;
        }
        for (int k = 0; k < n; ++k) {
          hcd x = A[p + n * k], y = A[q + n * k];
          A[p + n * k] = cc * x - s * e * y;
          A[q + n * k] = s * std::conj(e) * x + cc * y;
        }
        for (int k = 0; k < n; ++k) {
          hcd x = V[k + n * p], y = V[k + n * q];
          V[k + n * p] = cc * x - s * std::conj(e) * y;
          V[k + n * q] = s * e * x + cc * y;
        }
      }
  }
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      hcd sacc = 0;
      for (int k = 0; k < n; ++k) sacc += V[i + n * k] * std::exp(c * A[k + n * k].real()) * std::conj(V[j + n * k]);
      out[i + n * j] = sacc;
    }
}

struct UploadedWMats {
  std::vector<WMat> heff1, heff2, envL, envR;
};

// Copies all CSR matrices into one device buffer and fills WMat views.
int upload_wmats(yaqs_ctx* ctx, DevMem& dm, const std::vector<HostWMat>& all, std::vector<WMat>& views) {
  size_t nint = 0, nval = 0;
  for (auto& m : all) {
    nint += m.rowp.size() + m.col.size();
    nval += m.val.size();
  }
  int* di = nullptr;
  cplx* dv = nullptr;
  HPlan* dplan = nullptr;  // one slot a map
  std::vector<HPlan> hp;
  CUDA_TRY(ctx, dm.alloc(&dplan, all.size()));
  CUDA_TRY(ctx, dm.alloc(&di, nint));
  CUDA_TRY(ctx, dm.alloc(&dv, nval));
  std::vector<int> hi;
  std::vector<hcd> hv;
  hi.reserve(nint);
  hv.reserve(nval);
  views.clear();
  for (auto& m : all) {
    WMat w;
    w.no = m.no;
    w.ni = m.ni;
    w.nnz = (int)m.val.size();
    w.ident = m.ident;
    w.idc = m.idc;
    w.plan = m.planned ? dplan + views.size() : nullptr;
    if (m.planned) {
      hp.resize(views.size() + 1);
      hp.back() = m.plan;
    }
    w.rowp = di + hi.size();
    hi.insert(hi.end(), m.rowp.begin(), m.rowp.end());
    w.col = di + hi.size();
    hi.insert(hi.end(), m.col.begin(), m.col.end());
    w.val = dv + hv.size();
    hv.insert(hv.end(), m.val.begin(), m.val.end());
    views.push_back(w);
  }
  if (!hp.empty()) CUDA_TRY(ctx, cudaMemcpy(dplan, hp.data(), hp.size() * sizeof(HPlan), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(di, hi.data(), hi.size() * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(dv, hv.data(), hv.size() * sizeof(hcd), cudaMemcpyHostToDevice));
  return YAQS_OK;
}

inline hcd cload(const double* p, size_t k) { return hcd(p[2 * k], p[2 * k + 1]); }

// Noise processes for the device: jump operator and the dissipators
// exp(-0.5 dt_eff gamma L^dag L) for dt_eff = dt/2 and dt (Dissipation.jl:62-69).
int pack_noise(yaqs_ctx* ctx, const yaqs_noise_desc* noise, int nprocs, int L, double dt, std::vector<DevProc>& hp,
               bool& all_zero) {
  hp.assign(std::max(nprocs, 1), DevProc());
  all_zero = true;
  for (int k = 0; k < nprocs; ++k) {
    const yaqs_noise_proc& q = noise->procs[k];
    DevProc& d = hp[k];
    memset(&d, 0, sizeof(d));
    d.nsites = q.nsites;
    d.s0 = q.site[0];
    d.s1 = q.nsites == 2 ? q.site[1] : q.site[0];
    if (q.nsites < 1 || q.nsites > 2 || d.s0 < 0 || d.s1 >= L || (q.nsites == 2 && d.s1 <= d.s0))
      return set_err(ctx, YAQS_E_ARG, "noise processes must be 1-site or 2-site (ascending) with sites in range");
    d.gamma = q.strength;
    d.drate = q.strength;
    d.pauli_name = q.pauli_name;
    d.pauli_proc = q.pauli_proc;
    if (q.strength != 0.0) all_zero = false;
    if (q.nsites == 2 && d.s1 > d.s0 + 1) {  // long-range: sig, tau, alpha, beta, dissipation rate
      if (!q.pauli_name)
        return set_err(ctx, YAQS_E_UNSUPPORTED, "Non-Pauli long-range processes not fully implemented");
      d.lr = 1;
      for (int e = 0; e < 10; ++e) d.mat[e] = make_double2(q.matrix[2 * e], q.matrix[2 * e + 1]);
      d.drate = q.matrix[20];
      continue;
    }
    const int dd = q.nsites == 1 ? 2 : 4;
    hcd M[16], LdL[16], e1[16], e2[16];
    for (int e = 0; e < dd * dd; ++e) M[e] = cload(q.matrix, e);
    for (int i = 0; i < dd; ++i)
      for (int j = 0; j < dd; ++j) {
        hcd sacc = 0;
        for (int kk = 0; kk < dd; ++kk) sacc += std::conj(M[kk + dd * i]) * M[kk + dd * j];
        LdL[i + dd * j] = sacc;
      }
    double dev = 0.0;
    for (int i = 0; i < dd; ++i)
      for (int j = 0; j < dd; ++j) dev = std::max(dev, std::abs(LdL[i + dd * j] - (i == j ? 1.0 : 0.0)));
    d.unitary = dev < 1e-13 ? 1 : 0;
    herm_expm(dd, LdL, -0.5 * (dt / 2) * q.strength, e1);
    herm_expm(dd, LdL, -0.5 * dt * q.strength, e2);
    for (int e = 0; e < dd * dd; ++e) {
      d.mat[e] = make_double2(M[e].real(), M[e].imag());
      d.diss_half[e] = make_double2(e1[e].real(), e1[e].imag());
      d.diss_full[e] = make_double2(e2[e].real(), e2[e].imag());
    }
  }
  return YAQS_OK;
}

int pack_obs(yaqs_ctx* ctx, const yaqs_obs_desc* obs, int n_obs, int L, std::vector<DevObs>& ho) {
  ho.assign(std::max(n_obs, 1), DevObs());
  for (int k = 0; k < n_obs; ++k) {
    const yaqs_obs_desc& o = obs[k];
    DevObs& d = ho[k];
    memset(&d, 0, sizeof(d));
    d.kind = o.kind;
    d.s0 = o.site[0];
    d.s1 = o.site[1];
    bool ok = (o.kind == YAQS_OBS_LOCAL1 && d.s0 >= 0 && d.s0 < L) ||
              (o.kind == YAQS_OBS_LOCAL2 && d.s0 >= 0 && d.s0 + 1 < L && d.s1 == d.s0 + 1) ||
              (o.kind == YAQS_OBS_ENTROPY && d.s0 >= 0 && d.s0 + 1 < L);
    if (!ok) return set_err(ctx, YAQS_E_ARG, "bad observable descriptor");
    const int dd = o.kind == YAQS_OBS_LOCAL2 ? 4 : 2;
    for (int e = 0; e < dd * dd; ++e) d.mat[e] = make_double2(o.matrix[2 * e], o.matrix[2 * e + 1]);
  }
  return YAQS_OK;
}

// Structural capacities cap(b) = max(min(2^min(b, L-b), chi_max), chi0(b)) of
// every bond and the sizes that follow from them.
struct Caps {
  std::vector<int> cap;
  std::vector<long long> mps_off, env_off;
  long long mps_size = 0, env_size = 0, kry_n = 0, t_size = 0;
  int capmax = 1;
};

bool plan_caps(int L, const int* chi0, const int* w, int max_bond, Caps& c) {
  c.cap.assign(L + 1, 1);
  for (int b = 0; b <= L; ++b) {
    long long sz = 1;
    const int e = std::min(b, L - b);
    for (int k = 0; k < e && sz < (1 << 20); ++k) sz *= 2;
    c.cap[b] = (int)std::max<long long>(std::min<long long>(sz, max_bond), chi0 ? chi0[b] : 1);
    if (2 * c.cap[b] > SVD_MAX_COLS) return false;
  }
  c.capmax = *std::max_element(c.cap.begin(), c.cap.end());
  c.mps_off.assign(L, 0);
  c.env_off.assign(L + 1, 0);
  c.mps_size = c.env_size = c.kry_n = c.t_size = 0;
  for (int i = 0; i < L; ++i) {
    c.mps_off[i] = c.mps_size;
    c.mps_size += (long long)c.cap[i] * 2 * c.cap[i + 1];
  }
  for (int b = 0; b <= L; ++b) {
    c.env_off[b] = c.env_size;
    c.env_size += (long long)c.cap[b] * c.cap[b] * w[b];
  }
  for (int i = 0; i < L; ++i) {
    c.kry_n = std::max(c.kry_n, (long long)c.cap[i] * 2 * c.cap[i + 1]);
    c.t_size = std::max(c.t_size, (long long)c.cap[i] * c.cap[i + 1] * 2 * std::max(w[i], w[i + 1]));
    if (i + 2 <= L) {
      c.kry_n = std::max(c.kry_n, (long long)c.cap[i] * 4 * c.cap[i + 2]);
      c.t_size = std::max(c.t_size, (long long)c.cap[i] * c.cap[i + 2] * 4 * std::max(w[i], w[i + 2]));
    }
  }
  return true;
}

// Per-slot workspace of one trajectory's program (offsets in complex-double
// units, each buffer 32-byte aligned).  analog = false leaves out what the
// digital program does not use (the sampled copy, environments, Krylov basis,
// contraction intermediates).
// True when the noise model holds a long-range process (two sites that are
// not neighbours); its jumps need the long-range work buffers.
bool has_long_range(const yaqs_noise_desc* noise, int nprocs) {
  for (int k = 0; k < nprocs; ++k)
    if (noise->procs[k].nsites == 2 && noise->procs[k].site[1] > noise->procs[k].site[0] + 1) return true;
  return false;
}

WsLayout plan_layout(int L, const Caps& c, const int* w, bool analog, int kdim, bool mixed, bool lr = false,
                     bool tc = false) {
  const long long tmp = 4LL * c.capmax * c.capmax + 16;
  WsLayout lay;
  long long off = 0;
  auto take = [&](long long n) {
    long long o = off;
    off += (n + 1) & ~1LL;
    return o;
  };
  lay.psi = take(analog ? c.mps_size : 0);
  lay.EL = take(analog ? c.env_size : 0);
  lay.ER = take(analog ? c.env_size : 0);
  lay.Q = take(analog ? (long long)(kdim + 1) * c.kry_n : 0);
  lay.T1 = take(analog ? c.t_size : 0);
  lay.T2 = take(analog ? c.t_size : 0);
  lay.tA = take(tmp);
  lay.tB = take(tmp);
  lay.tC = take(tmp);
  lay.th = take(c.kry_n);
  lay.B = take(tmp);
  lay.X = take(tmp);
  lay.Yo = take(tmp);
  lay.Zo = take(tmp);
  lay.y = take(2 * c.capmax + 16);
  lay.dbl = take((SVD_MAX_COLS + MAX_PROCS) / 2 + 8);
  // mixed form: FP32 copies of one left and one right environment, of a site
  // tensor and of a Krylov vector, and FP32 contraction intermediates
  long long emax = 0, amax = 0;
  for (int b = 0; b <= L; ++b) emax = std::max(emax, (long long)c.cap[b] * c.cap[b] * w[b]);
  for (int i = 0; i < L; ++i) amax = std::max(amax, 2LL * c.cap[i] * c.cap[i + 1]);
  const bool mf = analog && mixed;
  auto takef = [&](long long nf) { return take(mf ? (nf + 1) / 2 : 0); };
  lay.Lf = takef(emax);
  lay.Rf = takef(emax);
  lay.xf = takef(c.kry_n);
  lay.T1f = takef(c.t_size);
  lay.T2f = takef(c.t_size);
  lay.Af = takef(amax);
  // tcgen05 operands of the H_eff products (rows x pitch complex FP32 each;
  // even pitches keep every staged row on a 16-byte boundary)
  int wmax = 1;
  for (int b = 0; b <= L; ++b) wmax = std::max(wmax, w[b]);
  auto even = [](long long v) { return (int)((v + 1) & ~1LL); };
  lay.pL = even((long long)c.capmax * wmax);
  lay.rL = c.capmax;
  lay.px = even(c.capmax);
  lay.rx = 4 * c.capmax;
  lay.pT2 = even(4LL * c.capmax);
  lay.rT2 = wmax * c.capmax;
  lay.pR = even(c.capmax);
  lay.rR = wmax * c.capmax;
  const bool st = mf && tc;
  lay.sL = takef(st ? (long long)lay.pL * lay.rL : 0);
  lay.sx = takef(st ? (long long)lay.px * lay.rx : 0);
  lay.sT2 = takef(st ? (long long)lay.pT2 * lay.rT2 : 0);
  lay.sR = takef(st ? (long long)lay.pR * lay.rR : 0);
  const long long big = lr ? 8LL * c.capmax * c.capmax + 16 : 0, small = lr ? tmp : 0;
  lay.lrQ = take(lr ? 4 * c.mps_size : 0);
  lay.lrPhi = take(big);
  lay.lrM = take(big);
  lay.lrH = take(big);
  lay.lrQh = take(big);
  lay.lrL = take(small);
  lay.lrR = take(small);
  lay.lrC0 = take(small);
  lay.lrC1 = take(small);
  lay.total = off;
  long long ioff = 0;
  lay.i_chi = ioff;
  ioff += L + 1;
  lay.i_oc = ioff;
  ioff += 1;
  lay.i_ord = ioff;
  ioff += SVD_MAX_COLS;
  lay.i_cand = ioff;
  ioff += MAX_PROCS;
  lay.i_lr = ioff;
  ioff += lr ? L + 1 : 0;
  lay.itotal = (ioff + 31) & ~31LL;
  return lay;
}

// Slot workspaces owned by a server and shared by every run it admits.
struct ServePool {
  int slots = 0;
  long long ws_stride = 0, wsi_stride = 0;
  cplx* ws = nullptr;
  int* wsi = nullptr;
  // servers that admit mixed runs: the tcgen05 operands of every slot sit at
  // fixed offsets at the end of the slot (sL, sx, sT2, sR and their pitches
  // and rows in `stage`), described by tmaps[4 slot .. 4 slot + 3]
  int tc = 0;
  WsLayout stage{};
  const CUtensorMap* tmaps = nullptr;
};

}  // namespace

// One analog run held on the device between yaqs_analog_begin and
// yaqs_analog_finish: trajectory states, workspaces and outputs.
struct yaqs_run {
  yaqs_ctx* ctx = nullptr;
  DevMem dm;
  DevParams P;
  int digital = 0;  // 0 analog TJM program, 1 digital (circuit) program
  int dg = 0;       // digital run on the 128-thread kernel (engine_dg.cu)
  DigParams D;
  int slots = 0;
  size_t smem = 0;
  int num_traj = 0, n_obs = 0, ncols = 0;
  std::vector<int> launches;
  size_t next = 0;
  // whether this kind of run keeps canonical states, and what is known of each trajectory's
  enum { GAUGE_CANONICAL = 0, GAUGE_UNKNOWN = 1, GAUGE_OTHER = 2 };
  bool canonical_kind = false;
  std::vector<char> gauge;
  double device_ms = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  double* d_traj_out = nullptr;
  int* d_chi_out = nullptr;
  int* d_status = nullptr;
  unsigned long long* d_counters = nullptr;
  double* d_flops = nullptr;
  unsigned long long* d_prof = nullptr;
  ~yaqs_run() {
    if (d_prof) {
      unsigned long long* z = nullptr;
      cudaMemcpyToSymbol(g_prof, &z, sizeof(z));
      tc_set_prof(nullptr);
      dg_set_prof(nullptr);
    }
    if (stream) cudaStreamSynchronize(stream);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (stream) cudaStreamDestroy(stream);
  }
};

// Uploads what the analog and digital programs share (site capacities and
// offsets, noise processes, observables, the initial state) and allocates
// the trajectory states, per-slot workspaces and outputs.  Expects P.L,
// P.num_traj, P.mps_size, P.lay, run->slots, run->n_obs and run->ncols set.
static int setup_run(yaqs_ctx* ctx, yaqs_run* run, const std::vector<int>& cap, const std::vector<int>& chi0,
              const std::vector<int>& w, const std::vector<long long>& mps_off, const std::vector<long long>& env_off,
              const yaqs_mps_desc* psi0, const std::vector<DevProc>& hp, const std::vector<DevObs>& ho,
              const yaqs_rng_desc* rng, int nqueue, const ServePool* pool) {
  DevMem& dm = run->dm;
  DevParams& P = run->P;
  const int L = P.L, num_traj = P.num_traj, slots = run->slots, n_obs = run->n_obs, ncols = run->ncols;
  const long long mps_size = P.mps_size;
  const WsLayout& lay = P.lay;
  int *d_cap, *d_w, *d_chi0;
  long long *d_mps_off, *d_env_off;
  CUDA_TRY(ctx, dm.alloc(&d_cap, L + 1));
  CUDA_TRY(ctx, dm.alloc(&d_w, L + 1));
  CUDA_TRY(ctx, dm.alloc(&d_chi0, L + 1));
  CUDA_TRY(ctx, dm.alloc(&d_mps_off, L));
  CUDA_TRY(ctx, dm.alloc(&d_env_off, L + 1));
  CUDA_TRY(ctx, cudaMemcpy(d_cap, cap.data(), (L + 1) * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_w, w.data(), (L + 1) * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_chi0, chi0.data(), (L + 1) * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_mps_off, mps_off.data(), L * sizeof(long long), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_env_off, env_off.data(), (L + 1) * sizeof(long long), cudaMemcpyHostToDevice));
  P.cap = d_cap;
  P.w = d_w;
  P.chi0 = d_chi0;
  P.mps_off = d_mps_off;
  P.env_off = d_env_off;

  DevProc* d_procs;
  DevObs* d_obs;
  CUDA_TRY(ctx, dm.alloc(&d_procs, hp.size()));
  CUDA_TRY(ctx, dm.alloc(&d_obs, ho.size()));
  CUDA_TRY(ctx, cudaMemcpy(d_procs, hp.data(), hp.size() * sizeof(DevProc), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_obs, ho.data(), ho.size() * sizeof(DevObs), cudaMemcpyHostToDevice));
  P.procs = d_procs;
  P.obs = d_obs;
  {  // processes and 1-site observables by site
    std::vector<int> idx;
    std::vector<size_t> at;
    auto by_site = [&](size_t n, auto site_of) {  // site_of(k): its site, or -1
      at.push_back(idx.size());
      std::vector<int> off(1, 0), list;
      for (int i = 0; i < L; ++i) {
        for (size_t k = 0; k < n; ++k)
          if (site_of(k) == i) list.push_back((int)k);
        off.push_back((int)list.size());
      }
      idx.insert(idx.end(), off.begin(), off.end());
      idx.insert(idx.end(), list.begin(), list.end());
    };
    const size_t np = (size_t)P.nprocs;
    by_site(np, [&](size_t k) { return hp[k].s0; });
    by_site(np, [&](size_t k) { return hp[k].nsites == 2 ? hp[k].s1 : -1; });
    by_site((size_t)n_obs, [&](size_t k) { return ho[k].kind == OBS_LOCAL1 ? ho[k].s0 : -1; });
    int* d_idx;
    CUDA_TRY(ctx, dm.alloc(&d_idx, idx.size()));
    CUDA_TRY(ctx, cudaMemcpy(d_idx, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice));
    P.p0_off = d_idx + at[0];
    P.p1_off = d_idx + at[1];
    P.ob_off = d_idx + at[2];
    P.p0_idx = P.p0_off + L + 1;
    P.p1_idx = P.p1_off + L + 1;
    P.ob_idx = P.ob_off + L + 1;
    P.scalar_all = 1;
    P.has_lr = 0;
    for (size_t k = 0; k < np; ++k) {
      if (!hp[k].pauli_name) P.scalar_all = 0;
      if (hp[k].lr) P.has_lr = 1;
    }
    // sweeps, splits and normalisations leave canonical states; what may not:
    // long-range jumps, non-unitary 1-qubit gates (digital_begin) and states
    // put in from outside (yaqs_run_restore, looked over by check_restored).
    // FP64 analog records keep their sums' order like the sweeps: a record
    // that a symmetry makes zero is nothing but its rounding.
    P.canonical = P.has_lr || !P.blocked ? 0 : 1;
  }

  // initial state arena (compact tensors at the site slots)
  std::vector<hcd> arena((size_t)mps_size, 0.0);
  for (int i = 0; i < L; ++i) {
    const size_t n = (size_t)chi0[i] * 2 * chi0[i + 1];
    if (!psi0->tensors[i]) return set_err(ctx, YAQS_E_ARG, "null MPS tensor");
    for (size_t e = 0; e < n; ++e) arena[mps_off[i] + e] = cload(psi0->tensors[i], e);
  }
  cplx* d_psi0;
  CUDA_TRY(ctx, dm.alloc(&d_psi0, mps_size));
  CUDA_TRY(ctx, cudaMemcpy(d_psi0, arena.data(), mps_size * sizeof(cplx), cudaMemcpyHostToDevice));
  P.psi0 = d_psi0;

  cplx* d_phi;
  int *d_phi_chi, *d_phi_oc, *d_status, *d_queue, *d_chi_out, *d_wsi;
  long long* d_rng_pos;
  double *d_traj_out, *d_flops, *d_uniforms = nullptr;
  unsigned long long* d_counters;
  cplx* d_ws;
  CUDA_TRY(ctx, dm.alloc(&d_phi, (size_t)num_traj * mps_size));
  CUDA_TRY(ctx, dm.alloc(&d_phi_chi, (size_t)num_traj * (L + 1)));
  CUDA_TRY(ctx, dm.alloc(&d_phi_oc, num_traj));
  CUDA_TRY(ctx, dm.alloc(&d_status, num_traj));
  CUDA_TRY(ctx, dm.alloc(&d_queue, nqueue));
  CUDA_TRY(ctx, dm.alloc(&d_chi_out, (size_t)num_traj * ncols));
  CUDA_TRY(ctx, dm.alloc(&d_rng_pos, num_traj));
  CUDA_TRY(ctx, dm.alloc(&d_traj_out, (size_t)num_traj * std::max(n_obs, 1) * ncols));
  CUDA_TRY(ctx, dm.alloc(&d_flops, slots));
  CUDA_TRY(ctx, dm.alloc(&d_counters, (size_t)slots * 8));
  if (pool) {
    d_ws = pool->ws;
    d_wsi = pool->wsi;
    P.lay.total = pool->ws_stride;
    P.lay.itotal = pool->wsi_stride;
  } else {
    CUDA_TRY(ctx, dm.alloc(&d_ws, (size_t)slots * lay.total));
    CUDA_TRY(ctx, dm.alloc(&d_wsi, (size_t)slots * lay.itotal));
  }
  CUDA_TRY(ctx, cudaMemset(d_status, 0, num_traj * sizeof(int)));
  CUDA_TRY(ctx, cudaMemset(d_queue, 0, nqueue * sizeof(int)));
  CUDA_TRY(ctx, cudaMemset(d_rng_pos, 0, num_traj * sizeof(long long)));
  CUDA_TRY(ctx, cudaMemset(d_traj_out, 0, (size_t)num_traj * std::max(n_obs, 1) * ncols * sizeof(double)));
  CUDA_TRY(ctx, cudaMemset(d_chi_out, 0, (size_t)num_traj * ncols * sizeof(int)));
  CUDA_TRY(ctx, cudaMemset(d_flops, 0, slots * sizeof(double)));
  CUDA_TRY(ctx, cudaMemset(d_counters, 0, (size_t)slots * 8 * sizeof(unsigned long long)));
  if (rng->mode == YAQS_RNG_INJECTED) {
    CUDA_TRY(ctx, dm.alloc(&d_uniforms, (size_t)num_traj * rng->stride));
    CUDA_TRY(ctx, cudaMemcpy(d_uniforms, rng->uniforms, (size_t)num_traj * rng->stride * sizeof(double),
                             cudaMemcpyHostToDevice));
  }
  P.phi = d_phi;
  P.phi_chi = d_phi_chi;
  P.phi_oc = d_phi_oc;
  P.status = d_status;
  P.queue = d_queue;
  P.chi_out = d_chi_out;
  P.rng_pos = d_rng_pos;
  P.traj_out = d_traj_out;
  P.flops = d_flops;
  P.counters = d_counters;
  P.ws = d_ws;
  P.wsi = d_wsi;
  P.uniforms = d_uniforms;

  run->num_traj = num_traj;
  run->gauge.assign(num_traj, yaqs_run::GAUGE_CANONICAL);
  run->d_traj_out = d_traj_out;
  run->d_chi_out = d_chi_out;
  run->d_status = d_status;
  run->d_counters = d_counters;
  run->d_flops = d_flops;
  const char* pe = getenv("YAQS_PROFILE");
  if (pe && pe[0] == '1') {
    CUDA_TRY(ctx, dm.alloc(&run->d_prof, (size_t)slots * PROF_N));
    CUDA_TRY(ctx, cudaMemset(run->d_prof, 0, (size_t)slots * PROF_N * sizeof(unsigned long long)));
    CUDA_TRY(ctx, cudaMemcpyToSymbol(g_prof, &run->d_prof, sizeof(run->d_prof)));
    CUDA_TRY(ctx, tc_set_prof(run->d_prof));  // the tensor-core kernel's translation unit
    CUDA_TRY(ctx, dg_set_prof(run->d_prof));  // the 128-thread digital kernel's
  }
  CUDA_TRY(ctx, cudaStreamCreateWithFlags(&run->stream, cudaStreamNonBlocking));
  CUDA_TRY(ctx, cudaEventCreate(&run->e0));
  CUDA_TRY(ctx, cudaEventCreate(&run->e1));
  return YAQS_OK;
}

// ||W - W^dag||_F^2 / ||W||_F^2 of an MPO (host arithmetic only), formed as
// (2 tr(W^dag W) - 2 Re tr(W W)) / tr(W^dag W) from two transfer
// contractions over the bonds of two copies.  Being a difference of squared
// norms it carries rounding of about 1e-15 relative, so only values well
// above that mean anything.  0 for the zero operator; NaN for non-finite
// tensors.
static double mpo_antihermitian_sq(const yaqs_mpo_desc* H) {
  std::vector<hcd> E1(1, 1.0), E2(1, 1.0);
  int wl = 1;
  for (int site = 0; site < H->L; ++site) {
    const int wr = H->w[site + 1];
    const double* T = H->tensors[site];
    auto at = [&](int a, int o, int i, int r) {
      return cload(T, (size_t)a + (size_t)wl * (o + 2 * (i + 2 * (size_t)r)));
    };
    std::vector<hcd> N1((size_t)wr * wr, 0.0), N2((size_t)wr * wr, 0.0);
    for (int b = 0; b < wl; ++b)
      for (int a = 0; a < wl; ++a) {
        const hcd e1 = E1[a + (size_t)wl * b], e2 = E2[a + (size_t)wl * b];
        for (int rb = 0; rb < wr; ++rb)
          for (int ra = 0; ra < wr; ++ra) {
            hcd s1 = 0.0, s2 = 0.0;
            for (int o = 0; o < 2; ++o)
              for (int i = 0; i < 2; ++i) {
                s1 += std::conj(at(a, o, i, ra)) * at(b, o, i, rb);  // tr(W^dag W)
                s2 += at(a, o, i, ra) * at(b, i, o, rb);             // tr(W W)
              }
            N1[ra + (size_t)wr * rb] += e1 * s1;
            N2[ra + (size_t)wr * rb] += e2 * s2;
          }
      }
    E1.swap(N1);
    E2.swap(N2);
    wl = wr;
  }
  const double n1 = E1[0].real();
  if (n1 == 0.0) return 0.0;
  return (2.0 * n1 - 2.0 * E2[0].real()) / n1;
}

// Looks over the gauge of the trajectories restored since the last call: the
// caller's tensors may be in any, and records are read from the canonical form
// only while every trajectory is in it (to 1e-10).  On the device, all of them
// in one launch: 256 trajectories at L = 30, chi 64 take under 2 ms, where
// host loops took 9 ms for each.
static int check_restored(yaqs_ctx* ctx, yaqs_run* run) {
  DevParams& P = run->P;
  std::vector<int> list;
  for (int t = 0; t < P.num_traj; ++t)
    if (run->gauge[t] == yaqs_run::GAUGE_UNKNOWN) list.push_back(t);
  if (list.empty()) return YAQS_OK;
  if (run->canonical_kind) {
    const int n = (int)list.size();
    const size_t smem = cta_smem_bytes();
    DevMem dm;
    dm.pool = ctx->pool;
    int* d_list;
    double* d_defect;
    std::vector<double> defect(n);
    CUDA_TRY(ctx, dm.alloc(&d_list, n));
    CUDA_TRY(ctx, dm.alloc(&d_defect, n));
    CUDA_TRY(ctx, cudaMemcpy(d_list, list.data(), n * sizeof(int), cudaMemcpyHostToDevice));
    CUDA_TRY(ctx, cudaFuncSetAttribute(gauge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    gauge_kernel<<<std::min(n, run->slots), NT, smem>>>(P, d_list, n, d_defect);
    CUDA_TRY(ctx, cudaGetLastError());
    CUDA_TRY(ctx, cudaMemcpy(defect.data(), d_defect, n * sizeof(double), cudaMemcpyDeviceToHost));
    for (int k = 0; k < n; ++k)
      run->gauge[list[k]] = defect[k] < 1e-10 ? yaqs_run::GAUGE_CANONICAL : yaqs_run::GAUGE_OTHER;
    P.canonical = 1;
    for (char g : run->gauge)
      if (g == yaqs_run::GAUGE_OTHER) P.canonical = 0;
  }
  return YAQS_OK;
}

// Largest squared relative anti-Hermitian part accepted for a Hamiltonian:
// a relative defect of 1e-5, far above the rounding of the estimate.
constexpr double HERMITIAN_TOL_SQ = 1e-10;

// Uploads the launch list (time index or layer per position) and marks no
// position done for any trajectory; the last step of a run's set-up.
static int upload_positions(yaqs_ctx* ctx, yaqs_run* run) {
  int *d_jlist, *d_done;
  const size_t np = run->launches.size();
  CUDA_TRY(ctx, run->dm.alloc(&d_jlist, std::max<size_t>(np, 1)));
  CUDA_TRY(ctx, run->dm.alloc(&d_done, run->P.num_traj));
  CUDA_TRY(ctx, cudaMemcpy(d_jlist, run->launches.data(), np * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemset(d_done, 0xff, run->P.num_traj * sizeof(int)));  // -1
  run->P.jlist = d_jlist;
  run->P.done = d_done;
  run->canonical_kind = run->P.canonical != 0;
  return YAQS_OK;
}

extern "C" {

static cudaError_t noalloc_prepare(int device);

const char* yaqs_version(void) { return "yaqs-b200 0.1.0 (sm_100a, FP64 trajectory engine)"; }

int yaqs_mpo_hermitian_defect(const yaqs_mpo_desc* H, double* defect) {
  if (!H || !defect || H->L < 1 || !H->w || !H->tensors) return set_err(nullptr, YAQS_E_ARG, "null MPO descriptor");
  if (H->w[0] != 1 || H->w[H->L] != 1) return set_err(nullptr, YAQS_E_ARG, "boundary bond dimensions must be 1");
  for (int b = 0; b <= H->L; ++b)
    if (H->w[b] < 1 || H->w[b] > 8) return set_err(nullptr, YAQS_E_UNSUPPORTED, "MPO bond width must be in [1, 8]");
  for (int i = 0; i < H->L; ++i)
    if (!H->tensors[i]) return set_err(nullptr, YAQS_E_ARG, "null MPO tensor");
  const double q = mpo_antihermitian_sq(H);
  *defect = q > 0.0 ? std::sqrt(q) : (q == q ? 0.0 : q);
  return YAQS_OK;
}

int yaqs_ctx_create(int32_t device, yaqs_ctx** out) {
  if (!out) return set_err(nullptr, YAQS_E_ARG, "null out pointer");
  int n = 0;
  cudaError_t e = cudaGetDeviceCount(&n);
  if (e != cudaSuccess || n == 0) return set_err(nullptr, YAQS_E_CUDA, "no CUDA device visible");
  if (device < 0 || device >= n) return set_err(nullptr, YAQS_E_ARG, "device index out of range");
  if (cudaSetDevice(device) != cudaSuccess) return set_err(nullptr, YAQS_E_CUDA, "cudaSetDevice failed");
  // Loads the module onto the device now (the no-allocation entry point's
  // scratch array is part of it) and caches that array's device address, so
  // no later call has to load the module mid-run.  Refreshed by every new
  // context: after a cudaDeviceReset, create a new context.
  e = noalloc_prepare(device);
  if (e != cudaSuccess) return set_err(nullptr, YAQS_E_CUDA, std::string("module set-up: ") + cudaGetErrorString(e));
  yaqs_ctx* c = new yaqs_ctx();
  c->device = device;
  cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, device);
  c->pool = make_pool(device);
  *out = c;
  return YAQS_OK;
}

int yaqs_ctx_destroy(yaqs_ctx* ctx) {
  delete ctx;
  return YAQS_OK;
}

void yaqs_ctx_trim(yaqs_ctx* ctx) {
  if (!ctx || !ctx->pool) return;
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (cudaSetDevice(ctx->device) != cudaSuccess || trim_pool(ctx->pool) != cudaSuccess) cudaGetLastError();
}

const char* yaqs_last_error(const yaqs_ctx* ctx) { return ctx ? ctx->err.c_str() : g_static_err.c_str(); }

// Autotuner of the mixed H_eff products: per shape bucket (tune_index) the
// tcgen05 form or the mma.sync form, whichever a launch over every slot of
// the run applying H_eff to synthetic operands of that shape finishes first
// (mma.sync only when it is more than 5 % faster).  Choices are measured once
// per device, shape and what the tcgen05 form does there (the structured
// product with its block counts where the MPO has a plan, the general one
// elsewhere) and kept for the process, so every run of a kind uses the same
// form and a run's results do not depend on what ran before it.  Solves that
// run in shared memory take neither form; their entry is fixed.
// YAQS_AUTOTUNE=0 keeps tcgen05 everywhere.
struct TuneRecord {
  unsigned char form;
  float us_tc, us_mma;
};
static std::mutex g_tune_mu;
static std::map<std::array<int, 10>, TuneRecord> g_tune_cache;

// all: the run's maps in the order append_mpo_wmats and the bonds give them.
static int autotune_products(yaqs_ctx* ctx, yaqs_run* run, const std::vector<int>& cap, const std::vector<int>& w,
                             const std::vector<HostWMat>& all) {
  const char* env = getenv("YAQS_AUTOTUNE");
  if (env && env[0] == '0') return YAQS_OK;
  DevParams& P = run->P;
  const int L = P.L;
  struct Shape {
    int bl, br, l, D, r, site;
  };
  std::map<int, Shape> buckets;  // first occurrence of every bucket
  for (int b = 1; b < L; ++b) buckets.emplace(tune_index(cap[b], 1, cap[b]), Shape{b, b, cap[b], 1, cap[b], b});
  for (int i = 0; i < L; ++i)
    buckets.emplace(tune_index(cap[i], 2, cap[i + 1]), Shape{i, i + 1, cap[i], 2, cap[i + 1], i});
  for (int i = 0; i + 2 <= L; ++i)
    buckets.emplace(tune_index(cap[i], 4, cap[i + 2]), Shape{i, i + 2, cap[i], 4, cap[i + 2], i});
  unsigned char *d_tune, *d_tc, *d_mma;
  CUDA_TRY(ctx, run->dm.alloc(&d_tune, TUNE_ENTRIES));
  CUDA_TRY(ctx, run->dm.alloc(&d_tc, TUNE_ENTRIES));
  CUDA_TRY(ctx, run->dm.alloc(&d_mma, TUNE_ENTRIES));
  CUDA_TRY(ctx, cudaMemset(d_tc, 0, TUNE_ENTRIES));
  CUDA_TRY(ctx, cudaMemset(d_mma, 1, TUNE_ENTRIES));
  std::vector<unsigned char> table(TUNE_ENTRIES, 0);
  std::lock_guard<std::mutex> lk(g_tune_mu);
  for (const auto& kv : buckets) {
    const Shape& sh = kv.second;
    const HostWMat& W = sh.D == 1 ? all[4 * L - 1 + sh.bl] : sh.D == 2 ? all[sh.site] : all[L + sh.site];
    const HPlan none{}, &pl = W.planned ? W.plan : none;
    const std::array<int, 10> key{ctx->device, sh.l,           sh.D,   sh.r,       w[sh.bl],
                                  w[sh.br],    (int)W.planned, pl.nt1, pl.left.nb, pl.right.nb};
    SmallPlan sp;
    const bool small =
        small_layout(sh.l, sh.D, sh.r, w[sh.bl], w[sh.br], W.ident, W.no, (int)W.val.size(), sp);
    auto it = g_tune_cache.find(key);
    if (it == g_tune_cache.end()) {
      TuneRecord rec{0, 0.f, 0.f};
      CUDA_TRY(ctx, tc_tune_time(P, run->slots, d_tc, sh.bl, sh.br, sh.l, sh.D, sh.r, sh.site, 4, &rec.us_tc));
      CUDA_TRY(ctx, tc_tune_time(P, run->slots, d_mma, sh.bl, sh.br, sh.l, sh.D, sh.r, sh.site, 4, &rec.us_mma));
      rec.us_tc *= 250.f;  // ms for 4 products -> us per product
      rec.us_mma *= 250.f;
      rec.form = !small && rec.us_mma < 0.95f * rec.us_tc ? 1 : 0;
      it = g_tune_cache.emplace(key, rec).first;
    }
    table[kv.first] = it->second.form;
  }
  CUDA_TRY(ctx, cudaMemcpy(d_tune, table.data(), TUNE_ENTRIES, cudaMemcpyHostToDevice));
  P.tune = d_tune;
  return YAQS_OK;
}

static int analog_begin_impl(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_mpo_desc* H,
                             const yaqs_noise_desc* noise, const yaqs_obs_desc* obs, int32_t n_obs,
                             const yaqs_tev_config* cfg, const yaqs_rng_desc* rng, yaqs_run** out,
                             const ServePool* pool) {
  if (!ctx) return set_err(nullptr, YAQS_E_ARG, "null context");
  if (!out) return set_err(ctx, YAQS_E_ARG, "null run handle");
  *out = nullptr;
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (!psi0 || !H || !cfg || !rng || (n_obs > 0 && !obs)) return set_err(ctx, YAQS_E_ARG, "null descriptor");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int L = psi0->L;
  if (L < 2 || L > MAX_L || H->L != L) return set_err(ctx, YAQS_E_ARG, "need 2 <= L <= 256 and matching MPO length");
  if (!psi0->chi || !psi0->tensors || !H->w || !H->tensors) return set_err(ctx, YAQS_E_ARG, "null tensor arrays");
  if (psi0->chi[0] != 1 || psi0->chi[L] != 1 || H->w[0] != 1 || H->w[L] != 1)
    return set_err(ctx, YAQS_E_ARG, "boundary bond dimensions must be 1");
  for (int b = 0; b <= L; ++b) {
    if (psi0->chi[b] < 1) return set_err(ctx, YAQS_E_ARG, "bond dimension < 1");
    if (H->w[b] < 1 || H->w[b] > 8) return set_err(ctx, YAQS_E_UNSUPPORTED, "MPO bond width must be in [1, 8]");
  }
  for (int i = 0; i < L; ++i)
    if (!H->tensors[i]) return set_err(ctx, YAQS_E_ARG, "null MPO tensor");
  {  // the Krylov solver is Lanczos: refuse what the reference would hand to Arnoldi
    const double q = mpo_antihermitian_sq(H);
    if (!(q <= HERMITIAN_TOL_SQ))
      return set_err(ctx, YAQS_E_UNSUPPORTED,
                     "the Hamiltonian MPO is not Hermitian (relative anti-Hermitian part " +
                         std::to_string(q > 0.0 ? std::sqrt(q) : q) +
                         "); the engine runs Lanczos, where the reference's :auto Krylov mode switches to Arnoldi");
  }
  if (cfg->n_times < 1 || cfg->num_traj < 1 || cfg->max_bond_dim < 1 || !(cfg->dt == cfg->dt))
    return set_err(ctx, YAQS_E_ARG, "bad config (n_times, num_traj, max_bond_dim, dt)");
  if (cfg->krylov_dim < 1 || cfg->krylov_dim > KRYLOV_MAX) return set_err(ctx, YAQS_E_ARG, "krylov_dim must be in [1, 32]");
  if (cfg->order != 1 && cfg->order != 2) return set_err(ctx, YAQS_E_ARG, "order must be 1 or 2");
  if (cfg->tdvp_mode < YAQS_TDVP_2SITE || cfg->tdvp_mode > YAQS_TDVP_DYNAMIC)
    return set_err(ctx, YAQS_E_ARG, "tdvp_mode must be YAQS_TDVP_2SITE, _1SITE or _DYNAMIC");
  if (cfg->precision != YAQS_PREC_FP64 && cfg->precision != YAQS_PREC_MIXED)
    return set_err(ctx, YAQS_E_ARG, "precision must be YAQS_PREC_FP64 or YAQS_PREC_MIXED");
  if (n_obs < 0 || n_obs > MAX_OBS) return set_err(ctx, YAQS_E_ARG, "n_obs out of range");
  if (rng->mode != YAQS_RNG_PHILOX && rng->mode != YAQS_RNG_INJECTED) return set_err(ctx, YAQS_E_ARG, "bad rng mode");
  if (rng->mode == YAQS_RNG_INJECTED && (!rng->uniforms || rng->stride < 1))
    return set_err(ctx, YAQS_E_ARG, "injected uniforms need a buffer and stride >= 1");
  const int nprocs = (noise && noise->present) ? noise->n : 0;
  if (nprocs < 0 || nprocs > MAX_PROCS || (nprocs > 0 && !noise->procs)) return set_err(ctx, YAQS_E_ARG, "bad noise descriptor");

  // ---- capacities and layouts ----
  std::vector<int> chi0(psi0->chi, psi0->chi + L + 1), w(H->w, H->w + L + 1);
  Caps caps;
  if (!plan_caps(L, chi0.data(), w.data(), cfg->max_bond_dim, caps))
    return set_err(ctx, YAQS_E_UNSUPPORTED, "bond dimension above 128 is not served");
  const bool mixed = cfg->precision == YAQS_PREC_MIXED;
  // the mixed H_eff products run on tcgen05 in direct runs (the tensor-core
  // kernel, engine_tc.cu); server slots are shared by runs of different
  // shapes and keep the mma.sync form
  const bool use_tc = mixed && (!pool || pool->tc);
  WsLayout lay =
      plan_layout(L, caps, w.data(), true, cfg->krylov_dim, mixed, has_long_range(noise, nprocs), use_tc && !pool);
  if (use_tc && pool) {  // the server's fixed staging region and tensor maps
    const WsLayout& g = pool->stage;
    if (lay.pL > g.pL || lay.rL > g.rL || lay.px > g.px || lay.rx > g.rx || lay.pT2 > g.pT2 || lay.rT2 > g.rT2 ||
        lay.pR > g.pR || lay.rR > g.rR)
      return set_err(ctx, YAQS_E_UNSUPPORTED, "the request's H_eff operands exceed the server's staging shape");
    lay.sL = g.sL;
    lay.sx = g.sx;
    lay.sT2 = g.sT2;
    lay.sR = g.sR;
    lay.pL = g.pL;
    lay.px = g.px;
    lay.pT2 = g.pT2;
    lay.pR = g.pR;
  }
  const std::vector<int>& cap = caps.cap;
  const std::vector<long long>& mps_off = caps.mps_off;
  const std::vector<long long>& env_off = caps.env_off;
  const long long mps_size = caps.mps_size, kry_n = caps.kry_n;

  // ---- MPO sparse matrices (merged two-site W of Algorithms.jl:639-643) ----
  auto Wat = [&](int i, int m, int po, int pi, int mr) {
    return cload(H->tensors[i], (size_t)m + (size_t)w[i] * (po + 2 * (pi + 2 * (size_t)mr)));
  };
  std::vector<HostWMat> all;
  append_mpo_wmats(L, w.data(), Wat, all);
  std::vector<int> left, right;
  identity_channels(L, w.data(), Wat, left, right);
  for (int b = 0; b <= L; ++b) {  // bond: identity on the MPO bond, physical dimension 1
    all.push_back(build_wmat(w[b], w[b], [&](int o, int in) { return hcd(o == in ? 1.0 : 0.0, 0.0); }));
    all.back().ident = 1;
    plan_heff(all.back(), 1, w[b], w[b], left[b], right[b]);
  }
  for (auto& m : all)
    if (m.ni > WAPPLY_MAXI || m.no > WAPPLY_MAXI || (int)m.val.size() > WAPPLY_MAXNNZ)
      return set_err(ctx, YAQS_E_UNSUPPORTED, "MPO too wide for the sparse MPO apply");

  // ---- noise and observables ----
  std::vector<DevProc> hp;
  std::vector<DevObs> ho;
  bool all_zero = true;
  {
    int st = pack_noise(ctx, noise, nprocs, L, cfg->dt, hp, all_zero);
    if (st != YAQS_OK) return st;
    st = pack_obs(ctx, obs, n_obs, L, ho);
    if (st != YAQS_OK) return st;
  }

  // ---- slots and memory admission ----
  const int num_traj = cfg->num_traj;
  const int ncols = cfg->sample_timesteps ? cfg->n_times : 1;
  size_t smem = cta_smem_bytes();
  int per_sm = 0;
  if (use_tc) {  // two programs per 512-thread CTA
    CUDA_TRY(ctx, tc_kernel_prepare(&per_sm, &smem));
    per_sm = std::min(per_sm, TMEM_PROGRAMS_PER_SM);
  } else {
    CUDA_TRY(ctx, cudaFuncSetAttribute(tjm_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tjm_step_kernel, NT, smem));
  }
  if (per_sm < 1) return set_err(ctx, YAQS_E_CUDA, "kernel does not fit on an SM");
  // a mixed request in a tensor-core server must end below the slot's staging region
  if (pool && (lay.total > (use_tc ? pool->stage.sL : pool->ws_stride) || lay.itotal > pool->wsi_stride))
    return set_err(ctx, YAQS_E_UNSUPPORTED, "the request's workspace exceeds the server's slot shape");
  size_t free_b = 0, total_b = 0;
  CUDA_TRY(ctx, cudaMemGetInfo(&free_b, &total_b));
  free_b += pool_idle(ctx);
  const size_t per_traj = (size_t)mps_size * sizeof(cplx) + (L + 2) * sizeof(int) + 64 +
                          (size_t)n_obs * ncols * sizeof(double) + ncols * sizeof(int);
  const size_t per_slot = (size_t)lay.total * sizeof(cplx) + lay.itotal * sizeof(int) + 8 * 8 + 8;
  const size_t fixed = (size_t)mps_size * sizeof(cplx) + (64u << 20);
  const size_t budget = free_b > (size_t)(1u << 30) ? free_b - (size_t)(1u << 30) : 0;
  if (fixed + (size_t)num_traj * per_traj + (pool ? 0 : per_slot) > budget)
    return set_err(ctx, YAQS_E_OOM, "trajectory states do not fit in device memory");
  int slots = std::min(num_traj, ctx->sms * per_sm);
  while (slots > 1 && fixed + (size_t)num_traj * per_traj + (size_t)slots * per_slot > budget) --slots;
  if (use_tc) slots = (slots + 1) & ~1;  // whole CTAs of two programs
  if (pool) slots = pool->slots;

  yaqs_run* run = new yaqs_run();
  std::unique_ptr<yaqs_run> guard(run);
  run->ctx = ctx;
  run->dm.pool = ctx->pool;
  DevMem& dm = run->dm;
  DevParams& P = run->P;
  memset(&P, 0, sizeof(P));
  P.L = L;
  P.n_times = cfg->n_times;
  P.order = cfg->order;
  P.mixed = mixed ? 1 : 0;
  P.tc = use_tc ? 1 : 0;
  P.tdvp_mode = cfg->tdvp_mode;
  // FP64 runs keep the order of their sums: a sweep follows basis vectors that
  // rounding decides wherever a bond's state has (nearly) null directions, so
  // another order moves the records far beyond rounding.  Between the two
  // orders, relative: one-site after a lowering jump right of the middle bond
  // 1.2e-7 (L = 16, chi 128), dynamic from a product state 1e-8 to 6e-7, a
  // padded start 2e-9 to 7e-7, a saturated XY state with Pauli jumps only
  // 1.8e-6, a 2-site cut between equal Schmidt values 1e-8.  The mixed form
  // rounds its products to FP32 whatever the order: on such problems its
  // two product forms differ by as much (1.7e-2) as the two orders do (1.6e-2).
  P.blocked = mixed ? 1 : 0;
  P.sample_ts = cfg->sample_timesteps != 0;
  P.max_bond = cfg->max_bond_dim;
  P.nobs = n_obs;
  P.nprocs = nprocs;
  P.noise_present = (noise && noise->present) ? 1 : 0;
  P.all_zero = all_zero ? 1 : 0;
  P.rng_mode = rng->mode;
  P.num_traj = num_traj;
  P.traj_offset = cfg->traj_offset;
  P.ncols = ncols;
  P.dt = cfg->dt;
  P.thr = cfg->truncation_threshold;
  P.kc.kdim = cfg->krylov_dim;
  P.kc.tol = cfg->krylov_tol;
  P.kc.exit_tol = cfg->krylov_exit_tol;
  P.seed = rng->seed;
  P.stride = rng->stride;
  P.mps_size = mps_size;
  P.kry_n = kry_n;
  P.lay = lay;

  run->slots = slots;
  run->smem = smem;
  run->n_obs = n_obs;
  run->ncols = ncols;
  int st = setup_run(ctx, run, cap, chi0, w, mps_off, env_off, psi0, hp, ho, rng, cfg->n_times, pool);
  if (st != YAQS_OK) return st;
  if (use_tc && pool) {
    P.tmaps = pool->tmaps;
  } else if (use_tc) {  // four tensor maps per slot over its staged operands
    std::vector<CUtensorMap> maps(4 * (size_t)slots);
    for (int sl = 0; sl < slots; ++sl) {
      const cplx* base = P.ws + (long long)sl * P.lay.total;
      const WsLayout& y = P.lay;
      if (!make_tc_map(&maps[4 * sl + 0], base + y.sL, y.pL, y.rL, TC_A_MN) ||
          !make_tc_map(&maps[4 * sl + 1], base + y.sx, y.px, y.rx, TC_B_K) ||
          !make_tc_map(&maps[4 * sl + 2], base + y.sT2, y.pT2, y.rT2, TC_A_MN) ||
          !make_tc_map(&maps[4 * sl + 3], base + y.sR, y.pR, y.rR, TC_B_MN))
        return set_err(ctx, YAQS_E_CUDA, "cuTensorMapEncodeTiled refused a staged H_eff operand");
    }
    CUtensorMap* d_maps;
    CUDA_TRY(ctx, dm.alloc(&d_maps, maps.size()));
    CUDA_TRY(ctx, cudaMemcpy(d_maps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
    P.tmaps = d_maps;
  }
  std::vector<WMat> views;
  st = upload_wmats(ctx, dm, all, views);
  if (st != YAQS_OK) return st;
  WMat* d_views;
  CUDA_TRY(ctx, dm.alloc(&d_views, views.size()));
  CUDA_TRY(ctx, cudaMemcpy(d_views, views.data(), views.size() * sizeof(WMat), cudaMemcpyHostToDevice));
  P.wm_heff1 = d_views;
  P.wm_heff2 = d_views + L;
  P.wm_envL = d_views + L + (L - 1);
  P.wm_envR = d_views + L + (L - 1) + L;
  P.wm_bond = d_views + L + (L - 1) + L + L;

  if (use_tc) {
    st = autotune_products(ctx, run, cap, w, all);
    if (st != YAQS_OK) return st;
  }
  run->launches.push_back(0);
  for (int j = (cfg->order == 2 ? 2 : 1); j < cfg->n_times; ++j) run->launches.push_back(j);
  st = upload_positions(ctx, run);
  if (st != YAQS_OK) return st;
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  *out = guard.release();
  return YAQS_OK;
}

int yaqs_analog_begin(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_mpo_desc* H, const yaqs_noise_desc* noise,
                      const yaqs_obs_desc* obs, int32_t n_obs, const yaqs_tev_config* cfg, const yaqs_rng_desc* rng,
                      yaqs_run** out) {
  return analog_begin_impl(ctx, psi0, H, noise, obs, n_obs, cfg, rng, out, nullptr);
}

static int collect_stats(yaqs_run* run, yaqs_run_stats* stats) {
  yaqs_ctx* ctx = run->ctx;
  const int slots = run->slots;
  std::vector<unsigned long long> cnt((size_t)slots * 8);
  std::vector<double> fl(slots);
  CUDA_TRY(ctx, cudaMemcpy(cnt.data(), run->d_counters, cnt.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(fl.data(), run->d_flops, fl.size() * sizeof(double), cudaMemcpyDeviceToHost));
  memset(stats, 0, sizeof(*stats));
  for (int s = 0; s < slots; ++s) {
    stats->matvecs += cnt[s * 8 + 0];
    stats->krylov_solves += cnt[s * 8 + 1];
    stats->svds += cnt[s * 8 + 2];
    stats->jumps += cnt[s * 8 + 3];
    stats->nonfinite_fixes += cnt[s * 8 + 4];
    stats->svd_sweeps += cnt[s * 8 + 5];
    stats->flops += fl[s];
  }
  stats->device_ms = run->device_ms;
  return YAQS_OK;
}

int yaqs_analog_stats(yaqs_run* run, yaqs_run_stats* stats) {
  if (!run || !stats) return set_err(nullptr, YAQS_E_ARG, "null argument");
  std::lock_guard<std::mutex> lk(run->ctx->mu);
  CUDA_TRY(run->ctx, cudaSetDevice(run->ctx->device));
  CUDA_TRY(run->ctx, cudaStreamSynchronize(run->stream));
  return collect_stats(run, stats);
}

int yaqs_run_state(yaqs_run* run, int32_t traj, int32_t* chi_out, int32_t* oc_out, double* tensors_out,
                   int64_t capacity, int64_t* needed) {
  if (!run || !chi_out || !oc_out || !needed) return set_err(nullptr, YAQS_E_ARG, "null argument");
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (traj < 0 || traj >= run->P.num_traj) return set_err(ctx, YAQS_E_ARG, "trajectory index out of range");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaStreamSynchronize(run->stream));
  const int L = run->P.L;
  std::vector<long long> off(L);
  CUDA_TRY(ctx, cudaMemcpy(off.data(), run->P.mps_off, L * sizeof(long long), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(chi_out, run->P.phi_chi + (size_t)traj * (L + 1), (L + 1) * sizeof(int32_t),
                           cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(oc_out, run->P.phi_oc + traj, sizeof(int32_t), cudaMemcpyDeviceToHost));
  long long need = 0;
  for (int i = 0; i < L; ++i) need += 4LL * chi_out[i] * chi_out[i + 1];
  *needed = need;
  if (!tensors_out || capacity < need) return YAQS_OK;
  const cplx* base = run->P.phi + (size_t)traj * run->P.mps_size;
  double* dst = tensors_out;
  for (int i = 0; i < L; ++i) {
    const size_t n = (size_t)chi_out[i] * 2 * chi_out[i + 1];
    CUDA_TRY(ctx, cudaMemcpy(dst, base + off[i], n * sizeof(cplx), cudaMemcpyDeviceToHost));
    dst += 2 * n;
  }
  return YAQS_OK;
}

int yaqs_run_position(const yaqs_run* run, int32_t* position) {
  if (!run || !position) return set_err(nullptr, YAQS_E_ARG, "null argument");
  *position = (int32_t)run->next;
  return YAQS_OK;
}

int yaqs_run_rng(yaqs_run* run, int32_t traj, int64_t* draws) {
  if (!run || !draws) return set_err(nullptr, YAQS_E_ARG, "null argument");
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (traj < 0 || traj >= run->P.num_traj) return set_err(ctx, YAQS_E_ARG, "trajectory index out of range");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaStreamSynchronize(run->stream));
  long long v = 0;
  CUDA_TRY(ctx, cudaMemcpy(&v, run->P.rng_pos + traj, sizeof(long long), cudaMemcpyDeviceToHost));
  *draws = v;
  return YAQS_OK;
}

int yaqs_run_restore(yaqs_run* run, int32_t traj, const int32_t* chi, int32_t oc, const double* tensors,
                     int64_t draws) {
  if (!run || !chi || !tensors) return set_err(nullptr, YAQS_E_ARG, "null argument");
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  const int L = run->P.L;
  if (traj < 0 || traj >= run->P.num_traj) return set_err(ctx, YAQS_E_ARG, "trajectory index out of range");
  if (oc < 0 || oc >= L || draws < 0) return set_err(ctx, YAQS_E_ARG, "bad centre or draw count");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaStreamSynchronize(run->stream));
  std::vector<int> cap(L + 1);
  std::vector<long long> off(L);
  CUDA_TRY(ctx, cudaMemcpy(cap.data(), run->P.cap, (L + 1) * sizeof(int), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(off.data(), run->P.mps_off, L * sizeof(long long), cudaMemcpyDeviceToHost));
  if (chi[0] != 1 || chi[L] != 1) return set_err(ctx, YAQS_E_ARG, "boundary bonds must be 1");
  for (int b = 0; b <= L; ++b)
    if (chi[b] < 1 || chi[b] > cap[b]) return set_err(ctx, YAQS_E_ARG, "bond dimension beyond this run's capacity");
  run->gauge[traj] = yaqs_run::GAUGE_UNKNOWN;
  cplx* base = run->P.phi + (size_t)traj * run->P.mps_size;
  const double* src = tensors;
  for (int i = 0; i < L; ++i) {
    const size_t n = (size_t)chi[i] * 2 * chi[i + 1];
    CUDA_TRY(ctx, cudaMemcpy(base + off[i], src, n * sizeof(cplx), cudaMemcpyHostToDevice));
    src += 2 * n;
  }
  const long long d = draws;
  CUDA_TRY(ctx, cudaMemcpy(run->P.phi_chi + (size_t)traj * (L + 1), chi, (L + 1) * sizeof(int32_t),
                           cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(run->P.phi_oc + traj, &oc, sizeof(int32_t), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(run->P.rng_pos + traj, &d, sizeof(long long), cudaMemcpyHostToDevice));
  // a copy from pageable memory may return before it has landed, and the run's
  // stream does not wait for the legacy one
  CUDA_TRY(ctx, cudaStreamSynchronize(0));
  return YAQS_OK;
}

int yaqs_run_seek(yaqs_run* run, int32_t position) {
  if (!run) return set_err(nullptr, YAQS_E_ARG, "null run");
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  const int np = (int)run->launches.size();
  if (position < 1 || position > np) return set_err(ctx, YAQS_E_ARG, "position must be in [1, positions]");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaStreamSynchronize(run->stream));
  // launches from here on pull fresh unit counters, and every trajectory
  // counts as having completed exactly the position before
  CUDA_TRY(ctx, cudaMemset(run->P.queue + position, 0, (size_t)(np - position) * sizeof(int)));
  std::vector<int> done(run->P.num_traj, position - 1);
  CUDA_TRY(ctx, cudaMemcpy(run->P.done, done.data(), done.size() * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaStreamSynchronize(0));  // the run's stream does not wait for the legacy one
  run->next = position;
  return YAQS_OK;
}

int yaqs_analog_profile(yaqs_run* run, double* cycles) {
  if (!run || !cycles) return set_err(nullptr, YAQS_E_ARG, "null argument");
  for (int k = 0; k < PROF_N; ++k) cycles[k] = 0.0;
  if (!run->d_prof) return YAQS_OK;
  std::vector<unsigned long long> h((size_t)run->slots * PROF_N);
  CUDA_TRY(run->ctx, cudaMemcpy(h.data(), run->d_prof, h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
  for (int sl = 0; sl < run->slots; ++sl)
    for (int k = 0; k < PROF_N; ++k) cycles[k] += (double)h[(size_t)sl * PROF_N + k];
  return YAQS_OK;
}

int yaqs_analog_remaining(const yaqs_run* run) {
  return run ? (int)(run->launches.size() - run->next) : 0;
}

int yaqs_analog_advance(yaqs_run* run, int32_t n, double* device_ms) {
  if (!run) return set_err(nullptr, YAQS_E_ARG, "null run");
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  if (n < 0) return set_err(ctx, YAQS_E_ARG, "negative step count");
  const int avail = (int)(run->launches.size() - run->next);
  n = std::min(n, avail);
  const int cs = n > 0 ? check_restored(ctx, run) : YAQS_OK;
  if (cs != YAQS_OK) return cs;
  CUDA_TRY(ctx, cudaEventRecord(run->e0, run->stream));
  // one launch for all n positions (several when position x trajectory
  // units would overflow the 32-bit unit counter)
  const int per_launch = (int)std::max<long long>(1, (1LL << 30) / std::max(1, run->P.num_traj));
  while (n > 0) {
    const int first = (int)run->next, cnt = std::min(n, per_launch);
    run->next += cnt;
    n -= cnt;
    if (run->digital && run->dg)
      CUDA_TRY(ctx, dg_kernel_launch(run->slots, run->smem, run->stream, run->P, run->D, first, cnt));
    else if (run->digital)
      digital_step_kernel<<<run->slots, NT, run->smem, run->stream>>>(run->P, run->D, first, cnt);
    else
      if (run->P.tc)
        CUDA_TRY(ctx, tc_kernel_launch(run->slots, run->smem, run->stream, run->P, first, cnt));
      else
        tjm_step_kernel<<<run->slots, NT, run->smem, run->stream>>>(run->P, first, cnt);
    cudaError_t le = cudaGetLastError();
    if (le != cudaSuccess) return set_err(ctx, YAQS_E_CUDA, std::string("launch: ") + cudaGetErrorString(le));
  }
  CUDA_TRY(ctx, cudaEventRecord(run->e1, run->stream));
  cudaError_t se = cudaEventSynchronize(run->e1);
  if (se != cudaSuccess) return set_err(ctx, YAQS_E_CUDA, std::string("run: ") + cudaGetErrorString(se));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, run->e0, run->e1);
  run->device_ms += ms;
  if (device_ms) *device_ms = ms;
  return YAQS_OK;
}

int yaqs_analog_finish(yaqs_run* run, double* traj_out, double* mean_out, int32_t* maxchi_out,
                       yaqs_run_stats* stats) {
  if (!run) return set_err(nullptr, YAQS_E_ARG, "null run");
  std::unique_ptr<yaqs_run> guard(run);
  yaqs_ctx* ctx = run->ctx;
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  CUDA_TRY(ctx, cudaStreamSynchronize(run->stream));
  const int num_traj = run->num_traj, n_obs = run->n_obs, ncols = run->ncols;
  std::vector<double> out((size_t)num_traj * std::max(n_obs, 1) * ncols);
  std::vector<int> status(num_traj);
  CUDA_TRY(ctx, cudaMemcpy(out.data(), run->d_traj_out, out.size() * sizeof(double), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(status.data(), run->d_status, num_traj * sizeof(int), cudaMemcpyDeviceToHost));
  if (maxchi_out)
    CUDA_TRY(ctx, cudaMemcpy(maxchi_out, run->d_chi_out, (size_t)num_traj * ncols * sizeof(int), cudaMemcpyDeviceToHost));
  if (traj_out) memcpy(traj_out, out.data(), (size_t)num_traj * n_obs * ncols * sizeof(double));
  if (mean_out) {
    for (int k = 0; k < n_obs; ++k)
      for (int c = 0; c < ncols; ++c) {
        double s = 0;
        for (int t = 0; t < num_traj; ++t) s += out[((size_t)t * n_obs + k) * ncols + c];
        mean_out[(size_t)k * ncols + c] = s / num_traj;
      }
  }
  if (stats) {
    int st = collect_stats(run, stats);
    if (st != YAQS_OK) return st;
  }
  for (int t = 0; t < num_traj; ++t) {
    if (status[t] != 0) {
      const char* why = status[t] == ST_RNG           ? "injected uniform stream exhausted"
                        : status[t] == ST_UNSUPPORTED ? "bond dimension exceeded its planned capacity"
                        : status[t] == ST_TIMEOUT     ? "a bounded device wait gave up"
                                                      : "trajectory failed";
      return set_err(ctx, status[t], std::string(why) + " (trajectory " + std::to_string(t) + ")");
    }
  }
  return YAQS_OK;
}

int yaqs_analog_run(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_mpo_desc* H, const yaqs_noise_desc* noise,
                    const yaqs_obs_desc* obs, int32_t n_obs, const yaqs_tev_config* cfg, const yaqs_rng_desc* rng,
                    double* traj_out, double* mean_out, int32_t* maxchi_out, yaqs_run_stats* stats) {
  yaqs_run* run = nullptr;
  int st = yaqs_analog_begin(ctx, psi0, H, noise, obs, n_obs, cfg, rng, &run);
  if (st != YAQS_OK) return st;
  st = yaqs_analog_advance(run, yaqs_analog_remaining(run), nullptr);
  if (st != YAQS_OK) {
    yaqs_analog_finish(run, nullptr, nullptr, nullptr, nullptr);
    return st;
  }
  return yaqs_analog_finish(run, traj_out, mean_out, maxchi_out, stats);
}

// ---- digital TJM ----
namespace {
struct HostCircuit {
  std::vector<std::vector<int>> layers;  // gate indices per layer
  bool sample_at_start = false;
  std::vector<char> sample_after;  // per layer
  int n_samples = 1;
};

// process_circuit (DigitalTJM.jl:86-145) and _sample_plan (:159-168): gates
// are packed greedily in program order, a new layer starting whenever a gate
// touches a site the current layer already uses; a barrier closes the current
// layer, and a sampling barrier requests a measurement after the layers
// completed so far (before the first layer when none is).
int plan_circuit(yaqs_ctx* ctx, const yaqs_gate_desc* gates, int n, int L, HostCircuit& c) {
  std::vector<int> cur;
  std::vector<char> busy(L, 0);
  std::vector<std::pair<int, bool>> barriers;
  for (int g = 0; g < n; ++g) {
    const yaqs_gate_desc& q = gates[g];
    if (q.kind == YAQS_GATE_BARRIER) {
      if (!cur.empty()) {
        c.layers.push_back(cur);
        cur.clear();
        std::fill(busy.begin(), busy.end(), 0);
      }
      barriers.push_back({(int)c.layers.size(), q.sample != 0});
      continue;
    }
    const int a = q.site[0], b = q.kind == YAQS_GATE_2Q ? q.site[1] : q.site[0];
    if ((q.kind != YAQS_GATE_1Q && q.kind != YAQS_GATE_2Q) || a < 0 || a >= L || b < 0 || b >= L ||
        (q.kind == YAQS_GATE_2Q && a == b))
      return set_err(ctx, YAQS_E_ARG, "bad gate descriptor (gate " + std::to_string(g) + ")");
    if (busy[a] || busy[b]) {
      c.layers.push_back(cur);
      cur.clear();
      std::fill(busy.begin(), busy.end(), 0);
    }
    cur.push_back(g);
    busy[a] = busy[b] = 1;
  }
  if (!cur.empty()) c.layers.push_back(cur);
  c.sample_after.assign(c.layers.size(), 0);
  for (auto& bs : barriers) {
    if (!bs.second) continue;
    if (bs.first == 0)
      c.sample_at_start = true;
    else
      c.sample_after[bs.first - 1] = 1;
  }
  int ns = c.sample_at_start ? 1 : 0;
  for (char x : c.sample_after) ns += x ? 1 : 0;
  c.n_samples = ns == 0 ? 1 : ns;
  return YAQS_OK;
}

int digital_begin(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_gate_desc* gates, int32_t n_gates,
                  const yaqs_noise_desc* noise, const yaqs_obs_desc* obs, int32_t n_obs,
                  const yaqs_circuit_config* cfg, const yaqs_rng_desc* rng, yaqs_run** out,
                  const ServePool* pool = nullptr) {
  if (!ctx) return set_err(nullptr, YAQS_E_ARG, "null context");
  *out = nullptr;
  std::lock_guard<std::mutex> lk(ctx->mu);
  if (!psi0 || !cfg || !rng || (n_obs > 0 && !obs) || n_gates < 0 || (n_gates > 0 && !gates))
    return set_err(ctx, YAQS_E_ARG, "null descriptor");
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int L = psi0->L;
  if (L < 2 || L > MAX_L) return set_err(ctx, YAQS_E_ARG, "need 2 <= L <= 256");
  if (!psi0->chi || !psi0->tensors) return set_err(ctx, YAQS_E_ARG, "null tensor arrays");
  if (psi0->chi[0] != 1 || psi0->chi[L] != 1) return set_err(ctx, YAQS_E_ARG, "boundary bond dimensions must be 1");
  for (int b = 0; b <= L; ++b)
    if (psi0->chi[b] < 1) return set_err(ctx, YAQS_E_ARG, "bond dimension < 1");
  if (cfg->num_traj < 1 || cfg->max_bond_dim < 1) return set_err(ctx, YAQS_E_ARG, "bad config (num_traj, max_bond_dim)");
  if (cfg->local_method < YAQS_METHOD_TEBD || cfg->local_method > YAQS_METHOD_TDVP ||
      cfg->long_range_method < YAQS_METHOD_TEBD || cfg->long_range_method > YAQS_METHOD_TDVP)
    return set_err(ctx, YAQS_E_ARG, "gate methods must be YAQS_METHOD_TEBD or YAQS_METHOD_TDVP");
  if (cfg->precision != YAQS_PREC_FP64)
    return set_err(ctx, YAQS_E_UNSUPPORTED,
                   "digital runs are served in ComplexF64 only (their work is SVD/QR, which stays FP64)");
  if (n_obs < 0 || n_obs > MAX_OBS) return set_err(ctx, YAQS_E_ARG, "n_obs out of range");
  if (rng->mode != YAQS_RNG_PHILOX && rng->mode != YAQS_RNG_INJECTED) return set_err(ctx, YAQS_E_ARG, "bad rng mode");
  if (rng->mode == YAQS_RNG_INJECTED && (!rng->uniforms || rng->stride < 1))
    return set_err(ctx, YAQS_E_ARG, "injected uniforms need a buffer and stride >= 1");
  const int nprocs = (noise && noise->present) ? noise->n : 0;
  if (nprocs < 0 || nprocs > MAX_PROCS || (nprocs > 0 && !noise->procs)) return set_err(ctx, YAQS_E_ARG, "bad noise descriptor");
  HostCircuit C;
  int st = plan_circuit(ctx, gates, n_gates, L, C);
  if (st != YAQS_OK) return st;
  // gates applied through a TDVP window need their generators
  auto by_tdvp = [&](const yaqs_gate_desc& q) {
    if (q.kind != YAQS_GATE_2Q) return false;
    const bool lr = std::abs(q.site[0] - q.site[1]) > 1;
    return (lr ? cfg->long_range_method : cfg->local_method) == YAQS_METHOD_TDVP;
  };
  bool any_tdvp = false;
  for (int g = 0; g < n_gates; ++g)
    if (by_tdvp(gates[g])) {
      any_tdvp = true;
      if (!gates[g].has_generator)
        return set_err(ctx, YAQS_E_ARG, "a gate applied by TDVP needs its generator (GateLibrary.generator)");
    }
  const int kdim = 25;  // expm_krylov(..., 25) of the circuit sweeps (Algorithms.jl:185)

  // ---- capacities and layout (environments and Krylov basis only for TDVP windows) ----
  std::vector<int> chi0(psi0->chi, psi0->chi + L + 1), w(L + 1, 1);
  Caps caps;
  if (!plan_caps(L, chi0.data(), w.data(), cfg->max_bond_dim, caps))
    return set_err(ctx, YAQS_E_UNSUPPORTED, "bond dimension above 128 is not served");
  const WsLayout lay = plan_layout(L, caps, w.data(), any_tdvp, kdim, false, has_long_range(noise, nprocs));
  const std::vector<int>& cap = caps.cap;
  const std::vector<long long>& mps_off = caps.mps_off;
  const std::vector<long long>& env_off = caps.env_off;
  const long long mps_size = caps.mps_size, kry_n = caps.kry_n;

  // gate noise uses dt = 1 (DigitalTJM.jl:412-413)
  std::vector<DevProc> hp;
  std::vector<DevObs> ho;
  bool all_zero = true;
  st = pack_noise(ctx, noise, nprocs, L, 1.0, hp, all_zero);
  if (st != YAQS_OK) return st;
  st = pack_obs(ctx, obs, n_obs, L, ho);
  if (st != YAQS_OK) return st;

  // ---- slots and memory admission ----
  const int num_traj = cfg->num_traj;
  const int ncols = C.n_samples;
  const int n_layers = (int)C.layers.size();
  // direct runs take the 128-thread program kernel (three CTAs per SM) unless
  // YAQS_DIGITAL_THREADS=256 asks for the 256-thread one; a server's pool
  // runs digital units in its own kernel
  const char* dg_env = getenv("YAQS_DIGITAL_THREADS");
  const bool use_dg = !pool && !(dg_env && atoi(dg_env) == 256);
  size_t smem = cta_smem_bytes();
  int per_sm = 0;
  if (use_dg) {
    CUDA_TRY(ctx, dg_kernel_prepare(&per_sm, &smem));
  } else {
    CUDA_TRY(ctx, cudaFuncSetAttribute(digital_step_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, digital_step_kernel, NT, smem));
  }
  if (per_sm < 1) return set_err(ctx, YAQS_E_CUDA, "kernel does not fit on an SM");
  if (pool && (lay.total > pool->ws_stride || lay.itotal > pool->wsi_stride))
    return set_err(ctx, YAQS_E_UNSUPPORTED, "the request's workspace exceeds the server's slot shape");
  size_t free_b = 0, total_b = 0;
  CUDA_TRY(ctx, cudaMemGetInfo(&free_b, &total_b));
  free_b += pool_idle(ctx);
  const size_t per_traj = (size_t)mps_size * sizeof(cplx) + (L + 2) * sizeof(int) + 64 +
                          (size_t)n_obs * ncols * sizeof(double) + ncols * sizeof(int);
  const size_t per_slot = (size_t)lay.total * sizeof(cplx) + lay.itotal * sizeof(int) + 8 * 8 + 8;
  const size_t fixed = (size_t)mps_size * sizeof(cplx) + (size_t)(n_gates + 1) * sizeof(DevGate) + (64u << 20);
  const size_t budget = free_b > (size_t)(1u << 30) ? free_b - (size_t)(1u << 30) : 0;
  if (fixed + (size_t)num_traj * per_traj + (pool ? 0 : per_slot) > budget)
    return set_err(ctx, YAQS_E_OOM, "trajectory states do not fit in device memory");
  int slots = std::min(num_traj, ctx->sms * per_sm);
  while (slots > 1 && fixed + (size_t)num_traj * per_traj + (size_t)slots * per_slot > budget) --slots;
  if (pool) slots = pool->slots;

  yaqs_run* run = new yaqs_run();
  std::unique_ptr<yaqs_run> guard(run);
  run->ctx = ctx;
  run->dm.pool = ctx->pool;
  run->digital = 1;
  run->dg = use_dg ? 1 : 0;
  DevParams& P = run->P;
  memset(&P, 0, sizeof(P));
  P.L = L;
  P.n_times = n_layers + 1;
  // TDVP windows are 2-site sweeps and keep the order of their sums like the
  // analog ones (a Trotterised Ising chain from x+, threshold 1e-6: 1e-4 between
  // the two orders, the oracle against itself 2e-5).  TEBD circuits do not need
  // it: within 1e-10 at a threshold of 1e-6 and 2e-12 below, over 500 runs;
  // where the bond cap cuts between equal Schmidt values (Clifford circuits past
  // their cap) rounding decides in any order.
  P.blocked = any_tdvp ? 0 : 1;
  P.max_bond = cfg->max_bond_dim;
  P.nobs = n_obs;
  P.nprocs = nprocs;
  P.noise_present = (noise && noise->present) ? 1 : 0;
  P.all_zero = all_zero ? 1 : 0;
  P.rng_mode = rng->mode;
  P.num_traj = num_traj;
  P.traj_offset = cfg->traj_offset;
  P.ncols = ncols;
  P.dt = 1.0;
  P.thr = cfg->truncation_threshold;
  P.kc.kdim = kdim;
  P.kc.tol = 1e-10;
  P.kc.exit_tol = 1e-12;
  P.seed = rng->seed;
  P.stride = rng->stride;
  P.mps_size = mps_size;
  P.kry_n = kry_n;
  P.lay = lay;
  run->slots = slots;
  run->smem = smem;
  run->n_obs = n_obs;
  run->ncols = ncols;
  st = setup_run(ctx, run, cap, chi0, w, mps_off, env_off, psi0, hp, ho, rng, n_layers + 1, pool);
  if (st != YAQS_OK) return st;

  // ---- gates in layer order; window maps of the TDVP gates ----
  std::vector<DevGate> hg;
  std::vector<HostWMat> wall;
  std::vector<int> layer_off(1, 0), sample_col(std::max(n_layers, 1), -1);
  int col = C.sample_at_start ? 1 : 0;
  for (int l = 0; l < n_layers; ++l) {
    for (int g : C.layers[l]) {
      const yaqs_gate_desc& q = gates[g];
      DevGate d;
      memset(&d, 0, sizeof(d));
      d.kind = q.kind;
      d.a = q.kind == YAQS_GATE_2Q ? std::min(q.site[0], q.site[1]) : q.site[0];
      d.b = q.kind == YAQS_GATE_2Q ? std::max(q.site[0], q.site[1]) : q.site[0];
      d.wm = -1;
      const int dd = q.kind == YAQS_GATE_2Q ? 4 : 2;
      for (int e = 0; e < dd * dd; ++e) d.mat[e] = make_double2(q.matrix[2 * e], q.matrix[2 * e + 1]);
      if (dd == 2) {  // applied off the centre: keeps the gauge only when unitary
        double dev = 0.0;
        for (int i = 0; i < 2; ++i)
          for (int j = 0; j < 2; ++j) {
            hcd v = i == j ? -1.0 : 0.0;
            for (int k = 0; k < 2; ++k) v += std::conj(cload(q.matrix, k + 2 * i)) * cload(q.matrix, k + 2 * j);
            dev = std::max(dev, std::abs(v));
          }
        if (!(dev < 1e-14)) P.canonical = 0;
      }
      if (by_tdvp(q)) {
        // construct_window_mpo (DigitalTJM.jl:192-236): coeff g(s1) on the
        // first window site, g(s2) on the last, identities between, bond 1
        const int n = d.b - d.a + 1;
        const double* gs1 = q.site[0] == d.a ? q.gen1 : q.gen2;
        const double* gs2 = q.site[0] == d.a ? q.gen2 : q.gen1;
        std::vector<int> wone(n + 1, 1);
        auto Wat = [&](int j, int, int po, int pi, int) {
          if (j == 0) return q.coeff * cload(gs1, po + 2 * pi);
          if (j == n - 1) return cload(gs2, po + 2 * pi);
          return hcd(po == pi ? 1.0 : 0.0, 0.0);
        };
        d.wm = (int)wall.size();
        append_mpo_wmats(n, wone.data(), Wat, wall);
      }
      hg.push_back(d);
    }
    layer_off.push_back((int)hg.size());
    if (C.sample_after[l]) sample_col[l] = col++;
  }
  if (hg.empty()) hg.resize(1);
  DevGate* d_gates;
  int *d_layer_off, *d_sample_col;
  CUDA_TRY(ctx, run->dm.alloc(&d_gates, hg.size()));
  CUDA_TRY(ctx, run->dm.alloc(&d_layer_off, layer_off.size()));
  CUDA_TRY(ctx, run->dm.alloc(&d_sample_col, sample_col.size()));
  CUDA_TRY(ctx, cudaMemcpy(d_gates, hg.data(), hg.size() * sizeof(DevGate), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_layer_off, layer_off.data(), layer_off.size() * sizeof(int), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(d_sample_col, sample_col.data(), sample_col.size() * sizeof(int), cudaMemcpyHostToDevice));
  DigParams& D = run->D;
  D.wm = nullptr;
  if (!wall.empty()) {
    std::vector<WMat> views;
    st = upload_wmats(ctx, run->dm, wall, views);
    if (st != YAQS_OK) return st;
    WMat* d_wm;
    CUDA_TRY(ctx, run->dm.alloc(&d_wm, views.size()));
    CUDA_TRY(ctx, cudaMemcpy(d_wm, views.data(), views.size() * sizeof(WMat), cudaMemcpyHostToDevice));
    D.wm = d_wm;
  }
  D.gates = d_gates;
  D.layer_off = d_layer_off;
  D.sample_col = d_sample_col;
  D.n_layers = n_layers;
  D.sample_at_start = C.sample_at_start ? 1 : 0;
  D.any_sample = (col > 0) ? 1 : 0;
  for (int j = 0; j <= n_layers; ++j) run->launches.push_back(j);
  st = upload_positions(ctx, run);
  if (st != YAQS_OK) return st;
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  *out = guard.release();
  return YAQS_OK;
}
}  // namespace

int yaqs_digital_plan(const yaqs_gate_desc* gates, int32_t n_gates, int32_t* n_layers, int32_t* n_samples) {
  if (n_gates < 0 || (n_gates > 0 && !gates) || !n_layers || !n_samples)
    return set_err(nullptr, YAQS_E_ARG, "null argument");
  int L = 1;
  for (int g = 0; g < n_gates; ++g)
    if (gates[g].kind != YAQS_GATE_BARRIER)
      L = std::max(L, std::max(gates[g].site[0], gates[g].kind == YAQS_GATE_2Q ? gates[g].site[1] : 0) + 1);
  HostCircuit C;
  int st = plan_circuit(nullptr, gates, n_gates, L, C);
  if (st != YAQS_OK) return st;
  *n_layers = (int32_t)C.layers.size();
  *n_samples = C.n_samples;
  return YAQS_OK;
}

int yaqs_digital_begin(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_gate_desc* gates, int32_t n_gates,
                       const yaqs_noise_desc* noise, const yaqs_obs_desc* obs, int32_t n_obs,
                       const yaqs_circuit_config* cfg, const yaqs_rng_desc* rng, yaqs_run** out) {
  if (!out) return set_err(ctx, YAQS_E_ARG, "null run handle");
  return digital_begin(ctx, psi0, gates, n_gates, noise, obs, n_obs, cfg, rng, out);
}

int yaqs_digital_run(yaqs_ctx* ctx, const yaqs_mps_desc* psi0, const yaqs_gate_desc* gates, int32_t n_gates,
                     const yaqs_noise_desc* noise, const yaqs_obs_desc* obs, int32_t n_obs,
                     const yaqs_circuit_config* cfg, const yaqs_rng_desc* rng, double* traj_out, double* mean_out,
                     int32_t* maxchi_out, yaqs_run_stats* stats) {
  yaqs_run* run = nullptr;
  int st = digital_begin(ctx, psi0, gates, n_gates, noise, obs, n_obs, cfg, rng, &run);
  if (st != YAQS_OK) return st;
  st = yaqs_analog_advance(run, yaqs_analog_remaining(run), nullptr);
  if (st != YAQS_OK) {
    yaqs_analog_finish(run, nullptr, nullptr, nullptr, nullptr);
    return st;
  }
  return yaqs_analog_finish(run, traj_out, mean_out, maxchi_out, stats);
}

// ---- component entry points ----
int yaqs_batched_svd(yaqs_ctx* ctx, int32_t batch, int32_t m, int32_t n, const double* M, double* U, double* S,
                     double* Vt) {
  if (!ctx || batch < 1 || m < 1 || n < 1 || std::min(m, n) > SVD_MAX_COLS || !M || !U || !S || !Vt)
    return set_err(ctx, YAQS_E_ARG, "bad svd arguments");
  if (2 * (m + n) > SVD_SMEM_CPLX) return set_err(ctx, YAQS_E_UNSUPPORTED, "svd needs m + n <= 2048");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int k = std::min(m, n);
  const long long big = (long long)std::max(m, n) * std::max(m, n);
  const long long wstride = 4 * big + std::max(m, n) + SVD_MAX_COLS;
  DevMem dm;
  cplx *dM, *dU, *dVt, *dw;
  double* dS;
  int* di;
  CUDA_TRY(ctx, dm.alloc(&dM, (size_t)batch * m * n));
  CUDA_TRY(ctx, dm.alloc(&dU, (size_t)batch * m * k));
  CUDA_TRY(ctx, dm.alloc(&dVt, (size_t)batch * k * n));
  CUDA_TRY(ctx, dm.alloc(&dS, (size_t)batch * k));
  CUDA_TRY(ctx, dm.alloc(&dw, (size_t)batch * wstride));
  CUDA_TRY(ctx, dm.alloc(&di, (size_t)batch * SVD_MAX_COLS));
  CUDA_TRY(ctx, cudaMemcpy(dM, M, (size_t)batch * m * n * sizeof(cplx), cudaMemcpyHostToDevice));
  const size_t smem = sizeof(CompSmem) + 1024;
  CUDA_TRY(ctx, cudaFuncSetAttribute(svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  svd_kernel<<<batch, NT, smem>>>(m, n, dM, dU, dS, dVt, dw, wstride, di);
  CUDA_TRY(ctx, cudaGetLastError());
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  CUDA_TRY(ctx, cudaMemcpy(U, dU, (size_t)batch * m * k * sizeof(cplx), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(Vt, dVt, (size_t)batch * k * n * sizeof(cplx), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(S, dS, (size_t)batch * k * sizeof(double), cudaMemcpyDeviceToHost));
  return YAQS_OK;
}

// ---------------------------------------------------------------------------
// SVD without allocation
// ---------------------------------------------------------------------------
// yaqs_batched_svd_noalloc is for callers whose device memory is owned by
// someone else (a Julia or PyTorch pool allocator that holds the whole
// device, or a code path where a cudaMalloc would synchronise the device or
// could fail mid-run): it takes device pointers and keeps its scratch in
// this fixed array.  The array is part of the module image, so every GPU
// that loads the library holds these 8 MiB until the process exits.  In host
// code `g_noalloc_scratch` names a host-side stand-in, not device memory: the
// kernel gets the device address from cudaGetSymbolAddress.
#define YAQS_NOALLOC_SCRATCH_BYTES (8u << 20)
static __device__ __align__(256) cplx g_noalloc_scratch[YAQS_NOALLOC_SCRATCH_BYTES / sizeof(cplx)];

namespace {
std::mutex g_noalloc_mu;
void* g_noalloc_base[64] = {};  // device address of g_noalloc_scratch, per device ordinal
}  // namespace

// With `device` current: looks up the array's device address (the first
// lookup on a device loads the module there) and sets svd_kernel's
// shared-memory limit.  Run by yaqs_ctx_create for its device.
static cudaError_t noalloc_prepare(int device) {
  if (device < 0 || device >= 64) return cudaSuccess;  // the entry point refuses such ordinals
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(CompSmem) + 1024));
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(g_noalloc_mu);
  g_noalloc_base[device] = p;
  return cudaSuccess;
}

int yaqs_batched_svd_noalloc(yaqs_ctx* ctx, int32_t batch, int32_t m, int32_t n, const double* M, double* U,
                             double* S, double* SVt, void* stream) {
  if (!ctx) return set_err(nullptr, YAQS_E_ARG, "null context");
  if (batch < 1 || m < 1 || n < 1 || std::min(m, n) > SVD_MAX_COLS || !M || !U || !S || !SVt)
    return set_err(ctx, YAQS_E_ARG, "bad svd arguments");
  if (2 * (m + n) > SVD_SMEM_CPLX) return set_err(ctx, YAQS_E_UNSUPPORTED, "svd needs m + n <= 2048");
  if (ctx->device < 0 || ctx->device >= 64) return set_err(ctx, YAQS_E_UNSUPPORTED, "device ordinal above 63");
  const long long big = (long long)std::max(m, n) * std::max(m, n);
  const long long wstride = 4 * big + std::max(m, n) + SVD_MAX_COLS;
  const unsigned long long need =
      (unsigned long long)batch * wstride * sizeof(cplx) + (unsigned long long)batch * SVD_MAX_COLS * sizeof(int);
  if (need > YAQS_NOALLOC_SCRATCH_BYTES)
    return set_err(ctx, YAQS_E_ARG,
                   "batch x (4 max(m,n)^2 + max(m,n) + 256) complex scratch exceeds the fixed 8 MiB of "
                   "yaqs_batched_svd_noalloc; use fewer or smaller problems per call");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const size_t smem = sizeof(CompSmem) + 1024;
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> g(g_noalloc_mu);
    base = g_noalloc_base[ctx->device];  // set when the context was created
  }
  if (!base) return set_err(ctx, YAQS_E_CUDA, "scratch address not resolved for this device");
  cplx* work = static_cast<cplx*>(base);
  int* iwork = reinterpret_cast<int*>(work + (long long)batch * wstride);
  svd_kernel<<<batch, NT, smem, static_cast<cudaStream_t>(stream)>>>(
      m, n, reinterpret_cast<const cplx*>(M), reinterpret_cast<cplx*>(U), S, reinterpret_cast<cplx*>(SVt), work,
      wstride, iwork);
  CUDA_TRY(ctx, cudaGetLastError());
  return YAQS_OK;
}

int yaqs_autotune_results(yaqs_ctx* ctx, double* rows, int32_t capacity, int32_t* count) {
  if (!ctx || !count || capacity < 0 || (capacity > 0 && !rows)) return set_err(ctx, YAQS_E_ARG, "bad arguments");
  std::lock_guard<std::mutex> lk(g_tune_mu);
  int n = 0;
  for (const auto& kv : g_tune_cache) {
    if (kv.first[0] != ctx->device) continue;
    if (n < capacity) {
      double* r = rows + 8LL * n;
      for (int k = 0; k < 5; ++k) r[k] = kv.first[k + 1];
      r[5] = kv.second.form;
      r[6] = kv.second.us_tc;
      r[7] = kv.second.us_mma;
    }
    ++n;
  }
  *count = n;
  return YAQS_OK;
}

int yaqs_fp64_peak(yaqs_ctx* ctx, double* tflops) {
  if (!ctx || !tflops) return set_err(ctx, YAQS_E_ARG, "null argument");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  DevMem dm;
  double* d;
  CUDA_TRY(ctx, dm.alloc(&d, 1));
  const int blocks = ctx->sms * 8, iters = 1 << 16;
  fp64_probe_kernel<<<blocks, 256>>>(d, 1024, 0.999999, 1e-7);  // warm-up
  cudaEvent_t e0, e1;
  CUDA_TRY(ctx, cudaEventCreate(&e0));
  CUDA_TRY(ctx, cudaEventCreate(&e1));
  float best = 1e30f;
  for (int rep = 0; rep < 5; ++rep) {
    cudaEventRecord(e0);
    fp64_probe_kernel<<<blocks, 256>>>(d, iters, 0.999999, 1e-7);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    best = std::min(best, ms);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  CUDA_TRY(ctx, cudaGetLastError());
  *tflops = 2.0 * 8.0 * iters * (double)blocks * 256 / (best * 1e-3) / 1e12;
  return YAQS_OK;
}

int yaqs_batched_qr(yaqs_ctx* ctx, int32_t batch, int32_t m, int32_t n, const double* M, double* Q, double* R) {
  if (!ctx || batch < 1 || m < 1 || n < 1 || std::min(m, n) > SVD_MAX_COLS || !M || !Q || !R)
    return set_err(ctx, YAQS_E_ARG, "bad qr arguments");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const int k = std::min(m, n);
  DevMem dm;
  cplx *dM, *dQ, *dR, *dw;
  CUDA_TRY(ctx, dm.alloc(&dM, (size_t)batch * m * n));
  CUDA_TRY(ctx, dm.alloc(&dQ, (size_t)batch * m * k));
  CUDA_TRY(ctx, dm.alloc(&dR, (size_t)batch * k * n));
  CUDA_TRY(ctx, dm.alloc(&dw, (size_t)batch * m * n));
  CUDA_TRY(ctx, cudaMemcpy(dM, M, (size_t)batch * m * n * sizeof(cplx), cudaMemcpyHostToDevice));
  const size_t smem = sizeof(CompSmem) + 1024;
  CUDA_TRY(ctx, cudaFuncSetAttribute(qr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  qr_kernel<<<batch, NT, smem>>>(m, n, dM, dQ, dR, dw);
  CUDA_TRY(ctx, cudaGetLastError());
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  CUDA_TRY(ctx, cudaMemcpy(Q, dQ, (size_t)batch * m * k * sizeof(cplx), cudaMemcpyDeviceToHost));
  CUDA_TRY(ctx, cudaMemcpy(R, dR, (size_t)batch * k * n * sizeof(cplx), cudaMemcpyDeviceToHost));
  return YAQS_OK;
}

static int expm_common(yaqs_ctx* ctx, int32_t batch, int32_t chil, int32_t D, int32_t chir, int32_t wl, int32_t wr,
                       const double* Lh, const double* Rh, const double* Wh, const double* x, double dt,
                       int32_t kdim, double tol, double exit_tol, double* out, int32_t* matvecs, int heff_only) {
  if (!ctx || batch < 1 || chil < 1 || chir < 1 || (D != 2 && D != 4) || wl < 1 || wr < 1 || wl * D > WAPPLY_MAXI ||
      wr * D > WAPPLY_MAXI || kdim < 1 || kdim > KRYLOV_MAX || !Lh || !Rh || !Wh || !x || !out)
    return set_err(ctx, YAQS_E_ARG, "bad expm arguments");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  const long long n = (long long)chil * D * chir;
  const long long tsz = (long long)chil * chir * std::max(wl, wr) * D;
  const long long wstride = 2 * tsz + (long long)(kdim + 1) * n;
  HostWMat hm = build_wmat(D * wr, wl * D, [&](int o, int in) {
    int pp = o % D, mp = o / D, m = in % wl, p = in / wl;
    return cload(Wh, (size_t)m + (size_t)wl * (pp + D * (p + D * (size_t)mp)));
  });
  if ((int)hm.val.size() > WAPPLY_MAXNNZ) return set_err(ctx, YAQS_E_UNSUPPORTED, "MPO too dense");
  DevMem dm;
  std::vector<WMat> views;
  int st = upload_wmats(ctx, dm, {hm}, views);
  if (st != YAQS_OK) return st;
  cplx *dL, *dR, *dx, *dw, *dout;
  int* dmv;
  CUDA_TRY(ctx, dm.alloc(&dL, (size_t)batch * chil * wl * chil));
  CUDA_TRY(ctx, dm.alloc(&dR, (size_t)batch * chir * wr * chir));
  CUDA_TRY(ctx, dm.alloc(&dx, (size_t)batch * n));
  CUDA_TRY(ctx, dm.alloc(&dout, (size_t)batch * n));
  CUDA_TRY(ctx, dm.alloc(&dw, (size_t)batch * wstride));
  CUDA_TRY(ctx, dm.alloc(&dmv, batch));
  CUDA_TRY(ctx, cudaMemcpy(dL, Lh, (size_t)batch * chil * wl * chil * sizeof(cplx), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(dR, Rh, (size_t)batch * chir * wr * chir * sizeof(cplx), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(dx, x, (size_t)batch * n * sizeof(cplx), cudaMemcpyHostToDevice));
  KrylovCfg kc;
  kc.kdim = kdim;
  kc.tol = tol;
  kc.exit_tol = exit_tol;
  const size_t smem = sizeof(CompSmem) + 1024;
  CUDA_TRY(ctx, cudaFuncSetAttribute(expm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  expm_kernel<<<batch, NT, smem>>>(chil, D, chir, wl, wr, dL, dR, views[0], dx, dt, kc, dw, wstride, dmv, heff_only,
                                   dout);
  CUDA_TRY(ctx, cudaGetLastError());
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  CUDA_TRY(ctx, cudaMemcpy(out, heff_only ? dout : dx, (size_t)batch * n * sizeof(cplx), cudaMemcpyDeviceToHost));
  if (matvecs && !heff_only) CUDA_TRY(ctx, cudaMemcpy(matvecs, dmv, batch * sizeof(int), cudaMemcpyDeviceToHost));
  return YAQS_OK;
}

int yaqs_batched_expm_site(yaqs_ctx* ctx, int32_t batch, int32_t chil, int32_t D, int32_t chir, int32_t wl, int32_t wr,
                           const double* L, const double* R, const double* W, const double* x, double dt,
                           int32_t krylov_dim, double krylov_tol, double krylov_exit_tol, double* out,
                           int32_t* matvecs) {
  return expm_common(ctx, batch, chil, D, chir, wl, wr, L, R, W, x, dt, krylov_dim, krylov_tol, krylov_exit_tol, out,
                     matvecs, 0);
}

int yaqs_batched_cgemm_tf32(yaqs_ctx* ctx, int32_t batch, int32_t M, int32_t N, int32_t K, const float* A,
                            int32_t a_kmajor, int32_t conj_a, const float* B, int32_t b_kmajor, int32_t conj_b,
                            float* C) {
  if (!ctx || batch < 1 || M < 1 || N < 1 || K < 1 || M > 4096 || N > 4096 || K > 4096 || !A || !B || !C)
    return set_err(ctx, YAQS_E_ARG, "bad cgemm arguments");
  std::lock_guard<std::mutex> lk(ctx->mu);
  CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  // staged layouts: A MN-major = rows k, inner m; K-major = rows m, inner k (likewise B with n)
  const int a_mn = a_kmajor ? 0 : 1, b_mn = b_kmajor ? 0 : 1;
  const long long a_rows = a_mn ? K : M, a_inner = a_mn ? M : K, b_rows = b_mn ? K : N, b_inner = b_mn ? N : K;
  const long long pa = (a_inner + 1) & ~1LL, pb = (b_inner + 1) & ~1LL;
  std::vector<float> ha((size_t)batch * a_rows * pa * 2, 0.f), hb((size_t)batch * b_rows * pb * 2, 0.f);
  for (long long b = 0; b < batch; ++b) {
    for (long long r = 0; r < a_rows; ++r)
      for (long long i = 0; i < a_inner; ++i)
        for (int c = 0; c < 2; ++c)
          ha[((b * a_rows + r) * pa + i) * 2 + c] = A[((b * a_rows + r) * a_inner + i) * 2 + c];
    for (long long r = 0; r < b_rows; ++r)
      for (long long i = 0; i < b_inner; ++i)
        for (int c = 0; c < 2; ++c)
          hb[((b * b_rows + r) * pb + i) * 2 + c] = B[((b * b_rows + r) * b_inner + i) * 2 + c];
  }
  DevMem dm;
  float *dA, *dB;
  float2* dC;
  CUtensorMap* dmaps;
  int* dst;
  CUDA_TRY(ctx, dm.alloc(&dA, ha.size()));
  CUDA_TRY(ctx, dm.alloc(&dB, hb.size()));
  CUDA_TRY(ctx, dm.alloc(&dC, (size_t)batch * M * N));
  CUDA_TRY(ctx, dm.alloc(&dmaps, 2 * (size_t)batch));
  CUDA_TRY(ctx, dm.alloc(&dst, batch));
  CUDA_TRY(ctx, cudaMemcpy(dA, ha.data(), ha.size() * sizeof(float), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, cudaMemcpy(dB, hb.data(), hb.size() * sizeof(float), cudaMemcpyHostToDevice));
  std::vector<CUtensorMap> maps(2 * (size_t)batch);
  for (long long b = 0; b < batch; ++b) {
    if (!make_tc_map(&maps[2 * b], dA + b * a_rows * pa * 2, pa, a_rows, a_mn ? TC_A_MN : TC_A_K) ||
        !make_tc_map(&maps[2 * b + 1], dB + b * b_rows * pb * 2, pb, b_rows, b_mn ? TC_B_MN : TC_B_K))
      return set_err(ctx, YAQS_E_CUDA, "cuTensorMapEncodeTiled refused a staged operand");
  }
  CUDA_TRY(ctx, cudaMemcpy(dmaps, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice));
  CUDA_TRY(ctx, tc_cgemm_launch(batch, M, N, K, dmaps, a_mn, conj_a ? 1 : 0, b_mn, conj_b ? 1 : 0, dC, dst));
  CUDA_TRY(ctx, cudaDeviceSynchronize());
  std::vector<int> st(batch);
  CUDA_TRY(ctx, cudaMemcpy(st.data(), dst, batch * sizeof(int), cudaMemcpyDeviceToHost));
  for (int v : st)
    if (v) return set_err(ctx, YAQS_E_TIMEOUT, "tensor-core pipeline wait gave up");
  CUDA_TRY(ctx, cudaMemcpy(C, dC, (size_t)batch * M * N * sizeof(float2), cudaMemcpyDeviceToHost));
  return YAQS_OK;
}

int yaqs_batched_project_site(yaqs_ctx* ctx, int32_t batch, int32_t chil, int32_t D, int32_t chir, int32_t wl,
                              int32_t wr, const double* L, const double* R, const double* W, const double* x,
                              double* out) {
  return expm_common(ctx, batch, chil, D, chir, wl, wr, L, R, W, x, 0.0, 1, 0.0, 0.0, out, nullptr, 1);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Serving (yaqs_server_*)
// ---------------------------------------------------------------------------
#include "server.cuh"
