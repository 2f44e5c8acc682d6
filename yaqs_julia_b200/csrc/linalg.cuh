// linalg.cuh — CTA-level Householder QR/LQ and one-sided Jacobi SVD (FP64).
//
// Restates the LAPACK factorizations the reference calls through Julia's
// LinearAlgebra (Decompositions.jl:18-73, MPS.jl:182-311 for QR/LQ;
// Algorithms.jl:420, Dissipation.jl:281, StochasticProcess.jl:280 for SVD).
// The conventions (zlarfg reflectors with real R diagonal; round-robin
// Jacobi pair order; stable descending sort; deterministic completion of
// null singular vectors) are identical to the CPU oracle so both produce the
// same gauge up to rounding.
#pragma once
#include "common.cuh"

#define QR_NULL_TOL 1e-14
#define SVD_NULL_TOL 1e-14
#define JACOBI_MAX_SWEEPS 60
#define SVD_MAX_COLS 256
#define QR_REG_ROWS 4  // Householder rows per lane kept in registers (m - j - 1 <= 128)
// The register-held reflector pays off from about this many rows; smaller
// factorisations (the short bonds of a growing chain) keep the plain column
// loop, which measured 10 % faster on the digital workload.
#define QR_REG_MIN_ROWS 48

struct LinalgSmem {
  cplx tau[SVD_MAX_COLS];
  int rot_count;
  int flag;
  int blocked;  // this run may reorder sums: panel QR and short rotations
};

// ---------------------------------------------------------------------------
// Householder QR
// ---------------------------------------------------------------------------
// Factor H (m x n, col-major, ld m) in place: R in the upper triangle,
// reflector vectors below, scalars in ls.tau.  SHARED: H lies in shared
// memory.  CTA-collective.
template <bool SHARED>
static __device__ __noinline__ void dev_qr_factor_at(cplx* H, int m, int n, LinalgSmem& ls, RedScratch& rs) {
  ProfScope prof_scope_(PF_QR);
  if (SHARED) ASSUME_SHARED(H);
  ASSUME_SHARED(&ls);
  const int tid = ltid(), lane = tid & 31, wid = tid >> 5;
  const int kq = min(m, n);
  double fro2 = cta_norm2(H, (long long)m * n, rs);
  const double null_abs = QR_NULL_TOL * sqrt(fro2);
  for (int j = 0; j < kq; ++j) {
    cplx* col = H + (long long)m * j;
    double s = 0.0;
    for (int i = j + 1 + tid; i < m; i += NT) s += cabs2(col[i]);
    const double xn2 = block_sum(s, rs);
    // col[j] is rewritten (by thread 0) only after the barrier that follows
    // the scaling below, so no barrier is needed between this read and it
    const cplx alpha = col[j];
    const double full = sqrt(cabs2(alpha) + xn2);
    if (full <= null_abs || (xn2 == 0.0 && alpha.y == 0.0)) {
      for (int i = j + 1 + tid; i < m; i += NT) col[i] = make_double2(0.0, 0.0);
      if (tid == 0) ls.tau[j] = make_double2(0.0, 0.0);
      cta_sync();
      continue;
    }
    const double beta = (alpha.x >= 0.0) ? -full : full;
    const cplx t = make_double2((beta - alpha.x) / beta, -alpha.y / beta);
    const cplx amb = make_double2(alpha.x - beta, alpha.y);
    const double d = cabs2(amb);
    const cplx scale = make_double2(amb.x / d, -amb.y / d);
    for (int i = j + 1 + tid; i < m; i += NT) col[i] = cmul(col[i], scale);
    cta_sync();
    if (tid == 0) {
      col[j] = make_double2(beta, 0.0);
      ls.tau[j] = t;
    }
    const cplx ct = cconj(t);
    if (m >= QR_REG_MIN_ROWS && m <= 32 * QR_REG_ROWS + 1) {
      // reflector rows held in registers; two trailing columns per warp pass
      cplx v[QR_REG_ROWS];
#pragma unroll
      for (int q = 0; q < QR_REG_ROWS; ++q) {
        const int i = j + 1 + lane + 32 * q;
        v[q] = i < m ? col[i] : make_double2(0.0, 0.0);
      }
      for (int c0 = j + 1 + wid; c0 < n; c0 += 2 * NW) {
        const int c1 = c0 + NW;
        const bool two = c1 < n;
        cplx* x0 = H + (long long)m * c0;
        cplx* x1 = H + (long long)m * (two ? c1 : c0);
        cplx a0 = make_double2(0.0, 0.0), a1 = make_double2(0.0, 0.0);
        if (lane == 0) {
          a0 = x0[j];
          a1 = x1[j];
        }
        cplx y0[QR_REG_ROWS], y1[QR_REG_ROWS];
#pragma unroll
        for (int q = 0; q < QR_REG_ROWS; ++q) {
          const int i = j + 1 + lane + 32 * q;
          y0[q] = i < m ? x0[i] : make_double2(0.0, 0.0);
          y1[q] = i < m ? x1[i] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int q = 0; q < QR_REG_ROWS; ++q) {
          cfmac(a0, v[q], y0[q]);
          cfmac(a1, v[q], y1[q]);
        }
        a0.x = warp_sum(a0.x);
        a0.y = warp_sum(a0.y);
        a1.x = warp_sum(a1.x);
        a1.y = warp_sum(a1.y);
        a0 = cmul(a0, ct);
        a1 = cmul(a1, ct);
#pragma unroll
        for (int q = 0; q < QR_REG_ROWS; ++q) {
          const int i = j + 1 + lane + 32 * q;
          if (i < m) {
            x0[i] = csub(y0[q], cmul(a0, v[q]));
            if (two) x1[i] = csub(y1[q], cmul(a1, v[q]));
          }
        }
        if (lane == 0) {
          x0[j] = csub(x0[j], a0);
          if (two) x1[j] = csub(x1[j], a1);
        }
      }
    } else {
      for (int c = j + 1 + wid; c < n; c += NW) {
        cplx* x = H + (long long)m * c;
        cplx acc = make_double2(0.0, 0.0);
        if (lane == 0) acc = x[j];
        for (int i = j + 1 + lane; i < m; i += 32) cfmac(acc, col[i], x[i]);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        acc = cmul(acc, ct);
        for (int i = j + 1 + lane; i < m; i += 32) x[i] = csub(x[i], cmul(acc, col[i]));
        if (lane == 0) x[j] = csub(x[j], acc);
      }
    }
    cta_sync();
  }
}

static __device__ __forceinline__ void dev_qr_factor(cplx* H, int m, int n, LinalgSmem& ls, RedScratch& rs) {
  dev_qr_factor_at<false>(H, m, n, ls, rs);
}

// Q (m x kq) of a factored H; SHARED: both in shared memory.  CTA-collective.
template <bool SHARED>
static __device__ __noinline__ void dev_qr_formq_at(const cplx* H, int m, int n, cplx* Q, LinalgSmem& ls) {
  ProfScope prof_scope_(PF_QRQ);
  if (SHARED) ASSUME_SHARED(H);
  if (SHARED) ASSUME_SHARED(Q);
  ASSUME_SHARED(&ls);
  const int tid = ltid(), lane = tid & 31, wid = tid >> 5;
  const int kq = min(m, n);
  for (int e = tid; e < m * kq; e += NT) {
    int r = (int)(e % m), c = (int)(e / m);
    Q[e] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  cta_sync();
  for (int j = kq - 1; j >= 0; --j) {
    const cplx t = ls.tau[j];
    if (t.x == 0.0 && t.y == 0.0) continue;
    const cplx* v = H + (long long)m * j;
    if (m >= QR_REG_MIN_ROWS && m <= 32 * QR_REG_ROWS + 1) {
      cplx vr[QR_REG_ROWS];
#pragma unroll
      for (int qq = 0; qq < QR_REG_ROWS; ++qq) {
        const int i = j + 1 + lane + 32 * qq;
        vr[qq] = i < m ? v[i] : make_double2(0.0, 0.0);
      }
      for (int c0 = j + wid; c0 < kq; c0 += 2 * NW) {
        const int c1 = c0 + NW;
        const bool two = c1 < kq;
        cplx* q0 = Q + (long long)m * c0;
        cplx* q1 = Q + (long long)m * (two ? c1 : c0);
        cplx a0 = make_double2(0.0, 0.0), a1 = make_double2(0.0, 0.0);
        if (lane == 0) {
          a0 = q0[j];
          a1 = q1[j];
        }
        cplx y0[QR_REG_ROWS], y1[QR_REG_ROWS];
#pragma unroll
        for (int qq = 0; qq < QR_REG_ROWS; ++qq) {
          const int i = j + 1 + lane + 32 * qq;
          y0[qq] = i < m ? q0[i] : make_double2(0.0, 0.0);
          y1[qq] = i < m ? q1[i] : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int qq = 0; qq < QR_REG_ROWS; ++qq) {
          cfmac(a0, vr[qq], y0[qq]);
          cfmac(a1, vr[qq], y1[qq]);
        }
        a0.x = warp_sum(a0.x);
        a0.y = warp_sum(a0.y);
        a1.x = warp_sum(a1.x);
        a1.y = warp_sum(a1.y);
        a0 = cmul(a0, t);
        a1 = cmul(a1, t);
#pragma unroll
        for (int qq = 0; qq < QR_REG_ROWS; ++qq) {
          const int i = j + 1 + lane + 32 * qq;
          if (i < m) {
            q0[i] = csub(y0[qq], cmul(a0, vr[qq]));
            if (two) q1[i] = csub(y1[qq], cmul(a1, vr[qq]));
          }
        }
        if (lane == 0) {
          q0[j] = csub(q0[j], a0);
          if (two) q1[j] = csub(q1[j], a1);
        }
      }
    } else {
      for (int c = j + wid; c < kq; c += NW) {
        cplx* q = Q + (long long)m * c;
        cplx acc = make_double2(0.0, 0.0);
        if (lane == 0) acc = q[j];
        for (int i = j + 1 + lane; i < m; i += 32) cfmac(acc, v[i], q[i]);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        acc = cmul(acc, t);
        for (int i = j + 1 + lane; i < m; i += 32) q[i] = csub(q[i], cmul(acc, v[i]));
        if (lane == 0) q[j] = csub(q[j], acc);
      }
    }
    cta_sync();
  }
}

static __device__ __forceinline__ void dev_qr_formq(const cplx* H, int m, int n, cplx* Q, LinalgSmem& ls) {
  dev_qr_formq_at<false>(H, m, n, Q, ls);
}

// R (kq x n) of a factored H into Rout (ld kq), zero below the diagonal.
static __device__ __forceinline__ void dev_qr_extract_r(const cplx* H, int m, int n, cplx* Rout) {
  const int kq = min(m, n);
  for (int e = ltid(); e < kq * n; e += NT) {
    int r = (int)(e % kq), c = (int)(e / kq);
    Rout[e] = (r <= c) ? H[r + (long long)m * c] : make_double2(0.0, 0.0);
  }
  cta_sync();
}

// ---------------------------------------------------------------------------
// Panel Householder QR
// ---------------------------------------------------------------------------
// The column loop above is a chain of four barriers and a pass over the
// trailing matrix in L2 per column: 128 x 64 took about 860 us with its Q.
// Here QR_PANEL columns are factored in shared memory, one barrier a column
// (each warp forms the reflector for itself), and every other column is
// loaded once a panel into the registers of one warp, which applies all
// reflectors of the panel to it without a barrier.  Q is formed the same way
// from the last panel to the first.  The sums run in another order than the
// column loop's, so it serves TEBD circuits and mixed runs (DevParams::blocked).
#define QR_PANEL 16
#define QR_PANEL_MAX_ROWS 256

// Applies the reflectors ja <= j < jb (their tails below the diagonal of the
// panel V, ld m, column ja first) to the columns c0 <= c < c1 of X: ascending
// with conj(tau) (Q^H X), or descending with tau (Q X).  Columns c < ident
// start as unit vectors e_c.  Each warp takes CG columns of 32 CH rows.
template <int CH, int CG>
static __device__ __noinline__ void qr_apply(cplx* X, int ld, int c0, int c1, const cplx* V, int m, int ja, int jb,
                                             bool ascending, int ident, const cplx* tau) {
  ASSUME_SHARED(V);
  ASSUME_SHARED(tau);
  constexpr int NV = 2 * CG;
  constexpr int SH = NV == 2 ? 4 : NV == 4 ? 3 : NV == 8 ? 2 : 1;  // lane of value v: v << SH
  const int lane = ltid() & 31, wid = ltid() >> 5;
#pragma unroll 1
  for (int cb = c0 + wid * CG; cb < c1; cb += NW * CG) {
    cplx x[CG][CH];
#pragma unroll
    for (int g = 0; g < CG; ++g)
#pragma unroll
      for (int q = 0; q < CH; ++q) {
        const int i = lane + 32 * q, c = cb + g;
        x[g][q] = make_double2(0.0, 0.0);
        if (c < c1 && i < m) {
          if (c < ident)
            x[g][q].x = i == c ? 1.0 : 0.0;
          else
            x[g][q] = X[i + ld * c];
        }
      }
#pragma unroll 1
    for (int jj = ja; jj < jb; ++jj) {
      const int j = ascending ? jj : jb - 1 - (jj - ja);
      cplx t = tau[j];
      if (ascending) t.y = -t.y;
      cplx v[CH];
      double d[NV];
#pragma unroll
      for (int e = 0; e < NV; ++e) d[e] = 0.0;
#pragma unroll
      for (int q = 0; q < CH; ++q) {
        const int i = lane + 32 * q;
        v[q] = make_double2(i == j ? 1.0 : 0.0, 0.0);
        if (i > j && i < m) v[q] = V[i + m * (j - ja)];
#pragma unroll
        for (int g = 0; g < CG; ++g) {
          cplx a = make_double2(d[2 * g], d[2 * g + 1]);
          cfmac(a, v[q], x[g][q]);
          d[2 * g] = a.x;
          d[2 * g + 1] = a.y;
        }
      }
      warp_sum_multi<NV>(d);
#pragma unroll
      for (int g = 0; g < CG; ++g) {
        const cplx a = cmul(make_double2(__shfl_sync(0xffffffffu, d[0], (2 * g) << SH),
                                         __shfl_sync(0xffffffffu, d[0], (2 * g + 1) << SH)),
                            t);
        const cplx na = make_double2(-a.x, -a.y);
#pragma unroll
        for (int q = 0; q < CH; ++q) cfma(x[g][q], na, v[q]);
      }
    }
#pragma unroll
    for (int g = 0; g < CG; ++g)
#pragma unroll
      for (int q = 0; q < CH; ++q) {
        const int i = lane + 32 * q;
        if (cb + g < c1 && i < m) X[i + ld * (cb + g)] = x[g][q];
      }
  }
}

// Householder factorisation of the columns ja .. jb-1 of the panel V (m x
// (pe - ja) in shared memory, ld m) with the columns up to pe updated.
template <int CH>
static __device__ __noinline__ void qr_panel(cplx* V, int m, int ja, int jb, int pe, double null_abs, cplx* tau) {
  ASSUME_SHARED(V);
  ASSUME_SHARED(tau);
  const int lane = ltid() & 31, wid = ltid() >> 5;
  cplx v[CH];
  double diag = 0.0;
  int pending = -1;  // column whose reflector warp 0 still holds
#pragma unroll 1
  for (int j = ja; j < jb; ++j) {
    if (wid == 0 && pending >= 0) {
      cplx* pc = V + m * (pending - ja);
#pragma unroll
      for (int q = 0; q < CH; ++q) {
        const int i = lane + 32 * q;
        if (i > pending && i < m) pc[i] = v[q];
        if (i == pending) pc[i] = make_double2(diag, 0.0);
      }
    }
    const cplx* col = V + m * (j - ja);
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      const int i = lane + 32 * q;
      v[q] = i > j && i < m ? col[i] : make_double2(0.0, 0.0);
      s += cabs2(v[q]);
    }
    const double xn2 = warp_sum(s);
    const cplx alpha = col[j];
    const double full = sqrt(cabs2(alpha) + xn2);
    cplx t = make_double2(0.0, 0.0);
    pending = j;
    if (full <= null_abs || (xn2 == 0.0 && alpha.y == 0.0)) {
#pragma unroll
      for (int q = 0; q < CH; ++q) v[q] = make_double2(0.0, 0.0);
      diag = alpha.x;
      // alpha keeps its (null) imaginary part in place of a real diagonal
      if (alpha.y != 0.0) pending = -2 - j;
    } else {
      const double beta = (alpha.x >= 0.0) ? -full : full;
      const double rb = 1.0 / beta;
      t = make_double2((beta - alpha.x) * rb, -alpha.y * rb);
      const cplx amb = make_double2(alpha.x - beta, alpha.y);
      const double rd = 1.0 / cabs2(amb);
      const cplx scale = make_double2(amb.x * rd, -amb.y * rd);
#pragma unroll
      for (int q = 0; q < CH; ++q) v[q] = cmul(v[q], scale);
      diag = beta;
      const cplx ct = cconj(t);
#pragma unroll 1
      for (int c = j + 1 + wid; c < pe; c += NW) {
        cplx* xc = V + m * (c - ja);
        cplx x[CH];
        cplx a = make_double2(0.0, 0.0);
        const cplx xj = xc[j];
#pragma unroll
        for (int q = 0; q < CH; ++q) {
          const int i = lane + 32 * q;
          x[q] = i > j && i < m ? xc[i] : make_double2(0.0, 0.0);
          cfmac(a, v[q], x[q]);
        }
        double d[2] = {a.x, a.y};
        warp_sum_multi<2>(d);
        a = cadd(xj, make_double2(__shfl_sync(0xffffffffu, d[0], 0), __shfl_sync(0xffffffffu, d[0], 16)));
        a = cmul(a, ct);
        const cplx na = make_double2(-a.x, -a.y);
#pragma unroll
        for (int q = 0; q < CH; ++q) {
          const int i = lane + 32 * q;
          if (i > j && i < m) {
            cfma(x[q], na, v[q]);
            xc[i] = x[q];
          }
        }
        if (lane == 0) xc[j] = csub(xj, a);
      }
    }
    if (wid == 0 && lane == 0) tau[j] = t;
    if (pending < -1) {  // null column with a complex head: zero its tail, leave the head
      cta_sync();        // every warp has read it
      if (wid == 0)
        for (int i = j + 1 + lane; i < m; i += 32) V[i + m * (j - ja)] = make_double2(0.0, 0.0);
      pending = -1;
    }
    cta_sync();
  }
  if (wid == 0 && pending >= 0) {
    cplx* pc = V + m * (pending - ja);
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      const int i = lane + 32 * q;
      if (i > pending && i < m) pc[i] = v[q];
      if (i == pending) pc[i] = make_double2(diag, 0.0);
    }
  }
  cta_sync();
}

static __device__ __forceinline__ void qr_panel_rows(cplx* V, int m, int ja, int jb, int pe, double null_abs, cplx* tau) {
  if (m <= 32)
    qr_panel<1>(V, m, ja, jb, pe, null_abs, tau);
  else if (m <= 64)
    qr_panel<2>(V, m, ja, jb, pe, null_abs, tau);
  else if (m <= 128)
    qr_panel<4>(V, m, ja, jb, pe, null_abs, tau);
  else
    qr_panel<8>(V, m, ja, jb, pe, null_abs, tau);
}

// m x n values by load(e) into V; returns the null threshold of their factorisation.
template <class Load>
static __device__ __forceinline__ double qr_load_panel(int m, int n, Load load, cplx* V, RedScratch& rs) {
  cta_sync();  // the buffer's last readers are done
  double s = 0.0;
  for (int e = ltid(); e < m * n; e += NT) {
    const cplx v = load(e);
    V[e] = v;
    s += cabs2(v);
  }
  return QR_NULL_TOL * sqrt(block_sum(s, rs));
}

static __device__ __forceinline__ void qr_apply_rows(cplx* X, int ld, int c0, int c1, const cplx* V, int m, int ja,
                                                     int jb, bool ascending, int ident, const cplx* tau) {
  if (m <= 32)
    qr_apply<1, 4>(X, ld, c0, c1, V, m, ja, jb, ascending, ident, tau);
  else if (m <= 64)
    qr_apply<2, 2>(X, ld, c0, c1, V, m, ja, jb, ascending, ident, tau);
  else if (m <= 128)
    qr_apply<4, 2>(X, ld, c0, c1, V, m, ja, jb, ascending, ident, tau);
  else
    qr_apply<8, 1>(X, ld, c0, c1, V, m, ja, jb, ascending, ident, tau);
}

// dev_qr_factor by panels: H (m x n) in place, m <= QR_PANEL_MAX_ROWS; sb
// holds m x QR_PANEL values.  CTA-collective.
static __device__ __noinline__ void dev_qr_factor_panel(cplx* H, int m, int n, cplx* sb, LinalgSmem& ls, RedScratch& rs) {
  ProfScope prof_scope_(PF_QR);
  const int kq = min(m, n);
  const double null_abs = QR_NULL_TOL * sqrt(cta_norm2(H, (long long)m * n, rs));
  for (int ja = 0; ja < kq; ja += QR_PANEL) {
    const int pe = min(ja + QR_PANEL, n), jb = min(ja + QR_PANEL, kq);
    cplx* P = H + m * ja;
    for (int e = ltid(); e < m * (pe - ja); e += NT) sb[e] = P[e];
    cta_sync();
    qr_panel_rows(sb, m, ja, jb, pe, null_abs, ls.tau);
    for (int e = ltid(); e < m * (pe - ja); e += NT) P[e] = sb[e];
    qr_apply_rows(H, m, pe, n, sb, m, ja, jb, true, 0, ls.tau);
    cta_sync();
  }
}

// dev_qr_formq by panels.  CTA-collective.
static __device__ __noinline__ void dev_qr_formq_panel(const cplx* H, int m, int n, cplx* Q, cplx* sb, LinalgSmem& ls) {
  ProfScope prof_scope_(PF_QRQ);
  const int kq = min(m, n), last = (kq - 1) / QR_PANEL * QR_PANEL;
  for (int ja = last; ja >= 0; ja -= QR_PANEL) {
    const int jb = min(ja + QR_PANEL, kq);
    if (kq > QR_PANEL || n > QR_PANEL)  // otherwise the panel is still there
      for (int e = ltid(); e < m * (jb - ja); e += NT) sb[e] = H[m * ja + e];
    cta_sync();
    qr_apply_rows(Q, m, ja, kq, sb, m, ja, jb, false, jb, ls.tau);
    cta_sync();
  }
}

template <class Load, class Store>
static __device__ __forceinline__ void qr_one_panel(int m, int n, Load load, Store store_q, cplx* Rout, cplx* sb,
                                                    LinalgSmem& ls, RedScratch& rs) {
  const int k = min(m, n);
  const double null_abs = qr_load_panel(m, n, load, sb, rs);
  {
    ProfScope prof_scope_(PF_QR);
    qr_panel_rows(sb, m, 0, k, n, null_abs, ls.tau);
  }
  ProfScope prof_scope_(PF_QRQ);
  cplx* q = sb + m * n;
  qr_apply_rows(q, m, 0, k, sb, m, 0, k, false, k, ls.tau);
  for (int e = ltid(); e < k * n; e += NT) {
    const int c = e / k, r = e - c * k;
    Rout[e] = (r <= c) ? sb[r + m * c] : make_double2(0.0, 0.0);
  }
  cta_sync();
  for (int e = ltid(); e < m * k; e += NT) store_q(e, q);
  cta_sync();
}

// Thin QR of M (m x n, col-major), load(e) its element e: store_q(e, q), e < m k,
// stores from Q (m x k) at q, Rout becomes R (k x n), k = min(m, n).  H and Qg
// are work matrices in global memory; a problem that fits runs in the shared buffer sb
// (cap values) instead, Q beside the factored matrix if both do: every
// column step reads what other threads wrote in the step before, which
// through L2 costs its latency each time.
template <class Load, class Store>
static __device__ __forceinline__ void dev_qr_thin(int m, int n, Load load, cplx* H, Store store_q, cplx* Qg, cplx* Rout,
                                                   cplx* sb, int cap, LinalgSmem& ls, RedScratch& rs) {
  const int k = min(m, n);
  if (ls.blocked && n <= QR_PANEL && m <= QR_PANEL_MAX_ROWS && m * (n + k) <= cap) {
    // one panel: never leaves shared memory, Q beside it
    qr_one_panel(m, n, load, store_q, Rout, sb, ls, rs);
    return;
  }
  if (ls.blocked && m <= QR_PANEL_MAX_ROWS) {
    cta_sync();
    for (int e = ltid(); e < m * n; e += NT) H[e] = load(e);
    cta_sync();
    dev_qr_factor_panel(H, m, n, sb, ls, rs);
    dev_qr_formq_panel(H, m, n, Qg, sb, ls);
    dev_qr_extract_r(H, m, n, Rout);
    for (int e = ltid(); e < m * k; e += NT) store_q(e, Qg);
    cta_sync();
    return;
  }
  cplx* h = m * n <= cap ? sb : H;
  cplx* q = (m * n + m * k <= cap) ? sb + m * n : Qg;
  cta_sync();  // the shared buffer's last readers are done
  for (int e = ltid(); e < m * n; e += NT) h[e] = load(e);
  cta_sync();
  if (h == sb)
    dev_qr_factor_at<true>(h, m, n, ls, rs);
  else
    dev_qr_factor_at<false>(h, m, n, ls, rs);
  if (h == sb && q != Qg)
    dev_qr_formq_at<true>(h, m, n, q, ls);
  else
    dev_qr_formq_at<false>(h, m, n, q, ls);
  dev_qr_extract_r(h, m, n, Rout);
  for (int e = ltid(); e < m * k; e += NT) store_q(e, q);
  cta_sync();
}

// ---------------------------------------------------------------------------
// One-sided Jacobi SVD
// ---------------------------------------------------------------------------
struct SvdWork {
  cplx* B;      // q x p
  cplx* X;      // p x p
  cplx* Yo;     // q x p (sorted, normalised left vectors of B)
  cplx* Zo;     // p x p (sorted right vectors)
  cplx* y;      // q (completion scratch)
  double* sig;  // p
  int* ord;     // p
};

struct SvdResult {
  bool tr;
  int q, p, rank;  // rank = number of non-null singular values
  int sweeps;
};

// Orthonormal completion of column k of Y (rows x *) against columns 0..k-1.
static __device__ __noinline__ void dev_complete_column(cplx* Y, int rows, int k, cplx* y, RedScratch& rs) {
  for (int c = 0; c < rows; ++c) {
    // pass 1: y = e_c - sum_h conj(Y_h[c]) Y_h
    for (int i = ltid(); i < rows; i += NT) {
      cplx v = make_double2(i == c ? 1.0 : 0.0, 0.0);
      for (int h = 0; h < k; ++h) {
        cplx yc = Y[c + (long long)rows * h];
        cplx yi = Y[i + (long long)rows * h];
        v = csub(v, cmulc(yc, yi));
      }
      y[i] = v;
    }
    cta_sync();
    // pass 2: y -= sum_h (Y_h^H y) Y_h, dot products in chunks of 8
    for (int h0 = 0; h0 < k; h0 += 8) {
      double d[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) d[e] = 0.0;
      for (int i = ltid(); i < rows; i += NT) {
        cplx yi = y[i];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (h0 + e < k) {
            cplx a = Y[i + (long long)rows * (h0 + e)];
            cplx p = cmulc(a, yi);
            d[2 * e] += p.x;
            d[2 * e + 1] += p.y;
          }
        }
      }
      block_sum_n<16>(d, rs);
      for (int i = ltid(); i < rows; i += NT) {
        cplx v = y[i];
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (h0 + e < k) v = csub(v, cmul(make_double2(d[2 * e], d[2 * e + 1]), Y[i + (long long)rows * (h0 + e)]));
        y[i] = v;
      }
      cta_sync();
    }
    double nr = sqrt(cta_norm2(y, rows, rs));
    if (nr > 0.5) {
      for (int i = ltid(); i < rows; i += NT) Y[i + (long long)rows * k] = cscale(y[i], 1.0 / nr);
      cta_sync();
      return;
    }
  }
}

// Block size of the block-cyclic Jacobi ordering: blocks of b columns of B
// (q rows) so that a pair of blocks fits the SVD_SMEM_CPLX shared buffer.
// The CPU oracle uses the same rule.
#define SVD_SMEM_CPLX 4096
__host__ __device__ __forceinline__ int svd_block_size(int q, int p) {
  int b = SVD_SMEM_CPLX / (2 * q);
  if (b > 32) b = 32;
  if (b > p) b = p;
  if (b < 1) b = 1;
  return b;
}

// Jacobi rotation parameters for columns with |b_i|^2 = al, |b_j|^2 = be,
// b_i^H b_j = (gx, gy).  Same rotation as the oracle's
//   zeta = (be-al)/(2|g|), t = sign(zeta)/(|zeta| + sqrt(1+zeta^2)),
//   c = 1/sqrt(1+t^2), s = c t, e = g/|g|,
// written with fewer dependent divisions/square roots:
//   t = sign(d) 2|g| / (|d| + sqrt(d^2 + 4|g|^2)),  d = be - al.
// Returns false when the pair is already orthogonal to tolerance.
static __device__ __forceinline__ bool jacobi_params(double al, double be, double gx, double gy, double tol, double& c,
                                              cplx& se, cplx& sec) {
  const double g2 = gx * gx + gy * gy;
  if (!(g2 > tol * tol * (al * be))) return false;
  const double rag = rsqrt(g2);
  const double ag = g2 * rag;
  const double d = be - al;
  const double R = sqrt(fma(d, d, 4.0 * g2));
  double t = 2.0 * ag / (fabs(d) + R);
  if (d < 0.0) t = -t;
  c = rsqrt(fma(t, t, 1.0));
  const double f = c * t * rag;
  se = make_double2(f * gx, f * gy);
  sec = make_double2(f * gx, -f * gy);
  return true;
}

// Pair k of round t of such a block as columns i < j; false when it has none.
static __device__ __forceinline__ bool block_pair(bool cross, int b, int n0, int n1, int joff, int t, int k, int& i,
                                                  int& j) {
  if (cross) {
    i = k;
    j = k + t < b ? k + t : k + t - b;
    if (i >= n0 || j >= n1) return false;
    j += joff;
    return true;
  }
  // place p holds column ((p - 1 - t) mod (be2 - 1)) + 1, place 0 column 0
  const int be2 = b + (b & 1), tb = be2 - 1 - k;
  int x = k == 0 ? 0 : k - t, y = tb == 0 ? 0 : tb - t;
  if (k != 0 && x < 1) x += be2 - 1;
  if (tb != 0 && y < 1) y += be2 - 1;
  i = min(x, y);
  j = max(x, y);
  return j < n0;
}

// All rounds of one diagonal block (cross = false: n0 columns, round-robin over
// be2 places) or of one pair of blocks (cross: columns kk < n0 against
// joff + (kk + t) mod b for t = 0 .. b-1) of columns held in shared memory, for
// the runs that keep the order of their sums.  Each half-warp takes one pair a
// round.  Out of line and with the columns as its only data pointer: it is told
// that they are shared memory, which its caller, choosing between the staging
// buffer and global memory elsewhere, must not be.
static __device__ __noinline__ void kept_rounds(cplx* cols, int ld, int q, bool cross, int b, int n0, int n1, int joff,
                                                double tol, int* rot) {
  ASSUME_SHARED(cols);
  const int hl = ltid() & 15, hw = ltid() >> 4;
  const unsigned mask = (ltid() & 16) ? 0xffff0000u : 0x0000ffffu;
  const int be2 = b + (b & 1);
  const int rounds = cross ? b : be2 - 1, npairs = cross ? b : be2 / 2;
#pragma unroll 1
  for (int t = 0; t < rounds; ++t) {
#pragma unroll 1
    for (int k = hw; k < npairs; k += NT / 16) {
      int i, j;
      if (!block_pair(cross, b, n0, n1, joff, t, k, i, j)) continue;
      cplx* bi = cols + ld * i;
      cplx* bj = cols + ld * j;
      double al = 0.0, be = 0.0, gx = 0.0, gy = 0.0;
      for (int r = hl; r < q; r += 16) {
        cplx x = bi[r], y = bj[r];
        al += cabs2(x);
        be += cabs2(y);
        gx += x.x * y.x + x.y * y.y;
        gy += x.x * y.y - x.y * y.x;
      }
      {  // the four trees over 16 lanes with the values halved twice: same pairs, 9 shuffles instead of 16
        const int base = (ltid() & 31) & 16;
        bool up = (hl & 8) != 0;
        double k0 = up ? gx : al, k1 = up ? gy : be;
        const double g0 = up ? al : gx, g1 = up ? be : gy;
        k0 += __shfl_xor_sync(mask, g0, 8);
        k1 += __shfl_xor_sync(mask, g1, 8);
        up = (hl & 4) != 0;
        double v = up ? k1 : k0;
        const double g = up ? k0 : k1;
        v += __shfl_xor_sync(mask, g, 4);
        v += __shfl_xor_sync(mask, v, 2);
        v += __shfl_xor_sync(mask, v, 1);
        al = __shfl_sync(mask, v, base);
        be = __shfl_sync(mask, v, base + 4);
        gx = __shfl_sync(mask, v, base + 8);
        gy = __shfl_sync(mask, v, base + 12);
      }
      double c;
      cplx se, sec;
      if (!jacobi_params(al, be, gx, gy, tol, c, se, sec)) continue;
      if (hl == 0) *rot = 1;  // any rotation keeps the sweeps going
      for (int r = hl; r < q; r += 16) {
        cplx x = bi[r], y = bj[r];
        bi[r] = csub(cscale(x, c), cmul(sec, y));
        bj[r] = cadd(cmul(se, x), cscale(y, c));
      }
    }
    cta_sync();
  }
}

// The same for the runs that may reorder sums, LP lanes a pair, RPL rows a lane.  A round is one dependent chain, so its
// length is its cost: both columns are loaded at once and stay in registers
// for the update, the four sums are reduced together, and the rotation comes
// from two reciprocal square roots: with R = sqrt(d^2 + 4 |g|^2),
//   cos^2 = (1 + |d| / R) / 2,  sin / |g| = 1 / (R cos),
// instead of a chain of rsqrt, sqrt, division and rsqrt.
template <int LP, int RPL>
static __device__ __noinline__ void jacobi_rounds(cplx* cols, int ld, int q, bool cross, int b, int n0, int n1, int joff,
                                                  double tol2, int* rot) {
  ASSUME_SHARED(cols);
  const int hl = ltid() & (LP - 1), grp = ltid() / LP;
  const int base = (ltid() & 31) & ~(LP - 1);
  const unsigned mask = LP == 32 ? 0xffffffffu : ((1u << (LP & 31)) - 1u) << base;
  const int be2 = b + (b & 1);
  const int rounds = cross ? b : be2 - 1, npairs = cross ? b : be2 / 2;
#pragma unroll 1
  for (int t = 0; t < rounds; ++t) {
#pragma unroll 1
    for (int k = grp; k < npairs; k += NT / LP) {
      int i, j;
      if (!block_pair(cross, b, n0, n1, joff, t, k, i, j)) continue;
      cplx* bi = cols + ld * i;
      cplx* bj = cols + ld * j;
      cplx x[RPL], y[RPL];
#pragma unroll
      for (int u = 0; u < RPL; ++u) {
        const int r = hl + LP * u;
        x[u] = r < q ? bi[r] : make_double2(0.0, 0.0);
        y[u] = r < q ? bj[r] : make_double2(0.0, 0.0);
      }
      double d4[4] = {0.0, 0.0, 0.0, 0.0};  // |b_i|^2, |b_j|^2, b_i^H b_j
#pragma unroll
      for (int u = 0; u < RPL; ++u) {
        d4[0] = fma(x[u].x, x[u].x, fma(x[u].y, x[u].y, d4[0]));
        d4[1] = fma(y[u].x, y[u].x, fma(y[u].y, y[u].y, d4[1]));
        d4[2] = fma(x[u].x, y[u].x, fma(x[u].y, y[u].y, d4[2]));
        d4[3] = fma(x[u].x, y[u].y, fma(-x[u].y, y[u].x, d4[3]));
      }
      {  // butterfly over the pair's lanes, halving the values twice
        bool up = (hl & (LP / 2)) != 0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double keep = up ? d4[e + 2] : d4[e], give = up ? d4[e] : d4[e + 2];
          d4[e] = keep + __shfl_xor_sync(mask, give, LP / 2);
        }
        up = (hl & (LP / 4)) != 0;
        const double keep = up ? d4[1] : d4[0], give = up ? d4[0] : d4[1];
        d4[0] = keep + __shfl_xor_sync(mask, give, LP / 4);
#pragma unroll
        for (int o = LP / 8; o > 0; o >>= 1) d4[0] += __shfl_xor_sync(mask, d4[0], o);
      }
      const double al = __shfl_sync(mask, d4[0], base), be = __shfl_sync(mask, d4[0], base + LP / 4);
      const double gx = __shfl_sync(mask, d4[0], base + LP / 2), gy = __shfl_sync(mask, d4[0], base + 3 * LP / 4);
      const double g2 = fma(gx, gx, gy * gy);
      if (!(g2 > tol2 * (al * be))) continue;
      if (hl == 0) *rot = 1;  // any rotation keeps the sweeps going
      const double d = be - al;
      const double h = rsqrt(fma(d, d, 4.0 * g2));
      const double c2 = fma(0.5 * fabs(d), h, 0.5);
      const double rc = rsqrt(c2);
      const double c = c2 * rc, f = d < 0.0 ? -h * rc : h * rc;
      const cplx se = make_double2(f * gx, f * gy);
#pragma unroll
      for (int u = 0; u < RPL; ++u) {
        const int r = hl + LP * u;
        if (r < q) {
          const cplx a = x[u], e = y[u];
          // b_i <- c b_i - conj(se) b_j,  b_j <- se b_i + c b_j
          bi[r] = make_double2(fma(c, a.x, fma(-se.x, e.x, -se.y * e.y)), fma(c, a.y, fma(-se.x, e.y, se.y * e.x)));
          bj[r] = make_double2(fma(c, e.x, fma(se.x, a.x, -se.y * a.y)), fma(c, e.y, fma(se.x, a.y, se.y * a.x)));
        }
      }
    }
    cta_sync();
  }
}

// A pair gets 16 lanes where a round's pairs leave that many, else 8, and at
// least as many as hold its rows in registers; q <= 256 (SVD_MAX_COLS).
template <int LP>
static __device__ __forceinline__ void jacobi_block_lp(cplx* cols, int ld, int q, bool cross, int b, int n0, int n1,
                                                       int joff, double tol2, int* rot) {
  if (q <= LP)
    jacobi_rounds<LP, 1>(cols, ld, q, cross, b, n0, n1, joff, tol2, rot);
  else if (q <= 2 * LP)
    jacobi_rounds<LP, 2>(cols, ld, q, cross, b, n0, n1, joff, tol2, rot);
  else if (q <= 4 * LP)
    jacobi_rounds<LP, 4>(cols, ld, q, cross, b, n0, n1, joff, tol2, rot);
  else
    jacobi_rounds<LP, 8>(cols, ld, q, cross, b, n0, n1, joff, tol2, rot);
}
static __device__ __forceinline__ void jacobi_block(cplx* cols, int ld, int q, bool cross, int b, int n0, int n1,
                                                    int joff, double tol, int* rot) {
  const int npairs = cross ? b : (b + 1) / 2;
  if (q > 128)  // up to 256 rows
    jacobi_rounds<32, 8>(cols, ld, q, cross, b, n0, n1, joff, tol * tol, rot);
  else if (npairs * 16 <= NT || q > 64)
    jacobi_block_lp<16>(cols, ld, q, cross, b, n0, n1, joff, tol * tol, rot);
  else
    jacobi_block_lp<8>(cols, ld, q, cross, b, n0, n1, joff, tol * tol, rot);
}

// Stage columns [c0, c0+nc0) and [c1, c1+nc1) of B into sb (ld = q), or
// write them back.
static __device__ __forceinline__ void svd_stage(cplx* sb, int ld, const SvdWork& w, int q, int c0, int nc0, int c1, int nc1,
                                          bool store) {
  const int nc = nc0 + nc1;
  for (int e = ltid(); e < nc * ld; e += NT) {
    int r = (int)(e % ld), lc = (int)(e / ld);
    int col = lc < nc0 ? c0 + lc : c1 + (lc - nc0);
    cplx* g = w.B + (long long)q * col + r;
    if (store) *g = sb[e];
    else sb[e] = *g;
  }
  cta_sync();
}

// SVD of M (m x n, col-major ld m), phase 1.  side LEFT asks for the left
// singular vectors (orthonormal U, m-vectors), side RIGHT for the right ones
// (orthonormal V, n-vectors).  QR-preconditioned one-sided Jacobi
// (Drmac-Veselic): LEFT factors M^H = Q R and orthogonalises the columns of
// B = R^H (m x k); RIGHT factors M = Q R and orthogonalises B = R^H
// (n x k); k = min(m, n).  Either way B's columns converge to (vectors) x
// Sigma.  Jacobi runs in the block-cyclic order (per sweep: every diagonal
// block with a round-robin pass, then every pair of blocks in round-robin
// order with b rounds of disjoint cross pairs) on blocks staged in the
// shared buffer sb (SVD_SMEM_CPLX elements), or on all of B held there when
// it fits: the sweeps then touch no global memory, where each block pair
// used to be read and written back every time it was rotated.  Leaves the sorted singular
// values in w.sig (nulls set to 0).  CTA-collective; returns metadata.
enum { SVD_LEFT = 0, SVD_RIGHT = 1 };
static __device__ __noinline__ SvdResult dev_svd(const cplx* M, int m, int n, int side, SvdWork& w, LinalgSmem& ls,
                                          RedScratch& rs, cplx* sb) {
  ProfScope prof_scope_(PF_SVD);
  const int tid = ltid();
  SvdResult res;
  res.tr = side == SVD_RIGHT;
  const int mm = res.tr ? m : n;  // rows of the factored matrix H
  const int nn = res.tr ? n : m;
  const int k = min(m, n);
  const int q = nn, p = k;
  res.q = q;
  res.p = p;
  res.sweeps = 0;
  // A problem that fits the shared buffer stays there: the factored matrix
  // (at the end of the buffer, or in global memory) and B for all sweeps.
  const bool resident = q * p <= SVD_SMEM_CPLX;
  const bool panel = ls.blocked && mm <= QR_PANEL_MAX_ROWS;
  const bool one_panel = panel && nn <= QR_PANEL && mm * nn + q * p <= SVD_SMEM_CPLX;
  const bool h_shared = one_panel || (!panel && mm * nn <= SVD_SMEM_CPLX);
  const bool both = resident && (panel || mm * nn + q * p <= SVD_SMEM_CPLX);
  cplx* H = h_shared ? sb + (SVD_SMEM_CPLX - mm * nn) : w.X;
  auto load = [&](int e) {
    const int c = e / mm, r = e - c * mm;
    return res.tr ? M[e] : cconj(M[c + m * r]);
  };
  if (one_panel) {
    const double null_abs = qr_load_panel(mm, nn, load, H, rs);
    ProfScope qr_scope_(PF_QR);
    qr_panel_rows(H, mm, 0, k, nn, null_abs, ls.tau);
  } else {
    for (int e = tid; e < mm * nn; e += NT) H[e] = load(e);
    cta_sync();
    if (panel)
      dev_qr_factor_panel(H, mm, nn, sb, ls, rs);
    else if (h_shared)
      dev_qr_factor_at<true>(H, mm, nn, ls, rs);
    else
      dev_qr_factor_at<false>(H, mm, nn, ls, rs);
  }
  // B = R^H (nn x k): B[r, c] = conj(R[c, r]) for c <= r
  cplx* B0 = both ? sb : w.B;
  for (int e = tid; e < q * p; e += NT) {
    const int c = e / q, r = e - c * q;
    B0[e] = (c <= r) ? cconj(H[c + mm * r]) : make_double2(0.0, 0.0);
  }
  cta_sync();
  if (resident && !both) {
    cta_copy(sb, w.B, (long long)q * p);
    cta_sync();
  }
  const double tol = 2.220446049250313e-16 * q;
  const bool blocked = ls.blocked != 0;
  const int ld = q;
  const int b = svd_block_size(q, p);
  const int nb = (p + b - 1) / b;
  const int nbe = nb + (nb & 1);
  for (int sweep = 0; sweep < JACOBI_MAX_SWEEPS; ++sweep) {
    if (tid == 0) ls.rot_count = 0;
    cta_sync();
    for (int I = 0; I < nb; ++I) {
      const int c0 = I * b, nc = min(b, p - c0);
      if (!resident) svd_stage(sb, ld, w, q, c0, nc, 0, 0, false);
      cplx* cols = resident ? sb + ld * c0 : sb;
      if (blocked)
        jacobi_block(cols, ld, q, false, b, nc, 0, 0, tol, &ls.rot_count);
      else
        kept_rounds(cols, ld, q, false, b, nc, 0, 0, tol, &ls.rot_count);
      if (!resident) svd_stage(sb, ld, w, q, c0, nc, 0, 0, true);
    }
    for (int round = 0; round < nbe - 1; ++round) {
      for (int pr = 0; pr < nbe / 2; ++pr) {
        int ta = pr, tb = nbe - 1 - pr;
        int A = ta == 0 ? 0 : ((ta - 1 - round + 2 * (nbe - 1)) % (nbe - 1)) + 1;
        int Bk = tb == 0 ? 0 : ((tb - 1 - round + 2 * (nbe - 1)) % (nbe - 1)) + 1;
        int I = min(A, Bk), J = max(A, Bk);
        if (J >= nb) continue;
        const int c0 = I * b, n0 = min(b, p - c0), c1 = J * b, n1 = min(b, p - c1);
        if (!resident) svd_stage(sb, ld, w, q, c0, n0, c1, n1, false);
        cplx* cols = resident ? sb + ld * c0 : sb;
        const int joff = resident ? c1 - c0 : n0;
        if (blocked)
          jacobi_block(cols, ld, q, true, b, n0, n1, joff, tol, &ls.rot_count);
        else
          kept_rounds(cols, ld, q, true, b, n0, n1, joff, tol, &ls.rot_count);
        if (!resident) svd_stage(sb, ld, w, q, c0, n0, c1, n1, true);
      }
    }
    int rc = ls.rot_count;
    cta_sync();
    res.sweeps = sweep + 1;
    if (rc == 0) break;
  }
  // singular values; the factorisation's scalars are done with, their room
  // holds the unsorted values and the order
  const cplx* Bv = resident ? sb : w.B;
  double* sig0 = reinterpret_cast<double*>(ls.tau);
  int* ord = reinterpret_cast<int*>(sig0 + SVD_MAX_COLS);
  if (resident) cta_copy(w.B, sb, (long long)q * p);
  const int lane = tid & 31, wid = tid >> 5;
  for (int c = wid; c < p; c += NW) {
    const cplx* bc = Bv + q * c;
    double s = 0.0;
    for (int r = lane; r < q; r += 32) s += cabs2(bc[r]);
    s = warp_sum(s);
    if (lane == 0) sig0[c] = sqrt(s);
  }
  cta_sync();
  // stable descending order
  for (int c = tid; c < p; c += NT) {
    double sc = sig0[c];
    int rank = 0;
    for (int c2 = 0; c2 < p; ++c2) {
      double s2 = sig0[c2];
      if (s2 > sc || (s2 == sc && c2 < c)) ++rank;
    }
    ord[rank] = c;
    w.ord[rank] = c;
  }
  cta_sync();
  // sorted singular values into sig (nulls zeroed); rank = their non-null prefix
  const double smax = p > 0 ? sig0[ord[0]] : 0.0;
  int cnt = 0;
  for (int k2 = tid; k2 < p; k2 += NT) {
    const double s = sig0[ord[k2]];
    const bool live = smax > 0.0 && s > SVD_NULL_TOL * smax;
    cnt += live ? 1 : 0;
    w.sig[k2] = live ? s : 0.0;
  }
  res.rank = (int)block_sum((double)cnt, rs);
  return res;
}

// Phase 2: the requested orthonormal vectors Yo (q x need): column k is
// B[:, ord[k]] / sigma_k for non-null k and an orthonormal completion for
// null k < need.  CTA-collective.
static __device__ __noinline__ void dev_svd_vectors(const SvdResult& res, int need, SvdWork& w, RedScratch& rs) {
  ProfScope prof_scope_(PF_SVDVEC);
  const int tid = ltid(), q = res.q, p = res.p;
  need = min(need, p);
  const int ng = min(need, res.rank);
  for (int e = tid; e < q * ng; e += NT) {
    const int k = e / q, r = e - k * q;
    w.Yo[e] = cscale(w.B[r + q * w.ord[k]], 1.0 / w.sig[k]);
  }
  cta_sync();
  for (int k = res.rank; k < need; ++k) dev_complete_column(w.Yo, q, k, w.y, rs);
}

// Truncation ranks (see the oracle for the reference lines they restate).
// split_mps_tensor_svd / two_site_svd: absolute, keep crossing value, min 2.
static __device__ __forceinline__ int keep_tdvp(const double* S, int n, double thr, int max_bond) {
  double disc = 0.0;
  int keep = n;
  for (int k = n; k >= 1; --k) {
    disc += S[k - 1] * S[k - 1];
    if (disc >= thr) {
      keep = max(k, 2);
      break;
    }
  }
  return max(1, min(keep, max_bond));
}
// Dissipation / jump split: relative, min 1.
static __device__ __forceinline__ int keep_relative(const double* S, int n, double thr, int max_bond) {
  double nsq = 0.0;
  for (int k = 0; k < n; ++k) nsq += S[k] * S[k];
  double cur = 0.0;
  int rank = n;
  for (int k = n; k >= 1; --k) {
    cur += S[k - 1] * S[k - 1];
    if (cur > thr * nsq) {
      rank = k;
      break;
    }
  }
  return max(1, min(rank, max_bond));
}

// apply_local_gate_exact! (DigitalTJM.jl:282-292): absolute, drop while the
// running sum plus s^2 stays <= thr, no minimum.
static __device__ __forceinline__ int keep_tebd(const double* S, int n, double thr, int max_bond) {
  double cur = 0.0;
  int keep = n;
  for (int k = n; k >= 1; --k) {
    if (cur + S[k - 1] * S[k - 1] > thr) break;
    cur += S[k - 1] * S[k - 1];
    --keep;
  }
  return max(1, min(keep, max_bond));
}
