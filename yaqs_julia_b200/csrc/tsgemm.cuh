// tsgemm.cuh — the structured effective-Hamiltonian product of the mixed form
// on the 5th-generation tensor cores (included by krylov.cuh in the
// tensor-core translation unit).
//
//   y[(a,p'), b]  =  sum_blocks X_b[(a,p'), c] R_b[c, b]        (right blocks)
//   y[a, (p',b)] +=  sum_blocks L_b[a, a'] X_b[a', (p',b)]      (left blocks)
//
// with X_b a slice permutation of x (or of T1 = L_m x) times a factor per p'
// (HPlan).  The left sum runs transposed, rows (p',b), so that both products
// have up to 128 rows and 64 columns a tile at chi = 64, D = 2.
//
// Arithmetic: every real product as three TF32 products (hi lo + lo hi + hi
// hi of the 3xTF32 split), accumulated in FP32 in tensor memory; a complex
// product as four real ones into two accumulators (the subtraction by the
// instruction's negate bit), 12 tcgen05.mma per 8 k.
//
// Bound: with tc_gemm (TMA-fed, nine MMAs in the three-product form, one
// 8-deep K step per barrier) a step took about 2600 clocks for 300 of MMAs:
// six planes to split and store, and a chain of mbarrier, split, fence,
// barrier and commit for every eight k.  Here a step is 16 deep, four planes
// are split (the sum plane is gone), and the operands come straight from FP32
// copies of x and the environments into registers, one step ahead, under the
// MMAs of the step before.  The product needs no MPO apply and no operand
// staging, and 64 K steps of 8 instead of 88 at chi = 64, w = 5.
#pragma once

#define TS_BK 16

static __device__ __forceinline__ void ts_split4(unsigned* planes, int plane_words, int r, int q, const cflt* v) {
  unsigned h0[4], l0[4], h1[4], l1[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    h0[j] = tf32_rna(v[j].x);
    l0[j] = tf32_rna(v[j].x - __uint_as_float(h0[j]));
    h1[j] = tf32_rna(v[j].y);
    l1[j] = tf32_rna(v[j].y - __uint_as_float(h1[j]));
  }
  const int w = tc_plane_off(r, q) >> 2;
  *reinterpret_cast<uint4*>(planes + 0 * plane_words + w) = make_uint4(h0[0], h0[1], h0[2], h0[3]);
  *reinterpret_cast<uint4*>(planes + 1 * plane_words + w) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
  *reinterpret_cast<uint4*>(planes + 2 * plane_words + w) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
  *reinterpret_cast<uint4*>(planes + 3 * plane_words + w) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
}

// Shared memory: [K step][plane][rows x 8 k] of A and B (48 KB of the union).
struct TsSmem {
  unsigned a[2][4][1024];
  unsigned b[2][4][512];
};
static_assert(sizeof(TsSmem) <= sizeof(TcSmem), "the planes must fit the tensor-core staging");

enum { TS_RIGHT = 0, TS_LEFT = 1, TS_T1 = 2 };

// One pass over all its tiles.  CTA-collective; false once a wait gave up.
//   TS_RIGHT: y = sum;  TS_LEFT: y += sum + local term;  TS_T1: T1f = L_m x.
template <int MODE>
static __device__ __noinline__ bool ts_pass(const HeffOp& h, const TsSide& side, const cplx* loc, const cplx* x,
                                            cplx* y, TcSmem& raw, TcState& st) {
  ProfScope prof_scope_(PF_GEMM);
  ASSUME_SHARED(&raw);
  ASSUME_SHARED(&side);
  ASSUME_SHARED(loc);
  TsSmem& s = reinterpret_cast<TsSmem&>(raw);
  const int tid = ltid(), lane = tid & 31, wid = tid >> 5;
  const int chil = h.chil, D = h.D, chir = h.chir;
  const int nt1 = h.plan->nt1, t1m = h.plan->t1m;
  const bool has_loc = h.plan->has_loc != 0;
  const int M = MODE == TS_RIGHT ? chil * D : MODE == TS_LEFT ? D * chir : chil * nt1;
  const int N = MODE == TS_RIGHT ? chir : MODE == TS_LEFT ? chil : D * chir;
  const int K = MODE == TS_RIGHT ? chir : chil;
  const int nb = MODE == TS_T1 ? 1 : side.nb;
  cta_sync();
  if (st.fatal) return false;
  unsigned phase = st.ph_mma & 1;
  bool ok = true;
  // this thread's share: A row ar, K half ah (8 values); B column bc, quad bq (4 values)
  const int ar = MODE == TS_LEFT ? tid >> 1 : tid & 127, ah = MODE == TS_LEFT ? tid & 1 : tid >> 7;
  const int bc = MODE == TS_T1 ? tid >> 2 : tid & 63, bq = MODE == TS_T1 ? tid & 3 : tid >> 6;
  const int steps = (K + TS_BK - 1) / TS_BK;
  for (int m0 = 0; m0 < M; m0 += TC_BM) {
    const int row = m0 + ar;
    const bool rok = row < M;
    const int pp = MODE == TS_RIGHT ? row / chil : MODE == TS_LEFT ? row % D : 0;
    const int r0 = MODE == TS_RIGHT ? row - pp * chil : MODE == TS_LEFT ? row / D : row;
    for (int n0 = 0; n0 < N; n0 += TC_BN) {
      const int nrem = min(TC_BN, N - n0);
      const unsigned idesc = tc_idesc((nrem + 15) & ~15), idneg = idesc | (1u << 13);
      const bool cok = n0 + bc < N;
      const cflt *pa = nullptr, *pb = nullptr;
      int ka = 0, kb = 0;  // strides over k
      float2 coef = make_float2(1.f, 0.f);
      auto block = [&](int b) {
        pa = pb = nullptr;
        if (MODE == TS_T1) {
          if (rok) pa = h.Lf + chil * t1m + row;
          ka = chil * h.wl;
          if (cok) pb = h.xf + (n0 + bc) * chil;
          kb = 1;
          return;
        }
        const int src = rok ? side.src[b][pp] : -1;
        if (MODE == TS_RIGHT) {
          const int g = rok ? side.t1[b][pp] : -1, ld = g < 0 ? chil : chil * nt1;
          if (src >= 0) pa = (g < 0 ? h.xf : h.T1f + chil * g) + ld * src + r0;
          ka = ld * D;
          if (cok) pb = h.Rf + chir * side.m[b] + n0 + bc;
          kb = chir * h.wr;
        } else {
          if (src >= 0) pa = h.xf + chil * (src + D * r0);
          ka = 1;
          if (cok) pb = h.Lf + chil * side.m[b] + n0 + bc;
          kb = chil * h.wl;
        }
        if (src >= 0) coef = side.coef[b][pp];
      };
      cflt va[8], vb[4];
      auto load = [&](int k0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int k = k0 + 8 * ah + j;
          va[j] = pa && k < K ? pa[k * ka] : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int k = k0 + 4 * bq + j;
          vb[j] = pb && k < K ? pb[k * kb] : make_float2(0.f, 0.f);
        }
      };
      block(0);
      load(0);
      int b = 0, ks = 0;
      const int total = nb * steps;
      for (int t = 0; t < total; ++t) {
        if (MODE != TS_T1 && !(coef.x == 1.f && coef.y == 0.f)) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const cflt v = va[j];
            va[j] = make_float2(fmaf(coef.x, v.x, -coef.y * v.y), fmaf(coef.x, v.y, coef.y * v.x));
          }
        }
        if (t > 0) {  // the MMAs that last read the planes are done
          ok &= mbar_wait(&st.bar_mma[0], phase);
          phase ^= 1;
        }
        ts_split4(&s.a[ah][0][0], 1024, ar, 0, va);
        ts_split4(&s.a[ah][0][0], 1024, ar, 1, va + 4);
        ts_split4(&s.b[bq >> 1][0][0], 512, bc, bq & 1, vb);
        fence_async_smem();
        cta_sync();
        if (tid == 0) {
          tc_fence_after();
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const unsigned long long a0 = tc_sdesc(&s.a[u][0][0], 128, 256), b0 = tc_sdesc(&s.b[u][0][0], 128, 256);
            // planes of one K step are 4096 (A) and 2048 (B) bytes apart: 256 and 128 in descriptor units
            const unsigned long long arh = a0, arl = a0 + 256, aih = a0 + 512, ail = a0 + 768;
            const unsigned long long brh = b0, brl = b0 + 128, bih = b0 + 256, bil = b0 + 384;
            const unsigned re = st.tmem_base, im = st.tmem_base + TC_BN;
            const unsigned acc = t > 0 || u > 0 ? 1u : 0u;
            tc_mma_tf32(re, arh, brl, idesc, acc);
            tc_mma_tf32(im, arh, bil, idesc, acc);
            tc_mma_tf32(re, arl, brh, idesc, 1u);
            tc_mma_tf32(im, arl, bih, idesc, 1u);
            tc_mma_tf32(re, arh, brh, idesc, 1u);
            tc_mma_tf32(im, arh, bih, idesc, 1u);
            tc_mma_tf32(re, aih, bil, idneg, 1u);
            tc_mma_tf32(im, aih, brl, idesc, 1u);
            tc_mma_tf32(re, ail, bih, idneg, 1u);
            tc_mma_tf32(im, ail, brh, idesc, 1u);
            tc_mma_tf32(re, aih, bih, idneg, 1u);
            tc_mma_tf32(im, aih, brh, idesc, 1u);
          }
          tc_commit(&st.bar_mma[0]);
        }
        if (++ks == steps) {
          ks = 0;
          if (++b < nb) block(b);
        }
        if (t + 1 < total) load(ks * TS_BK);  // in flight under the MMAs
      }
      ok &= mbar_wait(&st.bar_mma[0], phase);
      phase ^= 1;
      tc_fence_after();
      // epilogue: warp w reads lanes 32 (w % 4) .. +31, warps 0-3 the first 32
      // columns.  Loads and stores of y are dense and in batches: one element
      // at a time, each waiting for the one before, they took 200 of the 375 us
      // of a 64 x 2 x 64 product.
      const int quarter = wid & 3, half = wid >> 2;
      const int r_base = m0 + quarter * 32;
      const unsigned lane_addr = st.tmem_base + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
      for (int c16 = 0; c16 < 2; ++c16) {
        const int col = half * 32 + c16 * 16;
        if (col >= nrem || r_base >= M) break;  // uniform per warp
        float re[16], im[16];
        tmem_ld16(lane_addr + col, re);
        tmem_ld16(lane_addr + TC_BN + col, im);
        tmem_wait_ld();
        if (MODE != TS_LEFT) {  // lanes run along the output's fast index
          const int er = r_base + lane;
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const int n = n0 + col + j;
            if (er < M && n < N) {
              if (MODE == TS_T1)
                h.T1f[er + M * n] = make_float2(re[j], im[j]);
              else
                y[er + M * n] = make_double2(re[j], im[j]);
            }
          }
        } else {
          // turned in shared memory (the planes are free): the fast index of y is the column
          float2* turn = reinterpret_cast<float2*>(&s) + wid * (32 * 17);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 16; ++j) turn[lane * 17 + j] = make_float2(re[j], im[j]);
          __syncwarp();
          const int j = lane & 15, n = n0 + col + j;
#pragma unroll 1
          for (int i0 = lane >> 4; i0 < 32; i0 += 16) {
            cplx v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int er = r_base + i0 + 2 * u;
              v[u] = er < M && n < N ? y[n + chil * er] : make_double2(0.0, 0.0);
            }
            if (has_loc) {
#pragma unroll 1
              for (int p = 0; p < D; ++p) {
                cplx xv[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                  const int er = r_base + i0 + 2 * u, bb = er / D;
                  xv[u] = er < M && n < N ? x[n + chil * (p + D * bb)] : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                  const int er = r_base + i0 + 2 * u;
                  cfma(v[u], loc[er % D + D * p], xv[u]);
                }
              }
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
              const int er = r_base + i0 + 2 * u;
              const float2 t = turn[(i0 + 2 * u) * 17 + j];
              if (er < M && n < N) y[n + chil * er] = make_double2(v[u].x + t.x, v[u].y + t.y);
            }
          }
        }
      }
      tc_fence_before();
      cta_sync();
    }
  }
  if (!ok) st.fatal = 1;  // benign race: every writer stores 1
  cta_sync();
  if (tid == 0) st.ph_mma = (st.ph_mma & ~1u) | phase;
  const bool good = !st.fatal;
  cta_sync();
  return good;
}

// y = H_eff x by the plan of h; ts[0], ts[1] its left and right blocks.  h.xf
// holds x in FP32.
static __device__ __forceinline__ void ts_heff(const HeffOp& h, const cplx* x, cplx* y, const TsSide* ts,
                                               const cplx* loc, TcSmem& raw, TcState& st) {
  if (h.plan->nt1 > 0) ts_pass<TS_T1>(h, ts[0], loc, x, y, raw, st);
  ts_pass<TS_RIGHT>(h, ts[1], loc, x, y, raw, st);
  ts_pass<TS_LEFT>(h, ts[0], loc, x, y, raw, st);
}
