// fh_hline_df.cuh -- the implicit line solve of one 1D H_solver step in
// double-float, for the mixed-precision mode (FH_H_BLOCKED): the
// cancellation-free elimination of fh_hline.cuh with every operation on the
// FP32 pipe.
//
// Why: in FP64 the solve is bound by its ~80 FP64 instructions per equation
// (one FP64 warp instruction takes an SM 17 cycles, ~1400 cycles per 32
// equations); the ~400 FP32 instructions of this form take 100.  All factors
// are sums and products of non-negative terms, so an error of 2^-47 per
// operation stays that of the result relative to its size.
//
// Only lines of kHdfMinN intervals and more.  A line's coefficients carry the
// pairs' 2^-47 into the solution times ~N; the reference's order in FP64 loses
// ~N^2 2^-53 to cancellation.  Error of psi solves against 64 bits, reference
// order / pairs / the FP64 form of fh_hline.cuh: N = 256, 600 steps 1.4e-12 /
// 3.0e-12 / 1.4e-12; 512, 800 steps 4.1e-12 / 5.7e-12 / 0.9e-12; 640: 9.7e-12 /
// 7.8e-12 / 1.2e-12, single batches 5.9e-12 / 1.0e-11; 768: 2.2e-11 / 1.0e-11 /
// 1.3e-12; 1024: 3.2e-11 / 1.3e-11 / 1.0e-12 (1500 steps: 768 3.7e-11 / 1.5e-11).
// So pairs are no further off than the reference's order from 768 on, and shorter
// lines run in FP64: 512 psi instances of 64..1024 nodes, 1500 steps 111 -> 148 ms,
// 1.3e-11 -> 1.1e-11.
//
// Everything is divided by Dg kc / c (the row scale of A, B, R): A_i and B_i
// are then exp(gam u) of the neighbours, the row sum s is (Da c / (Dg kc)) wc,
// and the FP32 exponent range holds them.  Lines out of that range
// (kHdfExp, kHdfRow), with states or boundary values that FP32 pairs do not hold
// (above kHdfState, or all below kHdfFloor: a product of one with a row sum
// would lose its low word), with al_left outside [0, 1], or too long for one
// panel are left to the FP64 solve (the function returns false).
//
// exp: table and polynomial (Tang, ACM TOMS 15, 1989, here in pairs): 2^(j/16) from
// a table times a Taylor polynomial of degree 6 on |r| <= ln 2 / 32 (next term
// 2^-51), its terms above the third power in FP32.
#pragma once
#include "fh_df.cuh"
#include "fh_hline.cuh"

// |gam u| at most: a pair near 8 ends at 2^-44, and exp turns that into a relative
// error of K (2^-43.9 measured for 11, 2^-46 for 2)
constexpr float kHdfExp = 2.0f;
constexpr float kHdfRow = 0x1p16f;           // row sum at most, 2^-40 at least
constexpr float kHdfState = 0x1p60f;
constexpr float kHdfFloor = 0x1p-54f;        // the largest state or boundary value at least
constexpr int kHdfMinN = 768;                // intervals of a line at least

__device__ const float2 kHdfTab[16] = {  // 2^(j/16)
    {0x1.000000p+0f, 0.0f},           {0x1.0b5586p+0f, 0x1.9f3122p-25f},  {0x1.172b84p+0f, -0x1.c15742p-27f},
    {0x1.2387a6p+0f, 0x1.ceac48p-25f},  {0x1.306fe0p+0f, 0x1.4636e2p-25f},  {0x1.3dea64p+0f, 0x1.824684p-25f},
    {0x1.4bfdaep+0f, -0x1.593abcp-25f}, {0x1.5ab07ep+0f, -0x1.5bd5ecp-27f}, {0x1.6a09e6p+0f, 0x1.9fcef4p-26f},
    {0x1.7a1148p+0f, -0x1.829fd0p-25f}, {0x1.8ace54p+0f, 0x1.15506ep-27f},  {0x1.9c4918p+0f, 0x1.51f848p-27f},
    {0x1.ae89fap+0f, -0x1.a94b14p-26f}, {0x1.c199bep+0f, -0x1.3d56b2p-27f}, {0x1.d5818ep+0f, -0x1.822dbcp-27f},
    {0x1.ea4afap+0f, 0x1.52486cp-27f}};

// exp(x), |x| <= kHdfExp
__device__ __forceinline__ fh_df fh_df_exp(fh_df x, const float2 *tab) {
  const float n = rintf(x.h * 0x1.715476p+4f);  // 16 / ln 2
  const int k = (int)n;
  // r = x - n ln 2 / 16, ln 2 / 16 in parts of 15, 15 and 24 bits
  float s, e;
  fh_two_sum(fmaf(-n, 0x1.62e4p-5f, x.h), -n * 0x1.7f7cp-24f, s, e);
  e += fmaf(-n, 0x1.1cf79ap-40f, x.l);
  const fh_df r = fh_df_renorm(s, e);
  const float w = r.h * fmaf(r.h, fmaf(r.h, 0x1.6c16c2p-10f, 0x1.111112p-7f), 0x1.555556p-5f);
  const float t0 = 0x1.555556p-3f + w;
  fh_df t{t0, (w - (t0 - 0x1.555556p-3f)) - 0x1.555556p-28f};
  t = fh_df_fma(r, t, fh_df{0.5f, 0.f});
  t = fh_df_fma(fh_df_mul(r, r), t, r);
  const fh_df T = fh_df_from_pair(tab[k & 15]);
  t = fh_df_fma(T, t, T);
  const float sc = __int_as_float((127 + (k >> 4)) << 23);
  return fh_df{t.h * sc, t.l * sc};
}

// a / b for normal a, b and quotients that a pair holds (2^-78 and more): the FP32
// reciprocal's quotient, corrected twice by its remainder.
__device__ __forceinline__ fh_df fh_df_quot(fh_df a, fh_df b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b.h));
  const float q1 = a.h * r;
  float m, e;
  fh_two_sum(fmaf(-q1, b.h, a.h), fmaf(-q1, b.l, a.l), m, e);
  const float q2 = m * r;
  const float q3 = (fmaf(-q2, b.h, m) + e) * r;
  const fh_df q = fh_df_renorm(q1, q2);
  return fh_df_renorm(q.h, q.l + q3);
}

struct fh_dmob {
  fh_df m00, m01, m10, m11;
};
__device__ __forceinline__ fh_dmob fh_dmob_sel(bool c, fh_dmob a, fh_dmob b) {
  return fh_dmob{fh_df_sel(c, a.m00, b.m00), fh_df_sel(c, a.m01, b.m01), fh_df_sel(c, a.m10, b.m10),
                 fh_df_sel(c, a.m11, b.m11)};
}
__device__ __forceinline__ float fh_pow2_inv(float x) {  // 2^-exponent of x, |x| within 2^+-125
  const int e = (__float_as_int(x) >> 23) & 0xff;
  return __int_as_float(max(1, min(253, 254 - e)) << 23);
}
__device__ __forceinline__ fh_df fh_df_pow2(fh_df a, float s) { return fh_df{a.h * s, a.l * s}; }
__device__ __forceinline__ fh_dmob fh_dmob_rescale(fh_dmob m) {
  const float s = fh_pow2_inv(fmaxf(fmaxf(fabsf(m.m00.h), fabsf(m.m01.h)), fmaxf(fabsf(m.m10.h), fabsf(m.m11.h))));
  return fh_dmob{fh_df_pow2(m.m00, s), fh_df_pow2(m.m01, s), fh_df_pow2(m.m10, s), fh_df_pow2(m.m11, s)};
}
// f2 o f1
__device__ __forceinline__ fh_dmob fh_dmob_compose(fh_dmob f2, fh_dmob f1) {
  fh_dmob r;
  r.m00 = fh_df_fma(f2.m00, f1.m00, fh_df_mul(f2.m01, f1.m10));
  r.m01 = fh_df_fma(f2.m00, f1.m01, fh_df_mul(f2.m01, f1.m11));
  r.m10 = fh_df_fma(f2.m10, f1.m00, fh_df_mul(f2.m11, f1.m10));
  r.m11 = fh_df_fma(f2.m10, f1.m01, fh_df_mul(f2.m11, f1.m11));
  return r;
}

template <int NW>
struct fh_hline_df_scan {
  fh_dmob mob[NW];
  fh_daff fwd[NW], bwd[NW];
};

// fh_hl_scan in double-float.
template <int NW, bool REV>
__device__ __forceinline__ fh_df fh_hl_scan_df(fh_daff G, fh_df v, fh_daff *tot) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const fh_daff p = REV ? fh_daff{fh_df_shfl_down(G.a, d), fh_df_shfl_down(G.b, d)}
                          : fh_daff{fh_df_shfl_up(G.a, d), fh_df_shfl_up(G.b, d)};
    G = fh_daff_sel(REV ? lane + d < 32 : lane >= d, fh_daff_compose(G, p), G);
  }
  if (lane == (REV ? 0 : 31)) tot[warp] = G;
  fh_daff e = REV ? fh_daff{fh_df_shfl_down(G.a, 1), fh_df_shfl_down(G.b, 1)}
                  : fh_daff{fh_df_shfl_up(G.a, 1), fh_df_shfl_up(G.b, 1)};
  if (lane == (REV ? 31 : 0)) e = fh_daff{fh_df{1.f, 0.f}, fh_df{0.f, 0.f}};
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const int k = REV ? NW - 1 - j : j;
    if (k == warp) break;
    v = fh_df_fma(tot[k].a, v, tot[k].b);
  }
  return fh_df_fma(e.a, v, e.b);
}

// One step of instance I by a CTA of 32 NW threads: wc the weight of the
// current slot, part the history sums (pairs, state layout).  sm:
// fh_hline_smem(32 NW) bytes.  False, with nothing written, where the line is
// left to the FP64 solve.
template <int NW>
__device__ __forceinline__ bool fh_hline_df(const fh_h_dev_inst &I, double wc, const float2 *part, double *U,
                                            float2 *__restrict__ Dnew, float2 *sm,
                                            fh_hline_df_scan<NW> &sc) {
  constexpr int T = 32 * NW;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  __shared__ float2 tab[16];
  float2 *sE = sm, *sO = sE + fh_hline_len(T), *sU = sO + fh_hline_len(T);
  const long long o = I.off;
  const int N = I.N, n = N - 1;
  if (N < kHdfMinN || n > T * kHLineEq) return false;
  const fh_df zero{0.f, 0.f}, one{1.f, 0.f};
  if (t < 16) tab[t] = kHdfTab[t];
  __syncthreads();
  // ---- state and exp(gam u)
  const fh_df s = fh_df_bits(I.dq * wc), gam = fh_df_bits(I.kgam);
  const fh_df al0 = fh_df_bits(I.al_left), b0 = fh_df_bits(I.bt_left), uN = fh_df_bits(I.u_right);
  float big = fmaxf(fabsf(b0.h), fabsf(uN.h));
  bool ok = s.h >= 0x1p-40f && s.h <= kHdfRow && big <= kHdfState && I.al_left >= 0.0 && I.al_left <= 1.0;
  for (int k = t; k <= N + 1; k += T) {
    const fh_df x = fh_df_bits(U[o + k]);
    sU[fh_hsk(k)] = fh_df_pair(x);
    ok = ok && fabsf(x.h) <= kHdfState;
    big = fmaxf(big, fabsf(x.h));
    if (k <= N) {
      fh_df e = one;
      if (I.kmodel != FH_K_CONST) {
        const fh_df a = fh_df_mul(gam, x);
        ok = ok && fabsf(a.h) <= kHdfExp;
        e = fh_df_exp(fabsf(a.h) <= kHdfExp ? a : zero, tab);
      }
      sE[fh_hsk(k)] = fh_df_pair(e);
    }
  }
  if (!__syncthreads_and(ok) || !__syncthreads_or(big >= kHdfFloor)) return false;
  // ---- right parts
  {
    const fh_df q = fh_df_bits(I.dq), gq = fh_df_bits(I.gq);
    for (int k = t; k < n; k += T) {
      fh_df om = fh_df_neg(fh_df_mul(s, fh_df_from_pair(sU[fh_hsk(k + 1)])));
      if (I.gravity)
        om = fh_df_fma(gq, fh_df_sub(fh_df_from_pair(sE[fh_hsk(k + 1)]), fh_df_from_pair(sE[fh_hsk(k)])), om);
      sO[fh_hsk(k)] = fh_df_pair(fh_df_fma(q, fh_df_from_pair(part[o + 1 + k]), om));
    }
  }
  const int E = (n + T - 1) / T, s0 = t * E;
  const int c = max(0, min(E, n - s0));  // the thread's equations; those past the line's end are identities
  // ---- chunk map of d
  fh_dmob M{one, zero, zero, one};
#pragma unroll
  for (int e = 0; e < kHLineEq; ++e)
    if (e < E) {
      const int k = e < c ? s0 + e : 0;
      const fh_df A = fh_df_from_pair(sE[fh_hsk(k)]), B = fh_df_from_pair(sE[fh_hsk(k + 2)]);
      fh_dmob m;
      m.m00 = fh_df_fma(A, M.m00, fh_df_mul(s, M.m10));
      m.m01 = fh_df_fma(A, M.m01, fh_df_mul(s, M.m11));
      m.m10 = fh_df_fma(B, M.m10, m.m00);
      m.m11 = fh_df_fma(B, M.m11, m.m01);
      M = fh_dmob_sel(e < c, m, M);
      if (e == 3) M = fh_dmob_rescale(M);
    }
  // ---- scan of the maps
  M = fh_dmob_rescale(M);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const fh_dmob p{fh_df_shfl_up(M.m00, d), fh_df_shfl_up(M.m01, d), fh_df_shfl_up(M.m10, d), fh_df_shfl_up(M.m11, d)};
    M = fh_dmob_sel(lane >= d, fh_dmob_rescale(fh_dmob_compose(M, p)), M);
  }
  if (lane == 31) sc.mob[warp] = M;
  fh_dmob X{fh_df_shfl_up(M.m00, 1), fh_df_shfl_up(M.m01, 1), fh_df_shfl_up(M.m10, 1), fh_df_shfl_up(M.m11, 1)};
  if (lane == 0) X = fh_dmob{one, zero, zero, one};
  __syncthreads();
  fh_df P = fh_df_sub(one, al0), Q = one;  // d as P / Q, first at the line's start
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    if (k == warp) break;
    const fh_dmob W = sc.mob[k];
    const fh_df p = fh_df_fma(W.m00, P, fh_df_mul(W.m01, Q)), r = fh_df_fma(W.m10, P, fh_df_mul(W.m11, Q));
    const float f = fh_pow2_inv(r.h);
    P = fh_df_pow2(p, f);
    Q = fh_df_pow2(r, f);
  }
  {
    const fh_df p = fh_df_fma(X.m00, P, fh_df_mul(X.m01, Q));
    Q = fh_df_fma(X.m10, P, fh_df_mul(X.m11, Q));
    P = p;
    const float f = fh_pow2_inv(Q.h);
    P = fh_df_pow2(P, f);
    Q = fh_df_pow2(Q, f);
  }
  // ---- the thread's factors and the forward substitution from zero
  fh_df al[kHLineEq], bt[kHLineEq], pf[kHLineEq];
  fh_daff F{one, zero};
#pragma unroll
  for (int e = 0; e < kHLineEq; ++e)
    if (e < E) {
      const bool in = e < c;
      const int k = in ? s0 + e : 0;
      const fh_df A = fh_df_from_pair(sE[fh_hsk(k)]), B = fh_df_from_pair(sE[fh_hsk(k + 2)]);
      const fh_df Pn = fh_df_fma(A, P, fh_df_mul(s, Q)), Qn = fh_df_fma(B, Q, Pn);
      const fh_df g = fh_df_quot(Q, Qn);
      const float r = fh_pow2_inv(Qn.h);
      P = fh_df_pow2(Pn, r);
      Q = fh_df_pow2(Qn, r);
      al[e] = fh_df_sel(in, fh_df_mul(B, g), one);
      const fh_df f = fh_df_mul(g, A);
      const fh_df b = fh_df_fma(f, F.b, fh_df_neg(fh_df_mul(g, fh_df_from_pair(sO[fh_hsk(k)]))));
      F = fh_daff_sel(in, fh_daff{fh_df_mul(f, F.a), b}, F);
      pf[e] = F.a;
      bt[e] = fh_df_sel(in, F.b, zero);
    }
  {
    const fh_df S = fh_hl_scan_df<NW, false>(F, b0, sc.fwd);
#pragma unroll
    for (int e = 0; e < kHLineEq; ++e)
      if (e < E && e < c) bt[e] = fh_df_fma(pf[e], S, bt[e]);
  }
  // ---- back substitution
  fh_daff G{one, zero};
#pragma unroll
  for (int e = kHLineEq - 1; e >= 0; --e)
    if (e < E) {
      G.b = fh_df_fma(al[e], G.b, bt[e]);
      G.a = fh_df_mul(al[e], G.a);
      bt[e] = G.b;
      al[e] = G.a;
    }
  const fh_df S = fh_hl_scan_df<NW, true>(G, uN, sc.bwd);
#pragma unroll
  for (int e = 0; e < kHLineEq; ++e)
    if (e < E && e < c) sO[fh_hsk(s0 + e)] = fh_df_pair(fh_df_fma(al[e], S, bt[e]));
  __syncthreads();
  // ---- the new state and history entry; the ends of the line
  for (int k = t; k <= N + 1; k += T) {
    const fh_df x = k == 0   ? fh_df_fma(al0, fh_df_from_pair(sO[0]), b0)
                    : k <= n ? fh_df_from_pair(sO[fh_hsk(k - 1)])
                             : uN;
    U[o + k] = k <= n ? fh_df_to_double_bits(x) : I.u_right;
    if (Dnew) Dnew[o + k] = fh_df_pair(fh_df_sub(x, fh_df_from_pair(sU[fh_hsk(k)])));
  }
  return true;
}
