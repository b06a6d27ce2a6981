// fh_hline.cuh -- the implicit line solve of one 1D H_solver step by one CTA
// (al1, Om1, bt1, bottom Dirichlet, back substitution and history append of
// mt_psi_caputo.cpp:1262-1507 and mt_minimal.cpp:829-1031).
//
// The Thomas factors without cancellation.  The reference runs
//   Al[i+1] = B_i / (R_i - A_i Al[i]),  R_i = A_i + B_i + s_i,
// where s_i > 0 (the weight of the current time slot) is 1e-5 of R_i on a fine
// grid: Al is close to 1, and the difference R - A Al loses the digits of
// d = 1 - Al.  In d the same recurrence has no subtraction at all,
//   d_{i+1} = (A_i d_i + s_i) / (A_i d_i + B_i + s_i),
// the elimination of Grassmann, Taksar and Heyman (1985) for a matrix given by
// its off-diagonal entries and row sums.  As a Moebius map it is the matrix
// [[A, s], [A, B + s]] of non-negative entries, so products of any number of
// them, in any order of association, keep the relative accuracy of their
// factors: the serial chain becomes a scan.  s_i is the exact R - A - B of the
// rounded coefficients, so the system solved is the reference's own.  With
// al_left outside [0, 1] or negative kc or cinv the terms have either sign and the
// scan is an elimination like any other, as near to long double as the serial
// order (al_left = -0.5, 1.5, 3 and kc, cinv < 0: 2.7e-13 both).  Measured
// against a long-double elimination of the same rounded systems (160 psi
// instances, 300 steps, restated on the CPU): mean error 1.15e-13, the
// reference's order 1.38e-13; L1, N = 1000: 2.8e-13 against 4.2e-12.
//
// Why the scan: the serial order is a chain of FP64 products and divisions of
// ~650 cycles per equation on GB300, whatever the batch does beside it (one
// FP64 warp instruction per ~67 cycles and sub-partition, and the same again
// as latency).  Measured, 1000 psi instances of 64..1024 nodes: coefficients,
// serial factors and sweeps took 94 + 432 + 148 us per step in three launches;
// one launch of this form takes 114 us, the longest lines first (250-step solve
// 215 -> 79 ms with the history sums of fh_dp.cuh).  The
// FP64 pipe bounds it: ~70 FP64 instructions per equation, of which the
// exponential of K(u) and the division take half, and ~75 per warp for the
// scans.
//
// Layout: thread t owns E consecutive equations (registers); state, K(u),
// right parts and results pass through shared memory so that all global
// traffic is coalesced.  A line longer than kHLineEq equations per thread runs
// in panels, with Al and Bt of every panel kept in global memory between the
// forward and the backward pass.
#pragma once
#include "fh_common.cuh"
#include "fh_df.cuh"
#include "fh_linescan.cuh"

constexpr int kHLineEq = 8;  // equations per thread at most

struct fh_h_dev_inst {
  int N, weights, kmodel, gravity;
  int fixed;  // coefficients independent of u and of the step: factor once
  // the instance's own clock (fh_h_batch_restart): its step is tstep - tb and
  // its saved-layer count nsaved - ob; history slots below ob belong to an
  // earlier occupant and are never read
  int tb, ob;
  long long off;  // segment start in the concatenated state
  double dL, rdL, Dg, Da, tau, alpha, beta, kc, kgam, cinv, al_left, bt_left, u_right;
  // rdL = 1 / dL
  // space-fractional derivative in z (fh_h_batch_set_space_order): order
  // spg, spA = 1 - spg (0: classical second derivative), kbf = the
  // mt_psi_caputo factor kb(gamma, i-1, i, i) of A, B, R
  double spg, spA, kbf;
  // row scale of fh_hline_df.cuh: Da / (Dg kc / c) and 1 / (dL Dg / c)
  double dq, gq;
};

__device__ __forceinline__ double fh_h_K(const fh_h_dev_inst &I, double u) {
  return I.kmodel == FH_K_CONST ? I.kc : I.kc * exp(I.kgam * u);
}

// New history entry: FP64, or a (hi, lo) FP32 pair in the double-float modes.
__device__ __forceinline__ void fh_h_store_diff(double *D, long long i, double d, int dfstore) {
  if (dfstore)
    reinterpret_cast<float2 *>(D)[i] = fh_df_pair(fh_df_from_double(d));
  else
    D[i] = d;
}

// Skewed index of a staged array: threads walking chunks of up to eight
// consecutive entries stay on distinct banks.
__host__ __device__ constexpr int fh_hsk(int i) { return i + (i >> 3); }
// Doubles of one staged array (nodes of a panel and one neighbour each side).
__host__ __device__ constexpr int fh_hline_len(int threads) { return fh_hsk(threads * kHLineEq + 2) + 1; }
// Shared memory of fh_hline: K, right parts / results and the old state.
__host__ __device__ constexpr size_t fh_hline_smem(int threads) { return sizeof(double) * 3 * (size_t)fh_hline_len(threads); }

// Power-of-two rescaling to a largest entry in [1, 2) on the exponent fields
// (entries that fall below the normal range become 0).
__device__ __forceinline__ double fh_exp_shift(double x, int sh) {
  const int hi = __double2hiint(x), ex = (hi >> 20) & 0x7ff;
  if (ex == 0x7ff) return x;
  return ex + sh > 0 && ex > 0 ? __hiloint2double(hi + (sh << 20), __double2loint(x)) : 0.0;
}
__device__ __forceinline__ fh_mob fh_mob_rescale(fh_mob m) {
  const int e0 = __double2hiint(m.m00) & 0x7fffffff, e1 = __double2hiint(m.m01) & 0x7fffffff;
  const int e2 = __double2hiint(m.m10) & 0x7fffffff, e3 = __double2hiint(m.m11) & 0x7fffffff;
  const int ex = max(max(e0, e1), max(e2, e3)) >> 20;
  if (ex == 0 || ex == 0x7ff) return m;
  const int sh = 1023 - ex;
  return fh_mob{fh_exp_shift(m.m00, sh), fh_exp_shift(m.m01, sh), fh_exp_shift(m.m10, sh), fh_exp_shift(m.m11, sh)};
}

// x / y from r = RN(1 / y): the quotient corrected by its exact remainder
// (Markstein, IBM J. Res. Dev. 34, 1990), three operations.
__device__ __forceinline__ double fh_div_by(double x, double y, double r) {
  const double q = x * r;
  return fma(fma(-q, y, x), r, q);
}

// Scratch of the group scans.
template <int NW>
struct fh_hline_scan {
  fh_mob mob[NW];
  fh_aff fwd[NW], bwd[NW];
};

// Per-thread constants of the two affine scans for lines whose slopes do not
// change from step to step (fh_hline_res): entry k of thread t at
// lv[k 32 NW + t]; k = 0..4 the slope at each level of the forward scan, 5 its
// exclusive prefix, 6..11 the same of the backward scan.
constexpr int kHLineLv = 12;

// Start value of the thread's chunk under the maps of all threads before it
// (REV: after it), v at the line's first (last) one; total: v past the whole
// group's maps (only where the caller wants it).  lv: record the slopes.
template <int NW, bool REV>
__device__ __forceinline__ double fh_hl_scan(fh_aff G, double v, fh_aff *tot, double *total, double *lv) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int T = 32 * NW;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    if (lv) lv[k * T + t] = G.a;
    const double pa = REV ? __shfl_down_sync(0xffffffffu, G.a, d) : __shfl_up_sync(0xffffffffu, G.a, d);
    const double pb = REV ? __shfl_down_sync(0xffffffffu, G.b, d) : __shfl_up_sync(0xffffffffu, G.b, d);
    G = fh_aff_sel(REV ? lane + d < 32 : lane >= d, fh_aff_compose(G, fh_aff{pa, pb}), G);
  }
  if (lane == (REV ? 0 : 31)) tot[warp] = G;
  double ea = REV ? __shfl_down_sync(0xffffffffu, G.a, 1) : __shfl_up_sync(0xffffffffu, G.a, 1);
  double eb = REV ? __shfl_down_sync(0xffffffffu, G.b, 1) : __shfl_up_sync(0xffffffffu, G.b, 1);
  if (lane == (REV ? 31 : 0)) {
    ea = 1.0;
    eb = 0.0;
  }
  if (lv) lv[5 * T + t] = ea;
  fh_group_bar(1, T);
  double vw = v;
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const int k = REV ? NW - 1 - j : j;
    if (k == warp) {
      vw = v;
      if (!total) break;
    }
    v = fma(tot[k].a, v, tot[k].b);
  }
  if (total) *total = v;
  return fma(ea, vw, eb);
}

// The same for recorded slopes: only the offsets are scanned (one FP64
// operation and one shuffle per level instead of two each).
template <int NW, bool REV>
__device__ __forceinline__ double fh_hl_scan_fixed(double g, double v, fh_aff *tot, const double *lv) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  constexpr int T = 32 * NW;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    const double pb = REV ? __shfl_down_sync(0xffffffffu, g, d) : __shfl_up_sync(0xffffffffu, g, d);
    const double r = fma(lv[k * T + t], pb, g);
    g = (REV ? lane + d < 32 : lane >= d) ? r : g;
  }
  if (lane == (REV ? 0 : 31)) tot[warp].b = g;
  double eb = REV ? __shfl_down_sync(0xffffffffu, g, 1) : __shfl_up_sync(0xffffffffu, g, 1);
  if (lane == (REV ? 31 : 0)) eb = 0.0;
  fh_group_bar(1, T);
#pragma unroll
  for (int j = 0; j < NW; ++j) {
    const int k = REV ? NW - 1 - j : j;
    if (k == warp) break;
    v = fma(tot[k].a, v, tot[k].b);
  }
  return fma(lv[5 * T + t], v, eb);
}

// Shared memory of a line that stays resident over many steps (fh_hline_res):
// the three arrays of fh_hline, the newest layer difference, f, g, Al and the
// two prefix products of a constant-coefficient line, and its scan constants.
__host__ __device__ constexpr size_t fh_hline_res_smem(int threads) {
  return sizeof(double) * (9 * (size_t)fh_hline_len(threads) + (size_t)kHLineLv * threads);
}
// What fh_hline keeps there (RES): dn skewed by node.
struct fh_hline_keep {
  double *dn, *f, *g, *al, *pf, *pb, *lv;
  bool load;  // state and factors from global memory (the call's first step)
  bool last;  // state to global memory (its last)
};
struct fh_hline_no_sink {
  __device__ void operator()(int, double) const {}
};

// One step of instance I by the CTA (32 NW threads): DaW = Da wc, the weight
// of the current slot; ts(i) the history sum at node i.  fac_* (state layout):
// Al, f = g A and g of the constant-coefficient instances, written on the
// instance's first step; Al and Bt scratch of lines of several panels share
// fac_al and fac_bt.  sm: fh_hline_smem(32 NW) bytes.
// Only the CTA's first 32 NW threads call (named barrier 1).
// RES: a line of one panel whose state stays in shared memory between the
// steps of a launch (keep); a constant-coefficient line keeps its factors, the
// prefix products and the slopes of its scans there too.  The new differences
// go to keep.dn and sink(node, difference) instead of Dnew.
template <int NW, bool SPACE, bool RES, class TS, class SINK = fh_hline_no_sink>
__device__ __forceinline__ void fh_hline(const fh_h_dev_inst &I, double DaW, const TS &ts, double *__restrict__ U,
                                         double *__restrict__ fac_al, double *__restrict__ fac_bt,
                                         double *__restrict__ fac_f, double *__restrict__ fac_g, double *Dnew,
                                         bool first, int dfstore, const double *__restrict__ sV, double *sm,
                                         fh_hline_scan<NW> &sc, const fh_hline_keep &keep, const SINK &sink = SINK()) {
  constexpr int T = 32 * NW;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  double *sK = sm, *sO = sK + fh_hline_len(T), *sU = sO + fh_hline_len(T);
  const long long o = I.off;
  double *u = U + o;
  const int N = I.N, n = N - 1;
  const int npan = !RES && n > T * kHLineEq ? (n + T * kHLineEq - 1) / (T * kHLineEq) : 1;
  const int E = npan == 1 ? (n + T - 1) / T : kHLineEq;
  const bool factor = !I.fixed || first;
  const bool known = RES && I.fixed && !keep.load;  // factors and slopes in shared memory
  double *rec = RES && I.fixed && keep.load ? keep.lv : nullptr;
  double al[kHLineEq], bt[kHLineEq];        // Al[i+1], Bt[i+1] of the thread's equations
  double d0 = 1.0 - I.al_left, q0 = 1.0;    // d at the panel's first equation as d0 / q0
  double b0 = I.bt_left;                    // Bt there
  int i0 = 1, cnt = 0, c = 0;
  for (int pan = 0; pan < npan; ++pan) {
    i0 = 1 + pan * T * E;
    cnt = min(N - i0, T * E);
    if (pan > 0) fh_group_bar(1, T);
    // ---- state and K(u) of nodes i0 - 1 .. i0 + cnt
    for (int k = t; k < cnt + 2; k += T) {
      double x;
      if (!RES || keep.load) {
        x = u[i0 - 1 + k];
        sU[fh_hsk(k)] = x;
      } else {
        x = sU[fh_hsk(k)];
      }
      sK[fh_hsk(k)] = fh_h_K(I, x);
    }
    if (RES && keep.load && t == 0) sU[fh_hsk(N + 1)] = u[N + 1];
    fh_group_bar(1, T);
    // ---- right parts, in the reference's order, each operation rounded once
    for (int k = t; k < cnt; k += T) {
      const double x = sU[fh_hsk(k + 1)];
      double om = -DaW * x;
      if (SPACE || I.gravity) {
        const double Km = sK[fh_hsk(k)], Kc = sK[fh_hsk(k + 1)];
        if (SPACE && I.spA != 0.0) {  // space-fractional derivative (k_h_space_v)
          const double flux = __dsub_rn(__dmul_rn(Kc, sV[o + i0 + k]), __dmul_rn(Km, sV[o + i0 + k - 1]));
          om = __dsub_rn(-I.Dg * I.cinv * flux, DaW * x);
        }
        if (I.gravity) om = __dadd_rn(om, fh_div_by(Kc - Km, I.dL, I.rdL));
      }
      sO[fh_hsk(k)] = __dadd_rn(om, __dmul_rn(I.Da, ts(i0 + k)));
    }
    fh_group_bar(1, T);
    const int s0 = t * E;
    c = max(0, min(E, cnt - s0));
    const int i1 = i0 + s0;  // the thread's first equation
    double pf[kHLineEq];     // products of the forward slopes f = g A
    fh_aff F{1.0, 0.0};
    if (known) {
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e) {
        if (e < c) {
          const int k = fh_hsk(s0 + e);
          al[e] = keep.al[k];
          pf[e] = keep.pf[k];
          F.b = fma(keep.f[k], F.b, -(keep.g[k] * sO[k]));
          bt[e] = F.b;
        }
      }
    } else if (factor) {
      double rA[kHLineEq], rB[kHLineEq], rs[kHLineEq];
      fh_mob M{1.0, 0.0, 0.0, 1.0};
      double Km = sK[fh_hsk(s0)], Kc = sK[fh_hsk(s0 + 1)];
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e) {
        if (e < c) {
          const double Kp = sK[fh_hsk(s0 + e + 2)];
          double A = I.Dg * Km * I.cinv;
          double B = I.Dg * Kp * I.cinv;
          double R = I.cinv * (Kp + Km) * I.Dg;
          if (SPACE && I.spA != 0.0 && I.weights == FH_W_PSI) {
            A = A * I.kbf * I.spA;
            B = B * I.kbf * I.spA;
            R = R * I.kbf * I.spA;
          }
          R = __dadd_rn(R, DaW);
          const double r1 = __dsub_rn(R, A);
          const double s = __dadd_rn(__dsub_rn(r1, B), __dsub_rn(__dsub_rn(R, r1), A));  // R - A - B
          rA[e] = A;
          rB[e] = B;
          rs[e] = s;
          const double a = fma(A, M.m00, s * M.m10), b = fma(A, M.m01, s * M.m11);
          M.m10 = fma(B, M.m10, a);
          M.m11 = fma(B, M.m11, b);
          M.m00 = a;
          M.m01 = b;
          if (e == 3) M = fh_mob_rescale(M);
          Km = Kc;
          Kc = Kp;
        }
      }
      // ---- scan of the chunk maps, applied to the panel's first (d0 : q0)
      fh_mob G = fh_mob_rescale(M);
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        fh_mob p;
        p.m00 = __shfl_up_sync(0xffffffffu, G.m00, d);
        p.m01 = __shfl_up_sync(0xffffffffu, G.m01, d);
        p.m10 = __shfl_up_sync(0xffffffffu, G.m10, d);
        p.m11 = __shfl_up_sync(0xffffffffu, G.m11, d);
        const fh_mob m = fh_mob_compose(G, p);
        const bool in = lane >= d;
        G = fh_mob{in ? m.m00 : G.m00, in ? m.m01 : G.m01, in ? m.m10 : G.m10, in ? m.m11 : G.m11};
        if (d == 4 || d == 16) G = fh_mob_rescale(G);
      }
      if (lane == 31) sc.mob[warp] = G;
      fh_mob X;
      X.m00 = __shfl_up_sync(0xffffffffu, G.m00, 1);
      X.m01 = __shfl_up_sync(0xffffffffu, G.m01, 1);
      X.m10 = __shfl_up_sync(0xffffffffu, G.m10, 1);
      X.m11 = __shfl_up_sync(0xffffffffu, G.m11, 1);
      if (lane == 0) X = fh_mob{1.0, 0.0, 0.0, 1.0};
      fh_group_bar(1, T);
      double dw = d0, qw = q0;  // (d : q) at the warp's first equation
      double dl = d0, ql = q0;
#pragma unroll
      for (int k = 0; k < NW; ++k) {
        if (k == warp) {
          dw = dl;
          qw = ql;
          if (npan == 1) break;
        }
        const fh_mob W = sc.mob[k];
        const double dn = fma(W.m00, dl, W.m01 * ql), qn = fma(W.m10, dl, W.m11 * ql);
        const int ex = (__double2hiint(qn) >> 20) & 0x7ff;
        const int sh = ex > 0 && ex < 0x7ff ? 1023 - ex : 0;
        dl = fh_exp_shift(dn, sh);
        ql = sh ? fh_exp_shift(qn, sh) : qn;
      }
      if (npan > 1) {
        d0 = dl;
        q0 = ql;
      }
      double P = fma(X.m00, dw, X.m01 * qw), Q = fma(X.m10, dw, X.m11 * qw);
      // ---- the thread's factors: g = 1 / (A d + B + s) = Q_i / Q_{i+1}
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e) {
        if (e < c) {
          const double Pn = fma(rA[e], P, rs[e] * Q), Qn = fma(rB[e], Q, Pn);
          const double g = Q / Qn;
          P = Pn;
          Q = Qn;
          if (e == 3) {
            const int ex = (__double2hiint(Q) >> 20) & 0x7ff;
            const int sh = ex > 0 && ex < 0x7ff ? 1023 - ex : 0;
            P = fh_exp_shift(P, sh);
            Q = sh ? fh_exp_shift(Q, sh) : Q;
          }
          al[e] = rB[e] * g;
          const double f = g * rA[e];
          F.b = fma(f, F.b, -(g * sO[fh_hsk(s0 + e)]));
          F.a = f * F.a;
          pf[e] = F.a;
          bt[e] = F.b;
          if (I.fixed) {
            fac_al[o + i1 + e + 1] = al[e];
            fac_f[o + i1 + e] = f;
            fac_g[o + i1 + e] = g;
            if (RES) {
              const int k = fh_hsk(s0 + e);
              keep.f[k] = f;
              keep.g[k] = g;
              keep.al[k] = al[e];
              keep.pf[k] = F.a;
            }
          }
        }
      }
    } else {
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e) {
        if (e < c) {
          const double f = fac_f[o + i1 + e], g = fac_g[o + i1 + e];
          al[e] = fac_al[o + i1 + e + 1];
          F.b = fma(f, F.b, -(g * sO[fh_hsk(s0 + e)]));
          F.a = f * F.a;
          pf[e] = F.a;
          bt[e] = F.b;
          if (RES) {
            const int k = fh_hsk(s0 + e);
            keep.f[k] = f;
            keep.g[k] = g;
            keep.al[k] = al[e];
            keep.pf[k] = F.a;
          }
        }
      }
    }
    // ---- Bt: scan of the chunk maps, Bt = prefix slope * start + zero-start value
    {
      const double S = known ? fh_hl_scan_fixed<NW, false>(F.b, b0, sc.fwd, keep.lv)
                             : fh_hl_scan<NW, false>(F, b0, sc.fwd, npan > 1 ? &b0 : nullptr, rec);
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e)
        if (e < c) {
          bt[e] = fma(pf[e], S, bt[e]);
          if (npan > 1) {
            if (!I.fixed) fac_al[o + i1 + e + 1] = al[e];
            fac_bt[o + i1 + e + 1] = bt[e];
          }
        }
    }
  }
  // ---- back substitution u_i = Al[i+1] u_{i+1} + Bt[i+1], i = N-1..1, from u_N
  double un = I.u_right;
  for (int pan = npan - 1; pan >= 0; --pan) {
    if (npan > 1) {
      fh_group_bar(1, T);
      i0 = 1 + pan * T * E;
      cnt = min(N - i0, T * E);
      c = max(0, min(E, cnt - t * E));
      if (pan < npan - 1)
        for (int k = t; k < cnt + 1; k += T) sU[fh_hsk(k)] = u[i0 - 1 + k];
#pragma unroll
      for (int e = 0; e < kHLineEq; ++e)
        if (e < c) {
          al[e] = fac_al[o + i0 + t * E + e + 1];
          bt[e] = fac_bt[o + i0 + t * E + e + 1];
        }
    }
    const int s0 = t * E;
    fh_aff G{1.0, 0.0};
#pragma unroll
    for (int e = kHLineEq - 1; e >= 0; --e)
      if (e < c) {
        G.b = fma(al[e], G.b, bt[e]);
        bt[e] = G.b;
        if (known) {
          al[e] = keep.pb[fh_hsk(s0 + e)];
        } else {
          G.a = al[e] * G.a;
          al[e] = G.a;
          if (RES && I.fixed) keep.pb[fh_hsk(s0 + e)] = G.a;
        }
      }
    const double S = known ? fh_hl_scan_fixed<NW, true>(G.b, un, sc.bwd, keep.lv + 6 * T)  // u after the last equation
                           : fh_hl_scan<NW, true>(G, un, sc.bwd, npan > 1 ? &un : nullptr, rec ? rec + 6 * T : nullptr);
#pragma unroll
    for (int e = 0; e < kHLineEq; ++e)
      if (e < c) sO[fh_hsk(s0 + e)] = fma(al[e], S, bt[e]);
    fh_group_bar(1, T);
    // ---- the new state and history entry, coalesced; the ends of the line
    for (int k = t; k < cnt; k += T) {
      const double x = sO[fh_hsk(k)], dx = x - sU[fh_hsk(k + 1)];
      if (!RES || keep.last) u[i0 + k] = x;
      if (RES) {
        sU[fh_hsk(k + 1)] = x;
        keep.dn[fh_hsk(k + 1)] = dx;
        sink(i0 + k, dx);
      }
      if (Dnew) fh_h_store_diff(Dnew, o + i0 + k, dx, dfstore);
    }
    if (pan == 0 && t == 0) {
      const double x = fma(I.al_left, sO[0], I.bt_left), dx = x - sU[0];
      if (!RES || keep.last) u[0] = x;
      if (RES) {
        sU[0] = x;
        keep.dn[0] = dx;
        sink(0, dx);
      }
      if (Dnew) fh_h_store_diff(Dnew, o, dx, dfstore);
    }
  }
  if (t == T - 1) {
    const double uN = I.u_right;
    const double dN = uN - (RES ? sU[fh_hsk(N)] : u[N]), dG = uN - (RES ? sU[fh_hsk(N + 1)] : u[N + 1]);
    if (!RES || keep.last) {
      u[N] = uN;
      u[N + 1] = uN;
    }
    if (RES) {
      sU[fh_hsk(N)] = sU[fh_hsk(N + 1)] = uN;
      keep.dn[fh_hsk(N)] = dN;
      keep.dn[fh_hsk(N + 1)] = dG;
      sink(N, dN);
      sink(N + 1, dG);
    }
    if (Dnew) {
      fh_h_store_diff(Dnew, o + N, dN, dfstore);
      fh_h_store_diff(Dnew, o + N + 1, dG, dfstore);
    }
  }
}
