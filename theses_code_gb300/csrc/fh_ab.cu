// fh_ab.cu -- 1D Atangana-Baleanu convection-diffusion solve of
// MF_int_series.cpp:875-958 (solve_and_check, simple = 1): per step i
//   Rp_j = (Ii/(1-a)) C_j + f_j - (1/(1-a)) sum_{tt<=i-2} dC_tt/tau * I(i-tt)
//   A C_{j-1} + Bd C_j + Cc C_{j+1} = Rp_j, Dirichlet at both ends.
// The lag weights I(.) are computed once on the device (fh_weights_ab); the
// history stores dC_t/tau = (C^{t+1}-C^t)/tau per node.  The matrix is the same
// every step, so its elimination coefficients are built once and every step
// runs the two affine recurrences (see fh_linescan.cuh).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "fh_internal.h"
#include "fh_common.cuh"
#include "fh_linescan.cuh"
#include "fh_df.cuh"
#include "fh_cluster.cuh"
#include "fh_far64.h"

// blocked contraction helpers (fh_blocked.cu)
struct fh_blk;
fh_blk *fh_blk_new();
void fh_blk_delete(fh_blk *b);
int fh_blk_init(fh_ctx *ctx, fh_blk &b, long long P, int Kcap);
int fh_blk_convert(fh_ctx *ctx, fh_blk &b, const double *D, long long ldd, int k0, int df);
int fh_blk_toeplitz_weights(fh_ctx *ctx, fh_blk &b, const double *w, int base, int K, int mrows);
int fh_blk_gemm(fh_ctx *ctx, fh_blk &b, int K, float2 *out, long long ldo, int gbeg = 0);
long long fh_blk_ppad(const fh_blk &b);
static constexpr int kAbBlock = 128;  // steps per block: one weight row each

struct fh_ab_solver {
  fh_ctx *ctx = nullptr;
  int m = 0, max_steps = 0, step = 0, nrows = 0, max_splits = 1024;
  long long P = 0;  // m+1 rounded up to even
  double tau = 0, alpha = 0, A = 0, Bd = 0, Cc = 0;
  fh_dbuf w, ii, al, nal, den, inv, sl, pf, pb, C, D, W, part, S, src, bl, br;
  fh_graph_cache graph;
  int mode = FH_AB_FP64;
  fh_blk *blk = nullptr;  // blocked mode: bf16 slice planes of the history entries older than T0
  fh_dbuf far;            // far rows ((hi, lo) pairs) of the steps T0+1 .. T0+128
  long long ldfar = 0;
  int T0 = 0;
  // blocked mode, lines of at most 2560 nodes: all steps up to the next block
  // boundary in one launch of k_ab_resident in double-float; history entries,
  // lag weights, source rows and elimination tables as (hi, lo) FP32 pairs
  // FP64 mode, lines of at most 2049 nodes: the same in FP64, the entries
  // before the current 64-step block contracted at FP64 accuracy (f64)
  bool resident = false;
  fh_far64 *f64 = nullptr;
  double Ii = 0;          // current-step coefficient (host copy of ii)
  fh_dbuf w2, src2, tab2, dx;  // pairs: lag weights, source rows, tables sl, -al, inv, last change of C
  fh_dbuf derr;           // set when a device wait ran out
  ~fh_ab_solver() {
    if (blk) fh_blk_delete(blk);
    if (f64) fh_far64_delete(f64);
  }
};

constexpr int kAbThreads = 256;
constexpr int kAbSolveWarps = 8;  // the solve runs on eight warps (two per SM sub-partition), 8-equation chunks
constexpr int kAbSolveThreads = 32 * kAbSolveWarps;

// al[j] = Cc/(Bd - A al[j-1]), den[j] = Bd - A al[j-1], al[0] = 0 (MF_int_series.cpp:933-940).
// The matrix is fixed, so the step-independent parts of both recurrences are
// tabulated here once: inv[j] = 1/den[j], the forward slope sl[j] = -A inv[j],
// and the per-lane chunk prefix products of the forward slopes (pf) and of the
// backward slopes -al[j] (pb) in the chunking of k_ab_line.
// The pivots are a serial chain of FP64 divisions (thread 0); everything that
// follows from them runs over the threads of one CTA (1.4 -> 0.6 ms at 2048 nodes).
__global__ void __launch_bounds__(kAbSolveThreads) k_ab_factor(int m, double A, double Bd, double Cc,
                                                               double *__restrict__ al, double *__restrict__ den,
                                                               double *__restrict__ inv, double *__restrict__ sl,
                                                               double *__restrict__ pf, double *__restrict__ pb,
                                                               double *__restrict__ nal) {
  const int t = threadIdx.x;
  if (t == 0) {
    double a = 0.0;
    al[0] = 0.0;
    den[0] = 1.0;
    for (int j = 1; j <= m; ++j) {
      const double d = Bd - A * a;
      a = Cc / d;
      al[j] = a;
      den[j] = d;
    }
  }
  __syncthreads();
  for (int j = t; j <= m; j += kAbSolveThreads) {
    nal[j] = -al[j];
    if (j == 0) continue;
    inv[j] = 1.0 / den[j];
    sl[j] = -A * inv[j];
  }
  __syncthreads();
  const int ch = (m + kAbSolveThreads - 1) / kAbSolveThreads;
  double p = 1.0;
  for (int j = 1 + t * ch; j <= min(m, (t + 1) * ch); ++j) {
    p = j == 1 + t * ch ? sl[j] : p * sl[j];
    pf[j] = p;
  }
  double q = 1.0;
  const int b1 = min(m, (t + 1) * ch);
  for (int j = b1 - 1; j >= t * ch; --j) {
    q = j == b1 - 1 ? -al[j] : q * -al[j];
    pb[j] = q;
  }
}

// W[t] = w[i - (k0 + t)] for the history entries k0 + t, t < n
__global__ void k_ab_stepweights(int i, int k0, int n, const double *__restrict__ w, double *__restrict__ W) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) W[t] = w[i - k0 - t];
}

// One step of the tridiagonal solve (the line has m+1 nodes):
//   forward   bt[j] = (Rp_j - A bt[j-1]) / den_j = sl_j bt[j-1] + Rp_j inv_j
//   backward  C[j]  = bt[j] - al[j] C[j+1],  C[m] = right boundary value
// All threads stage the right parts and the tabulated coefficients into
// shared memory with coalesced loads (skewed by i / chunk so that the
// threads' chunks fall on distinct banks), kAbSolveWarps warps walk their
// threads' chunks from a zero start and add
// prefix * start value after a group scan of the chunk maps
// (fh_line_solve_prefix scheme), then all threads write C and the new history
// entry.
__global__ void __launch_bounds__(kAbThreads) k_ab_line(int m, double oma, const double *__restrict__ ii,
                                                        const double *__restrict__ alg,
                                                        const double *__restrict__ invg,
                                                        const double *__restrict__ slg,
                                                        const double *__restrict__ pfg,
                                                        const double *__restrict__ pbg,
                                                        const double *__restrict__ src,
                                                        const double *__restrict__ blp,
                                                        const double *__restrict__ brp, double *C,
                                                        const double *__restrict__ S,
                                                        const float2 *__restrict__ far, double *__restrict__ Dnew,
                                                        double tau) {
  extern __shared__ double sm[];
  const int ch = (m + kAbSolveThreads - 1) / kAbSolveThreads;
  const int Lm = m + 2 + m / ch + 1;
  double *rb = sm, *sl = rb + Lm, *pf = sl + Lm, *al = pf + Lm, *pb = al + Lm, *bt = pb + Lm, *cv = bt + Lm;
  auto sk = [ch](int j) { return j + j / ch; };
  // step constants computed once per CTA (FP64 divisions are scarce on this GPU)
  __shared__ double cst[3];
  if (threadIdx.x == 0) {
    cst[0] = ii[0] / oma;  // Ii/(1-a)
    cst[1] = 1.0 / oma;
    cst[2] = 1.0 / tau;
  }
  __syncthreads();
  const double cI = cst[0], ioma = cst[1], itau = cst[2];
  for (int j = threadIdx.x; j <= m; j += kAbThreads) {
    double r = fma(cI, C[j], src[j]);
    if (S || far) {  // MF_intF_simple returns ret/(1-a)
      double sv = S ? S[j] : 0.0;
      if (far) sv += (double)far[j].x + (double)far[j].y;
      r -= sv * ioma;
    }
    rb[sk(j)] = r * invg[j];
    sl[sk(j)] = slg[j];
    pf[sk(j)] = pfg[j];
    al[sk(j)] = alg[j];
    pb[sk(j)] = pbg[j];
  }
  __syncthreads();
  __shared__ fh_aff scan_sm[kAbSolveWarps];
  if (threadIdx.x < kAbSolveThreads) {
    const int t = threadIdx.x;
    const double bl = blp[0], br = brp[0];
    const int f0 = 1 + t * ch, f1 = min(m + 1, f0 + ch);
    double b = 0.0;
    for (int j = f0; j < f1; ++j) {
      b = fma(sl[sk(j)], b, rb[sk(j)]);
      bt[sk(j)] = b;
    }
    const fh_aff Pf =
        fh_group_exclusive_affine<kAbSolveWarps>(f1 > f0 ? fh_aff{pf[sk(f1 - 1)], b} : fh_aff{1.0, 0.0}, scan_sm, 1);
    const double s0 = fma(Pf.a, bl, Pf.b);  // bt[f0 - 1]
    for (int j = f0; j < f1; ++j) bt[sk(j)] = fma(pf[sk(j)], s0, bt[sk(j)]);
    if (t == 0) bt[sk(0)] = bl;
    fh_group_bar(1, kAbSolveThreads);
    const int b0 = t * ch, b1 = min(m, b0 + ch);
    double c = 0.0;
    for (int j = b1 - 1; j >= b0; --j) {
      c = fma(-al[sk(j)], c, bt[sk(j)]);
      cv[sk(j)] = c;
    }
    const fh_aff Pb = fh_group_exclusive_affine_rev<kAbSolveWarps>(b1 > b0 ? fh_aff{pb[sk(b0)], c} : fh_aff{1.0, 0.0},
                                                                   scan_sm, 1);
    const double tv = fma(Pb.a, br, Pb.b);  // C[b1]
    for (int j = b0; j < b1; ++j) cv[sk(j)] = fma(pb[sk(j)], tv, cv[sk(j)]);
    if (t == 0) cv[sk(m)] = br;
  }
  __syncthreads();
  for (int j = threadIdx.x; j <= m; j += kAbThreads) {
    const double v = cv[sk(j)];
    const double old = C[j];
    C[j] = v;
    if (Dnew) Dnew[j] = (v - old) * itau;
  }
}

// ------------------------------------------------ resident solve of a block
// All steps of a call up to the next block boundary in one launch of one
// cluster.  The entries older than the block (tt < T0) come as far rows from
// the tensor cores; the block's own entries are summed here.
//   CTA 0 solves the line, step after step: field, elimination tables, prefix
//     products and the slopes of both scans stay in registers and shared
//     memory.  Of the right part times 1/den it adds only what needs the last
//     step, Ii/(1-a) C and the newest entry.
//   CTAs 1 .. 15 own a range of the line's threads each and prepare the rest
//     for the nodes of those threads: source, far row and every entry of the
//     block but the newest, times 1/den.  They keep their nodes' entries in
//     shared memory, made from the field differences CTA 0 sends, and store
//     them for the block's contraction.
// Both directions are one-sided (fh_cluster.cuh): the difference of step s goes
// out when it is solved, the right parts of step s + 2 come back while CTA 0
// solves step s + 1.  Buffers alternate with the parity of the step: CTA 0
// sends the difference of step s after it has the right parts of step s, which
// their owner sent after it had read the difference of step s - 2; and an
// owner sends right parts of step s + 2 after it has the difference of step s,
// sent when CTA 0 had read the right parts of step s.  A cluster barrier before
// the first and after the last message; waits are bounded (*err on expiry).
// With one cluster barrier a step instead, reading each other's shared memory,
// 2048 nodes took 4.4-5.4 us a step, of which a 200-node line still took 2.9.
//
// The matrix is fixed, so the slopes of both substitutions are too: a thread
// owns E consecutive equations, walks them from a zero start and adds prefix
// product x start value, and the scans move offsets only (one multiply-add and
// one shuffle of a value per level).  What bounds a step is CTA 0: ~100 FP32
// instructions per equation and ~20 per scan level and warp, and their
// dependent chain.
// Arithmetic A: double-float on the FP32 pipe (blocked mode) or FP64 (fh_ab_f64).
//
struct fh_ab_df {
  using S = float2;  // stored
  using V = fh_df;   // computed with
  static __device__ __forceinline__ V ld(S s) { return fh_df_from_pair(s); }
  static __device__ __forceinline__ S st(V v) { return fh_df_pair(v); }
  static __device__ __forceinline__ V of(double x) { return fh_df_from_double(x); }
  static __device__ __forceinline__ double to(V v) { return fh_df_to_double(v); }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return fh_df_fma(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return fh_df_mul(a, b); }
  static __device__ __forceinline__ V add(V a, V b) { return fh_df_add(a, b); }
  static __device__ __forceinline__ V sub(V a, V b) { return fh_df_sub(a, b); }
  static __device__ __forceinline__ V shfl(V v, int lane) {
    return fh_df{__shfl_sync(0xffffffffu, v.h, lane), __shfl_sync(0xffffffffu, v.l, lane)};
  }
  static __device__ __forceinline__ V sel(bool c, V a, V b) { return fh_df_sel(c, a, b); }
};

// FP64 (FP64 mode).
struct fh_ab_f64 {
  using S = double;
  using V = double;
  static __device__ __forceinline__ V ld(S s) { return s; }
  static __device__ __forceinline__ S st(V v) { return v; }
  static __device__ __forceinline__ V of(double x) { return x; }
  static __device__ __forceinline__ double to(V v) { return v; }
  static __device__ __forceinline__ V fma(V a, V b, V c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ V mul(V a, V b) { return a * b; }
  static __device__ __forceinline__ V add(V a, V b) { return a + b; }
  static __device__ __forceinline__ V sub(V a, V b) { return a - b; }
  static __device__ __forceinline__ V shfl(V v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
  static __device__ __forceinline__ V sel(bool c, V a, V b) { return c ? a : b; }
};

constexpr int kAbResThreads = 512;
constexpr int kAbResMaxCtas = 16;
constexpr int kAbResMaxSteps = 128;  // entries of a block
constexpr int kAbResLv = 12;         // scan constants per thread: 5 levels and the exclusive prefix, both ways

struct fh_ab_res_args {
  int m, nrows, T0, K0, ns;    // history entries older than T0 in the far rows; steps K0 .. K0 + ns - 1
  long long P, ldfar;
  const void *sl, *nal, *inv;  // forward slopes, -al and 1/den (S per node)
  void *dx;                    // C minus C of the step before at the end of a call (S per node)
  const void *src;             // source rows (S), m + 1 per row
  const double *bl, *br;       // boundary values per row
  const void *w;               // lag weights (S)
  int *err;
  const void *far;             // far row of step T0 + r at far + r ldfar (S), null: none
  void *D;                     // entry tt at D + tt P (S)
  double *C;
  double cI, nioma, itau;      // Ii/(1-a), -1/(1-a), 1/tau
};

// Shared memory: CTA 0 the tables [6][E][T], scan constants [12][T], prepared
// right parts [2][E][T]; the others their nodes' differences [2][E][TW],
// partial sums and entries [128][E TW].
__host__ __device__ inline int ab_res_tw(int nw, int ctas) { return (32 * nw + ctas - 2) / (ctas - 1); }
static size_t ab_res_smem(int nw, int E, int ctas) {
  const int T = 32 * nw, nn = E * ab_res_tw(nw, ctas);
  const size_t line = 8 * ((size_t)8 * E * T + (size_t)kAbResLv * T);
  const size_t work = 8 * ((size_t)2 * nn + kAbResThreads + (size_t)kAbResMaxSteps * nn);
  return line > work ? line : work;
}

// Scan of the chunk maps' offsets over 32 NW threads with recorded slopes lv
// (and lw: the same for the NW warp totals, [5][32]); v: value at the line's
// first (REV: last) end; returns the value at the thread's chunk.
template <class A, int NW, bool REV>
__device__ __forceinline__ typename A::V ab_scan(typename A::V g, typename A::V v, typename A::S *tot,
                                                 const typename A::S *lv, const typename A::S *lw) {
  using V = typename A::V;
  constexpr int T = 32 * NW;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    const V p = A::shfl(g, REV ? lane + d : lane - d);
    g = A::sel(REV ? lane + d < 32 : lane >= d, A::fma(A::ld(lv[k * T + t]), p, g), g);
  }
  if (lane == (REV ? 0 : 31)) tot[warp] = A::st(g);
  V e = A::shfl(g, REV ? lane + 1 : lane - 1);
  if (lane == (REV ? 31 : 0)) e = A::of(0.0);
  fh_group_bar(1, T);
  // warp totals: lane l holds warp l's (REV: warp NW-1-l's)
  const int wl = lane < NW ? (REV ? NW - 1 - lane : lane) : 0;
  V q = A::ld(tot[wl]);
#pragma unroll
  for (int k = 0; (1 << k) < NW; ++k) {
    const int d = 1 << k;
    const V p = A::shfl(q, lane - d);
    q = A::sel(lane >= d, A::fma(A::ld(lw[k * 32 + lane]), p, q), q);
  }
  // start of this warp: the inclusive scan up to the warp before it
  const int wi = REV ? NW - 1 - warp : warp;
  const V off = A::shfl(q, wi > 0 ? wi - 1 : 0);
  if (wi > 0) v = A::fma(A::ld(lw[4 * 32 + wi - 1]), v, off);
  return A::fma(A::ld(lv[5 * T + t]), v, e);
}

// The constants of ab_scan from the chunks' slopes a (once per launch).
template <class A, int NW, bool REV>
__device__ __forceinline__ void ab_scan_setup(typename A::V a, typename A::S *tot, typename A::S *lv,
                                              typename A::S *lw) {
  using V = typename A::V;
  constexpr int T = 32 * NW;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    lv[k * T + t] = A::st(a);
    const V p = A::shfl(a, REV ? lane + d : lane - d);
    if (REV ? lane + d < 32 : lane >= d) a = A::mul(a, p);
  }
  if (lane == (REV ? 0 : 31)) tot[warp] = A::st(a);
  V e = A::shfl(a, REV ? lane + 1 : lane - 1);
  if (lane == (REV ? 31 : 0)) e = A::of(1.0);
  lv[5 * T + t] = A::st(e);
  fh_group_bar(1, T);
  if (warp == 0) {
    V q = lane < NW ? A::ld(tot[REV ? NW - 1 - lane : lane]) : A::of(1.0);
#pragma unroll
    for (int k = 0; (1 << k) < NW; ++k) {
      const int d = 1 << k;
      lw[k * 32 + lane] = A::st(q);
      const V p = A::shfl(q, lane - d);
      if (lane >= d) q = A::mul(q, p);
    }
    lw[4 * 32 + lane] = A::st(q);
  }
  fh_group_bar(1, T);
}

template <class A, int NW, int EM>
__global__ void __launch_bounds__(kAbResThreads, 1) k_ab_resident(const fh_ab_res_args a) {
  namespace cg = cooperative_groups;
  using S = typename A::S;
  using V = typename A::V;
  constexpr int T = 32 * NW;  // threads of the line solve
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double2 ab_sm2[];
  S *sm = reinterpret_cast<S *>(ab_sm2);
  __shared__ S tot[2][NW], lw[2][5 * 32], wl[kAbResMaxSteps + 2];
  __shared__ uint64_t bars[2];  // CTA 0: right parts here; the others: differences here
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank(), t = threadIdx.x;
  const int m = a.m, n = m - 1;  // equations 1 .. m - 1
  const int E = (n + T - 1) / T;
  const int TW = ab_res_tw(NW, C);
  S *D = reinterpret_cast<S *>(a.D);
  const S *w = reinterpret_cast<const S *>(a.w);
  const uint32_t bar = fh_smem_u32(bars), smb = fh_smem_u32(sm);
  if (t == 0) {
    fh_mbar_init(bar, 1);
    fh_mbar_init(bar + 8, 1);
    fh_fence_mbar_init();
  }
  bool ok = true;
  if (r == 0) {
    // forward slope, Ii/(1-a)/den, newest entry's factor, -al, prefix products
    S *tf = sm, *tc = tf + E * T, *tw = tc + E * T, *tn = tw + E * T, *pf = tn + E * T, *pb = pf + E * T;
    S *lvf = pb + E * T, *lvb = lvf + 6 * T, *rp = lvf + kAbResLv * T;  // rp: [2][E][T]
    const bool solving = t < T;  // whole warps; the others only keep the cluster barriers
    const int j0 = 1 + t * E;    // the thread's first equation
    const int c = solving ? max(0, min(E, m - j0)) : 0;
    V Cv[EM], dv[EM];  // field, its last change
    const V zero = A::of(0.0), one = A::of(1.0);
    if (solving) {
      const V cI = A::of(a.cI);
      // the newest entry, lag 2: -1/(1-a) w dC / tau
      const V cw = A::mul(A::ld(w[2]), A::of(a.nioma * a.itau));
      V pa = one;
#pragma unroll
      for (int e = 0; e < EM; ++e)
        if (e < E) {
          const bool in = e < c;
          const int q = e * T + t, j = in ? j0 + e : 0;
          const V f = in ? A::ld(reinterpret_cast<const S *>(a.sl)[j]) : zero;
          tf[q] = A::st(f);
          const V iv = in ? A::ld(reinterpret_cast<const S *>(a.inv)[j]) : zero;
          tc[q] = A::st(A::mul(cI, iv));
          tw[q] = A::st(A::mul(cw, iv));
          tn[q] = in ? reinterpret_cast<const S *>(a.nal)[j] : A::st(one);
          pa = A::mul(pa, f);
          pf[q] = A::st(pa);
          Cv[e] = in ? A::of(a.C[j]) : zero;
          dv[e] = in && a.K0 > a.T0 ? A::ld(reinterpret_cast<const S *>(a.dx)[j]) : zero;
        }
      V pq = one;
#pragma unroll
      for (int e = EM - 1; e >= 0; --e)
        if (e < E) {
          const int q = e * T + t;
          pq = A::mul(pq, A::ld(tn[q]));
          pb[q] = A::st(pq);
        }
      ab_scan_setup<A, NW, false>(pa, tot[0], lvf, lw[0]);
      ab_scan_setup<A, NW, true>(pq, tot[1], lvb, lw[1]);
    }
    V c0 = A::of(a.C[0]), cm = A::of(a.C[m]);  // the boundary nodes (thread 0 keeps them)
    const V itau = A::of(a.itau);
    int row = -1;
    V bl = zero, br = zero;
    auto load_row = [&](int K) {  // boundary values of the step with K entries
      const int nr = K < a.nrows - 1 ? K : a.nrows - 1;
      if (!solving || nr == row) return;
      row = nr;
      bl = A::of(a.bl[row]);
      br = A::of(a.br[row]);
    };
    load_row(a.K0);
    // the thread's differences in its owner's buffer
    const uint32_t own = 1 + t / TW, obar = fh_mapa(bar, own), odst = fh_mapa(smb, own) + 8 * (t % TW);
    cl.sync();
    for (int s = 0; s < a.ns; ++s) {
      const int K = a.K0 + s, par = s & 1;
      if (solving) {
        if (t == 0) fh_mbar_arrive_expect_tx(bar + 8 * par, 8 * E * T);
        ok = fh_group_and(1, T, fh_mbar_wait(bar + 8 * par, (s >> 1) & 1));
        if (!ok) break;
        V bt[EM];
        {
          const bool newest = K > a.T0;
          V v = zero;
#pragma unroll
          for (int e = 0; e < EM; ++e)
            if (e < E) {
              const int q = e * T + t;
              V x = A::fma(A::ld(tc[q]), Cv[e], A::ld(rp[par * E * T + q]));
              if (newest) x = A::fma(A::ld(tw[q]), dv[e], x);
              v = A::fma(A::ld(tf[q]), v, x);
              bt[e] = v;
            }
          const V st = ab_scan<A, NW, false>(v, bl, tot[0], lvf, lw[0]);  // bt before the thread's equations
#pragma unroll
          for (int e = 0; e < EM; ++e)
            if (e < E) bt[e] = A::fma(A::ld(pf[e * T + t]), st, bt[e]);
        }
        V v = zero;
#pragma unroll
        for (int e = EM - 1; e >= 0; --e)
          if (e < E) {
            v = A::fma(A::ld(tn[e * T + t]), v, e < c ? bt[e] : zero);
            bt[e] = v;
          }
        const V st = ab_scan<A, NW, true>(v, br, tot[1], lvb, lw[1]);  // C after the thread's equations
#pragma unroll
        for (int e = 0; e < EM; ++e)
          if (e < E) {
            const V x = A::fma(A::ld(pb[e * T + t]), st, bt[e]);
            dv[e] = A::sub(x, Cv[e]);
            if (e < c) Cv[e] = x;
            fh_st_async8(odst + 8 * (par * E + e) * TW, A::st(dv[e]), obar + 8 * par);
          }
        if (t == 0) {
          S *Dk = D + (long long)K * a.P;
          Dk[0] = A::st(A::mul(A::sub(bl, c0), itau));
          Dk[m] = A::st(A::mul(A::sub(br, cm), itau));
          c0 = bl;
          cm = br;
        }
        if (s + 1 < a.ns) load_row(K + 1);
      }
    }
    if (!ok) atomicOr(a.err, 1);
    if (solving) {
#pragma unroll
      for (int e = 0; e < EM; ++e)
        if (e < c) {
          a.C[j0 + e] = A::to(Cv[e]);
          reinterpret_cast<S *>(a.dx)[j0 + e] = A::st(dv[e]);
        }
      if (t == 0) {
        a.C[0] = A::to(c0);
        a.C[m] = A::to(cm);
      }
    }
    cl.sync();
    return;
  }
  // ---- history of the nodes of threads [t0, t0 + TW): item i = e TW + (thread - t0)
  const int t0 = (r - 1) * TW, nn = E * TW, tw = max(0, min(TW, T - t0));
  S *dxb = sm, *pt = dxb + 2 * nn, *ent = pt + kAbResThreads;
  // thread t sums run p of the block's entries for item i; run 0 also fetches,
  // stores and sends
  const int i = t % nn, p = t / nn, parts = kAbResThreads / nn;
  const int ti = t0 + i % TW, node = 1 + ti * E + i / TW;
  const bool mine = ti < T, live = mine && node < m;
  const int K0 = a.K0, T0 = a.T0;
  for (int k = t; k < kAbResMaxSteps + 2; k += kAbResThreads) wl[k] = k < K0 - T0 + a.ns + 2 ? w[k] : A::st(A::of(0.0));
  if (p < parts)
    for (int tt = p; tt < K0 - T0; tt += parts)
      ent[tt * nn + i] = live ? D[(long long)(T0 + tt) * a.P + node] : A::st(A::of(0.0));
  const V itau = A::of(a.itau);
  const V iv = live ? A::ld(reinterpret_cast<const S *>(a.inv)[node]) : A::of(0.0);
  const V ni = A::mul(A::of(a.nioma), iv);  // MF_intF_simple returns ret/(1-a)
  const uint32_t rbar = fh_mapa(bar, 0);
  const uint32_t rdst = fh_mapa(smb, 0) + 8 * ((6 * E + kAbResLv) * T + (i / TW) * T + ti);
  int row = -1;
  V sr = A::of(0.0);  // source times 1/den
  cl.sync();
  for (int s = -2; s < a.ns; ++s) {
    if (s >= 0) {  // the difference of step s: own copy and the stored history
      const int K = K0 + s;
      if (t == 0) fh_mbar_arrive_expect_tx(bar + 8 * (s & 1), 8 * E * tw);
      if (tw > 0) ok = fh_mbar_wait(bar + 8 * (s & 1), (s >> 1) & 1);
      if (p == 0) {
        S d = A::st(A::of(0.0));
        if (live) {
          d = A::st(A::mul(A::ld(dxb[(s & 1) * nn + i]), itau));
          D[(long long)K * a.P + node] = d;
        }
        ent[(K - T0) * nn + i] = d;
      }
    }
    ok = __syncthreads_and(ok);
    if (!ok) break;
    const int sn = s + 2;  // the step to prepare
    if (sn < a.ns) {
      const int K = K0 + sn, no = max(K - 1 - T0, 0);  // entries T0 .. K - 2
      const int nr = K < a.nrows - 1 ? K : a.nrows - 1;
      if (nr != row) {
        row = nr;
        if (live) sr = A::mul(A::ld(reinterpret_cast<const S *>(a.src)[(long long)row * (m + 1) + node]), iv);
      }
      const int per = (no + parts - 1) / parts;
      const int b = min(no, p * per), e = p < parts ? min(no, b + per) : b;
      V s0 = A::of(0.0), s1 = A::of(0.0);
      if (p == 0 && a.far && live) s0 = A::ld(reinterpret_cast<const S *>(a.far)[(long long)(K - T0) * a.ldfar + node]);
      int tt = b;
      for (; tt + 2 <= e; tt += 2) {  // entry tt has lag K + 1 - (T0 + tt)
        s0 = A::fma(A::ld(wl[K + 1 - T0 - tt]), A::ld(ent[tt * nn + i]), s0);
        s1 = A::fma(A::ld(wl[K - T0 - tt]), A::ld(ent[(tt + 1) * nn + i]), s1);
      }
      if (tt < e) s0 = A::fma(A::ld(wl[K + 1 - T0 - tt]), A::ld(ent[tt * nn + i]), s0);
      s0 = A::add(s0, s1);
      if (parts > 1) {
        if (p > 0 && p < parts) pt[t] = A::st(s0);
        __syncthreads();
        if (p == 0)
          for (int q = 1; q < parts; ++q) s0 = A::add(s0, A::ld(pt[q * nn + i]));
      }
      if (p == 0 && mine)
        fh_st_async8(rdst + 8 * (sn & 1) * E * T, A::st(A::fma(ni, s0, sr)), rbar + 8 * (sn & 1));
    }
  }
  if (!ok) atomicOr(a.err, 1);
  cl.sync();
}

// (hi, lo) pairs of n doubles; neg: of their negatives
__global__ void k_ab_pairs(const double *__restrict__ x, float2 *__restrict__ y, long long n, int neg) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fh_df_pair(fh_df_from_double(neg ? -x[i] : x[i]));
}

// Pair copies for the double-float launches: elimination tables (after every
// factorization), lag weights, source rows.
static int ab_pairs(fh_ctx *ctx, const double *x, float2 *y, long long n, int neg) {
  k_ab_pairs<<<(unsigned)fh_ceil_div(n, 256), 256, 0, ctx->stream>>>(x, y, n, neg);
  return fh_after_launch(ctx, "k_ab_pairs");
}
static int ab_table_pairs(fh_ab_solver *s) {
  if (!s->resident || s->mode != FH_AB_BLOCKED) return FH_OK;
  const long long n = s->m + 1;
  float2 *t = s->tab2.as<float2>();
  int rc;
  if ((rc = ab_pairs(s->ctx, s->sl.as<double>(), t, n, 0)) || (rc = ab_pairs(s->ctx, s->al.as<double>(), t + s->P, n, 1)) ||
      (rc = ab_pairs(s->ctx, s->inv.as<double>(), t + 2 * s->P, n, 0)))
    return rc;
  return FH_OK;
}
static int ab_src_pairs(fh_ab_solver *s) {
  if (!s->resident || s->mode != FH_AB_BLOCKED || s->nrows < 1) return FH_OK;
  int rc = fh_alloc(s->ctx, s->src2, sizeof(float2) * (size_t)s->nrows * (s->m + 1), false);
  if (rc) return rc;
  return ab_pairs(s->ctx, s->src.as<double>(), s->src2.as<float2>(), (long long)s->nrows * (s->m + 1), 0);
}

static size_t ab_line_smem(int m) {
  const int ch = (m + kAbSolveThreads - 1) / kAbSolveThreads;
  return sizeof(double) * 7 * (size_t)(m + 2 + m / ch + 1);
}

static int ab_res_steps(fh_ab_solver *s, int max_n, int *done);

static int ab_one_step(fh_ab_solver *s, int max_n, int *done) {
  *done = 1;
  fh_ctx *ctx = s->ctx;
  const int i = s->step + 1;  // reference step index (1-based)
  const int K = i - 1;        // history entries dC_0 .. dC_{i-2}
  const int row = (i - 1 < s->nrows - 1) ? i - 1 : s->nrows - 1;
  int rc;
  if (s->blk && K > 0 && K % kAbBlock == 0) {
    // new block: entries [K-128, K) into the slice planes, Toeplitz rows of the
    // next 128 steps, far rows S_far[r] = sum_{tt<K} w[K+1+r-tt] dC_tt
    const int dfh = s->resident ? 1 : 0;  // the resident solve stores the entries as (hi, lo) pairs
    if ((rc = fh_blk_convert(ctx, *s->blk, s->D.as<double>(), s->P, K - kAbBlock, dfh)) ||
        (rc = fh_blk_convert(ctx, *s->blk, s->D.as<double>(), s->P, K - kAbBlock / 2, dfh)))
      return rc;
    const int mrows = s->max_steps - K < kAbBlock ? s->max_steps - K : kAbBlock;
    if ((rc = fh_blk_toeplitz_weights(ctx, *s->blk, s->w.as<double>(), K + 1, K, mrows))) return rc;
    if ((rc = fh_blk_gemm(ctx, *s->blk, K, s->far.as<float2>(), s->ldfar))) return rc;
    s->T0 = K;
  }
  if (s->f64 && K > 0 && K % kF64Rows == 0) {
    // new block: the newest 64 entries join the exponents, then the rows of the
    // next 64 steps, S_far[r] = sum_{tt<K} w[K+1+r-tt] dC_tt
    const int nrows = std::min(kF64Rows, s->max_steps - K);
    if ((rc = fh_far64_append(ctx, *s->f64, s->D.p, s->P, K - 2 * kF64Block)) ||
        (rc = fh_far64_append(ctx, *s->f64, s->D.p, s->P, K - kF64Block)) ||
        (rc = fh_far64_weights_lag(ctx, *s->f64, K, s->w.as<double>(), K + 1, nrows)) ||
        (rc = fh_far64_run(ctx, *s->f64, s->D.p, s->P, K)))
      return rc;
    s->T0 = K;
  }
  if (s->resident) return ab_res_steps(s, max_n, done);
  const int k0 = s->blk ? s->T0 : 0;  // entries summed on the CUDA cores this step
  const int kn = K - k0;
  const float2 *far = (s->blk && s->T0 > 0) ? s->far.as<float2>() + (long long)(K - s->T0) * s->ldfar : nullptr;
  const double *S = nullptr;
  if (kn > 0) {
    k_ab_stepweights<<<(unsigned)fh_ceil_div(kn, 256), 256, 0, ctx->stream>>>(i, k0, kn, s->w.as<double>(),
                                                                             s->W.as<double>());
    if ((rc = fh_after_launch(ctx, "k_ab_stepweights"))) return rc;
    int splits, kchunk;
    fh_hist_plan(s->P, kn, s->max_splits, &splits, &kchunk);
    if ((rc = fh_launch_hist_sum_partials(ctx, 1, kn, s->P, s->W.as<double>(), s->max_steps + 1,
                                          s->D.as<double>() + (long long)k0 * s->P, s->P, splits, kchunk,
                                          s->part.as<double>(), s->P)))
      return rc;
    if ((rc = fh_launch_reduce_splits(ctx, splits, s->P, s->part.as<double>(), s->P, s->S.as<double>()))) return rc;
    S = s->S.as<double>();
  }
  fh_prof_mark(ctx, FH_PROF_SWEEP, false);
  k_ab_line<<<1, kAbThreads, ab_line_smem(s->m), ctx->stream>>>(
      s->m, 1.0 - s->alpha, s->ii.as<double>(), s->al.as<double>(), s->inv.as<double>(), s->sl.as<double>(),
      s->pf.as<double>(), s->pb.as<double>(), s->src.as<double>() + (long long)row * (s->m + 1),
      s->bl.as<double>() + row, s->br.as<double>() + row, s->C.as<double>(), S, far,
      s->D.as<double>() + (long long)s->step * s->P, s->tau);
  fh_prof_mark(ctx, FH_PROF_SWEEP, true);
  if ((rc = fh_after_launch(ctx, "k_ab_line"))) return rc;
  s->step++;
  return FH_OK;
}

// The block-start work of step K is already enqueued; runs up to max_n steps, to
// the end of the block at most.  Solving warps, double-float: the fewest that
// take the line at four equations a thread, sixteen (five) for the longest.
// FP64 (one warp instruction per 17 cycles and SM: fewer warps, fewer scans):
// eight equations a thread, up to 2049 nodes.
template <class F>
static auto ab_res_pick(const fh_ab_solver *s, F f) {
  const int n = s->m - 1;
  if (s->mode == FH_AB_BLOCKED) {
    if (n <= 4 * 32 * 4) return f(k_ab_resident<fh_ab_df, 4, 4>, 4, 4);
    if (n <= 8 * 32 * 4) return f(k_ab_resident<fh_ab_df, 8, 4>, 8, 4);
    return f(k_ab_resident<fh_ab_df, 16, 5>, 16, 5);
  }
  if (n <= 4 * 32 * 8) return f(k_ab_resident<fh_ab_f64, 4, 8>, 4, 8);
  return f(k_ab_resident<fh_ab_f64, 8, 8>, 8, 8);
}

static cudaLaunchConfig_t ab_res_config(cudaLaunchAttribute *at, size_t smem, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kAbResMaxCtas);
  cfg.blockDim = dim3(kAbResThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kAbResMaxCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Whether the solver's mode and line run the resident solve, on a device that
// takes its clusters (sixteen CTAs with this much shared memory); sets the
// kernel's attributes (to the kernel's largest size: solvers share them).
static bool ab_res_ok(const fh_ab_solver *s) {
  return ab_res_pick(s, [&](auto kern, int nw, int em) {
    if (s->m - 1 > 32 * nw * em) return false;
    const int smem = (int)ab_res_smem(nw, em, kAbResMaxCtas);
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = ab_res_config(at, (size_t)smem, nullptr);
    int active = 0;
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
                    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&active, kern, &cfg) == cudaSuccess && active >= 1;
    cudaGetLastError();
    return ok;
  });
}

static int ab_block(const fh_ab_solver *s) { return s->f64 ? kF64Rows : kAbBlock; }

static int ab_res_steps(fh_ab_solver *s, int max_n, int *done) {
  fh_ctx *ctx = s->ctx;
  const bool df = s->mode == FH_AB_BLOCKED;
  const int K = s->step, T0 = s->T0, ns = std::min(max_n, T0 + ab_block(s) - K);
  FH_REQUIRE(ctx, K >= T0 && ns >= 1, FH_EINVAL, "fh_ab_step: step %d outside its block at %d", K, T0);
  FH_REQUIRE(ctx, !df || s->src2.p, FH_ENOMEM, "fh_ab_step: the last source rows found no memory");
  fh_ab_res_args a;
  a.m = s->m;
  a.nrows = s->nrows;
  a.T0 = T0;
  a.K0 = K;
  a.ns = ns;
  a.P = s->P;
  const float2 *tab = s->tab2.as<float2>();
  a.sl = df ? (const void *)tab : s->sl.p;
  a.nal = df ? (const void *)(tab + s->P) : s->nal.p;
  a.inv = df ? (const void *)(tab + 2 * s->P) : s->inv.p;
  a.src = df ? s->src2.p : s->src.p;
  a.w = df ? s->w2.p : s->w.p;
  a.dx = s->dx.p;
  a.err = s->derr.as<int>();
  a.bl = s->bl.as<double>();
  a.br = s->br.as<double>();
  a.far = T0 == 0 ? nullptr : s->f64 ? fh_far64_rows(*s->f64) : s->far.p;
  a.ldfar = s->f64 ? fh_far64_pitch(*s->f64) : s->ldfar;
  a.D = s->D.p;
  a.C = s->C.as<double>();
  a.cI = s->Ii / (1.0 - s->alpha);
  a.nioma = -1.0 / (1.0 - s->alpha);
  a.itau = 1.0 / s->tau;
  fh_prof_mark(ctx, FH_PROF_SWEEP, false);
  const cudaError_t e = ab_res_pick(s, [&](auto kern, int nw, int) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg =
        ab_res_config(at, ab_res_smem(nw, (s->m - 1 + 32 * nw - 1) / (32 * nw), kAbResMaxCtas), ctx->stream);
    return cudaLaunchKernelEx(&cfg, kern, a);
  });
  fh_prof_mark(ctx, FH_PROF_SWEEP, true);
  if (e != cudaSuccess) return fh_set_error(ctx, FH_ECUDA, "k_ab_resident: %s", cudaGetErrorString(e));
  const int rc = fh_after_launch(ctx, "k_ab_resident");
  if (rc) return rc;
  s->step += ns;
  *done = ns;
  return FH_OK;
}

static int ab_res_buffers(fh_ab_solver *s);

// The resident solve's buffers and, in the FP64 mode, the contraction of older
// entries (without memory for it every step sums every entry).  Where a buffer
// fails, the solver is left to step by step solves.
static int ab_res_setup(fh_ab_solver *s) {
  const int rc = ab_res_buffers(s);
  if (rc) {
    if (s->f64) fh_far64_delete(s->f64);
    s->f64 = nullptr;
    s->resident = false;
  }
  return rc;
}
static int ab_res_buffers(fh_ab_solver *s) {
  fh_ctx *ctx = s->ctx;
  int rc;
  s->graph.reset();
  if (s->f64) fh_far64_delete(s->f64);
  s->f64 = nullptr;
  s->resident = ab_res_ok(s);
  if (s->resident && s->mode == FH_AB_FP64 && s->max_steps > kF64Rows &&
      fh_far64_create(ctx, s->P, (int)fh_ceil_div(s->max_steps, kF64Rows) * kF64Rows, false, &s->f64)) {
    s->resident = false;
    cudaGetLastError();
  }
  if (!s->resident) return FH_OK;
  if (!s->derr.p && (rc = fh_alloc(ctx, s->derr, sizeof(int)))) return rc;
  if (!s->dx.p && (rc = fh_alloc(ctx, s->dx, sizeof(double) * (size_t)s->P))) return rc;
  if (s->mode != FH_AB_BLOCKED) return FH_OK;
  if (!s->tab2.p && (rc = fh_alloc(ctx, s->tab2, sizeof(float2) * 3 * (size_t)s->P))) return rc;
  if (!s->w2.p) {
    if ((rc = fh_alloc(ctx, s->w2, sizeof(float2) * (size_t)(s->max_steps + 2)))) return rc;
    if ((rc = ab_pairs(ctx, s->w.as<double>(), s->w2.as<float2>(), s->max_steps + 2, 0))) return rc;
  }
  if ((rc = ab_table_pairs(s))) return rc;
  return ab_src_pairs(s);
}

// The error flags of the solver's device waits: cleared when a solve starts (set:
// as an expired wait leaves them, for tests).
static int ab_mark(fh_ab_solver *s, int expired) {
  if (s->derr.p) FH_CUDA_TRY(s->ctx, cudaMemsetAsync(s->derr.p, expired, sizeof(int), s->ctx->stream));
  return s->f64 ? fh_far64_mark(s->ctx, *s->f64, expired) : (int)FH_OK;
}

extern "C" {

int fh_ab_test_expire(fh_ab_solver *s) { return ab_mark(s, 1); }

int fh_ab_create(fh_ctx *ctx, int m, int max_steps, double tau, double alpha, fh_ab_solver **out) {
  FH_REQUIRE(ctx, ctx && out, FH_EINVAL, "fh_ab_create: null argument");
  *out = nullptr;
  FH_REQUIRE(ctx, m >= 2 && m <= 3500 && max_steps >= 1 && tau > 0 && alpha > 0 && alpha < 1, FH_EINVAL,
             "fh_ab_create: need 2 <= m <= 3500, max_steps >= 1, tau > 0, 0 < alpha < 1");
  {
    const size_t sm = ab_line_smem(m);
    FH_REQUIRE(ctx, sm <= 200 * 1024, FH_EINVAL, "fh_ab_create: m too large for the staged line (m <= 3500)");
    FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ab_line, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
  }
  fh_ab_solver *s = new fh_ab_solver();
  s->ctx = ctx;
  s->m = m;
  s->max_steps = max_steps;
  s->tau = tau;
  s->alpha = alpha;
  s->P = ((long long)m + 1 + 1) & ~1LL;
  const double h = 1.0 / m;
  s->A = -(1.0 / (h * h)) - (1.0 / (2.0 * h));
  s->Cc = -(1.0 / (h * h)) + (1.0 / (2.0 * h));
  int rc;
  const size_t fld = sizeof(double) * (size_t)s->P;
  if ((rc = fh_alloc(ctx, s->w, sizeof(double) * (size_t)(max_steps + 2))) || (rc = fh_alloc(ctx, s->ii, 16)) ||
      (rc = fh_alloc(ctx, s->al, fld)) || (rc = fh_alloc(ctx, s->nal, fld)) || (rc = fh_alloc(ctx, s->den, fld)) || (rc = fh_alloc(ctx, s->inv, fld)) ||
      (rc = fh_alloc(ctx, s->sl, fld)) || (rc = fh_alloc(ctx, s->pf, fld)) || (rc = fh_alloc(ctx, s->pb, fld)) ||
      (rc = fh_alloc(ctx, s->C, fld)) ||
      (rc = fh_alloc(ctx, s->D, fld * (size_t)max_steps)) ||
      (rc = fh_alloc(ctx, s->W, sizeof(double) * (size_t)(max_steps + 1))) ||
      (rc = fh_alloc(ctx, s->part, fld * (size_t)s->max_splits, false)) || (rc = fh_alloc(ctx, s->S, fld))) {
    delete s;
    return rc;
  }
  if ((rc = fh_weights_ab(ctx, max_steps + 1, tau, alpha, s->w.as<double>()))) {
    delete s;
    return rc;
  }
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->ii.p, s->w.p, sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream));
  // Bd = Ii/(1-a) + 2/h^2 with Ii from the device weights
  double ii_h = 0.0;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(&ii_h, s->w.p, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  s->Ii = ii_h;
  s->Bd = (ii_h / (1.0 - alpha)) + (2.0 / (h * h));
  k_ab_factor<<<1, kAbSolveThreads, 0, ctx->stream>>>(m, s->A, s->Bd, s->Cc, s->al.as<double>(), s->den.as<double>(),
                                        s->inv.as<double>(), s->sl.as<double>(), s->pf.as<double>(),
                                        s->pb.as<double>(), s->nal.as<double>());
  if ((rc = fh_after_launch(ctx, "k_ab_factor")) || (rc = ab_res_setup(s))) {
    delete s;
    return rc;
  }
  *out = s;
  return FH_OK;
}

int fh_ab_destroy(fh_ab_solver *s) {
  if (!s) return FH_OK;
  if (s->ctx) cudaStreamSynchronize(s->ctx->stream);
  delete s;
  return FH_OK;
}

int fh_ab_set_source_host(fh_ab_solver *s, int nrows, const double *src_host, const double *bl_host,
                          const double *br_host) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, nrows >= 1 && src_host && bl_host && br_host, FH_EINVAL, "fh_ab_set_source_host: bad args");
  int rc;
  if ((rc = fh_alloc(ctx, s->src, sizeof(double) * (size_t)nrows * (s->m + 1), false)) ||
      (rc = fh_alloc(ctx, s->bl, sizeof(double) * nrows, false)) ||
      (rc = fh_alloc(ctx, s->br, sizeof(double) * nrows, false)))
    return rc;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->src.p, src_host, sizeof(double) * (size_t)nrows * (s->m + 1),
                                   cudaMemcpyHostToDevice, ctx->stream));
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->bl.p, bl_host, sizeof(double) * nrows, cudaMemcpyHostToDevice, ctx->stream));
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->br.p, br_host, sizeof(double) * nrows, cudaMemcpyHostToDevice, ctx->stream));
  s->nrows = nrows;
  s->graph.reset();  // the rows' addresses and count are in the captured launches
  if ((rc = ab_src_pairs(s))) return rc;
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return FH_OK;
}

int fh_ab_set_c_host(fh_ab_solver *s, const double *C_host) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, C_host, FH_EINVAL, "fh_ab_set_c_host: null pointer");
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->C.p, C_host, sizeof(double) * (s->m + 1), cudaMemcpyHostToDevice, ctx->stream));
  if (int rc = ab_mark(s, 0)) return rc;
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  s->step = 0;
  s->T0 = 0;
  return FH_OK;
}

int fh_ab_set_c(fh_ab_solver *s, const double *C) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, C, FH_EINVAL, "fh_ab_set_c: null pointer");
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->C.p, C, sizeof(double) * (s->m + 1), cudaMemcpyDeviceToDevice, ctx->stream));
  if (int rc = ab_mark(s, 0)) return rc;
  s->step = 0;
  s->T0 = 0;
  return FH_OK;
}

int fh_ab_set_current_coef(fh_ab_solver *s, double Ii) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->ii.p, &Ii, sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  const double h = 1.0 / s->m;
  s->Ii = Ii;
  s->Bd = (Ii / (1.0 - s->alpha)) + (2.0 / (h * h));
  k_ab_factor<<<1, kAbSolveThreads, 0, ctx->stream>>>(s->m, s->A, s->Bd, s->Cc, s->al.as<double>(), s->den.as<double>(),
                                        s->inv.as<double>(), s->sl.as<double>(), s->pf.as<double>(),
                                        s->pb.as<double>(), s->nal.as<double>());
  s->graph.reset();  // the coefficient is an argument of the captured launches
  const int rc = fh_after_launch(ctx, "k_ab_factor");
  return rc ? rc : ab_table_pairs(s);
}

int fh_ab_set_lag_weights_host(fh_ab_solver *s, int n, const double *w_host) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, w_host && n >= 1 && n <= s->max_steps + 1, FH_EINVAL,
             "fh_ab_set_lag_weights_host: need 1 <= n <= max_steps + 1 and a table");
  FH_REQUIRE(ctx, s->step == 0, FH_EINVAL, "fh_ab_set_lag_weights_host: only before the first step");
  for (int l = 0; l < n; ++l)
    FH_REQUIRE(ctx, std::isfinite(w_host[l]), FH_ENONFINITE, "fh_ab_set_lag_weights_host: weight of lag %d", l + 1);
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(s->w.as<double>() + 1, w_host, sizeof(double) * (size_t)n, cudaMemcpyHostToDevice,
                                   ctx->stream));
  int rc;
  if (s->w2.p && (rc = ab_pairs(ctx, s->w.as<double>(), s->w2.as<float2>(), s->max_steps + 2, 0))) return rc;
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  s->graph.reset();
  return FH_OK;
}

int fh_ab_set_mode(fh_ab_solver *s, int mode) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, mode == FH_AB_FP64 || mode == FH_AB_BLOCKED, FH_EINVAL, "fh_ab_set_mode: unknown mode %d", mode);
  FH_REQUIRE(ctx, s->step == 0, FH_EINVAL, "fh_ab_set_mode: only before the first step");
  if (mode == FH_AB_BLOCKED && !s->blk && s->max_steps > kAbBlock) {
    // on failure the solver keeps its previous mode
    fh_blk *blk = fh_blk_new();
    const int kcap = (int)fh_ceil_div(s->max_steps, kAbBlock) * kAbBlock;
    int rc = fh_blk_init(ctx, *blk, s->P, kcap);
    if (rc || (rc = fh_alloc(ctx, s->far, sizeof(float2) * kAbBlock * (size_t)fh_blk_ppad(*blk), false))) {
      fh_blk_delete(blk);
      return rc;
    }
    s->ldfar = fh_blk_ppad(*blk);
    s->blk = blk;
  }
  s->mode = mode;
  if (mode == FH_AB_FP64 && s->blk) {
    fh_blk_delete(s->blk);
    s->blk = nullptr;
  }
  return ab_res_setup(s);
}

int fh_ab_step(fh_ab_solver *s, int nsteps) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, s->nrows >= 1, FH_EINVAL, "fh_ab_step: source not set");
  FH_REQUIRE(ctx, nsteps >= 0 && s->step + nsteps <= s->max_steps, FH_ENOMEM, "fh_ab_step: history full");
  if (ctx->graphs && s->step == 0 && nsteps > 1) {
    int rc = fh_graph_run(ctx, s->graph, nsteps, [&]() {
      for (int n = 0, d = 1; n < nsteps; n += d) {
        int r = ab_one_step(s, nsteps - n, &d);
        if (r) return r;
      }
      return (int)FH_OK;
    });
    if (rc) return rc;
    s->step = nsteps;
    s->T0 = s->blk || s->f64 ? ((nsteps - 1) / ab_block(s)) * ab_block(s) : 0;  // where the replayed steps left it
    return FH_OK;
  }
  for (int n = 0, d = 1; n < nsteps; n += d) {
    int rc = ab_one_step(s, nsteps - n, &d);
    if (rc) return rc;
  }
  return FH_OK;
}

int fh_ab_get_c_host(fh_ab_solver *s, double *C_host) {
  FH_REQUIRE(nullptr, s, FH_EINVAL, "null solver");
  fh_ctx *ctx = s->ctx;
  FH_REQUIRE(ctx, C_host, FH_EINVAL, "fh_ab_get_c_host: null pointer");
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(C_host, s->C.p, sizeof(double) * (s->m + 1), cudaMemcpyDeviceToHost, ctx->stream));
  int err = 0;
  if (s->derr.p) FH_CUDA_TRY(ctx, cudaMemcpyAsync(&err, s->derr.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  FH_REQUIRE(ctx, err == 0, FH_ETIMEOUT, "fh_ab_step: a wait of the resident solve ran out");
  return s->f64 ? fh_far64_check(ctx, *s->f64) : (int)FH_OK;
}

}  // extern "C"
