// fh_h.cu -- batched 1D H_solver path (mt_minimal.cpp:276-1048 and
// mt_psi_caputo.cpp:369-1507 with gamma = 1): per step
//   1. k_h_weights      per-instance history weights and current weight
//   2. k_hist_tiles     history sum per instance segment (split-K partials)
//   3. k_h_line         one CTA per instance: coefficients, right part,
//                       elimination and substitutions as scans, history
//                       append (fh_hline.cuh)
//
// All instances advance in lock step.  The concatenated state holds each
// instance's N_i+2 nodes in a segment padded to an even length; the history
// stores layer differences d_t = layer[t+1] - layer[t] at slot t for the
// concatenated state (layer-major), so the history loads coalesce across
// neighbouring nodes and instances.
#include <algorithm>
#include <cooperative_groups.h>

#include <utility>
#include <vector>

#include "fh_internal.h"
#include "fh_common.cuh"
#include "fh_linescan.cuh"
#include "fh_df.cuh"
#include "fh_slices.cuh"
#include "fh_weights.cuh"
#include "fh_hline.cuh"
#include "fh_hline_df.cuh"
#include "fh_dp.cuh"
#include "fh_cluster.cuh"

// batched far contraction on the tensor cores (fh_blocked.cu)
struct fh_hblk;
fh_hblk *fh_hblk_new();
void fh_hblk_delete(fh_hblk *b);
int fh_hblk_init(fh_ctx *ctx, fh_hblk &b, long long P, int Kcap, int ninst, const long long *tile_p0,
                 const int *tile_inst, const int *tile_np, int ntiles);
int fh_hblk_convert(fh_ctx *ctx, fh_hblk &b, const float2 *ring, long long ldd, int c);
int fh_hblk_gemm(fh_ctx *ctx, fh_hblk &b, int K, float2 *far, long long ldf);
int fh_hblk_check(fh_ctx *ctx, fh_hblk &b);
__nv_bfloat16 *fh_hblk_wplanes(fh_hblk &b);
int8_t *fh_hblk_wexp(fh_hblk &b);
int fh_hblk_kcap(const fh_hblk &b);
size_t fh_hblk_bytes(const fh_hblk &b);

struct fh_h_tile {
  int inst;
  int start;  // first node of the tile inside the segment
  int len;    // nodes in the tile (even)
};

struct fh_h_batch {
  fh_ctx *ctx = nullptr;
  int n = 0, max_steps = 0, tstep = 1, nsaved = 0, max_splits = 64, max_weights = 0;
  // history-sum launch shape (fh_h_batch_autotune): threads per tile CTA (two
  // nodes each) and the cap on K splits; one tile list per candidate shape
  int tile_threads = 256, split_cap = 64;
  std::vector<fh_h_tile> tiles_by[3];
  fh_dbuf tl_by[3];
  long long Ptot = 0;
  std::vector<fh_h_params> hp;
  std::vector<long long> off;
  fh_dbuf inst, U, D, W, Lb, ibt, lgt, wc, part, Al, Bt, fF, fG;  // fF, fG: factors of fixed instances
  fh_graph_cache graph;
  bool use_graph = true;
  int mode = FH_H_FP64;  // FH_H_DF64: history as (hi, lo) FP32 pairs; FH_H_BLOCKED: below
  bool persistent = true;  // small FP64 batches: one launch per call (k_h_persistent)
  int pers_ctas[2] = {4, 4};  // CTAs per instance there (k_h_persistent, k_h_pers_own)
  int *perr = nullptr;     // pinned: set when a wait of the persistent solve ran out
  std::vector<fh_h_dev_inst> di;  // host copy of inst
  std::vector<int> cap;           // nodes a restarted occupant of each instance may have (segment - 2)
  // space-fractional instances: Toeplitz weights wsp and the sums sV per
  // node (state layout), shared memory of k_h_space_v
  bool space = false;
  size_t space_smem = 0;
  fh_dbuf wsp, sV;
  // weights of the next step on hs (h_one_step): two buffer pairs of W and
  // wc, selected by the parity of the step; w_ready = step whose weights
  // are pending on hs behind ev_w
  cudaStream_t hs = nullptr;
  cudaEvent_t ev_main = nullptr, ev_w = nullptr;
  int w_ready = -1;
  // FH_H_BLOCKED: history slots older than the current 64-step block in bf16
  // slice planes (hb), contracted once per block for its 64 steps into far
  // rows; the slots of the last two chunks as (hi, lo) pairs in a 128-layer
  // ring (slot t in row t mod 128)
  fh_hblk *hb = nullptr;
  fh_dbuf ring, far, cheb;  // cheb: interpolation tables of k_hb_wcheb
  fh_dbuf ord;              // instances by falling N
  fh_dbuf wb, wcb;          // the block's near and current weights (k_h_weights_block)
  long long lined = -1;     // ctx->launches after the last k_h_line_df of this call
  int max_n = 0;            // the longest instance's N
  bool has_l1 = false;      // some instance has L1 weights (k_hb_weights covers every group)
  double *Wp(int par) const { return W.as<double>() + (long long)par * n * max_weights; }
  double *wcp(int par) const { return wc.as<double>() + (long long)par * n; }
  ~fh_h_batch() {
    if (hb) fh_hblk_delete(hb);
    if (hs) cudaStreamDestroy(hs);
    if (ev_main) cudaEventDestroy(ev_main);
    if (ev_w) cudaEventDestroy(ev_w);
    if (perr) cudaFreeHost(perr);
  }
};

static constexpr int kTileThreads = 512;  // largest tile CTA (1024 nodes)
static constexpr int kTileShapes[3] = {128, 256, 512};  // candidate tile CTAs
static inline int tile_shape_index(int threads) { return threads == 128 ? 0 : threads == 256 ? 1 : 2; }
static constexpr int kLineCtaMaxInst = 152;  // batches below this many instances: eight warps per line, weights ahead on the side stream
static constexpr int kSpaceMaxN = 2048;  // nodes of a space-fractional instance (shared-memory sums)
static constexpr int kHWeightThreads = 128;                 // slots per weights CTA
// per psi instance: Lc[kIbTerms] | Uc[kIbTerms] | B(a, b) | kIbLowMax^(1/beta) |
// log tau | 1/beta
static constexpr int kIbStride = 2 * kIbTerms + 4;

// ------------------------------------------------------------------ kernels

// Row b of W: the weights of instance b for the history slots t = 0..os-2,
// and wc[b], the weight of the current slot [tstep, tstep + 1].  The
// reference's t = 0 term multiplies layer1 - layer1 (its layer pointer starts
// at old[1], mt_minimal.cpp:913-917), so slot 0 carries weight 0.
// Thread i of CTA (x, b) owns slot i = x*128 + threadIdx.x; i = max(os - 1, 0)
// is the current slot.
// Weight of slot i of instance b at its step tstep with os saved layers
// (cur: the current slot's weight, the factor of the newest difference);
// invX = 1 / (tstep + 1).  The arithmetic of every weight kind as described
// at k_h_weights.
__device__ __forceinline__ double h_slot_weight(const fh_h_dev_inst &I, int b, int i, bool cur, int tstep, int os,
                                                double invX, int ldw, const double *__restrict__ Lb,
                                                const double *__restrict__ ibt, const double2 *__restrict__ lgt) {
  if (I.weights == FH_W_PSI && I.beta != 1.0) {
    // psi = t^beta: the interval [x0, x0 + 1] in the divided-difference form of
    // fh_ib_diff, with the per-instance series tables and the logs as
    // double-doubles from the table of log(x)
    if (i == 0 && !cur) return 0.0;
    const double *Lc = ibt + (long long)b * kIbStride, *Uc = Lc + kIbTerms;
    const int X = tstep + 1, x0 = cur ? tstep : i, x1 = x0 + 1;
    // p - q as a double-double for log values 0 <= p <= q (fast two-sum)
    auto dd_sub = [](double2 p, double2 q, double &h, double &l) {
      h = p.x - q.x;
      l = (p.x - (h + q.x)) + (p.y - q.y);
    };
    const double2 lX = lgt[X], l0 = lgt[x0], l1 = lgt[x1];
    fh_ib_slot q;
    q.zero0 = x0 == 0;
    q.top = x1 == X;
    q.r0 = (double)x0 * invX;
    q.r1 = (double)x1 * invX;
    q.dr = invX;
    dd_sub(l1, lX, q.l1h, q.l1l);  // log(x1/X)
    dd_sub(l0, lX, q.l0h, q.l0l);  // log(x0/X)
    dd_sub(l0, l1, q.ldh, q.ldl);  // log(x0/x1) = -log(x1/x0)
    q.ldh = -q.ldh;
    q.ldl = -q.ldl;
    const double bb = 1.0 - I.alpha;
    const double diff = fh_ib_diff(q, I.beta, bb, Lc[2 * kIbTerms + 1], [&] { return Lc[2 * kIbTerms]; },
                                   fh_ib_coef_tab{Lc}, fh_ib_coef_tab{Uc});
    // (X tau)^(1 - alpha beta) / beta with log X from the table: one exp
    const double sc = exp((1.0 - I.alpha * I.beta) * (lX.x + Lc[2 * kIbTerms + 2])) * Lc[2 * kIbTerms + 3];
    return sc * diff * (1 - I.alpha);
  }
  if (cur)
    return (I.weights == FH_W_L1)
               ? 1.0
               : fh_psi_int_t((double)tstep, (double)tstep + 1.0, (double)(tstep + 1), I.tau, I.alpha) *
                     (1 - I.alpha);
  const int t = i;
  if (t == 0) return 0.0;
  if (I.weights == FH_W_L1) return Lb[(long long)b * ldw + (os - t - 1)];  // L1 weights depend on the lag only
  return fh_psi_int_t((double)t, (double)t + 1.0, (double)(tstep + 1), I.tau, I.alpha) * (1 - I.alpha);
}

__global__ void k_h_weights(const fh_h_dev_inst *__restrict__ inst, int n, int tstep_g, int os_g,
                            double *__restrict__ W_g, int ldw, double *__restrict__ wc, const double *__restrict__ Lb,
                            const double *__restrict__ ibt, const double2 *__restrict__ lgt, double invX_g) {
  const int b = blockIdx.y;
  const fh_h_dev_inst I = inst[b];
  // the instance's own step and slot numbers; its slot i is column I.ob + i
  const int tstep = tstep_g - I.tb, os = os_g - I.ob;
  double *W = W_g + I.ob;
  const double invX = I.tb == 0 ? invX_g : 1.0 / (double)(tstep + 1);
  const int i = blockIdx.x * kHWeightThreads + threadIdx.x;
  const int nh = os > 1 ? os - 1 : 0;  // history slots
  if (i > nh) return;
  const bool cur = i == nh;
  const double w = h_slot_weight(I, b, i, cur, tstep, os, invX, ldw, Lb, ibt, lgt);
  if (cur)
    wc[b] = w;
  else
    W[(long long)b * ldw + i] = w;
}

// Blocked mode: the near weights of every step of the block whose older slots
// are [0, K0), in one launch (2145 weights per instance; a launch per step held
// at most 64 and took 19 us of its latency).  Row q is step os_first + q,
// os_first = K0 + 1, or 0 in the first block, whose steps 0 and 1 both have no
// slot: its history slots from K0 at wb[inst][q][.], its current weight at
// wcb[q][inst].
constexpr int kNearRows = 65, kNearLd = 64;
__global__ void __launch_bounds__(kHWeightThreads) k_h_weights_block(
    const fh_h_dev_inst *__restrict__ inst, int n, int K0, int max_steps, double *__restrict__ wb,
    double *__restrict__ wcb, const double *__restrict__ Lb, int ldw, const double *__restrict__ ibt,
    const double2 *__restrict__ lgt) {
  const int b = blockIdx.y, x = blockIdx.x * kHWeightThreads + threadIdx.x;
  int q = (int)((sqrtf(8.0f * x + 1.0f) - 1.0f) * 0.5f);  // x = q (q + 1) / 2 + r, r <= q
  if (q * (q + 1) / 2 > x) --q;
  if ((q + 1) * (q + 2) / 2 <= x) ++q;
  const int r = x - q * (q + 1) / 2, os = (K0 > 0 ? K0 + 1 : 0) + q, K = max(os - 1, 0);
  if (q >= kNearRows || os >= max_steps || K - K0 >= kNearLd || r > K - K0) return;
  const fh_h_dev_inst I = inst[b];
  const int tstep = os + 1;
  const bool cur = r == K - K0;
  const double w = h_slot_weight(I, b, K0 + r, cur, tstep, os, 1.0 / (double)(tstep + 1), ldw, Lb, ibt, lgt);
  if (cur)
    wcb[(long long)q * n + b] = w;
  else
    wb[((long long)b * kNearRows + q) * kNearLd + r] = w;
}

// Incomplete-beta series coefficients of every psi instance (fh_ib_tables).
__global__ void k_h_ibtab(const fh_h_dev_inst *__restrict__ inst, int n, double *__restrict__ ibt) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= n) return;
  const fh_h_dev_inst I = inst[b];
  if (I.weights != FH_W_PSI) return;
  const double a = 1.0 / I.beta, bb = 1.0 - I.alpha;
  double *row = ibt + (long long)b * kIbStride;
  fh_ib_tables(a, bb, row, row + kIbTerms);
  row[2 * kIbTerms] = exp(lgamma(a) + lgamma(bb) - lgamma(a + bb));  // B(a, b)
  row[2 * kIbTerms + 1] = pow(kIbLowMax, a);                         // y <= kIbLowMax <=> x/X <= this
  row[2 * kIbTerms + 2] = log(I.tau);
  row[2 * kIbTerms + 3] = a;                                          // 1/beta
}

// Segments of instances first .. first + gridDim.x - 1 of the state to (get) or
// from their packed order, one CTA each.  A copy per instance costs ~5 us: 1000
// psi instances over 250 steps 96.8 -> 87.0 ms, 32 of them 6.59 -> 6.27 ms; below
// four a launch costs as much as the copies.
constexpr int kHPackMin = 4;
__global__ void k_h_pack(const fh_h_dev_inst *__restrict__ inst, int first, double *U, double *packed, bool get) {
  __shared__ long long part[8];
  long long o = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += 256) o += inst[first + k].N + 2;
  for (int d = 16; d > 0; d >>= 1) o += __shfl_xor_sync(0xffffffffu, o, d);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = o;
  __syncthreads();
  o = 0;
  for (int k = 0; k < 8; ++k) o += part[k];
  const fh_h_dev_inst &I = inst[first + blockIdx.x];
  double *u = U + I.off;
  for (int k = threadIdx.x; k < I.N + 2; k += 256) {
    if (get)
      packed[o + k] = u[k];
    else
      u[k] = packed[o + k];
  }
}

// Lag table of the L1 instances: Lb[b][l] = (l+1)^(1-a) - l^(1-a) (mt_minimal.cpp:930),
// the weight of the layer difference l steps back.
__global__ void k_h_lagtab(const fh_h_dev_inst *__restrict__ inst, int nlag, double *__restrict__ Lb, int ldw) {
  const int b = blockIdx.y;
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  const fh_h_dev_inst I = inst[b];
  if (I.weights != FH_W_L1 || l >= nlag) return;
  Lb[(long long)b * ldw + l] = pow((double)(l + 1), 1.0 - I.alpha) - pow((double)l, 1.0 - I.alpha);
}

// part[s][p] = sum_{k in split s} W[inst][k] * D[k][p] over one tile of one instance.
__global__ void __launch_bounds__(kTileThreads) k_hist_tiles(const fh_h_tile *__restrict__ tiles,
                                                             const fh_h_dev_inst *__restrict__ inst,
                                                             const double *__restrict__ D, long long ldd, int K,
                                                             const double *__restrict__ W, int ldw, int kchunk,
                                                             double *__restrict__ part, long long ldpart) {
  extern __shared__ double ws[];
  const fh_h_tile T = tiles[blockIdx.x];
  const int s = blockIdx.y;
  const int k0 = s * kchunk;
  const int nk = min(K, k0 + kchunk) - k0;
  const double *wrow = W + (long long)T.inst * ldw + k0;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) ws[i] = wrow[i];
  __syncthreads();
  const int q = threadIdx.x * 2;
  if (q >= T.len) return;
  const fh_h_dev_inst &I = inst[T.inst];
  const long long p = I.off + T.start + q;
  double a0 = 0.0, a1 = 0.0;
  int k = max(0, I.ob - k0);  // slots of the instance's current occupant only
  const double *d = D + (long long)(k0 + k) * ldd + p;
  for (; k + 4 <= nk; k += 4) {
    const double2 v0 = fh_ld_stream2(d), v1 = fh_ld_stream2(d + ldd);
    const double2 v2 = fh_ld_stream2(d + 2 * ldd), v3 = fh_ld_stream2(d + 3 * ldd);
    d += 4 * ldd;
    a0 = fma(ws[k], v0.x, a0);
    a1 = fma(ws[k], v0.y, a1);
    a0 = fma(ws[k + 1], v1.x, a0);
    a1 = fma(ws[k + 1], v1.y, a1);
    a0 = fma(ws[k + 2], v2.x, a0);
    a1 = fma(ws[k + 2], v2.y, a1);
    a0 = fma(ws[k + 3], v3.x, a0);
    a1 = fma(ws[k + 3], v3.y, a1);
  }
  for (; k < nk; ++k) {
    const double2 v = fh_ld_stream2(d);
    d += ldd;
    a0 = fma(ws[k], v.x, a0);
    a1 = fma(ws[k], v.y, a1);
  }
  double2 o;
  o.x = a0;
  o.y = a1;
  *reinterpret_cast<double2 *>(part + (long long)s * ldpart + p) = o;
}

// The same for kDpMin layers and more (fh_dp.cuh): half a 256-node tile per CTA.
__global__ void __launch_bounds__(kDpThreads, 6) k_hist_tiles_dp(const fh_h_tile *__restrict__ tiles,
                                                                 const fh_h_dev_inst *__restrict__ inst,
                                                                 const double *__restrict__ D, long long ldd, int K,
                                                                 const double *__restrict__ W, int ldw, int kchunk,
                                                                 double *__restrict__ part, long long ldpart) {
  const fh_h_tile T = tiles[blockIdx.x >> 1];
  const int q = ((int)blockIdx.x & 1) * kDpThreads + threadIdx.x, s = blockIdx.y, k0 = s * kchunk;
  if (((int)blockIdx.x & 1) * kDpThreads >= T.len) return;  // whole CTA
  const fh_h_dev_inst &I = inst[T.inst];
  const long long p = I.off + T.start + q;
  double acc[1] = {};
  dp_sum<1>(D + (long long)k0 * ldd + p, ldd, max(0, I.ob - k0), min(K, k0 + kchunk) - k0,
            W + (long long)T.inst * ldw + k0, ldw, q < T.len, acc);
  if (q < T.len) part[(long long)s * ldpart + p] = acc[0];
}

// Double-float history ((hi, lo) FP32 pairs): the same tile sum with the
// weights split into pairs in shared memory and the sums carried in
// double-float on the FP32 pipe (2^-48 storage precision, HBM-bound).
__global__ void __launch_bounds__(kTileThreads) k_hist_tiles_df(const fh_h_tile *__restrict__ tiles,
                                                                const fh_h_dev_inst *__restrict__ inst,
                                                                const float2 *__restrict__ D, long long ldd, int K,
                                                                const double *__restrict__ W, int ldw, int kchunk,
                                                                double *__restrict__ part, long long ldpart) {
  extern __shared__ float2 wsf2[];
  const fh_h_tile T = tiles[blockIdx.x];
  const int s = blockIdx.y;
  const int k0 = s * kchunk;
  const int nk = min(K, k0 + kchunk) - k0;
  const double *wrow = W + (long long)T.inst * ldw + k0;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) wsf2[i] = fh_df_pair(fh_df_from_double(wrow[i]));
  __syncthreads();
  const int q = threadIdx.x * 2;
  if (q >= T.len) return;
  const fh_h_dev_inst &I = inst[T.inst];
  const long long p = I.off + T.start + q;
  fh_df a0{0.f, 0.f}, a1{0.f, 0.f};
  int k = max(0, I.ob - k0);  // slots of the instance's current occupant only
  const float4 *d = reinterpret_cast<const float4 *>(D + (long long)(k0 + k) * ldd + p);
  const long long ld4 = ldd / 2;
  for (; k + 4 <= nk; k += 4) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldcs(d + u * ld4);
    d += 4 * ld4;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const fh_df w = fh_df_from_pair(wsf2[k + u]);
      a0 = fh_df_fma(w, fh_df{v[u].x, v[u].y}, a0);
      a1 = fh_df_fma(w, fh_df{v[u].z, v[u].w}, a1);
    }
  }
  for (; k < nk; ++k) {
    const float4 v = __ldcs(d);
    d += ld4;
    const fh_df w = fh_df_from_pair(wsf2[k]);
    a0 = fh_df_fma(w, fh_df{v.x, v.y}, a0);
    a1 = fh_df_fma(w, fh_df{v.z, v.w}, a1);
  }
  double2 o;
  o.x = fh_df_to_double(a0);
  o.y = fh_df_to_double(a1);
  *reinterpret_cast<double2 *>(part + (long long)s * ldpart + p) = o;
}

// Space-fractional Caputo derivative in z (gamma < 1): H_solver::Om1 adds
// -Dg/(dw/dh) (K_i V_i - K_{i-1} V_{i-1}) with V_i = sum_{j<i} w_{i-j} F_j over
// the first differences F_j = u_{j+1} - u_j of the current state
// (calc_v, mt_minimal.cpp:228-271, mt_psi_caputo.cpp:749-777, with_zero 1).
// The weights depend on i - j only: mt_minimal (m+1)^A - m^A, mt_psi_caputo
// A kb_space of one interval at distance m+1 (1461-1472; psi = x in space;
// the reference tabulates kb_space[i][j-1], equal up to rounding).
// wsp[off + m], m = 1..N-1, per instance.
__global__ void k_h_spw(const fh_h_dev_inst *__restrict__ inst, double *__restrict__ wsp) {
  const fh_h_dev_inst I = inst[blockIdx.y];
  if (I.spA == 0.0) return;
  for (int m = 1 + blockIdx.x * blockDim.x + threadIdx.x; m < I.N; m += gridDim.x * blockDim.x)
    wsp[I.off + m] = I.weights == FH_W_L1
                         ? pow((double)m + 1, I.spA) - pow((double)m, I.spA)
                         : I.spA * fh_psi_int_t(0.0, 1.0, (double)m + 1.0, I.dL, I.spg);
}

// V_i of one instance per CTA (F and the weights in shared memory), i =
// 1..N-1; V_0 = 0.  O(N^2) FP64 FMAs per instance and step, as the reference
// (FP64-pipe-bound; a double-float form on the FP32 pipe ran 3.4x faster but
// the flux difference K_i V_i - K_{i-1} V_{i-1} amplified its 2^-48 products
// to 1e-10 of the solution at N ~ 1000).  Rows go to threads in snake order
// (t, 2T-1-t, 2T+t, ...) so that every thread sums about as many terms.
__global__ void __launch_bounds__(256) k_h_space_v(const fh_h_dev_inst *__restrict__ inst, const double *__restrict__ U,
                                                   const double *__restrict__ wsp, double *__restrict__ V) {
  extern __shared__ double spm[];
  const fh_h_dev_inst I = inst[blockIdx.x];
  if (I.spA == 0.0) return;
  const int N = I.N;
  const double *u = U + I.off;
  double *F = spm, *w = spm + N;
  for (int j = threadIdx.x; j < N; j += blockDim.x) {
    F[j] = u[j + 1] - u[j];
    w[j] = wsp[I.off + j];
  }
  __syncthreads();
  const int T = blockDim.x;
  for (int r = 0; r * T < N - 1; ++r) {
    const int i = 1 + r * T + ((r & 1) ? T - 1 - (int)threadIdx.x : (int)threadIdx.x);
    if (i >= N) continue;
    double v = 0.0;
    for (int j = 0; j < i; ++j) v = fma(w[i - j], F[j], v);
    V[I.off + i] = v;
  }
  if (threadIdx.x == 0) V[I.off] = 0.0;
}

// The line solves of one step (fh_hline), one CTA of NW warps per instance.
// Four warps at 152 instances or more, where the FP64 pipe is shared by
// several CTAs per SM and fewer, longer chunks cost less in scans; eight
// below, where each instance has an SM to itself.  CTA x solves instance
// ord[x], the longest first, so that no long line starts in the last wave.
template <int NW, bool SPACE>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 3 : 1) k_h_line(
    const fh_h_dev_inst *__restrict__ inst, double *__restrict__ U, const double *__restrict__ wc,
    const double *__restrict__ part, long long ldpart, int splits, double *__restrict__ Al, double *__restrict__ Bt,
    double *__restrict__ fF, double *__restrict__ fG, double *__restrict__ Dnew, int os, int dfstore,
    const double *__restrict__ sV, const int *__restrict__ ord) {
  extern __shared__ double hsm[];
  __shared__ fh_hline_scan<NW> sc;
  const int b = ord[blockIdx.x];
  const fh_h_dev_inst I = inst[b];
  const double *pp = part + I.off;
  auto ts = [&](int i) {  // split order
    double a = 0.0;
    for (int s = 0; s < splits; ++s) a += pp[(long long)s * ldpart + i];
    return a;
  };
  fh_hline<NW, SPACE, false>(I, I.Da * wc[b], ts, U, Al, Bt, fF, fG, Dnew, os == I.ob, dfstore, sV, hsm, sc,
                             fh_hline_keep{});
}
static constexpr int kLineWarps = 4, kLineWarpsSmall = 8;

// The same in double-float, for the blocked mode: history sums and the new
// layer as pairs.  A line out of its range runs the FP64 solve (its factors
// are never kept here, so it always makes them).
template <int NW>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 4 : 2) k_h_line_df(
    const fh_h_dev_inst *__restrict__ inst, double *U, const double *__restrict__ wc, const float2 *part,
    double *__restrict__ Al, double *__restrict__ Bt, double *__restrict__ fF,
    double *__restrict__ fG, float2 *__restrict__ Dnew, const int *__restrict__ ord) {
  fh_grid_wait_prev();
  fh_grid_start_next();  // the next step's near sums: after the wait, see k_h_near_df
  extern __shared__ double hsm[];
  __shared__ union {
    fh_hline_df_scan<NW> d;
    fh_hline_scan<NW> f;
  } sc;
  const int b = ord[blockIdx.x];
  const fh_h_dev_inst I = inst[b];
  if (fh_hline_df<NW>(I, wc[b], part, U, Dnew, reinterpret_cast<float2 *>(hsm), sc.d)) return;
  __syncthreads();
  const float2 *pp = part + I.off;
  fh_hline<NW, false, false>(I, I.Da * wc[b], [&](int i) { return fh_df_to_double(fh_df_from_pair(pp[i])); }, U,
                             Al, Bt, fF, fG, reinterpret_cast<double *>(Dnew), true, 1, nullptr, hsm, sc.f,
                             fh_hline_keep{});
}

// ------------------------------------------- persistent solves of small batches
// Batches of few instances run all the steps of a call in one launch: one
// cluster of C CTAs per instance.  CTA 0 solves the line of step s (fh_hline,
// state, newest layer and constant factors resident in shared memory) while
// CTAs 1 .. C - 1 prepare step s + 1: everything in it that does not depend on
// step s, that is all its weights (they depend on the step number only) and
// the sums over all its history slots but the newest, each CTA its share of
// the slots for all nodes.  CTA 0 reads those partial sums, the newest slot's
// weight and the current slot's through distributed shared memory, adds them
// in rank order and the newest layer last.  One hardware cluster barrier per
// step publishes the new layer and the partial sums (double-buffered by the
// parity of the step); the instances are independent, and every CTA of a
// cluster reaches the barrier the same number of times.
// The sums of a step are split by its slot count alone, so a solve does not
// depend on how its steps are spread over calls.
// Measured against the form that summed and solved one after the other (two
// barriers a step, eight CTAs for any batch, serial factors): one L1 instance
// of N = 200 over 1000 steps 13.6 -> 6.6 ms, 32 psi instances of N = 512 over
// 250 steps 60.8 -> 8.3 ms.
constexpr int kPersThreads = 32 * kLineWarpsSmall;
constexpr int kPersMaxNodes = 2048;  // nodes of an instance (N + 2) in the partial sums
constexpr int kPersMaxInst = 32;     // larger batches step kernel by kernel
constexpr int kPersMaxSteps = 30400;
constexpr int kPersStage = 1024;     // slots of a CTA whose weights are staged at a time
constexpr int kPersMaxCtas = 16;
constexpr int kPersNodes = kPersMaxNodes / kPersThreads;  // nodes per thread at most
// dynamic shared memory: CTA 0 the resident line, the others the partial sums
// of two steps and the staged weights; all of them the two weights of a step
constexpr size_t kPersSmem = fh_hline_res_smem(kPersThreads) > sizeof(double) * (2 * kPersMaxNodes + kPersStage)
                                 ? fh_hline_res_smem(kPersThreads)
                                 : sizeof(double) * (2 * kPersMaxNodes + kPersStage);

// Phase stamps of the persistent solve for profiling builds (-DFH_H_STAMPS):
// %clock64 of CTA 0 (phases 0, 1) and CTA 1 (2, 3) at the start and the end of
// their part of the first 1024 steps of instance 0, read with
// fh_h_stamps_read.  Empty otherwise.
#ifdef FH_H_STAMPS
__device__ long long g_h_stamps[1024 * 8];
#define H_STAMP(p)                                                              \
  if (b == 0 && threadIdx.x == 0 && s >= 0 && s < 1024) g_h_stamps[s * 8 + (p)] = clock64();
extern "C" int fh_h_stamps_read(long long *h) {
  return (int)cudaMemcpyFromSymbol(h, g_h_stamps, sizeof(g_h_stamps));
}
#else
#define H_STAMP(p)
#endif

__global__ void __launch_bounds__(kPersThreads, 1)
    k_h_persistent(const fh_h_dev_inst *__restrict__ inst, int tstep0, int os0, int nsteps, double *D, long long ldd,
                   int ldw, const double *__restrict__ Lb, const double *__restrict__ ibt,
                   const double2 *__restrict__ lgt, double *U, double *Al, double *Bt, double *fF, double *fG) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double psm[];
  __shared__ fh_hline_scan<kLineWarpsSmall> sc;
  __shared__ double wstep[2][2];  // newest slot's and current slot's weight of a step (rank C - 1)
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank();
  const int b = blockIdx.x / C, t = threadIdx.x;
  const fh_h_dev_inst I = inst[b];
  const int np = I.N + 2;
  // history slots of the occupant before the newest one, at step s of the call
  auto older = [&](int s) { return max(os0 + s - I.ob - 2, 0); };
  if (r == 0) {
    constexpr int L = fh_hline_len(kPersThreads);
    fh_hline_keep keep;
    keep.dn = psm + 3 * L;
    keep.f = psm + 4 * L;
    keep.g = psm + 5 * L;
    keep.al = psm + 6 * L;
    keep.pf = psm + 7 * L;
    keep.pb = psm + 8 * L;
    keep.lv = psm + 9 * L;
    {  // the newest layer before the call
      const bool has = os0 - I.ob >= 2;
      const double *d = D + (long long)(has ? os0 - 2 : 0) * ldd + I.off;
      for (int p = t; p < np; p += kPersThreads) keep.dn[fh_hsk(p)] = has ? __ldcg(d + p) : 0.0;
    }
    cl.sync();  // step 0 is prepared
    for (int s = 0; s < nsteps; ++s) {
      H_STAMP(0);
      const int os_g = os0 + s, os = os_g - I.ob, par = s & 1;
      const double *ws = cl.map_shared_rank(&wstep[par][0], C - 1);
      const double wnew = ws[0], DaW = I.Da * ws[1];
      const double *pq = psm + par * kPersMaxNodes;
      auto ts = [&](int i) {
        double a = 0.0;
        if (os >= 2) {
          double v[kPersMaxCtas - 1];
#pragma unroll
          for (int q = 0; q < kPersMaxCtas - 1; ++q) v[q] = q + 1 < C ? cl.map_shared_rank(pq, q + 1)[i] : 0.0;
          // pairwise in a fixed order
          a = (v[0] + v[1]) + v[2];
          if (C > 4) a = a + ((v[3] + v[4]) + (v[5] + v[6]));
          if (C > 8) a = a + (((v[7] + v[8]) + (v[9] + v[10])) + ((v[11] + v[12]) + (v[13] + v[14])));
          a = fma(wnew, keep.dn[fh_hsk(i)], a);
        }
        return a;
      };
      keep.load = s == 0;
      keep.last = s == nsteps - 1;
      fh_hline<kLineWarpsSmall, false, true>(I, DaW, ts, U, Al, Bt, fF, fG,
                                             os_g >= 1 ? D + (long long)(os_g - 1) * ldd : nullptr, os == 0, 0, nullptr,
                                             psm, sc, keep);
      H_STAMP(1);
      cl.sync();
    }
    return;
  }
  double *wsh = psm + 2 * kPersMaxNodes;
  for (int s = -1; s < nsteps; ++s) {  // while CTA 0 solves step s: step s + 1
    const int sn = s + 1, par = sn & 1;
    H_STAMP(2);
    if (sn < nsteps) {
      const int tstep = tstep0 + sn - I.tb, os = os0 + sn - I.ob;
      const int K = older(sn), kch = (K + C - 2) / (C - 1);
      const int k0 = min(K, (r - 1) * kch), nk = min(K, k0 + kch) - k0;
      const double invX = I.weights == FH_W_PSI ? 1.0 / (double)(tstep + 1) : 0.0;
      // the newest slot's and the current slot's weight on the last CTA's last two warps
      if (r == C - 1 && (t == kPersThreads - 32 || t == kPersThreads - 64)) {
        const int j = t == kPersThreads - 32;
        const int slot = j ? (os > 1 ? os - 1 : 0) : os - 2;
        wstep[par][j] =
            j || os >= 2 ? h_slot_weight(I, b, slot, j != 0, tstep, os, invX, ldw, Lb, ibt, lgt) : 0.0;
      }
      double acc[kPersNodes];
#pragma unroll
      for (int q = 0; q < kPersNodes; ++q) acc[q] = 0.0;
      for (int kb = 0; kb < nk; kb += kPersStage) {
        const int ns = min(kPersStage, nk - kb);
        if (kb > 0) __syncthreads();
        for (int k = t; k < ns; k += kPersThreads)
          wsh[k] = h_slot_weight(I, b, k0 + kb + k, false, tstep, os, invX, ldw, Lb, ibt, lgt);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kPersNodes; ++q) {
          const int p = t + q * kPersThreads;
          if (p < np) {
            // slots of the instance's occupant start at global slot I.ob; 16
            // independent loads ahead of the multiply-adds
            const double *d = D + (long long)(I.ob + k0 + kb) * ldd + I.off + p;
            double a = acc[q];
            int k = 0;
            for (; k + 16 <= ns; k += 16, d += 16 * ldd) {
              double v[16];
#pragma unroll
              for (int w = 0; w < 16; ++w) v[w] = __ldcg(d + w * ldd);
#pragma unroll
              for (int w = 0; w < 16; ++w) a = fma(wsh[k + w], v[w], a);
            }
            double v[16];
#pragma unroll
            for (int w = 0; w < 16; ++w) v[w] = k + w < ns ? __ldcg(d + w * ldd) : 0.0;
#pragma unroll
            for (int w = 0; w < 16; ++w)
              if (k + w < ns) a = fma(wsh[k + w], v[w], a);
            acc[q] = a;
          }
        }
      }
#pragma unroll
      for (int q = 0; q < kPersNodes; ++q)
        if (t + q * kPersThreads < np) psm[par * kPersMaxNodes + t + q * kPersThreads] = acc[q];
    }
    H_STAMP(3);
    cl.sync();
  }
}

// The same for lines of at most kOwnMaxN nodes and solves of at most
// kOwnMaxSteps steps, with the nodes instead of the slots shared out and without
// a cluster barrier in the step:
//   CTA 0 solves the line, step after step (fh_hline: state, newest layer and
//     constant factors stay in shared memory).  Of a step's history sum it adds
//     the newest layer; the rest arrives in its shared memory.
//   CTAs 1 .. C - 1 own a range of the nodes each: they sum every slot but the
//     newest for them (first 256 threads; the slots in runs side by side when
//     there are fewer nodes), keep their nodes' layers in shared memory as far
//     as it goes (the first ones; later ones are read back from the history),
//     and store new layers to the history.  psi weights are evaluated by the
//     owners' other 128 threads, a share of the slots each, one step ahead, and
//     sent to every owner; L1 weights come from the lag table in shared memory.
// Messages are one-sided (fh_cluster.cuh).  The layer of step s goes out when it
// is solved, the sums of step s + 2 come back while CTA 0 solves step s + 1.
// Sums and layers alternate between two buffers: CTA 0 sends layer s after it
// has the sums of step s, which their owner sent after it had copied layer
// s - 2; an owner sends the sums of step s + 2 after it has layer s, which CTA 0
// sent when it had read the sums of step s.  Weights rotate through three
// buffers: an owner that has layer s - 2 (preparing step s, sending weights of
// s + 1) knows every owner has finished step s - 2.  A cluster barrier before the
// first and after the last message; waits are bounded (*err on expiry).
// The sums of a step are split by its slot count alone, so a solve does not
// depend on how its steps are spread over calls.
// Measured: one L1 instance of N = 200 over 1000 steps 13.6 ms with sums and
// solves one after the other and serial factors, 6.6 ms with the solve beside the
// next step's sums behind one cluster barrier a step, 4.5 ms in this form; 40
// steps of N = 64 404, 266, 189 us; 32 psi instances of N = 512 over 250 steps
// 60.6, 8.3, 6.3 ms.
constexpr int kOwnLine = 32 * kLineWarps;     // threads of the line solve
constexpr int kOwnSum = 256;                  // threads of the sums
constexpr int kOwnThreads = kOwnSum + 128;    // and of the weights
constexpr int kOwnMaxN = kOwnLine * kHLineEq + 1;  // one panel
constexpr int kOwnMaxSteps = 4096;            // weights of three steps in shared memory; k_h_persistent above
constexpr size_t kOwnSmem = 200 * 1024;       // dynamic shared memory
// CTA 0: the resident line, then the sums [2][nodes]; their skewed lengths fit
static_assert(fh_hline_res_smem(kOwnLine) + sizeof(double) * 2 * (kOwnMaxN + 2) <= kOwnSmem, "line and sums");

__global__ void __launch_bounds__(kOwnThreads, 1)
    k_h_pers_own(const fh_h_dev_inst *__restrict__ inst, int tstep0, int os0, int nsteps, double *D, long long ldd,
                   int ldw, const double *__restrict__ Lb, const double *__restrict__ ibt,
                   const double2 *__restrict__ lgt, double *U, double *Al, double *Bt, double *fF, double *fG,
                   int *err) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double psm[];
  __shared__ fh_hline_scan<kLineWarps> sc;
  __shared__ double wst[3][2];  // CTA 0: psi weights of the newest and the current slot
  __shared__ uint64_t bars[5];  // 0, 1: sums (CTA 0) or layers (owners); 2..4: psi weights
  const int C = (int)cl.num_blocks(), r = (int)cl.block_rank();
  const int b = blockIdx.x / C, t = threadIdx.x;
  const fh_h_dev_inst I = inst[b];
  const int np = I.N + 2, PW = (np + C - 2) / (C - 1);  // nodes per owner
  const int Q = (np + PW - 1) / PW;                      // owners that have any
  const uint32_t bar = fh_smem_u32(bars), smb = fh_smem_u32(psm);
  if (t == 0) {
    for (int k = 0; k < 5; ++k) fh_mbar_init(bar + 8 * k, 1);
    fh_fence_mbar_init();
  }
  bool ok = true;
  const bool psi = I.weights == FH_W_PSI;
  if (r == 0) {
    constexpr int L = fh_hline_len(kOwnLine);
    fh_hline_keep keep;
    keep.dn = psm + 3 * L;
    keep.f = psm + 4 * L;
    keep.g = psm + 5 * L;
    keep.al = psm + 6 * L;
    keep.pf = psm + 7 * L;
    keep.pb = psm + 8 * L;
    keep.lv = psm + 9 * L;
    double *rp = keep.lv + kHLineLv * kOwnLine;  // sums [2][np]
    if (t < kOwnLine) {  // the newest layer before the call
      const bool has = os0 - I.ob >= 2;
      const double *d = D + (long long)(has ? os0 - 2 : 0) * ldd + I.off;
      for (int p = t; p < np; p += kOwnLine) keep.dn[fh_hsk(p)] = has ? __ldcg(d + p) : 0.0;
    }
    const double l1new = psi ? 0.0 : Lb[(long long)b * ldw + min(1, ldw - 1)];
    cl.sync();
    if (t < kOwnLine) {
      for (int s = 0; s < nsteps; ++s) {
        const int os = os0 + s - I.ob, par = s & 1, w3 = s % 3;
        if (t == 0) {
          fh_mbar_arrive_expect_tx(bar + 8 * par, 8 * np);
          if (psi) fh_mbar_arrive_expect_tx(bar + 8 * (2 + w3), 16);
        }
        ok = fh_mbar_wait(bar + 8 * par, (s >> 1) & 1);
        if (psi) ok &= fh_mbar_wait(bar + 8 * (2 + w3), (s / 3) & 1);
        ok = fh_group_and(1, kOwnLine, ok);
        if (!ok) break;
        H_STAMP(0);
        const double wnew = psi ? wst[w3][0] : l1new, DaW = I.Da * (psi ? wst[w3][1] : 1.0);
        const double *rs = rp + par * np;
        auto ts = [&](int i) { return os > 2 ? fma(wnew, keep.dn[fh_hsk(i)], rs[i]) : 0.0; };
        auto sink = [&](int p, double dx) {
          const int q = p / PW;
          fh_st_async8(fh_mapa(smb, 1 + q) + 8 * (par * PW + p - q * PW), dx, fh_mapa(bar, 1 + q) + 8 * par);
        };
        keep.load = s == 0;
        keep.last = s == nsteps - 1;
        fh_hline<kLineWarps, false, true>(I, DaW, ts, U, Al, Bt, fF, fG, nullptr, os == 0, 0, nullptr, psm, sc, keep,
                                          sink);
        H_STAMP(1);
        fh_group_bar(1, kOwnLine);  // the state is read by other threads next
      }
    }
    if (!ok && t == 0) {
      *(volatile int *)err = 1;
      __threadfence_system();
    }
    cl.sync();
    return;
  }
  if (r > Q) {
    cl.sync();
    cl.sync();
    return;
  }
  // ---- owner of nodes [n0, n0 + nn)
  const int n0 = (r - 1) * PW, nn = min(np, n0 + PW) - n0;
  // dx [2][PW] | partial sums [256] | weights: psi [3][kw], L1 the lag table [kw] | layers [cap][PW]
  const int kw = os0 - I.ob + nsteps + 1;
  double *dxb = psm, *pt = dxb + 2 * PW, *wb = pt + kOwnSum, *hist = wb + (psi ? 3 : 1) * (size_t)kw;
  const int cap = (int)((kOwnSmem / sizeof(double) - (size_t)(hist - psm)) / PW);
  double *Dn = D + I.off + n0;
  // (at most 64 runs, which one thread adds: of 256, on a line of 8 nodes, the
  // additions alone took 7 of a step's 11.7 us)
  const int parts = min(max(1, kOwnSum / PW), 64), rows = min(PW, kOwnSum);
  const int i = t % rows, p = t / rows;  // node and run of a summing thread (nodes i, i + 256, ... when PW > 256)
  // layers of the occupant before the call
  const int have = max(os0 - I.ob - 1, 0);
  for (int x = t; x < min(have, cap) * PW; x += kOwnThreads) {
    const int k = x / PW, j = x - k * PW;
    hist[x] = j < nn ? __ldcg(Dn + (long long)(I.ob + k) * ldd + j) : 0.0;
  }
  if (!psi)
    for (int k = t; k < kw; k += kOwnThreads) wb[k] = k < ldw ? Lb[(long long)b * ldw + k] : 0.0;
  auto older = [&](int s) { return max(os0 + s - I.ob - 2, 0); };  // slots but the newest at step s of the call
  // in CTA 0
  const uint32_t rbar = fh_mapa(bar, 0), rdst = fh_mapa(smb, 0) + 8 * (9 * fh_hline_len(kOwnLine) + kHLineLv * kOwnLine);
  const uint32_t wdst = fh_mapa(fh_smem_u32(wst), 0);
  // psi weights of step s of the call: this owner's share of the older slots to
  // every owner, of the newest and the current one (last) to CTA 0
  auto weights = [&](int s) {
    const int tstep = tstep0 + s - I.tb, os = os0 + s - I.ob, K = older(s), sh = (K + 2 + Q - 1) / Q, w3 = s % 3;
    const int k0 = (r - 1) * sh, k1 = min(K + 2, k0 + sh);
    const double invX = 1.0 / (double)(tstep + 1);
    for (int k = k0 + t - kOwnSum; k < k1; k += kOwnThreads - kOwnSum) {
      const bool cur = k == K + 1;
      const int slot = cur ? max(os - 1, 0) : k == K ? max(os - 2, 0) : k;
      const double w = h_slot_weight(I, b, slot, cur, tstep, os, invX, ldw, Lb, ibt, lgt);
      if (k < K) {
        const uint32_t off = (uint32_t)(8 * ((wb - psm) + (size_t)w3 * kw + k));
        for (int q = 1; q <= Q; ++q) fh_st_async8(fh_mapa(smb, q) + off, w, fh_mapa(bar, q) + 8 * (2 + w3));
      } else {
        fh_st_async8(wdst + 8 * (2 * w3 + k - K), w, rbar + 8 * (2 + w3));
      }
    }
  };
  cl.sync();
  if (psi && t >= kOwnSum) weights(0);
  for (int s = -2; s < nsteps; ++s) {
    if (s >= 0) {  // the layer of step s: slot os0 + s - 1
      H_STAMP(2);
      if (t == 0) fh_mbar_arrive_expect_tx(bar + 8 * (s & 1), 8 * nn);
      ok = fh_mbar_wait(bar + 8 * (s & 1), (s >> 1) & 1);
      const int slot = os0 + s - 1;
      if (ok && slot >= 0)
        for (int j = t; j < nn; j += kOwnThreads) {
          const double d = dxb[(s & 1) * PW + j];
          if (slot - I.ob >= 0 && slot - I.ob < cap) hist[(slot - I.ob) * PW + j] = d;
          Dn[(long long)slot * ldd + j] = d;
        }
    }
    const int sn = s + 2;  // the step to prepare
    if (psi && sn < nsteps) {
      if (t == 0) fh_mbar_arrive_expect_tx(bar + 8 * (2 + sn % 3), 8 * older(sn));
      ok &= fh_mbar_wait(bar + 8 * (2 + sn % 3), (sn / 3) & 1);
    }
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (sn >= nsteps) continue;
    const int os = os0 + sn - I.ob, K = older(sn), per = (K + parts - 1) / parts;
    if (t >= kOwnSum) {
      if (psi && sn + 1 < nsteps) weights(sn + 1);
    } else {
      const double *w = wb + (psi ? (size_t)(sn % 3) * kw : 0);
      auto wt = [&](int k) { return psi ? w[k] : w[os - 1 - k]; };  // L1: by the lag
      for (int j = i; j < PW; j += rows) {  // one round unless PW > 256
        double a0 = 0.0, a1 = 0.0;
        if (p < parts && j < nn) {
          // slot 0 carries no weight; even places from k to a0, odd ones to a1
          int k = max(1, p * per);
          const int k1 = min(K, (p + 1) * per), kc = k1 <= cap ? k1 : k + (max(cap - k, 0) & ~1);
          for (; k + 2 <= kc; k += 2) {
            a0 = fma(wt(k), hist[k * PW + j], a0);
            a1 = fma(wt(k + 1), hist[(k + 1) * PW + j], a1);
          }
          if (k < kc) {
            a0 = fma(wt(k), hist[k * PW + j], a0);
            ++k;
          }
          const double *d = Dn + (long long)(I.ob + k) * ldd + j;
          for (; k + 8 <= k1; k += 8, d += 8 * ldd) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = __ldcg(d + u * ldd);
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
              a0 = fma(wt(k + u), v[u], a0);
              a1 = fma(wt(k + u + 1), v[u + 1], a1);
            }
          }
          for (; k + 2 <= k1; k += 2, d += 2 * ldd) {
            a0 = fma(wt(k), __ldcg(d), a0);
            a1 = fma(wt(k + 1), __ldcg(d + ldd), a1);
          }
          if (k < k1) a0 = fma(wt(k), __ldcg(d), a0);
        }
        double a = a0 + a1;
        if (parts > 1) {
          pt[t] = a;
          fh_group_bar(2, kOwnSum);
          if (p == 0) {
            double v = 0.0;
            for (int q = 1; q + 1 < parts; q += 2) {
              a += pt[q * rows + j];
              v += pt[(q + 1) * rows + j];
            }
            if (!(parts & 1)) a += pt[(parts - 1) * rows + j];
            a += v;
          }
        }
        if (p == 0 && j < nn) fh_st_async8(rdst + 8 * ((sn & 1) * np + n0 + j), a, rbar + 8 * (sn & 1));
      }
    }
    H_STAMP(3);
  }
  if (!ok && t == 0) {
    *(volatile int *)err = 1;
    __threadfence_system();
  }
  cl.sync();
}

// ---------------------------------------------------- blocked history mode
// psi = t^beta node value F(x) = B(y(x); 1/beta, 1-alpha) at X (lower series
// r P(y), flag low = 1) or its upper tail U(c) = c^b Q(c) (low = 0), from the
// per-instance tables and the log table: one exp or expm1 + log + exp and one
// Horner polynomial per node.  A slot weight is the difference of its two
// nodes; the difference loses ~log10(X) digits, which is far below the 2^-32
// of the bf16 slices the blocked contraction uses these weights at.
// h_psi_node_at: the same at a real X (0 < x < X) given log x and log X as
// double-doubles and r = x/X.
__device__ __forceinline__ void h_psi_node_at(const fh_h_dev_inst &I, const double *__restrict__ Lc, double2 lx,
                                              double2 lX, double r, double &v, int &low) {
  const double *Uc = Lc + kIbTerms;
  const double sh = lx.x - lX.x;
  const double sl = (lx.x - (sh + lX.x)) + (lx.y - lX.y);
  const double th = I.beta * sh;
  const double tl = fma(I.beta, sh, -th) + I.beta * sl;
  if (r <= Lc[2 * kIbTerms + 1]) {  // y <= kIbLowMax: lower series in y
    const double ey = exp(th);
    const double y = fma(ey, tl, ey);
    v = r * fh_series(fh_ib_coef_tab{Lc}, fh_ib_nterms(y), y);
    low = 1;
  } else {  // upper tail in c = 1 - y
    const double em = expm1(th);
    const double c = -fma(em + 1.0, tl, em);
    v = c <= 0.0 ? 0.0 : exp((1.0 - I.alpha) * log(c)) * fh_series(fh_ib_coef_tab{Uc}, fh_ib_nterms(c), c);
    low = 0;
  }
}

__device__ __forceinline__ void h_psi_node(const fh_h_dev_inst &I, const double *__restrict__ Lc,
                                           const double2 *__restrict__ lgt, int x, int X, double invX, double &v,
                                           int &low) {
  if (x <= 0) {
    v = 0.0;
    low = 1;
    return;
  }
  if (x >= X) {  // c = 0
    v = 0.0;
    low = 0;
    return;
  }
  h_psi_node_at(I, Lc, lgt[x], lgt[X], (double)x * invX, v, low);
}

// Far slots by interpolation across the block's steps.  For a fixed slot
// [t, t + 1] the weight w(X) over the block's X in [K + 3, K + 66] is
// analytic off the branch points X = t, t + 1, so within the Bernstein
// ellipse of the interval with parameter rho = D + sqrt(D^2 - 1),
// D = 1 + 2 d / 63, d = K + 2 - t the distance of the nearer branch point:
// the interpolant at m first-kind Chebyshev points is within ~rho^-m of w
// (Trefethen, Approximation Theory and Approximation Practice, ch. 8).  A
// chunk group takes the order of its last slot for kHbChebBits bits (2^-38,
// far below the 2^-31 of the group's bf16 slices); groups that would need
// more than kHbChebMax points are evaluated exactly per step.
constexpr int kHbChebMax = 16;
constexpr double kHbChebBits = 38.0;
constexpr int kHbGroupSlots = 2 * kSlcK;  // slots of a chunk group
__host__ __device__ inline int hb_cheb_order(int d) {
  const double D = 1.0 + 2.0 * (double)d / 63.0;
  const double rho = D + sqrt(D * D - 1.0);
  return (int)ceil(kHbChebBits * 0.6931471805599453 / log(rho)) + 1;
}
// The same in the slot direction: the group's slot starts t in
// [t0, t0 + 127] (half length 63.5) with the nearer of the branch points
// t = 0 (at t0) and t = X - 1 (beyond the group's last slot by at least d).
__host__ __device__ inline int hb_cheb_order_t(int dt) {
  const double D = 1.0 + (double)dt / 63.5;
  const double rho = D + sqrt(D * D - 1.0);
  return (int)ceil(kHbChebBits * 0.6931471805599453 / log(rho)) + 1;
}
// Leading chunk groups of the block at K that are interpolated.
static int hb_cheb_groups(int K) {
  const int ng = fh_ngroups(K / kSlcK);
  int g = 0;
  while (g < ng - 1 && hb_cheb_order(K + 2 - (g * kHbGroupSlots + kHbGroupSlots - 1)) <= kHbChebMax) ++g;
  return g;
}
// Interpolation tables for m = 1..kHbChebMax points: block m holds the
// Lagrange basis L[r][j] at the block's steps r < 64 (x_r = -1 + 2 r / 63;
// row stride kHbChebMax) and, in row 64, the X offsets 31.5 (1 + x_j) of the
// points x_j = cos((2 j + 1) pi / (2 m)) from K + 3.
static constexpr size_t kHbChebBlock = (size_t)(kSlcK + 1) * kHbChebMax;
// Slot-direction tables after them: block m holds L[k][i] at the group's 128
// slots (x_k = -1 + 2 k / 127) and, in row 128, the slot offsets
// 63.5 (1 + x_i) from the group's first slot.
static constexpr size_t kHbChebTBlock = (size_t)(kHbGroupSlots + 1) * kHbChebMax;
static constexpr size_t kHbChebTBase = (kHbChebMax + 1) * kHbChebBlock;
static void hb_cheb_table(std::vector<double> &t) {
  t.assign(kHbChebTBase + (kHbChebMax + 1) * kHbChebTBlock, 0.0);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int m = 1; m <= kHbChebMax; ++m) {
    double *T = t.data() + (size_t)m * kHbChebBlock;
    long double xj[kHbChebMax];
    for (int j = 0; j < m; ++j) {
      xj[j] = cosl((long double)(2 * j + 1) * pi / (long double)(2 * m));
      T[kSlcK * kHbChebMax + j] = (double)(31.5L * (1.0L + xj[j]));
    }
    for (int r = 0; r < kSlcK; ++r) {
      const long double x = -1.0L + 2.0L * (long double)r / 63.0L;
      for (int j = 0; j < m; ++j) {
        long double l = 1.0L;
        for (int i = 0; i < m; ++i)
          if (i != j) l *= (x - xj[i]) / (xj[j] - xj[i]);
        T[r * kHbChebMax + j] = (double)l;
      }
    }
    double *Tt = t.data() + kHbChebTBase + (size_t)m * kHbChebTBlock;
    for (int j = 0; j < m; ++j) Tt[kHbGroupSlots * kHbChebMax + j] = (double)(63.5L * (1.0L + xj[j]));
    for (int k = 0; k < kHbGroupSlots; ++k) {
      const long double x = -1.0L + 2.0L * (long double)k / 127.0L;
      for (int j = 0; j < m; ++j) {
        long double l = 1.0L;
        for (int i = 0; i < m; ++i)
          if (i != j) l *= (x - xj[i]) / (xj[j] - xj[i]);
        Tt[k * kHbChebMax + j] = (double)l;
      }
    }
  }
}

// Weight planes of the interpolated chunk groups G < gridDim.x of the psi
// instances (one CTA per (group, instance)): the group's 129 node values at
// each of the m points X_j (h_psi_node_at; psi = t: (1 - x/X)^(1 - alpha)),
// the 128 slot weights at each X_j, then per step r of the block the
// interpolated weights sum_j L[r][j] w_j, sliced into W3/Ew as k_hb_weights
// does.  Rows past the last step are zero.  The 64 x 128 interpolated weights
// and their slices are formed in double-float (2^-45; the slices hold 2^-32):
// in FP64 they were 84 % of the kernel's FP64 work.
__global__ void __launch_bounds__(256) k_hb_wcheb(const fh_h_dev_inst *__restrict__ inst, int K, int max_steps,
                                                  const double *__restrict__ ibt, const double2 *__restrict__ lgt,
                                                  const double *__restrict__ cheb, long long R, int Kcap,
                                                  __nv_bfloat16 *__restrict__ W3, int8_t *__restrict__ Ew) {
  __shared__ double sv[kHbChebMax][kHbGroupSlots + 1];
  __shared__ float2 sw[kHbChebMax][kHbGroupSlots];
  __shared__ float2 sL[kSlcK * kHbChebMax];
  __shared__ double sX[kHbChebMax][3];  // log X_j, 1/X_j, scale of X_j
  __shared__ double sn[kHbChebMax][kHbChebMax];  // 2D path: weights at the (slot, step) points
  __shared__ unsigned char slo[kHbChebMax][kHbGroupSlots + 1];
  const int b = blockIdx.y, G = blockIdx.x;
  const fh_h_dev_inst I = inst[b];
  if (I.weights != FH_W_PSI) return;  // whole CTA
  const int x0 = G * kHbGroupSlots;
  const int m = min(hb_cheb_order(K + 2 - (x0 + kHbGroupSlots - 1)), kHbChebMax);
  const double *tab = cheb + (size_t)m * kHbChebBlock;
  for (int i = threadIdx.x; i < kSlcK * kHbChebMax; i += blockDim.x) sL[i] = fh_df_pair(fh_df_bits(tab[i]));
  const double *Lc = ibt + (long long)b * kIbStride;
  const bool psi_t = I.beta == 1.0;
  if (threadIdx.x < m) {
    const int j = threadIdx.x;
    const double X = (double)(K + 3) + tab[kSlcK * kHbChebMax + j];
    const double lX = log(X);
    sX[j][0] = lX;
    sX[j][1] = 1.0 / X;
    // (X tau)^(1 - alpha beta) (1 - alpha) / beta; psi = t: (X tau)^(1 - alpha)
    sX[j][2] = psi_t ? exp((1.0 - I.alpha) * (lX + Lc[2 * kIbTerms + 2]))
                     : exp((1.0 - I.alpha * I.beta) * (lX + Lc[2 * kIbTerms + 2])) * Lc[2 * kIbTerms + 3] *
                           (1.0 - I.alpha);
  }
  __syncthreads();
  // Groups after the first (slot starts t >= 128, away from the branch point
  // t = 0) are interpolated in the slot direction too: the weights at
  // mt x m points (t_i, X_j) of the interval [t_i, t_i + 1] (the
  // divided-difference form at real t), then the group's 128 slots at each
  // X_j from those
  const int mt = G >= 1 ? hb_cheb_order_t(min(K + 2 - (x0 + kHbGroupSlots - 1), x0)) : kHbChebMax + 1;
  if (mt <= kHbChebMax) {
    const double *tabt = cheb + kHbChebTBase + (size_t)mt * kHbChebTBlock;
    double *sLt = &sv[0][0];  // L[k][i], 128 x kHbChebMax (fits in sv)
    for (int i = threadIdx.x; i < kHbGroupSlots * kHbChebMax; i += blockDim.x) sLt[i] = tabt[i];
    const double *Uc = Lc + kIbTerms;
    for (int i = threadIdx.x; i < mt * m; i += blockDim.x) {
      const int ti = i / m, j = i - ti * m;
      const double t = (double)x0 + tabt[kHbGroupSlots * kHbChebMax + ti];
      const double X = (double)(K + 3) + tab[kSlcK * kHbChebMax + j];
      double w;
      if (psi_t) {
        w = fh_psi_int_t(t, t + 1.0, X, I.tau, I.alpha) * (1.0 - I.alpha);
      } else {
        auto lrat = [](double x, double Xv) { return 2.0 * x <= Xv ? log(x / Xv) : log1p((x - Xv) / Xv); };
        fh_ib_slot q;
        q.zero0 = false;
        q.top = false;
        q.r0 = t * sX[j][1];
        q.r1 = (t + 1.0) * sX[j][1];
        q.dr = sX[j][1];
        q.l1h = lrat(t + 1.0, X);
        q.l1l = 0.0;
        q.l0h = lrat(t, X);
        q.l0l = 0.0;
        q.ldh = log1p(1.0 / t);
        q.ldl = 0.0;
        const double diff = fh_ib_diff(q, I.beta, 1.0 - I.alpha, Lc[2 * kIbTerms + 1],
                                       [&] { return Lc[2 * kIbTerms]; }, fh_ib_coef_tab{Lc}, fh_ib_coef_tab{Uc});
        w = sX[j][2] * diff;
      }
      sn[ti][j] = w;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < m * kHbGroupSlots; i += blockDim.x) {
      const int j = i / kHbGroupSlots, k = i - j * kHbGroupSlots;
      const double *Lk = sLt + k * kHbChebMax;
      double acc = 0.0;
      for (int ti = 0; ti < mt; ++ti) acc = fma(Lk[ti], sn[ti][j], acc);
      sw[j][k] = fh_df_pair(fh_df_bits(acc));
    }
    __syncthreads();
  } else {
  for (int i = threadIdx.x; i < m * (kHbGroupSlots + 1); i += blockDim.x) {
    const int j = i / (kHbGroupSlots + 1), k = i - j * (kHbGroupSlots + 1);
    const int x = x0 + k;  // x < K + 3 <= X_j
    double v;
    int lo;
    if (psi_t) {
      v = exp((1.0 - I.alpha) * log1p(-(double)x * sX[j][1]));
      lo = 0;
    } else if (x == 0) {
      v = 0.0;
      lo = 1;
    } else {
      h_psi_node_at(I, Lc, lgt[x], make_double2(sX[j][0], 0.0), (double)x * sX[j][1], v, lo);
    }
    sv[j][k] = v;
    slo[j][k] = (unsigned char)lo;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < m * kHbGroupSlots; i += blockDim.x) {
    const int j = i / kHbGroupSlots, k = i - j * kHbGroupSlots;
    const double v0 = sv[j][k], v1 = sv[j][k + 1];
    const int l0 = slo[j][k], l1 = slo[j][k + 1];
    double diff;
    if (l0 && l1)
      diff = v1 - v0;
    else if (!l0)
      diff = v0 - v1;
    else
      diff = (Lc[2 * kIbTerms] - v1) - v0;
    sw[j][k] = fh_df_pair(fh_df_bits(x0 + k >= 1 ? sX[j][2] * diff : 0.0));  // slot 0 weighs nothing
  }
  __syncthreads();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nchunks = K / kSlcK;
  for (int r = warp; r < kSlcK; r += blockDim.x >> 5) {
    float2 w[4] = {};
    if (K + r + 2 <= max_steps) {
      const float2 *Lr = sL + r * kHbChebMax;
      for (int j = 0; j < m; ++j) {
        const fh_df l = fh_df_from_pair(Lr[j]);
#pragma unroll
        for (int h = 0; h < 4; ++h)
          w[h] = fh_df_pair(fh_df_fma(l, fh_df_from_pair(sw[j][lane + 32 * h]), fh_df_from_pair(w[h])));
      }
    }
    fh_slice_group_pairs(w, G, nchunks, (long long)b * kSlcK + r, R, Kcap, W3, Ew);
  }
}

// Weight planes of the block whose first step has K = 64 blk history slots:
// row m = 64 inst + r is step tstep = K + r + 2 (X = K + r + 3) of instance
// inst, weighing the slots t < K (slot 0: weight 0, as in k_h_weights); rows
// past the last step are zero.  One warp per (row, chunk group G >= G0), sliced
// into W3/Ew (fh_slices.cuh); the groups below gcheb of the psi instances are
// k_hb_wcheb's.
__global__ void k_hb_weights(const fh_h_dev_inst *__restrict__ inst, int K, int max_steps, int G0, int gcheb,
                             const double *__restrict__ Lb, int ldw, const double *__restrict__ ibt,
                             const double2 *__restrict__ lgt, long long R, int Kcap, __nv_bfloat16 *__restrict__ W3,
                             int8_t *__restrict__ Ew) {
  const long long m = (long long)blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (m >= R) return;  // whole warp
  const int lane = threadIdx.x & 31;
  const int b = (int)(m / kSlcK), r = (int)(m % kSlcK);
  const fh_h_dev_inst I = inst[b];
  const int G = G0 + blockIdx.x, nchunks = K / kSlcK;
  if (I.weights == FH_W_PSI && G < gcheb) return;  // interpolated (k_hb_wcheb); whole warp
  const int tstep = K + r + 2, X = tstep + 1, os = K + r + 1;
  const bool live = tstep <= max_steps;
  double w[4];
  const int k0 = 2 * G * kSlcK + lane;
  if (I.weights == FH_W_L1) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int k = k0 + 32 * h;
      w[h] = (live && k >= 1 && k < K) ? Lb[(long long)b * ldw + (os - k - 1)] : 0.0;
    }
  } else if (I.beta == 1.0) {
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int k = k0 + 32 * h;
      w[h] = (live && k >= 1 && k < K)
                 ? fh_psi_int_t((double)k, (double)k + 1.0, (double)X, I.tau, I.alpha) * (1 - I.alpha)
                 : 0.0;
    }
  } else {
    const double *Lc = ibt + (long long)b * kIbStride;
    const double invX = 1.0 / (double)X;
    double v[5];
    int lo[5];
    // nodes k0 + 32 h (h < 4) and, for lane 31, the upper node 128 G + 128 of
    // the group's last slot
#pragma unroll
    for (int h = 0; h < 5; ++h) {
      v[h] = 0.0;
      lo[h] = 1;
      if (live && (h < 4 || lane == 31))
        h_psi_node(I, Lc, lgt, h < 4 ? k0 + 32 * h : 2 * G * kSlcK + 128, X, invX, v[h], lo[h]);
    }
    const double sc = live ? exp((1.0 - I.alpha * I.beta) * (lgt[X].x + Lc[2 * kIbTerms + 2])) *
                                 Lc[2 * kIbTerms + 3] * (1 - I.alpha)
                           : 0.0;
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      // upper node of slot k = k0 + 32 h: node k + 1 (the next lane, or lane 0 of the next h)
      double v1 = __shfl_down_sync(0xffffffffu, v[h], 1);
      int l1 = __shfl_down_sync(0xffffffffu, lo[h], 1);
      const double vn = __shfl_sync(0xffffffffu, v[h + 1], 0);
      const int ln = __shfl_sync(0xffffffffu, lo[h + 1], 0);
      if (lane == 31) {
        v1 = h < 3 ? vn : v[4];
        l1 = h < 3 ? ln : lo[4];
      }
      const int k = k0 + 32 * h;
      double diff;
      if (lo[h] && l1)
        diff = v1 - v[h];
      else if (!lo[h])
        diff = v[h] - v1;
      else
        diff = (Lc[2 * kIbTerms] - v1) - v[h];
      w[h] = (live && k >= 1 && k < K) ? sc * diff : 0.0;
    }
  }
  float2 wp[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) wp[h] = fh_df_pair(fh_df_bits(w[h]));
  fh_slice_group_pairs(wp, G, nchunks, m, R, Kcap, W3, Ew);
}

// History sum of the blocked mode at one step: part[p] = far[p] + sum over
// the near slots t in [t_lo, K) of W[inst][t - t_lo] * ring[t mod 128][p], in
// double-float (the far row holds the contraction of the older slots; null
// before the first block has one), two points per thread over the
// per-instance tiles; written as FP64 or, for k_h_line_df, as pairs.
// Launched beside the line solves of the step before (fh_launch_after): all
// layers but the newest, the one those solves make, are summed meanwhile.  They
// are complete, as k_h_line_df lets this kernel start only after its own wait.
// 512 psi instances of 64..1024 nodes, 1500 steps: 116.5 -> 110.6 ms (with every
// line in double-float).
__global__ void __launch_bounds__(kTileThreads) k_h_near_df(const fh_h_tile *__restrict__ tiles,
                                                            const fh_h_dev_inst *__restrict__ inst,
                                                            const float2 *ring, long long ldr, int t_lo,
                                                            int K, const double *__restrict__ W, int ldw,
                                                            const float2 *__restrict__ far,
                                                            double *__restrict__ part, bool pairs) {
  __shared__ float2 wsf2[kSlcK];
  const fh_h_tile T = tiles[blockIdx.x];
  const int nk = K - t_lo;  // < 64
  const double *wrow = W + (long long)T.inst * ldw;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) wsf2[i] = fh_df_pair(fh_df_from_double(wrow[i]));
  __syncthreads();
  const int q = threadIdx.x * 2;
  if (q >= T.len) {
    fh_grid_wait_prev();
    return;
  }
  const long long p = inst[T.inst].off + T.start + q;
  fh_df a0{0.f, 0.f}, a1{0.f, 0.f};
  if (far) {
    const float4 f = *reinterpret_cast<const float4 *>(far + p);
    a0 = fh_df{f.x, f.y};
    a1 = fh_df{f.z, f.w};
  }
  auto add = [&](int k, float4 v) {
    const fh_df w = fh_df_from_pair(wsf2[k]);
    a0 = fh_df_fma(w, fh_df{v.x, v.y}, a0);
    a1 = fh_df_fma(w, fh_df{v.z, v.w}, a1);
  };
  auto layer = [&](int k) { return reinterpret_cast<const float4 *>(ring + (long long)((t_lo + k) & 127) * ldr + p); };
  for (int k = 0; k < nk - 1; ++k) add(k, __ldcs(layer(k)));
  fh_grid_wait_prev();
  if (nk > 0) {  // the newest layer
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(layer(nk - 1))
                 : "memory");
    add(nk - 1, v);
  }
  if (pairs) {
    *reinterpret_cast<float4 *>(part + p) = make_float4(a0.h, a0.l, a1.h, a1.l);
    return;
  }
  double2 o;
  o.x = fh_df_to_double(a0);
  o.y = fh_df_to_double(a1);
  *reinterpret_cast<double2 *>(part + p) = o;
}

// ------------------------------------------------------------------- host

// K splits of the batch history sum: enough CTAs for ~3 waves of 8 resident
// CTAs on 152 SMs, at least 32 layers per split, at most `cap` splits.
// Chunks of at most kHistMaxChunk layers in any case: the chunk's weights sit
// in shared memory, and larger chunks cost resident CTAs (4096 instances at
// K = 5000 without splits: 40 KB per CTA, 5 CTAs per SM, 71 % of HBM).
static constexpr int kHistMaxChunk = 512;
static constexpr int kHistMaxSplits = 64;  // partial-sum buffers of a batch
// FP64 sums of kDpMin layers and more: enough CTAs for ~4 waves of 6, chunks of
// whole groups (1000 psi instances at 250 layers: one split instead of three).
static bool h_dp(const fh_h_batch *B, int K) { return B->mode == FH_H_FP64 && K >= kDpMin; }
static void h_plan(const fh_h_batch *B, int ti, int K, int cap, int *splits, int *kchunk) {
  if (h_dp(B, K)) {
    const long long ctas = 2LL * (long long)B->tiles_by[0].size();
    const int s = (int)std::max(1LL, std::min((long long)std::min(cap, K / 32), (long long)fh_ceil_div(4LL * 152 * 6, ctas)));
    *kchunk = (int)fh_ceil_div((int)fh_ceil_div(K, s), kDpGroup) * kDpGroup;
    *splits = (int)fh_ceil_div(K, *kchunk);
    return;
  }
  const size_t ntiles = B->tiles_by[ti].size();
  const long long target = 3LL * 152 * 8;
  int s = (int)fh_ceil_div(target, (long long)(ntiles > 0 ? ntiles : 1));
  if (s > cap) s = cap;
  if (s > K / 32) s = K / 32;
  const int smin = (int)fh_ceil_div(K, kHistMaxChunk);
  if (s < smin) s = smin < kHistMaxSplits ? smin : kHistMaxSplits;
  if (s < 1) s = 1;
  int kc = (int)fh_ceil_div(K, s);
  kc = (int)fh_ceil_div(kc, 4) * 4;
  *splits = (int)fh_ceil_div(K, kc);
  *kchunk = kc;
}

// History sum over K layers with the weights W into part (tile shape ti).
static int h_hist(fh_h_batch *B, int ti, int K, int splits, int kchunk, const double *W, cudaStream_t st) {
  fh_ctx *ctx = B->ctx;
  if (h_dp(B, K)) {
    k_hist_tiles_dp<<<dim3(2 * (unsigned)B->tiles_by[0].size(), (unsigned)splits), kDpThreads, 0, st>>>(
        B->tl_by[0].as<fh_h_tile>(), B->inst.as<fh_h_dev_inst>(), B->D.as<double>(), B->Ptot, K, W, B->max_weights, kchunk,
        B->part.as<double>(), B->Ptot);
    return fh_after_launch(ctx, "k_hist_tiles_dp");
  }
  const dim3 g((unsigned)B->tiles_by[ti].size(), (unsigned)splits);
  const size_t smem = sizeof(double) * (size_t)kchunk;
  FH_REQUIRE(ctx, smem <= 48 * 1024, FH_EINVAL, "history chunk too large");
  if (B->mode == FH_H_DF64)
    k_hist_tiles_df<<<g, kTileShapes[ti], smem, st>>>(  // float2 weights: same bytes as FP64
        B->tl_by[ti].as<fh_h_tile>(), B->inst.as<fh_h_dev_inst>(), reinterpret_cast<const float2 *>(B->D.as<double>()),
        B->Ptot, K, W, B->max_weights, kchunk, B->part.as<double>(), B->Ptot);
  else
    k_hist_tiles<<<g, kTileShapes[ti], smem, st>>>(B->tl_by[ti].as<fh_h_tile>(), B->inst.as<fh_h_dev_inst>(),
                                                   B->D.as<double>(), B->Ptot, K, W, B->max_weights, kchunk,
                                                   B->part.as<double>(), B->Ptot);
  return fh_after_launch(ctx, "k_hist_tiles");
}

// Weights of step `tstep` (os saved layers) into the buffer pair `par`: the
// history slots and the current weight.
static int h_weights(fh_h_batch *B, int tstep, int os, int par, cudaStream_t st) {
  fh_ctx *ctx = B->ctx;
  FH_REQUIRE(ctx, tstep + 1 < B->max_steps + 2, FH_EINVAL, "h_weights: step %d beyond the log table", tstep);
  const int nh = os > 1 ? os - 1 : 0;
  dim3 gw((unsigned)(nh / kHWeightThreads + 1), (unsigned)B->n);  // slots 0 .. nh
  fh_prof_mark(ctx, FH_PROF_WEIGHTS, false, st);
  k_h_weights<<<gw, kHWeightThreads, 0, st>>>(B->inst.as<fh_h_dev_inst>(), B->n, tstep, os, B->Wp(par),
                                              B->max_weights, B->wcp(par), B->Lb.as<double>(), B->ibt.as<double>(),
                                              B->lgt.as<double2>(), 1.0 / (double)(tstep + 1));
  fh_prof_mark(ctx, FH_PROF_WEIGHTS, true, st);
  return fh_after_launch(ctx, "k_h_weights");
}

// Whether the long lines are solved in double-float (fh_hline_df.cuh): the
// blocked mode, classical derivative, lines of one panel, some long enough.
static bool h_line_in_df(const fh_h_batch *B) {
  return B->mode == FH_H_BLOCKED && !B->space && B->max_n >= kHdfMinN && B->max_n - 1 <= 32 * kLineWarps * kHLineEq;
}

// One step.  The weights depend on the step number only, so with `next` (and
// a small batch) the weights of the following step are computed on the side
// stream hs (high priority) beside this step's history sum and line solves,
// into the other buffer pair; the following call waits for them.
static int h_one_step(fh_h_batch *B, bool next) {
  fh_ctx *ctx = B->ctx;
  const int os = B->nsaved;
  const int K = os >= 2 ? os - 1 : 0;
  const int par = B->tstep & 1;
  const bool blk = B->mode == FH_H_BLOCKED;
  // blocked mode: slots below t_lo (whole 64-slot chunks) are in the far rows,
  // this step is row q of its block's near weights
  const int t_lo = blk ? (K / kSlcK) * kSlcK : 0, q = os - (t_lo > 0 ? t_lo + 1 : 0);
  const double *wcur = B->wcp(par);
  int rc;
  if (blk) {
    wcur = B->wcb.as<double>() + (long long)q * B->n;
    if (q == 0) {
      fh_prof_mark(ctx, FH_PROF_WEIGHTS, false);
      k_h_weights_block<<<dim3((unsigned)fh_ceil_div(kNearRows * (kNearRows + 1) / 2, kHWeightThreads), (unsigned)B->n),
                          kHWeightThreads, 0, ctx->stream>>>(
          B->inst.as<fh_h_dev_inst>(), B->n, t_lo, B->max_steps, B->wb.as<double>(), B->wcb.as<double>(),
          B->Lb.as<double>(), B->max_weights, B->ibt.as<double>(), B->lgt.as<double2>());
      fh_prof_mark(ctx, FH_PROF_WEIGHTS, true);
      if ((rc = fh_after_launch(ctx, "k_h_weights_block"))) return rc;
    }
  } else if (B->w_ready == B->tstep) {
    FH_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->stream, B->ev_w, 0));
  } else if ((rc = h_weights(B, B->tstep, os, par, ctx->stream))) {
    return rc;
  }
  B->w_ready = -1;
  // only for small batches: in large ones the FP64-bound weights take SM
  // slots from the HBM-bound history sum (measured: 4096 instances, 5000
  // steps, the history sum fell from 92 % to 58 % of HBM beside them)
  if (!blk && next && B->hs && B->n < kLineCtaMaxInst) {
    FH_CUDA_TRY(ctx, cudaEventRecord(B->ev_main, ctx->stream));
    FH_CUDA_TRY(ctx, cudaStreamWaitEvent(B->hs, B->ev_main, 0));
    if ((rc = h_weights(B, B->tstep + 1, os + 1, par ^ 1, B->hs))) return rc;
    FH_CUDA_TRY(ctx, cudaEventRecord(B->ev_w, B->hs));
    B->w_ready = B->tstep + 1;
  }
  int splits = 0, kchunk = 0;
  if (blk) {
    float2 *ring = B->ring.as<float2>(), *far = B->far.as<float2>();
    if (K >= kSlcK && K == t_lo) {
      // first step of a block: the chunk just completed into the planes, the
      // weight planes of the block's 64 steps, and their far rows
      fh_prof_mark(ctx, FH_PROF_HISTORY, false);
      rc = fh_hblk_convert(ctx, *B->hb, ring, B->Ptot, K / kSlcK - 1);
      fh_prof_mark(ctx, FH_PROF_HISTORY, true);
      if (rc) return rc;
      fh_prof_mark(ctx, FH_PROF_WEIGHTS, false);
      const long long R = (long long)B->n * kSlcK;
      const int ng = fh_ngroups(K / kSlcK), gcheb = hb_cheb_groups(K), G0 = B->has_l1 ? 0 : gcheb;
      if (gcheb > 0) {
        k_hb_wcheb<<<dim3((unsigned)gcheb, (unsigned)B->n), 256, 0, ctx->stream>>>(
            B->inst.as<fh_h_dev_inst>(), K, B->max_steps, B->ibt.as<double>(), B->lgt.as<double2>(),
            B->cheb.as<double>(), R, fh_hblk_kcap(*B->hb), fh_hblk_wplanes(*B->hb), fh_hblk_wexp(*B->hb));
        if ((rc = fh_after_launch(ctx, "k_hb_wcheb"))) return rc;
      }
      k_hb_weights<<<dim3((unsigned)(ng - G0), (unsigned)fh_ceil_div(R, 8)), 256, 0, ctx->stream>>>(
          B->inst.as<fh_h_dev_inst>(), K, B->max_steps, G0, gcheb, B->Lb.as<double>(), B->max_weights,
          B->ibt.as<double>(), B->lgt.as<double2>(), R, fh_hblk_kcap(*B->hb), fh_hblk_wplanes(*B->hb),
          fh_hblk_wexp(*B->hb));
      fh_prof_mark(ctx, FH_PROF_WEIGHTS, true);
      if ((rc = fh_after_launch(ctx, "k_hb_weights"))) return rc;
      if ((rc = fh_hblk_gemm(ctx, *B->hb, K, far, B->Ptot))) return rc;
    }
    const int ti = tile_shape_index(B->tile_threads);
    fh_prof_mark(ctx, FH_PROF_HISTORY, false);
    fh_launch_after(
        ctx->launches == B->lined, k_h_near_df, (unsigned)B->tiles_by[ti].size(), kTileShapes[ti], 0, ctx->stream,
        B->tl_by[ti].as<fh_h_tile>(), B->inst.as<fh_h_dev_inst>(), ring, B->Ptot, t_lo, K,
        B->wb.as<double>() + (long long)q * kNearLd, kNearRows * kNearLd, t_lo >= kSlcK ? far + (long long)(K - t_lo) * B->Ptot : nullptr, B->part.as<double>(), h_line_in_df(B));
    fh_prof_mark(ctx, FH_PROF_HISTORY, true);
    if ((rc = fh_after_launch(ctx, "k_h_near_df"))) return rc;
    splits = 1;
  } else if (K > 0) {
    const int ti = tile_shape_index(B->tile_threads);
    h_plan(B, ti, K, B->split_cap, &splits, &kchunk);
    fh_prof_mark(ctx, FH_PROF_HISTORY, false);
    rc = h_hist(B, ti, K, splits, kchunk, B->Wp(par), ctx->stream);
    fh_prof_mark(ctx, FH_PROF_HISTORY, true);
    if (rc) return rc;
  }
  fh_prof_mark(ctx, FH_PROF_SWEEP, false);  // right parts (incl. the space-fractional sums) and line solves
  if (B->space) {
    k_h_space_v<<<(unsigned)B->n, 256, B->space_smem, ctx->stream>>>(B->inst.as<fh_h_dev_inst>(), B->U.as<double>(),
                                                                   B->wsp.as<double>(), B->sV.as<double>());
    if ((rc = fh_after_launch(ctx, "k_h_space_v"))) return rc;
  }
  double *Dnew = os < 1 ? nullptr
                 : blk   ? reinterpret_cast<double *>(B->ring.as<float2>() + (long long)((os - 1) & 127) * B->Ptot)
                         : B->D.as<double>() + (long long)(os - 1) * B->Ptot;
  {
    const int dfs = (B->mode == FH_H_DF64 || blk) ? 1 : 0;
    auto line = [&](auto kern, int nw) {
      kern<<<(unsigned)B->n, 32 * nw, fh_hline_smem(32 * nw), ctx->stream>>>(
          B->inst.as<fh_h_dev_inst>(), B->U.as<double>(), wcur, B->part.as<double>(), B->Ptot, splits,
          B->Al.as<double>(), B->Bt.as<double>(), B->fF.as<double>(), B->fG.as<double>(), Dnew, os, dfs,
          B->sV.as<double>(), B->ord.as<int>());
    };
    auto line_df = [&](auto kern, int nw) {
      fh_launch_after(
          true, kern, (unsigned)B->n, 32 * nw, fh_hline_smem(32 * nw), ctx->stream,
          B->inst.as<fh_h_dev_inst>(), B->U.as<double>(), wcur, B->part.as<float2>(), B->Al.as<double>(),
          B->Bt.as<double>(), B->fF.as<double>(), B->fG.as<double>(), reinterpret_cast<float2 *>(Dnew),
          B->ord.as<int>());
    };
    if (h_line_in_df(B))
      B->n < kLineCtaMaxInst ? line_df(k_h_line_df<kLineWarpsSmall>, kLineWarpsSmall)
                             : line_df(k_h_line_df<kLineWarps>, kLineWarps);
    else if (B->n < kLineCtaMaxInst)
      B->space ? line(k_h_line<kLineWarpsSmall, true>, kLineWarpsSmall)
               : line(k_h_line<kLineWarpsSmall, false>, kLineWarpsSmall);
    else
      B->space ? line(k_h_line<kLineWarps, true>, kLineWarps) : line(k_h_line<kLineWarps, false>, kLineWarps);
  }
  fh_prof_mark(ctx, FH_PROF_SWEEP, true);
  if ((rc = fh_after_launch(ctx, "k_h_line"))) return rc;
  B->lined = h_line_in_df(B) ? ctx->launches : -1;
  B->nsaved++;
  B->tstep++;
  return FH_OK;
}

// A new solve of the whole batch: every instance on the batch's clock again.
static int h_reset_clocks(fh_h_batch *b) {
  bool any = false;
  for (auto &I : b->di)
    if (I.tb || I.ob) {
      I.tb = I.ob = 0;
      any = true;
    }
  if (!any) return FH_OK;
  FH_CUDA_TRY(b->ctx, cudaMemcpyAsync(b->inst.p, b->di.data(), sizeof(fh_h_dev_inst) * b->n, cudaMemcpyHostToDevice,
                                      b->ctx->stream));
  FH_CUDA_TRY(b->ctx, cudaStreamSynchronize(b->ctx->stream));
  b->w_ready = -1;
  b->graph.reset();
  return FH_OK;
}

static bool h_params_ok(const fh_h_params &p) {
  return p.N >= 2 && p.N <= (1 << 20) && p.L > 0 && p.tau > 0 && p.alpha > 0 && p.alpha < 1 &&
         (p.weights == FH_W_L1 || p.weights == FH_W_PSI) && (p.kmodel == FH_K_CONST || p.kmodel == FH_K_EXP) &&
         (p.weights == FH_W_L1 || p.beta > 0);
}

// Device record of one instance (segment at `off`, own clock at zero).
static void h_fill_inst(const fh_h_params &p, long long off, fh_h_dev_inst &I) {
  I.N = p.N;
  I.weights = p.weights;
  I.kmodel = p.kmodel;
  I.gravity = p.gravity;
  I.fixed = (p.kmodel == FH_K_CONST) && (p.weights == FH_W_L1 || p.beta == 1.0);
  I.tb = 0;
  I.ob = 0;
  I.off = off;
  I.dL = p.L / p.N;
  I.rdL = 1.0 / I.dL;
  I.Dg = pow(I.dL, -2.0);
  I.Da = p.weights == FH_W_L1 ? pow(p.tau, -p.alpha) / tgamma(2.0 - p.alpha) : pow(p.tau, -1.0) / tgamma(2.0 - p.alpha);
  I.tau = p.tau;
  I.alpha = p.alpha;
  I.beta = p.beta;
  I.kc = p.kc;
  I.kgam = p.kgam;
  I.cinv = p.cinv;
  I.al_left = p.al_left;
  I.bt_left = p.bt_left;
  I.u_right = p.u_right;
  I.spg = 1.0;
  I.spA = 0.0;
  I.kbf = 1.0;
  I.dq = I.Da / (I.Dg * p.kc * p.cinv);
  I.gq = 1.0 / (I.dL * I.Dg * p.cinv);
}

// Shared memory above 48 KiB: the eight-warp line solve and the persistent
// solve (their largest size, the same for every batch).
static int h_set_smem_attrs(fh_ctx *ctx) {
  constexpr auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const int sl = (int)fh_hline_smem(32 * kLineWarpsSmall);
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_line<kLineWarpsSmall, false>, at, sl));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_line<kLineWarpsSmall, true>, at, sl));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_line_df<kLineWarpsSmall>, at, sl));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_persistent, at, (int)kPersSmem));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_persistent, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_pers_own, at, (int)kOwnSmem));
  FH_CUDA_TRY(ctx, cudaFuncSetAttribute(k_h_pers_own, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  return FH_OK;
}

// CTAs per instance of the persistent solve: the largest cluster of which the
// device holds all n at once (a second wave would double the step time; with
// few instances more CTAs share the history sums), at least four.
template <class K>
static int h_pers_ctas(int n, K kern, int threads, size_t smem) {
  for (int c = kPersMaxCtas; c > 4; c /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(n * c));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, kern, &cfg) == cudaSuccess && active >= n) return c;
    cudaGetLastError();
  }
  return 4;
}

extern "C" {

int fh_h_batch_create(fh_ctx *ctx, int ninst, const fh_h_params *params_host, int max_steps, fh_h_batch **out) {
  FH_REQUIRE(ctx, ctx && params_host && out, FH_EINVAL, "fh_h_batch_create: null argument");
  *out = nullptr;
  FH_REQUIRE(ctx, ninst >= 1 && max_steps >= 1, FH_EINVAL, "fh_h_batch_create: need ninst >= 1, max_steps >= 1");
  {
    const int rc0 = h_set_smem_attrs(ctx);
    if (rc0) return rc0;
  }
  fh_h_batch *B = new fh_h_batch();
  B->ctx = ctx;
  B->n = ninst;
  B->max_steps = max_steps;
  B->max_weights = max_steps + 1;
  B->hp.assign(params_host, params_host + ninst);
  std::vector<fh_h_dev_inst> di(ninst);
  long long off = 0;
  for (int b = 0; b < ninst; ++b) {
    const fh_h_params &p = params_host[b];
    if (!h_params_ok(p)) {
      delete B;
      return fh_set_error(ctx, FH_EINVAL, "fh_h_batch_create: bad parameters for instance %d", b);
    }
    fh_h_dev_inst &I = di[b];
    h_fill_inst(p, off, I);
    if (I.weights == FH_W_L1) B->has_l1 = true;
    if (p.N > B->max_n) B->max_n = p.N;
    B->off.push_back(off);
    const int seg = ((p.N + 2) + 1) & ~1;
    B->cap.push_back(seg - 2);
    for (int k = 0; k < 3; ++k) {
      const int tn = 2 * kTileShapes[k];
      for (int st = 0; st < seg; st += tn) B->tiles_by[k].push_back({b, st, seg - st < tn ? seg - st : tn});
    }
    off += seg;
  }
  B->Ptot = off;
  int rc;
  if (ninst <= kPersMaxInst) {
    B->pers_ctas[0] = h_pers_ctas(ninst, k_h_persistent, kPersThreads, kPersSmem);
    B->pers_ctas[1] = h_pers_ctas(ninst, k_h_pers_own, kOwnThreads, kOwnSmem);
    if (cudaHostAlloc(&B->perr, sizeof(int), cudaHostAllocMapped) != cudaSuccess) {
      cudaGetLastError();
      delete B;
      return fh_set_error(ctx, FH_ENOMEM, "fh_h_batch_create: no pinned memory");
    }
    *B->perr = 0;
  }
  const size_t st = sizeof(double) * (size_t)B->Ptot;
  if ((rc = fh_alloc(ctx, B->inst, sizeof(fh_h_dev_inst) * ninst, false)) ||
      (rc = fh_alloc(ctx, B->ord, sizeof(int) * ninst, false)) ||
      (rc = fh_alloc(ctx, B->tl_by[0], sizeof(fh_h_tile) * B->tiles_by[0].size(), false)) ||
      (rc = fh_alloc(ctx, B->tl_by[1], sizeof(fh_h_tile) * B->tiles_by[1].size(), false)) ||
      (rc = fh_alloc(ctx, B->tl_by[2], sizeof(fh_h_tile) * B->tiles_by[2].size(), false)) || (rc = fh_alloc(ctx, B->U, st)) ||
      (rc = fh_alloc(ctx, B->Al, st)) || (rc = fh_alloc(ctx, B->Bt, st)) || (rc = fh_alloc(ctx, B->fF, st)) ||
      (rc = fh_alloc(ctx, B->fG, st)) ||
      (rc = fh_alloc(ctx, B->D, st * (size_t)max_steps)) ||
      (rc = fh_alloc(ctx, B->W, sizeof(double) * 2 * (size_t)ninst * B->max_weights)) ||
      (rc = fh_alloc(ctx, B->Lb, sizeof(double) * (size_t)ninst * B->max_weights, false)) ||
      (rc = fh_alloc(ctx, B->ibt, sizeof(double) * kIbStride * (size_t)ninst, false)) ||
      (rc = fh_alloc(ctx, B->lgt, sizeof(double2) * (size_t)(max_steps + 2), false)) ||
      (rc = fh_alloc(ctx, B->wc, sizeof(double) * 2 * (size_t)ninst)) ||
      (rc = fh_alloc(ctx, B->part, st * (size_t)B->max_splits, false))) {
    delete B;
    return rc;
  }
  {
    int plo = 0, phi = 0;
    cudaError_t es = cudaDeviceGetStreamPriorityRange(&plo, &phi);
    if (es == cudaSuccess) es = cudaStreamCreateWithPriority(&B->hs, cudaStreamNonBlocking, phi);
    if (es == cudaSuccess) es = cudaEventCreateWithFlags(&B->ev_main, cudaEventDisableTiming);
    if (es == cudaSuccess) es = cudaEventCreateWithFlags(&B->ev_w, cudaEventDisableTiming);
    if (es != cudaSuccess) {
      delete B;
      return fh_set_error(ctx, FH_ECUDA, "fh_h_batch_create: weights stream: %s", cudaGetErrorString(es));
    }
  }
  // log(x) as (head, tail) doubles for x = 0..max_steps+1: the psi weights form
  // beta log(x/X) from it as a double-double; long double carries the tail
  std::vector<double2> lg((size_t)max_steps + 2);
  lg[0] = make_double2(0.0, 0.0);
  for (int x = 1; x < max_steps + 2; ++x) {
    const long double l = logl((long double)x);
    const double h = (double)l;
    lg[x] = make_double2(h, (double)(l - (long double)h));
  }
  B->di = di;
  std::vector<int> ord(ninst);
  for (int b = 0; b < ninst; ++b) ord[b] = b;
  std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return di[x].N > di[y].N; });
  cudaError_t e1 = cudaMemcpyAsync(B->inst.p, di.data(), sizeof(fh_h_dev_inst) * ninst, cudaMemcpyHostToDevice, ctx->stream);
  if (e1 == cudaSuccess)
    e1 = cudaMemcpyAsync(B->lgt.p, lg.data(), sizeof(double2) * lg.size(), cudaMemcpyHostToDevice, ctx->stream);
  cudaError_t e2 = cudaMemcpyAsync(B->ord.p, ord.data(), sizeof(int) * ninst, cudaMemcpyHostToDevice, ctx->stream);
  for (int k = 0; k < 3 && e2 == cudaSuccess; ++k)
    e2 = cudaMemcpyAsync(B->tl_by[k].p, B->tiles_by[k].data(), sizeof(fh_h_tile) * B->tiles_by[k].size(),
                         cudaMemcpyHostToDevice, ctx->stream);
  cudaError_t e3 = cudaStreamSynchronize(ctx->stream);
  if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) {
    delete B;
    return fh_set_error(ctx, FH_ECUDA, "fh_h_batch_create: upload failed");
  }
  k_h_lagtab<<<dim3((unsigned)fh_ceil_div(B->max_weights, 128), (unsigned)ninst), 128, 0, ctx->stream>>>(
      B->inst.as<fh_h_dev_inst>(), B->max_weights, B->Lb.as<double>(), B->max_weights);
  if ((rc = fh_after_launch(ctx, "k_h_lagtab"))) {
    delete B;
    return rc;
  }
  k_h_ibtab<<<(unsigned)fh_ceil_div(ninst, 128), 128, 0, ctx->stream>>>(B->inst.as<fh_h_dev_inst>(), ninst,
                                                                        B->ibt.as<double>());
  if ((rc = fh_after_launch(ctx, "k_h_ibtab"))) {
    delete B;
    return rc;
  }
  *out = B;
  return FH_OK;
}

int fh_h_batch_destroy(fh_h_batch *b) {
  if (!b) return FH_OK;
  if (b->ctx) cudaStreamSynchronize(b->ctx->stream);
  delete b;
  return FH_OK;
}

long long fh_h_batch_device_bytes(const fh_h_batch *b) {
  if (!b) return -1;
  const fh_dbuf *bufs[] = {&b->inst, &b->U, &b->D, &b->W, &b->Lb, &b->ibt, &b->lgt, &b->wc, &b->part, &b->Al,
                           &b->Bt, &b->fF, &b->fG, &b->wsp, &b->sV, &b->ring, &b->far, &b->cheb, &b->wb, &b->wcb, &b->ord,
                           &b->tl_by[0], &b->tl_by[1], &b->tl_by[2]};
  size_t s = 0;
  for (const fh_dbuf *d : bufs) s += d->bytes;
  if (b->hb) s += fh_hblk_bytes(*b->hb);
  return (long long)s;
}

long long fh_h_batch_state_size(const fh_h_batch *b) {
  if (!b) return -1;
  long long s = 0;
  for (const auto &p : b->hp) s += p.N + 2;
  return s;
}

// Waits for the stream; FH_ETIMEOUT once a wait of the persistent solve ran out.
static int h_sync_check(fh_h_batch *b) {
  fh_ctx *ctx = b->ctx;
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  FH_REQUIRE(ctx, !b->perr || *(volatile int *)b->perr == 0, FH_ETIMEOUT, "fh_h_batch_step: a wait of the persistent solve ran out");
  return FH_OK;
}

// The flag of an expired wait, in stream order: cleared when a solve starts (set:
// as an expired wait leaves it, for tests).
static __global__ void k_h_mark(volatile int *err, int expired) {
  *err = expired;
  __threadfence_system();
}
static int h_mark(fh_h_batch *b, int expired) {
  if (!b->perr) return FH_OK;
  k_h_mark<<<1, 1, 0, b->ctx->stream>>>(b->perr, expired);
  return fh_after_launch(b->ctx, "k_h_mark");
}
int fh_h_batch_test_expire(fh_h_batch *b) { return h_mark(b, 1); }

// The states of instances first .. first + count - 1 between the host's packed
// order and the device's segments: from kHPackMin instances on one copy and a
// gather or scatter, below a copy per instance.
static int h_copy_u(fh_h_batch *b, int first, int count, double *host, bool to_host) {
  fh_ctx *ctx = b->ctx;
  const bool pack = count >= kHPackMin;
  double *buf = nullptr;
  size_t total = 0;
  for (int i = first; i < first + count; ++i) total += (size_t)b->hp[i].N + 2;
  if (pack) {
    buf = b->Bt.as<double>();  // free between the steps
    if (!to_host)
      FH_CUDA_TRY(ctx, cudaMemcpyAsync(buf, host, sizeof(double) * total, cudaMemcpyHostToDevice, ctx->stream));
    k_h_pack<<<(unsigned)count, 256, 0, ctx->stream>>>(b->inst.as<fh_h_dev_inst>(), first, b->U.as<double>(), buf,
                                                       to_host);
    const int rc = fh_after_launch(ctx, "k_h_pack");
    if (rc) return rc;
    if (to_host)
      FH_CUDA_TRY(ctx, cudaMemcpyAsync(host, buf, sizeof(double) * total, cudaMemcpyDeviceToHost, ctx->stream));
    return FH_OK;
  }
  for (int i = first; i < first + count; ++i) {
    const size_t cnt = (size_t)b->hp[i].N + 2;
    double *d = b->U.as<double>() + b->off[i];
    FH_CUDA_TRY(ctx, to_host ? cudaMemcpyAsync(host, d, sizeof(double) * cnt, cudaMemcpyDeviceToHost, ctx->stream)
                             : cudaMemcpyAsync(d, host, sizeof(double) * cnt, cudaMemcpyHostToDevice, ctx->stream));
    host += cnt;
  }
  return FH_OK;
}

int fh_h_batch_set_u_host(fh_h_batch *b, const double *U_host) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, U_host, FH_EINVAL, "fh_h_batch_set_u_host: null pointer");
  const int rc = h_copy_u(b, 0, b->n, const_cast<double *>(U_host), false);
  if (rc) return rc;
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  if (b->perr) *(volatile int *)b->perr = 0;
  b->tstep = 1;
  b->nsaved = 0;
  return h_reset_clocks(b);
}

int fh_h_batch_restart(fh_h_batch *b, int i, const fh_h_params *p, const double *U0_host) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, p && U0_host && i >= 0 && i < b->n, FH_EINVAL, "fh_h_batch_restart: bad arguments");
  FH_REQUIRE(ctx, h_params_ok(*p), FH_EINVAL, "fh_h_batch_restart: bad parameters");
  FH_REQUIRE(ctx, p->N <= b->cap[i], FH_EINVAL, "fh_h_batch_restart: N = %d above the instance's %d nodes", p->N,
             b->cap[i]);
  FH_REQUIRE(ctx, b->mode != FH_H_BLOCKED && !b->space, FH_EINVAL,
             "fh_h_batch_restart: FP64 or DF64 history, no space-fractional instances");
  FH_REQUIRE(ctx, b->nsaved + 1 < b->max_steps, FH_ENOMEM, "fh_h_batch_restart: no history slots left (%d of %d)",
             b->nsaved, b->max_steps);
  fh_h_dev_inst I;
  h_fill_inst(*p, b->off[i], I);
  I.tb = b->tstep - 1;  // the occupant's first step is its step 1
  I.ob = b->nsaved;
  b->di[i] = I;
  b->hp[i] = *p;
  if (I.weights == FH_W_L1) b->has_l1 = true;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(b->U.as<double>() + b->off[i], U0_host, sizeof(double) * ((size_t)p->N + 2),
                                   cudaMemcpyHostToDevice, ctx->stream));
  fh_h_dev_inst *di = b->inst.as<fh_h_dev_inst>() + i;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(di, &b->di[i], sizeof(fh_h_dev_inst), cudaMemcpyHostToDevice, ctx->stream));
  // the occupant's lag and series tables
  k_h_lagtab<<<dim3((unsigned)fh_ceil_div(b->max_weights, 128), 1), 128, 0, ctx->stream>>>(
      di, b->max_weights, b->Lb.as<double>() + (long long)i * b->max_weights, b->max_weights);
  int rc = fh_after_launch(ctx, "k_h_lagtab");
  if (rc) return rc;
  k_h_ibtab<<<1, 32, 0, ctx->stream>>>(di, 1, b->ibt.as<double>() + (long long)i * kIbStride);
  if ((rc = fh_after_launch(ctx, "k_h_ibtab"))) return rc;
  // the host copy of the initial state and the records are read before return
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  b->w_ready = -1;  // weights prepared ahead used the previous occupant's clock
  b->graph.reset();
  return FH_OK;
}

int fh_h_batch_set_u(fh_h_batch *b, const double *U) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, U, FH_EINVAL, "fh_h_batch_set_u: null pointer");
  long long src = 0;
  for (int i = 0; i < b->n; ++i) {
    const size_t cnt = (size_t)b->hp[i].N + 2;
    FH_CUDA_TRY(ctx, cudaMemcpyAsync(b->U.as<double>() + b->off[i], U + src, sizeof(double) * cnt,
                                     cudaMemcpyDeviceToDevice, ctx->stream));
    src += (long long)cnt;
  }
  if (int rc = h_mark(b, 0)) return rc;
  b->tstep = 1;
  b->nsaved = 0;
  return h_reset_clocks(b);
}

int fh_h_batch_get_u_host(fh_h_batch *b, double *U_host) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  FH_REQUIRE(b->ctx, U_host, FH_EINVAL, "fh_h_batch_get_u_host: null pointer");
  const int rc = h_copy_u(b, 0, b->n, U_host, true);
  return rc ? rc : h_sync_check(b);
}

int fh_h_batch_get_u_range_host(fh_h_batch *b, int first, int count, double *U_host) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  FH_REQUIRE(b->ctx, U_host && first >= 0 && count >= 0 && first + count <= b->n, FH_EINVAL,
             "fh_h_batch_get_u_range_host: bad range");
  const int rc = h_copy_u(b, first, count, U_host, true);
  return rc ? rc : h_sync_check(b);
}

// The persistent path: FP64 history, no space-fractional instances, few
// instances of at most kPersMaxNodes nodes each.
static bool h_persistent_ok(const fh_h_batch *b) {
  if (!b->persistent || b->mode != FH_H_FP64 || b->space || b->n > kPersMaxInst) return false;
  if (b->max_steps > kPersMaxSteps) return false;
  for (const auto &p : b->hp)
    if (p.N + 2 > kPersMaxNodes) return false;
  return true;
}

static int h_persistent_run(fh_h_batch *b, int nsteps) {
  fh_ctx *ctx = b->ctx;
  b->w_ready = -1;
  // nodes or slots shared out (see the kernels)
  bool own = b->max_steps <= kOwnMaxSteps;
  for (const auto &p : b->hp) own = own && p.N <= kOwnMaxN;
  const int ctas = b->pers_ctas[own];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(b->n * ctas));
  cfg.blockDim = dim3(own ? kOwnThreads : kPersThreads);
  cfg.dynamicSmemBytes = own ? kOwnSmem : kPersSmem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  fh_prof_mark(ctx, FH_PROF_HISTORY, false);
  auto launch = [&](auto kern, auto... last) {
    return cudaLaunchKernelEx(&cfg, kern, (const fh_h_dev_inst *)b->inst.as<fh_h_dev_inst>(), b->tstep, b->nsaved,
                              nsteps, b->D.as<double>(), b->Ptot, b->max_weights, (const double *)b->Lb.as<double>(),
                              (const double *)b->ibt.as<double>(), (const double2 *)b->lgt.as<double2>(),
                              b->U.as<double>(), b->Al.as<double>(), b->Bt.as<double>(), b->fF.as<double>(),
                              b->fG.as<double>(), last...);
  };
  FH_CUDA_TRY(ctx, own ? launch(k_h_pers_own, b->perr) : launch(k_h_persistent));
  fh_prof_mark(ctx, FH_PROF_HISTORY, true);
  int rc = fh_after_launch(ctx, "k_h_persistent");
  if (rc) return rc;
  b->nsaved += nsteps;
  b->tstep += nsteps;
  return FH_OK;
}

int fh_h_batch_step(fh_h_batch *b, int nsteps) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, nsteps >= 0, FH_EINVAL, "fh_h_batch_step: nsteps < 0");
  FH_REQUIRE(ctx, b->nsaved + nsteps <= b->max_steps, FH_ENOMEM, "fh_h_batch_step: history full (%d + %d > %d)",
             b->nsaved, nsteps, b->max_steps);
  if (nsteps >= 1 && h_persistent_ok(b)) return h_persistent_run(b, nsteps);
  b->lined = -1;
  if (b->use_graph && ctx->graphs && b->nsaved == 0 && nsteps > 1) {
    // whole solve from the initial state: capture once, replay afterwards
    b->w_ready = -1;
    int rc = fh_graph_run(ctx, b->graph, nsteps, [&]() {
      for (int i = 0; i < nsteps; ++i) {
        int r = h_one_step(b, i + 1 < nsteps);
        if (r) return r;
      }
      return (int)FH_OK;
    });
    if (rc) return rc;
    b->tstep = 1 + nsteps;
    b->nsaved = nsteps;
    return FH_OK;
  }
  b->w_ready = -1;
  for (int i = 0; i < nsteps; ++i) {
    int rc = h_one_step(b, i + 1 < nsteps);
    if (rc) return rc;
  }
  return FH_OK;
}



int fh_h_batch_tstep(const fh_h_batch *b) { return b ? b->tstep : -1; }

int fh_h_batch_set_persistent(fh_h_batch *b, int enable) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  b->persistent = enable != 0;
  b->graph.reset();
  return FH_OK;
}

int fh_h_batch_set_space_order(fh_h_batch *b, const double *gamma_host) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, gamma_host, FH_EINVAL, "fh_h_batch_set_space_order: null pointer");
  FH_REQUIRE(ctx, b->nsaved == 0, FH_EINVAL, "fh_h_batch_set_space_order: only before the first step");
  int maxN = 0;
  for (int i = 0; i < b->n; ++i) {
    const double g = gamma_host[i];
    FH_REQUIRE(ctx, g > 0.0 && g <= 1.0, FH_EINVAL, "fh_h_batch_set_space_order: gamma[%d] = %g not in (0, 1]", i, g);
    FH_REQUIRE(ctx, g == 1.0 || b->hp[i].N <= kSpaceMaxN, FH_EINVAL,
               "fh_h_batch_set_space_order: instance %d: N = %d > %d with gamma < 1", i, b->hp[i].N, kSpaceMaxN);
    if (g != 1.0 && b->hp[i].N > maxN) maxN = b->hp[i].N;
  }
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  // new buffers first: on failure the batch keeps its previous configuration
  fh_dbuf nw, nv;
  int rc;
  if (maxN > 0 && ((rc = fh_alloc(ctx, nw, sizeof(double) * (size_t)b->Ptot)) ||
                   (rc = fh_alloc(ctx, nv, sizeof(double) * (size_t)b->Ptot))))
    return rc;
  std::swap(b->wsp.p, nw.p);
  std::swap(b->wsp.bytes, nw.bytes);
  std::swap(b->sV.p, nv.p);
  std::swap(b->sV.bytes, nv.bytes);
  for (int i = 0; i < b->n; ++i) {
    fh_h_dev_inst &I = b->di[i];
    const double g = gamma_host[i];
    I.spg = g;
    I.spA = g == 1.0 ? 0.0 : 1.0 - g;
    if (g == 1.0) {
      I.Dg = pow(I.dL, -2.0);
      I.kbf = 1.0;
    } else {
      // reset_D: mt_minimal.cpp:744-749 dL^(-1-gamma)/Gamma(2-gamma),
      // mt_psi_caputo.cpp:1176-1181 dL^-2/Gamma(2-gamma)
      I.Dg = (I.weights == FH_W_L1 ? pow(I.dL, -1.0 - g) : pow(I.dL, -2.0)) / tgamma(2.0 - g);
      // kb(gamma, i-1, i, i, dL) of one interval at distance 1 (psi = x)
      const double gtj = I.dL, v = (gtj / gtj) * pow(gtj, 1.0 - g);
      const double v4 = pow(fabs(1.0 - 0.0 / gtj), 1.0 - g), v3 = pow(fabs(1.0 - gtj / gtj), 1.0 - g);
      I.kbf = (-(v3 - v4) / (1.0 - g)) * v;
    }
  }
  b->space = maxN > 0;
  b->space_smem = sizeof(double) * 2 * (size_t)maxN;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(b->inst.p, b->di.data(), sizeof(fh_h_dev_inst) * b->n, cudaMemcpyHostToDevice,
                                   ctx->stream));
  if (b->space) {
    k_h_spw<<<dim3((unsigned)fh_ceil_div(maxN, 128), (unsigned)b->n), 128, 0, ctx->stream>>>(
        b->inst.as<fh_h_dev_inst>(), b->wsp.as<double>());
    if ((rc = fh_after_launch(ctx, "k_h_spw"))) return rc;
  }
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  b->graph.reset();
  return FH_OK;
}

// Mean time of two launches of the batch history sum over K layers (after one
// that warms up); history contents do not change it.
static int h_time_hist(fh_h_batch *b, int ti, int K, int cap, cudaEvent_t e0, cudaEvent_t e1, float *ms) {
  fh_ctx *ctx = b->ctx;
  int splits, kchunk;
  h_plan(b, ti, K, cap < b->max_splits ? cap : b->max_splits, &splits, &kchunk);
  *ms = 1e30f;
  if (!h_dp(b, K) && (size_t)kchunk * sizeof(double) > 48 * 1024) return FH_OK;
  float sum = 0.f;
  for (int rep = 0; rep < 3; ++rep) {
    cudaEventRecord(e0, ctx->stream);
    const int rc = h_hist(b, ti, K, splits, kchunk, b->W.as<double>(), ctx->stream);
    if (rc) return rc;
    cudaEventRecord(e1, ctx->stream);
    FH_CUDA_TRY(ctx, cudaEventSynchronize(e1));
    float t = 0.f;
    if (rep > 0) FH_CUDA_TRY(ctx, cudaEventElapsedTime(&t, e0, e1));
    sum += t;
  }
  *ms = sum / 2;
  return FH_OK;
}

// Times the batch history sum for the candidate launch shapes (tile CTA of
// 128/256/512 threads, K split cap 1/8/64) at a probe depth of
// min(max_steps - 1, 512) layers on the batch's own buffers and keeps the fastest.
// FP64 sums of kDpMin layers and more have no tile shape: theirs is chosen at the
// deepest sum that has one, the cap at the probe depth.
int fh_h_batch_autotune(fh_h_batch *b, float *best_ms) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, !ctx->capturing, FH_EINVAL, "fh_h_batch_autotune: not during a capture");
  FH_REQUIRE(ctx, b->mode != FH_H_BLOCKED, FH_EINVAL, "fh_h_batch_autotune: the blocked mode has no split history sum");
  const int K = b->max_steps - 1 < 512 ? b->max_steps - 1 : 512;
  if (K < 32) return FH_OK;
  static const int caps[3] = {1, 8, 64};
  cudaEvent_t e0, e1;
  FH_CUDA_TRY(ctx, cudaEventCreate(&e0));
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return fh_set_error(ctx, FH_ECUDA, "fh_h_batch_autotune: no event");
  }
  float best = 1e30f, ms;
  int rc = FH_OK, shape = tile_shape_index(b->tile_threads), cap = b->split_cap;
  auto search = [&](int depth, int t0, int t1, int c0, int c1) {
    best = 1e30f;
    for (int ti = t0; ti < t1 && !rc; ++ti)
      for (int ci = c0; ci < c1 && !rc; ++ci)
        if (!(rc = h_time_hist(b, ti, depth, caps[ci], e0, e1, &ms)) && ms < best) {
          best = ms;
          shape = ti;
          cap = caps[ci];
        }
  };
  if (h_dp(b, K)) {
    search(kDpMin - 1, 0, 3, 2, 3);
    search(K, shape, shape + 1, 0, 3);
  } else {
    search(K, 0, 3, 0, 3);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc) return rc;
  b->tile_threads = kTileShapes[shape];
  b->split_cap = cap;
  b->graph.reset();
  if (best_ms) *best_ms = best;
  return FH_OK;
}

int fh_h_batch_launch_shape(const fh_h_batch *b, int *tile_threads, int *split_cap) {
  if (!b) return FH_EINVAL;
  if (tile_threads) *tile_threads = b->tile_threads;
  if (split_cap) *split_cap = b->split_cap;
  return FH_OK;
}

int fh_h_batch_set_mode(fh_h_batch *b, int mode) {
  FH_REQUIRE(nullptr, b, FH_EINVAL, "null batch");
  fh_ctx *ctx = b->ctx;
  FH_REQUIRE(ctx, mode == FH_H_FP64 || mode == FH_H_DF64 || mode == FH_H_BLOCKED, FH_EINVAL,
             "fh_h_batch_set_mode: unknown mode %d", mode);
  FH_REQUIRE(ctx, b->nsaved == 0, FH_EINVAL, "fh_h_batch_set_mode: only before the first step");
  int rc;
  if (mode == FH_H_BLOCKED && !b->hb) {
    // the weight-plane grids have n (interpolated groups) and 8 n rows
    FH_REQUIRE(ctx, (long long)b->n * 8 <= 65535, FH_EINVAL,
               "fh_h_batch_set_mode: the blocked mode takes at most 8191 instances (%d)", b->n);
    // 128-point tiles of every instance's segment
    std::vector<long long> tp0;
    std::vector<int> tin, tnp;
    for (int i = 0; i < b->n; ++i) {
      const int seg = b->hp[i].N + 2;
      for (int k = 0; k < seg; k += 128) {
        tp0.push_back(b->off[i] + k);
        tin.push_back(i);
        tnp.push_back(seg - k < 128 ? seg - k : 128);
      }
    }
    const int kcap = (int)fh_ceil_div(b->max_steps, kSlcK) * kSlcK;
    std::vector<double> ct;
    hb_cheb_table(ct);
    b->hb = fh_hblk_new();
    if ((rc = fh_hblk_init(ctx, *b->hb, b->Ptot, kcap, b->n, tp0.data(), tin.data(), tnp.data(), (int)tp0.size())) ||
        (rc = fh_alloc(ctx, b->ring, sizeof(float2) * 128 * (size_t)b->Ptot)) ||
        (rc = fh_alloc(ctx, b->far, sizeof(float2) * kSlcK * (size_t)b->Ptot, false)) ||
        (rc = fh_alloc(ctx, b->wb, sizeof(double) * kNearRows * kNearLd * (size_t)b->n, false)) ||
        (rc = fh_alloc(ctx, b->wcb, sizeof(double) * kNearRows * (size_t)b->n, false)) ||
        (rc = fh_alloc(ctx, b->cheb, sizeof(double) * ct.size(), false)) ||
        (rc = cudaMemcpy(b->cheb.p, ct.data(), sizeof(double) * ct.size(), cudaMemcpyHostToDevice) != cudaSuccess
                  ? fh_set_error(ctx, FH_ECUDA, "fh_h_batch_set_mode: upload of the interpolation tables failed")
                  : FH_OK)) {
      fh_hblk_delete(b->hb);
      b->hb = nullptr;
      b->ring.release();
      b->far.release();
      b->cheb.release();
      b->wb.release();
      b->wcb.release();
      return rc;
    }
    b->D.release();  // the full-precision history is not kept in this mode
  }
  if (mode != FH_H_BLOCKED && b->hb) {
    fh_hblk_delete(b->hb);
    b->hb = nullptr;
    b->ring.release();
    b->far.release();
    b->cheb.release();
    b->wb.release();
    b->wcb.release();
    if ((rc = fh_alloc(ctx, b->D, sizeof(double) * (size_t)b->Ptot * (size_t)b->max_steps))) return rc;
  }
  b->mode = mode;
  b->graph.reset();
  return FH_OK;
}

}  // extern "C"
