// fh_far64.cu -- S[n][p] = sum_{k < K} w_n(k) D[k][p] for 64 weight rows at FP64
// accuracy on the tensor cores: the layers before a block of future steps,
// contracted once for all its steps instead of once per step.
//
// Why: one FP64 warp instruction takes an SM 17 cycles on GB300, so a history
// sum on the FP64 pipe stops at 2.4 TB/s (two sums per 8-byte difference), and
// in double-float at HBM speed it still reads every layer every step.  A block
// of 32 steps x 2 half-step rows reads each layer once.
//
// Exact products (Ozaki, Ogita, Oishi, Rump 2012, with bf16 digits): per point
// and group of 128 layers a power of two scales the values below 2^6, and a
// value is cut into seven balanced base-256 digits, x = 2^E sum_i a_i 256^-i
// with integers |a_i| <= 128, which bf16 holds exactly; weights per row and
// group likewise.  The cut is at 2^-55 of the group's largest value, half the
// last place of an FP64 number of that size; the error of a group's sum is
// relative to its largest value times its largest weight.  Weights of the newest
// lags are up to 2^11 times those 128 layers back (alpha 0.95), so in each row and
// group those above 2^kSpread times the least take FP64 FMAs instead
// (k_far64_fix), as in fh_dp.cuh: a group whose values fall like k^-1 then comes
// out within ~1e-15 of the sum of its terms' magnitudes (k^-2: ~6e-15; FMAs 5e-16;
// without the rule 1e-13 and 8e-13 at alpha 0.95).  Every product a_i b_j is an
// integer <= 2^14 and a level sum (i + j = l, at most seven products a layer,
// 128 layers) stays below 2^24: exact in the FP32 accumulators.  Levels 0..6
// are kept (28 of 49 products; level 7 starts at 2^-56 of the largest
// product).  The epilogue turns the seven level sums into an unevaluated sum of
// three FP32 numbers, scales it by 2^(Ed + Ew) and adds it to a three-word
// running sum (72 bits), so groups of very different size add up without loss;
// one rounding to FP64 (or to an (hi, lo) pair) at the end.
//
// Digits without floating point: with w = v + 0x8080...80 (v the value as a
// 64-bit integer, top digit in the top byte) the balanced digits are the bytes
// of w minus 128, and bf16(byte - 128) = bf16(128 + (byte & 127)) - bf16(128 or
// 256): per pair of layers and digit one byte permute, two logical operations
// and one packed subtraction.
//
// One CTA of 512 threads per 128 points (and K split when there are few
// points).  A = 128 points x 64 layers in seven K-major planes which the CTA
// cuts itself from the stored layers, half (32 layers) by half, so that the
// MMAs of one half run while the next is cut; B = the 64-layer image of the
// weight digits, 7 digits x 32 rows stacked per row group, copied in bulk two
// chunks ahead.  The MMA of data digit ia takes the first 7 - ia weight digits
// (N = 32 (7 - ia)) and writes TMEM columns from 32 ia of its row group: the
// product (ia, ib) lands on level ia + ib.  Thread t cuts eight layers of point
// t & 127 and holds in the epilogue the sums of that point for 16 rows.  The
// cutting (~45 instructions per value) and the sums (~60 per row, point and
// group) take about as long as the MMAs; sixteen warps keep both going (eight,
// with twice the registers: 77k cycles per tile of 256 layers at 0.31
// instructions per cycle and scheduler).
// Waits are bounded; on expiry *err is set and nothing is stored.
//
// Measured, whole solves, before and now (with the sweeps' changes since): 2D 251 x
// 187, 500 steps, FP64 34.9 -> 12.1 ms (the sums of a step 49 -> ~9 us); 512 x
// 512, 500 steps, DF64 65.1 -> 25.4 ms; one line of 1024 nodes, 2500 steps, FP64
// 55.0 -> 12.1 ms with the resident solve of fh_ab.cu.  The results differ from the
// FP64 sums' by 1e-16 (relative).  A layer that is not finite makes its point's rows
// NaN, as it makes the point's own field one step later.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "fh_common.cuh"
#include "fh_df.cuh"
#include "fh_far64.h"
#include "fh_slices.cuh"
#include "fh_sm100.cuh"

namespace {
constexpr int kSl = 7;                         // digits per value
constexpr int kPts = 128;                      // points per CTA
constexpr int kThr = 512;
constexpr int kLay = 32 * kPts / kThr;         // layers of a half a thread cuts
constexpr int kRows = kF64Rows * kPts / kThr;  // rows a thread sums
constexpr int kGroup = 128;                    // layers of a group (one exponent)
constexpr uint32_t kPlane = kPts * 128;        // one digit of 128 points x 64 layers
constexpr uint32_t kABytes = kSl * kPlane;
constexpr uint32_t kBRows = 32;                // weight rows of a row group
constexpr uint32_t kBTile = kBRows * 128;      // one digit of a row group x 64 layers
constexpr uint32_t kBGroup = kSl * kBTile;
constexpr uint32_t kBBytes = 2 * kBGroup;      // a chunk's weight image (56 KiB)
constexpr uint32_t kLevCols = kSl * kBRows;    // TMEM columns of a row group
constexpr size_t kSmem = 1024 + kABytes + 2 * kBBytes + 64;
constexpr int kNonFinite = 0x7ff;
constexpr int kSpread = 3;                     // exponents of a row's weights in a group: the rest by FMAs
constexpr int kRowBlock = 8;                   // rows of a CTA that cuts weights
constexpr int kFixRows = 16;                   // rows of a CTA of k_far64_fix
static_assert(kLay == 8 && kRows == 16, "one 16-byte digit store per thread and half, two threads per row group");
}  // namespace

// ------------------------------------------------------------------ digits
// 64-bit digit word of x 2^-E, E from the group's largest biased exponent
// emax: digit i is byte 7 - i minus 128.
__device__ __forceinline__ unsigned long long f64_word(double x, int emax) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (hi >> 20) & 0x7ff;
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo;
  m = e == 0 ? 0ull : (m << 9) >> min(emax - e, 63);
  const unsigned long long sg = (long long)(int)hi >> 63;
  return (m ^ sg) - sg + 0x8080808080808080ull;
}
// The same for an (hi, lo) FP32 pair (emax still a double's biased exponent).
__device__ __forceinline__ unsigned long long f64_part(float x, int emax) {
  const unsigned b = __float_as_uint(x);
  const int e = (int)((b >> 23) & 0xff) + (1023 - 127);
  unsigned long long m = (unsigned long long)((b & 0x7fffffu) | 0x800000u) << 38;
  m = (b & 0x7f800000u) == 0 ? 0ull : m >> min(emax - e, 63);
  const unsigned long long sg = (long long)(int)b >> 63;
  return (m ^ sg) - sg;
}
__device__ __forceinline__ unsigned long long f64_word(float2 x, int emax) {
  return f64_part(x.x, emax) + f64_part(x.y, emax) + 0x8080808080808080ull;
}
// Biased exponent of the largest magnitude; 0x7ff when not finite.
__device__ __forceinline__ int f64_exp(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ int f64_exp(float2 x) {
  const int e = (__float_as_uint(x.x) >> 23) & 0xff;
  return e == 0xff || ((__float_as_uint(x.y) >> 23) & 0xff) == 0xff ? kNonFinite : e ? e + (1023 - 127) : 0;
}
// Digit i of two words as a bf16 pair (first word in the low half).
__device__ __forceinline__ uint32_t f64_digits(unsigned long long a, unsigned long long b, int i) {
  const int by = 7 - i;  // compile-time
  const uint32_t wa = by >= 4 ? (uint32_t)(a >> 32) : (uint32_t)a, wb = by >= 4 ? (uint32_t)(b >> 32) : (uint32_t)b;
  const uint32_t bb = __byte_perm(wa, wb, ((by & 3) + 4) << 8 | (by & 3));
  const uint32_t x = (bb & 0x007f007fu) | 0x43004300u, y = (bb & 0x00800080u) ^ 0x43804380u;
  const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&x), *reinterpret_cast<const __nv_bfloat162 *>(&y));
  return *reinterpret_cast<const uint32_t *>(&d);
}

// Exponents of layers [k0, k0 + 32) into the group's row of ed (the first
// layers of a group overwrite it).
template <class S>
__global__ void __launch_bounds__(256) k_far64_exp(const S *__restrict__ D, long long ldd, long long P, int k0,
                                                   int16_t *__restrict__ ed, long long lde) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  int e = 0;
#pragma unroll 8
  for (int k = 0; k < kF64Block; ++k) e = max(e, f64_exp(D[(long long)(k0 + k) * ldd + p]));
  int16_t *q = ed + (long long)(k0 / kGroup) * lde + p;
  if (k0 % kGroup) e = max(e, (int)*q);
  *q = (int16_t)e;
}

// Where row n, layer k of the weights stands: as fh_far64_weights and
// fh_far64_weights_lag take them.
struct f64_src {
  const double *w;
  long long row_step, ldw;
  int base, nrows;
  bool lag;
  __device__ __forceinline__ double at(int n, int k) const {
    if (n >= nrows) return 0.0;
    return lag ? w[base + n - k] : w[(long long)(n >> 1) * row_step + (long long)(n & 1) * ldw + k];
  }
};

// Weight digits of row n (one warp) in group G: image byte of (row group g,
// digit i, row r of the group, layer k of the chunk) at
// chunk * kBBytes + g * kBGroup + i * kBTile + fh_sw128_off(r, k).  Weights above
// 2^kSpread times the row's least are left out of the digits: bit `lane` of word
// h of hv[G][n] is layer 4 lane + h; hany[G][n / kRowBlock]: any in those rows.
__global__ void __launch_bounds__(32 * kRowBlock) k_far64_wrows(int K, const f64_src src, uint8_t *__restrict__ img,
                                                                int16_t *__restrict__ ew, uint4 *__restrict__ hv,
                                                                int *__restrict__ hany) {
  const int n = blockIdx.y * kRowBlock + (threadIdx.x >> 5), G = blockIdx.x, lane = threadIdx.x & 31;
  double w[4];
  int lo = kNonFinite;
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const int k = G * kGroup + 4 * lane + h;
    w[h] = k < K ? src.at(n, k) : 0.0;
    if (w[h] != 0.0) lo = min(lo, f64_exp(w[h]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
  int e = 0;
  uint32_t hm[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    const bool heavy = f64_exp(w[h]) > lo + kSpread;
    hm[h] = __ballot_sync(0xffffffffu, heavy);
    if (heavy) w[h] = 0.0;
    e = max(e, f64_exp(w[h]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  const uint32_t any = hm[0] | hm[1] | hm[2] | hm[3];
  if (lane == 0) {
    ew[(long long)G * kF64Rows + n] = (int16_t)e;
    hv[(long long)G * kF64Rows + n] = make_uint4(hm[0], hm[1], hm[2], hm[3]);
  }
  const int blk = __syncthreads_or(any != 0);
  if (threadIdx.x == 0) hany[G * (kF64Rows / kRowBlock) + blockIdx.y] = blk;
  unsigned long long q[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) q[h] = f64_word(w[h], e);
  const int k = 4 * lane, c = 2 * G + (k >> 6);
  if (c * 64 >= K) return;
  uint8_t *dst = img + (size_t)c * kBBytes + (size_t)(n >> 5) * kBGroup + fh_sw128_off(n & 31, k & 63);
#pragma unroll
  for (int i = 0; i < kSl; ++i)
    *reinterpret_cast<uint2 *>(dst + i * kBTile) = make_uint2(f64_digits(q[0], q[1], i), f64_digits(q[2], q[3], i));
}

// --------------------------------------------------------------- contraction
__device__ __forceinline__ void f64_two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
// A normal float's value as a double, by its bits (conversions run on the FP64 pipe).
__device__ __forceinline__ double f64_of(float x) {
  const unsigned b = __float_as_uint(x);
  if ((b & 0x7f800000u) == 0) return 0.0;
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
}
// x 2^e (e far from the limits of int); 0 below the normal range, infinite above.
__device__ __forceinline__ double f64_scale(double x, int e) {
  const int hi = __double2hiint(x), ex = (hi >> 20) & 0x7ff, en = ex + e;
  if (ex == 0 || en <= 0) return 0.0;
  if (en >= 0x7ff) return __hiloint2double((hi & 0x80000000) | 0x7ff00000, 0);
  return __hiloint2double(hi + (e << 20), __double2loint(x));
}
__device__ __forceinline__ void f64_store(double *o, float s0, float s1, float s2, int e, bool bad) {
  *o = bad ? __hiloint2double(0x7ff80000, 0) : f64_scale(f64_of(s0) + (f64_of(s1) + f64_of(s2)), e);
}
__device__ __forceinline__ float f64_scalef(float x, int e) {  // |e| up to ~2^10, in two steps
  const int a = max(-126, min(127, e)), b = max(-126, min(127, e - a));
  return x * fh_exp2f_int(a) * fh_exp2f_int(b);
}
__device__ __forceinline__ void f64_store(float2 *o, float s0, float s1, float s2, int e, bool bad) {
  float h0, l0;  // s1 may be far above the last place of s0 (cancelling level sums)
  f64_two_sum(s0, s1, h0, l0);
  const float t = l0 + s2, h = h0 + t;
  float2 v = make_float2(f64_scalef(h, e), f64_scalef(t - (h - h0), e));
  if (bad) v = make_float2(__int_as_float(0x7fc00000), 0.f);
  *o = v;
}

template <class S>
__global__ void __launch_bounds__(kThr, 1)
    k_far64(const S *__restrict__ D, long long ldd, long long P, int K, const uint8_t *__restrict__ img,
            const int16_t *__restrict__ ew, const int16_t *__restrict__ ed, long long lde, int gps,
            S *__restrict__ out, long long ldo, int *__restrict__ err) {
  extern __shared__ uint8_t f64_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t raw = fh_smem_u32(f64_raw);
  const uint32_t sA = (raw + 1023u) & ~1023u;
  uint8_t *gA = f64_raw + (sA - raw);
  const uint32_t sB = sA + kABytes, bars = sB + 2 * kBBytes;
  const uint32_t mdone = bars, bfull = bars + 16, tslot = bars + 32;  // two mbarriers each
  volatile uint32_t *tslot_g = reinterpret_cast<volatile uint32_t *>(gA + kABytes + 2 * kBBytes + 32);
  const int pt = tid & 127, q = tid >> 7;
  const long long p = (long long)blockIdx.x * kPts + pt;
  const bool live = p < P;
  // the thread's rows: [16 q, 16 q + 16), columns of their row group
  const uint32_t rcol = (uint32_t)(q >> 1) * kLevCols + (uint32_t)(q & 1) * kRows;
  const int ng = (K + kGroup - 1) / kGroup;
  const int G0 = min(ng, (int)blockIdx.y * gps), G1 = min(ng, G0 + gps);
  const int h0 = 4 * G0, h1 = min(K / 32, 4 * G1);  // halves: 32 layers each
  const int c1 = (h1 + 1) / 2;                      // chunks end
  out += (long long)blockIdx.y * kF64Rows * ldo;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      fh_mbar_init(mdone + 8 * i, 1);
      fh_mbar_init(bfull + 8 * i, 1);
    }
    fh_fence_mbar_init();
  }
  if (warp == 0) {
    fh_tmem_alloc(tslot, 512);
    fh_tmem_relinquish();
  }
  // largest exponents of the point and of row 16 q + lane % 16
  int eb = 1, wb = 1;
  bool bad = false;
  for (int g = G0; g < G1; ++g) {
    const int e = live ? ed[(long long)g * lde + p] : 0, w = ew[(long long)g * kF64Rows + kRows * q + lane % kRows];
    bad |= e == kNonFinite;
    eb = max(eb, e);
    wb = max(wb, w);
  }
  fh_tc_fence_before();
  __syncthreads();
  fh_tc_fence_after();
  const uint32_t tmem = *tslot_g;
  int last_c = -1, last_i = -1;  // thread 0: the last chunk copied, the last half committed
  auto load_b = [&](int c) {  // chunk c's weight image (thread 0)
    last_c = c - 2 * G0;
    const int b = last_c & 1;
    fh_mbar_arrive_expect_tx(bfull + 8 * b, kBBytes);
    fh_bulk_load(sB + b * kBBytes, img + (size_t)c * kBBytes, kBBytes, bfull + 8 * b);
  };
  if (tid == 0)
    for (int c = 2 * G0; c < min(c1, 2 * G0 + 2); ++c) load_b(c);
  // the thread's layers of a half: [8 q, 8 q + 8)
  S v[kLay];
  auto load_v = [&](int h) {
    const S *d = D + (long long)(32 * h + kLay * q) * ldd + (live ? p : 0);
#pragma unroll
    for (int i = 0; i < kLay; ++i) v[i] = __ldcs(d + i * ldd);
  };
  float s0[kRows], s1[kRows], s2[kRows];
#pragma unroll
  for (int n = 0; n < kRows; ++n) s0[n] = s1[n] = s2[n] = 0.f;
  // level sums of group G into the running sums
  auto epilogue = [&](int G) {
    const int e = (live ? (int)ed[(long long)G * lde + p] : 0) - eb;
    const int w = ew[(long long)G * kF64Rows + kRows * q + lane % kRows] - wb;
    const uint32_t cols = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + rcol;
#pragma unroll
    for (int nb = 0; nb < kRows; nb += 4) {
      float L[kSl][4];
#pragma unroll
      for (int l = 0; l < kSl; ++l) fh_tmem_ld4(cols + (uint32_t)(kBRows * l + nb), L[l]);
      fh_tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float sc = fh_exp2i(e + __shfl_sync(0xffffffffu, w, nb + i));
        float h, e1, m, e2, u, e3, a, b, c;
        f64_two_sum(L[0][i], L[1][i] * 0x1p-8f, h, e1);
        f64_two_sum(L[2][i], L[3][i] * 0x1p-8f, m, e2);
        const float lo = fmaf(L[6][i], 0x1p-16f, fmaf(L[5][i], 0x1p-8f, L[4][i]));
        f64_two_sum(e1, m * 0x1p-16f, u, e3);
        const float r = e3 + fmaf(e2, 0x1p-16f, lo * 0x1p-32f);
        f64_two_sum(s0[nb + i], h * sc, s0[nb + i], a);
        f64_two_sum(s1[nb + i], u * sc, u, b);
        f64_two_sum(u, a, s1[nb + i], c);
        s2[nb + i] += fmaf(r, sc, b + c);
      }
    }
  };
  bool ok = true;
  if (h1 > h0) load_v(h0);
  for (int h = h0; h < h1; ++h) {
    const int i = h - h0, slot = i & 1;
    if (i >= 2) ok &= fh_mbar_wait(mdone + 8 * slot, ((i >> 1) - 1) & 1);  // the slot's last MMAs
    // both halves of the chunk before the last are consumed: its buffer takes the next chunk
    if (tid == 0 && slot == 1 && i >= 2 && (h >> 1) + 1 < c1) load_b((h >> 1) + 1);
    const int emax = live ? max((int)ed[(long long)(h >> 2) * lde + p], 1) : 1;
    const bool cut = live && emax != kNonFinite;
    {
      unsigned long long w[kLay];
#pragma unroll
      for (int j = 0; j < kLay; ++j) w[j] = cut ? f64_word(v[j], emax) : 0x8080808080808080ull;
      const uint32_t off = fh_sw128_off(pt, 32 * slot + kLay * q);
#pragma unroll
      for (int d = 0; d < kSl; ++d)
        *reinterpret_cast<uint4 *>(gA + d * kPlane + off) =
            make_uint4(f64_digits(w[0], w[1], d), f64_digits(w[2], w[3], d), f64_digits(w[4], w[5], d),
                       f64_digits(w[6], w[7], d));
    }
    if (h + 1 < h1) load_v(h + 1);
    fh_fence_proxy_async_smem();
    if (i > 0 && (i & 3) == 0) {  // a new group: the last one's sums out of TMEM first
      ok &= fh_mbar_wait(mdone + 8 * (slot ^ 1), ((i - 1) >> 1) & 1);
      fh_tc_fence_after();
      epilogue((h >> 2) - 1);
    }
    fh_tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (tid == 0) {
      fh_tc_fence_after();
      const int b = (i >> 1) & 1;
      ok = fh_mbar_wait(bfull + 8 * b, (i >> 2) & 1);
      if (ok) {
#pragma unroll
        for (int kk = 2 * slot, n = 0; n < 2; ++n, ++kk)
#pragma unroll
          for (int g = 0; g < 2; ++g)
#pragma unroll
            for (int d = 0; d < kSl; ++d)
              fh_mma_bf16(tmem + (uint32_t)g * kLevCols + (uint32_t)d * kBRows,
                          fh_desc_kmajor_sw128(sA + d * kPlane + kk * 32),
                          fh_desc_kmajor_sw128(sB + b * kBBytes + g * kBGroup + kk * 32),
                          fh_idesc_bf16_f32(128, (kSl - d) * kBRows), (d > 0 || n > 0 || (i & 3)) ? 1u : 0u);
        fh_mma_commit(mdone + 8 * slot);
        last_i = i;
      }
    }
    __syncwarp();
  }
  if (h1 > h0) {
    const int i = h1 - 1 - h0;
    if (ok) ok = fh_mbar_wait(mdone + 8 * (i & 1), (i >> 1) & 1);
    fh_tc_fence_after();
    ok = __syncthreads_and(ok);
    if (ok) epilogue((h1 - 1) >> 2);
  }
  if (!ok && tid == 0) {  // after an expired wait: the copies and MMAs still in flight, bounded too
    if (last_c >= 0) fh_mbar_wait(bfull + 8 * (last_c & 1), (last_c >> 1) & 1);
    if (last_i >= 0) fh_mbar_wait(mdone + 8 * (last_i & 1), (last_i >> 1) & 1);
  }
  if (ok) {
    S *o = out + (long long)(kRows * q) * ldo + p;
#pragma unroll
    for (int n = 0; n < kRows; ++n) {
      const int w = __shfl_sync(0xffffffffu, wb, n);
      // unit of digit 0: 2^(exponent - 1028) each
      if (live) f64_store(o + n * ldo, s0[n], s1[n], s2[n], eb + w - 2 * 1028, bad || w == kNonFinite);
    }
  }
  if (!ok && tid == 0) atomicOr(err, 1);
  fh_tc_fence_before();
  __syncthreads();
  if (warp == 0) fh_tmem_dealloc(tmem, 512);
}

// out[i] = sum over splits of part[s][i], in split order
__global__ void __launch_bounds__(256) k_far64_reduce(const double *__restrict__ part, int splits, long long n,
                                                      double *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double a = part[i];
  for (int s = 1; s < splits; ++s) a += part[(long long)s * n + i];
  out[i] = a;
}
__global__ void __launch_bounds__(256) k_far64_reduce(const float2 *__restrict__ part, int splits, long long n,
                                                      float2 *__restrict__ out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fh_df a = fh_df_from_pair(part[i]);
  for (int s = 1; s < splits; ++s) a = fh_df_add(a, fh_df_from_pair(part[(long long)s * n + i]));
  out[i] = fh_df_pair(a);
}

// Adds the layers that a row's digits leave out (hv), in FP64: thread = one
// point, rows [16 y, 16 y + 16).  psi = t, alpha 0.7: 4 layers of the first row, none
// from the fifth step on; alpha 0.95: 7 to 11 layers of the first sixteen steps.
__device__ __forceinline__ double f64_value(double x) { return x; }
__device__ __forceinline__ double f64_value(float2 x) { return (double)x.x + (double)x.y; }
__device__ __forceinline__ void f64_add(double *o, double x) { *o += x; }
__device__ __forceinline__ void f64_add(float2 *o, double x) {
  *o = fh_df_pair(fh_df_add(fh_df_from_pair(*o), fh_df_from_double(x)));
}
template <class S>
__global__ void __launch_bounds__(256) k_far64_fix(const S *__restrict__ D, long long ldd, long long P, int K,
                                                   const f64_src src, const uint4 *__restrict__ hv,
                                                   const int *__restrict__ hany, S *__restrict__ out, long long ldo) {
  __shared__ double sw[kGroup][kFixRows];
  __shared__ uint32_t un[4];
  const int n0 = blockIdx.y * kFixRows, ng = (K + kGroup - 1) / kGroup, t = threadIdx.x;
  const long long p = (long long)blockIdx.x * blockDim.x + t;
  double acc[kFixRows] = {};
  bool any = false;
  uint32_t gm = 0;  // groups with such layers among 32
  for (int G = 0; G < ng; ++G) {
    if (G % 32 == 0) {
      const int g = G + (t & 31);
      const int *ha = hany + g * (kF64Rows / kRowBlock) + n0 / kRowBlock;
      gm = __ballot_sync(0xffffffffu, g < ng && (ha[0] | ha[1]));
    }
    if (!(gm >> (G % 32) & 1u)) continue;  // every thread of the CTA
    any = true;
    __syncthreads();
    if (t < 4) un[t] = 0;
    __syncthreads();
    for (int i = t; i < kFixRows * kGroup; i += blockDim.x) {
      const int n = i / kGroup, k = i % kGroup;
      const uint4 m = hv[(long long)G * kF64Rows + n0 + n];
      const uint32_t mh = (k & 3) == 0 ? m.x : (k & 3) == 1 ? m.y : (k & 3) == 2 ? m.z : m.w;
      const bool heavy = mh >> (k >> 2) & 1u;
      sw[k][n] = heavy ? src.at(n0 + n, G * kGroup + k) : 0.0;
      if (heavy) atomicOr(&un[k >> 5], 1u << (k & 31));
    }
    __syncthreads();
    if (p < P) {
      const S *d = D + (long long)G * kGroup * ldd + p;
      for (int q = 0; q < 4; ++q)
        for (uint32_t m = un[q]; m; m &= m - 1) {
          const int k = 32 * q + __ffs(m) - 1;
          const double x = f64_value(__ldcs(d + k * ldd));
#pragma unroll
          for (int n = 0; n < kFixRows; ++n) {
            const double w = sw[k][n];
            if (w != 0.0) acc[n] = fma(w, x, acc[n]);
          }
        }
    }
  }
  if (!any || p >= P) return;
#pragma unroll
  for (int n = 0; n < kFixRows; ++n)
    if (acc[n] != 0.0) f64_add(out + (long long)(n0 + n) * ldo + p, acc[n]);
}

// -------------------------------------------------------------------- host
struct fh_far64 {
  long long P = 0, ld = 0;  // ld: points rounded up to whole tiles
  int Kcap = 0;
  bool df = false;
  int nsm = 1, max_splits = 1;
  fh_dbuf img, ew, ed, rows, part, hv, hany, err;
  f64_src src = {};  // of the weights in img
};

namespace {
constexpr int kMaxSplits = 8;
// Splits of K: when the tiles alone leave SMs idle.
int splits_for(long long P, int nsm) {
  const long long tiles = fh_ceil_div(P, kPts);
  return (int)std::max(1LL, std::min((long long)kMaxSplits, nsm / tiles));
}
void sizes(long long P, int Kcap, int splits, size_t (&b)[7]) {
  const long long ld = fh_ceil_div(P, kPts) * kPts;
  const size_t ng = (size_t)fh_ceil_div(Kcap, kGroup);
  b[0] = ng * 2 * kBBytes;
  b[1] = ng * kF64Rows * 2;
  b[2] = ng * (size_t)ld * 2;
  b[3] = 8 * kF64Rows * (size_t)ld;
  b[4] = splits > 1 ? splits * b[3] : 0;
  b[5] = ng * kF64Rows * sizeof(uint4);
  b[6] = ng * (kF64Rows / kRowBlock) * sizeof(int);
}
}  // namespace

int fh_far64_create(fh_ctx *ctx, long long P, int Kcap, bool df, fh_far64 **out) {
  *out = nullptr;
  fh_far64 *f = new fh_far64();
  f->P = P;
  f->ld = fh_ceil_div(P, kPts) * kPts;
  f->Kcap = Kcap;
  f->df = df;
  int nsm = 0;
  if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, ctx->device) == cudaSuccess && nsm > 0) f->nsm = nsm;
  f->max_splits = splits_for(P, f->nsm);
  size_t b[7];
  sizes(P, Kcap, f->max_splits, b);
  int rc;
  if ((rc = fh_alloc(ctx, f->img, b[0])) || (rc = fh_alloc(ctx, f->ew, b[1])) || (rc = fh_alloc(ctx, f->ed, b[2])) ||
      (rc = fh_alloc(ctx, f->rows, b[3], false)) || (b[4] && (rc = fh_alloc(ctx, f->part, b[4], false))) ||
      (rc = fh_alloc(ctx, f->hv, b[5], false)) || (rc = fh_alloc(ctx, f->hany, b[6], false)) ||
      (rc = fh_alloc(ctx, f->err, sizeof(int)))) {
    delete f;
    return rc;
  }
  auto at = cudaFuncAttributeMaxDynamicSharedMemorySize;
  const cudaError_t e = df ? cudaFuncSetAttribute(k_far64<float2>, at, (int)kSmem)
                           : cudaFuncSetAttribute(k_far64<double>, at, (int)kSmem);
  if (e != cudaSuccess) {
    delete f;
    return fh_set_error(ctx, FH_ECUDA, "fh_far64_create: %s", cudaGetErrorString(e));
  }
  *out = f;
  return FH_OK;
}
void fh_far64_delete(fh_far64 *f) { delete f; }
size_t fh_far64_bytes(const fh_far64 &f) {
  return f.img.bytes + f.ew.bytes + f.ed.bytes + f.rows.bytes + f.part.bytes + f.hv.bytes + f.hany.bytes +
         f.err.bytes;
}
long long fh_far64_pitch(const fh_far64 &f) { return f.ld; }
const void *fh_far64_rows(const fh_far64 &f) { return f.rows.p; }

int fh_far64_append(fh_ctx *ctx, fh_far64 &f, const void *D, long long ldd, int k0) {
  FH_REQUIRE(ctx, k0 >= 0 && k0 % kF64Block == 0 && k0 + kF64Block <= f.Kcap, FH_EINVAL, "fh_far64_append: layer %d", k0);
  const unsigned g = (unsigned)fh_ceil_div(f.P, 256);
  if (f.df)
    k_far64_exp<<<g, 256, 0, ctx->stream>>>(static_cast<const float2 *>(D), ldd, f.P, k0, f.ed.as<int16_t>(), f.ld);
  else
    k_far64_exp<<<g, 256, 0, ctx->stream>>>(static_cast<const double *>(D), ldd, f.P, k0, f.ed.as<int16_t>(), f.ld);
  return fh_after_launch(ctx, "k_far64_exp");
}

static int far64_wrows(fh_ctx *ctx, fh_far64 &f, int K, const f64_src &src) {
  f.src = src;
  k_far64_wrows<<<dim3((unsigned)fh_ceil_div(K, kGroup), kF64Rows / kRowBlock), 32 * kRowBlock, 0, ctx->stream>>>(
      K, src, f.img.as<uint8_t>(), f.ew.as<int16_t>(), f.hv.as<uint4>(), f.hany.as<int>());
  return fh_after_launch(ctx, "k_far64_wrows");
}
int fh_far64_weights(fh_ctx *ctx, fh_far64 &f, int K, const double *W, long long row_step, long long ldw, int nrows) {
  return far64_wrows(ctx, f, K, f64_src{W, row_step, ldw, 0, nrows, false});
}
int fh_far64_weights_lag(fh_ctx *ctx, fh_far64 &f, int K, const double *lag, int base, int nrows) {
  return far64_wrows(ctx, f, K, f64_src{lag, 0, 0, base, nrows, true});
}

int fh_far64_run(fh_ctx *ctx, fh_far64 &f, const void *D, long long ldd, int K) {
  FH_REQUIRE(ctx, K >= kF64Block && K % kF64Block == 0 && K <= f.Kcap, FH_EINVAL, "fh_far64_run: K = %d", K);
  const int ng = (int)fh_ceil_div(K, kGroup);
  const int gps = (int)fh_ceil_div(ng, std::min(f.max_splits, ng)), splits = (int)fh_ceil_div(ng, gps);
  const dim3 grid((unsigned)(f.ld / kPts), (unsigned)splits);
  const long long n = kF64Rows * f.ld;
  auto go = [&](auto *d) {
    using S = std::remove_const_t<std::remove_pointer_t<decltype(d)>>;
    S *o = splits > 1 ? f.part.as<S>() : f.rows.as<S>();
    k_far64<S><<<grid, kThr, kSmem, ctx->stream>>>(d, ldd, f.P, K, f.img.as<uint8_t>(), f.ew.as<int16_t>(),
                                                   f.ed.as<int16_t>(), f.ld, gps, o, f.ld, f.err.as<int>());
    int rc = fh_after_launch(ctx, "k_far64");
    if (rc) return rc;
    if (splits > 1) {
      k_far64_reduce<<<(unsigned)fh_ceil_div(n, 256), 256, 0, ctx->stream>>>(f.part.as<S>(), splits, n, f.rows.as<S>());
      if ((rc = fh_after_launch(ctx, "k_far64_reduce"))) return rc;
    }
    k_far64_fix<S><<<dim3((unsigned)fh_ceil_div(f.P, 256), kF64Rows / kFixRows), 256, 0, ctx->stream>>>(
        d, ldd, f.P, K, f.src, f.hv.as<uint4>(), f.hany.as<int>(), f.rows.as<S>(), f.ld);
    return fh_after_launch(ctx, "k_far64_fix");
  };
  fh_prof_mark(ctx, FH_PROF_GEMM, false);
  const int rc = f.df ? go(static_cast<const float2 *>(D)) : go(static_cast<const double *>(D));
  fh_prof_mark(ctx, FH_PROF_GEMM, true);
  return rc;
}

int fh_far64_check(fh_ctx *ctx, const fh_far64 &f) {
  int h = 0;
  FH_CUDA_TRY(ctx, cudaMemcpyAsync(&h, f.err.p, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  FH_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  FH_REQUIRE(ctx, h == 0, FH_ETIMEOUT, "history contraction: a device wait ran out");
  return FH_OK;
}
int fh_far64_mark(fh_ctx *ctx, const fh_far64 &f, int expired) {
  FH_CUDA_TRY(ctx, cudaMemsetAsync(f.err.p, expired, sizeof(int), ctx->stream));
  return FH_OK;
}
