// fh_dp.cuh -- FP64-accurate history sums by exact integer dot products
// (k_hist_dp in fh_history.cu, k_hist_tiles_dp in fh_h.cu).
#pragma once
#include <stdint.h>

#include "fh_common.cuh"

// The sums of K >= kDpMin layers by exact integer products on the integer pipe
// (four-way byte dot products): one FP64 warp instruction takes an SM 17
// cycles, so M FMAs per 8-byte value stop plain sums at 2.4 TB/s (M = 2) and
// 4.7 TB/s (M = 1).  Ozaki's splitting (Ozaki, Ogita, Oishi, Rump 2012) as in
// fh_far64.cu, here with byte digits: per point and group of 16 layers a value
// is cut into eight balanced base-256 digits below the group's largest exponent
// (the last ends 2^-63 below it), weights per row and group likewise; the digit
// products of level i + j <= 7 are summed exactly in 32 bits, a group's eight
// level sums make one number of ~60 bits, rounded to FP64 and added to the
// running sum: two roundings per group instead of sixteen.  ~42 instructions
// per value and pair of rows, almost half of them dot products.  (Seven digits
// and levels 223 us below, but 2^-53 of a group's largest product is cut, and
// the error against extended precision was 4.8e-16, that of the FMAs 3.0e-16.)
//
// A digit is cut relative to the largest value and the largest weight of its
// group, so a group whose weights' exponents differ by more than kDpSpread
// (the few newest layers of an L1-like history) takes FP64 FMAs, as does a
// point whose values are not finite or too small for the digits' scale.
//
// Measured, 777 layers x 148,996 points: M = 2 392 -> 246 us, M = 1 203 -> 168
// us; 64 layers x 2000 points, M = 2, 16.5 -> 10.4 us.  Bound by the integer
// and the FMA pipe, which run at half the issue rate (0.62 instructions per
// cycle and scheduler, 53 % HBM at M = 2, 82 % at M = 1); the next group's
// loads issued between this one's work gained nothing, two points per thread
// lost up to 30 % on small sums.
static constexpr int kDpThreads = 128;  // one point each
static constexpr int kDpMin = 64;       // fewer layers: plain FMAs
static constexpr int kDpGroup = 16;     // layers of a group
static constexpr int kDpStage = 512;    // layers whose weight digits are in shared memory at a time
static constexpr int kDpSpread = 3;
static constexpr int kDpDigits = 8;  // and levels
// Of a group's four quads of layers the last dp_fma(M) take FP64 FMAs, issued
// between the integer work of the others (M = 1: 200 us above without, 175
// with one quad; M = 2: 254 without, 266 with one).
__host__ __device__ constexpr int dp_fma(int M) { return M == 2 ? 0 : 1; }

// sum of the four products of a's unsigned and b's signed bytes, plus c
__device__ __forceinline__ int dp_u8s8(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// x 2^-E as a 62-bit integer plus the bias that makes its bytes digits + 128; emax <= e + 63 gives 0
__device__ __forceinline__ uint64_t dp_word(double x, int emax) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 9;
  const uint64_t v = m >> min(emax - (int)((hi >> 20) & 0x7ff), 63);
  const uint64_t sg = (uint64_t)(int64_t)((int)hi >> 31);
  return (v ^ sg) - sg + 0x8080808080808080ull;
}
// The bytes 3..0 of four words as four words.
__device__ __forceinline__ void dp_bytes(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, uint32_t (&o)[4]) {
  const uint32_t a = __byte_perm(x0, x1, 0x5140), b = __byte_perm(x2, x3, 0x5140);
  const uint32_t c = __byte_perm(x0, x1, 0x7362), d = __byte_perm(x2, x3, 0x7362);
  o[0] = __byte_perm(c, d, 0x7632);
  o[1] = __byte_perm(c, d, 0x5410);
  o[2] = __byte_perm(a, b, 0x7632);
  o[3] = __byte_perm(a, b, 0x5410);
}
// An integer below 2^51 as a double, exactly.
__device__ __forceinline__ double dp_double(long long a) {
  return __longlong_as_double(a + 0x4338000000000000ll) - 6755399441055744.0;
}

// One group: the layers [lo, n) at d, weight digits dig, corrections corr,
// exponents wexp and weights wf (row m at wf + m ldw) of the group.
template <int M>
__device__ __forceinline__ void dp_group(const double *__restrict__ d, long long ldd, int lo, int n,
                                         const uint32_t (*dig)[M][8], const int (*corr)[8], const int *wexp,
                                         const double *wf, int ldw, double (&acc)[M]) {
  constexpr int F = dp_fma(M), Q = 4 - F, ND = 4 * Q, NF = 4 * F;  // quads and layers in digits, layers by FMAs
  double v[kDpGroup];
  if (lo <= 0 && n >= kDpGroup) {
#pragma unroll
    for (int k = 0; k < kDpGroup; ++k) v[k] = fh_ld_stream(d + k * ldd);
  } else {
#pragma unroll
    for (int k = 0; k < kDpGroup; ++k) v[k] = k >= lo && k < n ? fh_ld_stream(d + k * ldd) : 0.0;
  }
  auto fmas = [&](int k0, int k1) {
#pragma unroll
    for (int k = 0; k < kDpGroup; ++k)
      if (k >= k0 && k < k1)
#pragma unroll
        for (int m = 0; m < M; ++m) acc[m] = fma(wf[m * ldw + k], v[k], acc[m]);
  };
  uint32_t mx = 0;
#pragma unroll
  for (int k = 0; k < ND; ++k) mx = max(mx, (uint32_t)__double2hiint(v[k]) & 0x7fffffffu);
  const int emax = (int)(mx >> 20);
  int L[M][kDpDigits];
  bool ok = emax > 64 && emax != 0x7ff;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int we = wexp[m];
    ok = ok && we >= 0 && emax + we >= 1098 && emax + we <= 3000;
    const int4 c0 = *reinterpret_cast<const int4 *>(&corr[m][0]);
    const int4 c1 = *reinterpret_cast<const int4 *>(&corr[m][4]);
    L[m][0] = c0.x;
    L[m][1] = c0.y;
    L[m][2] = c0.z;
    L[m][3] = c0.w;
    L[m][4] = c1.x;
    L[m][5] = c1.y;
    L[m][6] = c1.z;
    L[m][7] = c1.w;
  }
  if (ok) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      fmas(ND + q * NF / Q, ND + (q + 1) * NF / Q);
      uint32_t a[kDpDigits];
      {
        uint64_t x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = dp_word(v[4 * q + u], emax);
        uint32_t o[4];
        dp_bytes((uint32_t)(x[0] >> 32), (uint32_t)(x[1] >> 32), (uint32_t)(x[2] >> 32), (uint32_t)(x[3] >> 32), o);
        a[0] = o[0], a[1] = o[1], a[2] = o[2], a[3] = o[3];
        dp_bytes((uint32_t)x[0], (uint32_t)x[1], (uint32_t)x[2], (uint32_t)x[3], o);
        a[4] = o[0], a[5] = o[1], a[6] = o[2], a[7] = o[3];
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const uint4 b0 = *reinterpret_cast<const uint4 *>(&dig[q][m][0]);
        const uint4 b1 = *reinterpret_cast<const uint4 *>(&dig[q][m][4]);
        const uint32_t b[kDpDigits] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int i = 0; i < kDpDigits; ++i)
#pragma unroll
          for (int j = 0; i + j < kDpDigits; ++j) L[m][i + j] = dp_u8s8(a[i], b[j], L[m][i + j]);
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) {
      // unit of digit 0: 2^(exponent - 1028) each
      const long long h =
          (long long)L[m][0] * (1 << 24) + (long long)L[m][1] * (1 << 16) + (long long)L[m][2] * 256 + L[m][3];
      const long long l =
          (long long)L[m][4] * (1 << 24) + (long long)L[m][5] * (1 << 16) + (long long)L[m][6] * 256 + L[m][7];
      const double sc = __hiloint2double((emax + wexp[m] - 1057) << 20, 0);
      acc[m] = fma(fma(dp_double(l), 0x1p-32, dp_double(h)), sc, acc[m]);
    }
  } else {
    bool any = mx != 0;  // zeros add nothing to finite weights' sums
#pragma unroll
    for (int k = 0; k < ND; ++k) any = any || __double2loint(v[k]) != 0;
#pragma unroll
    for (int m = 0; m < M; ++m) any = any || wexp[m] < 0;
    if (any) fmas(0, ND);
    fmas(ND, kDpGroup);
  }
}

// acc += sum_{lo <= k < nk} W[m][k] D[k] for the CTA's points, D[k] of this
// thread's at d + k ldd (live: it has one).  All kDpThreads threads call.
template <int M>
__device__ __forceinline__ void dp_sum(const double *__restrict__ d, long long ldd, int lo, int nk,
                                       const double *__restrict__ W, int ldw, bool live, double (&acc)[M]) {
  __shared__ __align__(16) uint32_t dig[kDpStage / 4][M][8];     // weight digits of four layers, signed bytes
  __shared__ __align__(16) int corr[kDpStage / kDpGroup][M][8];  // -128 x the digit sums met by each level
  __shared__ int wexp[kDpStage / kDpGroup][M];                   // largest exponent; -1: FP64
  __shared__ double wf[M][kDpStage];
  const int t = threadIdx.x;
  for (int kb = 0; kb < nk; kb += kDpStage) {
    const int ns = min(kDpStage, nk - kb), ng = (ns + kDpGroup - 1) / kDpGroup;
    const double *w = W + kb;
    __syncthreads();  // every thread is done with the previous stage
    for (int i = t; i - (t & 31) < M * ng * kDpGroup; i += kDpThreads) {
      const int m = min(i / (ng * kDpGroup), M - 1), k = i - m * ng * kDpGroup;  // 16 lanes: one row, one group
      const double x0 = k < ns && kb + k >= lo ? w[(long long)m * ldw + k] : 0.0;
      const double x = (k & 15) < kDpGroup - 4 * dp_fma(M) ? x0 : 0.0;
      const int e = (__double2hiint(x) >> 20) & 0x7ff;
      int mx = e, mn = e || x != 0.0 ? e : 0x7ff;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
      }
      const bool zero = __all_sync(0xffffu << (t & 16), x == 0.0);
      if (k < ng * kDpGroup) {
        const uint64_t v = dp_word(x, mx) ^ 0x8080808080808080ull;
#pragma unroll
        for (int j = 0; j < kDpDigits; ++j)
          reinterpret_cast<uint8_t *>(&dig[k >> 2][m][j])[k & 3] = e ? (uint8_t)(v >> (56 - 8 * j)) : 0;
        wf[m][k] = x0;
        if ((k & 15) == 0) wexp[k >> 4][m] = zero || (mx != 0x7ff && mx - mn <= kDpSpread && mx > 64) ? mx : -1;
      }
    }
    __syncthreads();
    for (int i = t; i < M * ng; i += kDpThreads) {
      const int g = i / M, m = i - g * M;
      int c = 0;
#pragma unroll
      for (int j = 0; j < kDpDigits; ++j) {
#pragma unroll
        for (int q = 0; q < 4; ++q) c = __dp4a((int)dig[4 * g + q][m][j], 0x01010101, c);
        corr[g][m][j] = -128 * c;
      }
    }
    __syncthreads();
    if (!live) continue;
    const double *dg = d + (long long)kb * ldd;
    for (int g = 0; g < ng; ++g, dg += kDpGroup * ldd)
      dp_group<M>(dg, ldd, lo - kb - g * kDpGroup, ns - g * kDpGroup, &dig[4 * g], corr[g], wexp[g], &wf[0][g * kDpGroup], kDpStage, acc);
  }
}
