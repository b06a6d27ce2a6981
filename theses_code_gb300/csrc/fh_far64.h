// fh_far64.h -- the history sum of a block of future steps at FP64 accuracy on
// the tensor cores (fh_far64.cu): 64 weight rows x the layers before the block.
#pragma once
#include "fh_internal.h"

constexpr int kF64Rows = 64;   // weight rows of a block
constexpr int kF64Block = 32;  // layers a block's history grows by (and K's unit)

struct fh_far64;
// P points, up to Kcap layers; df: layers and results as (hi, lo) FP32 pairs,
// else FP64.  *out is null and the code FH_OK's opposite when memory is short.
int fh_far64_create(fh_ctx *ctx, long long P, int Kcap, bool df, fh_far64 **out);
void fh_far64_delete(fh_far64 *f);
size_t fh_far64_bytes(const fh_far64 &f);
long long fh_far64_pitch(const fh_far64 &f);  // points per result row
// The newest kF64Block layers [k0, k0 + kF64Block) join the exponent table (in
// order from k0 = 0; layer k at D + k ldd points).
int fh_far64_append(fh_ctx *ctx, fh_far64 &f, const void *D, long long ldd, int k0);
// Weight rows: row n weighs layer k < K by W[(n >> 1) row_step + (n & 1) ldw + k]
// (rows n < nrows, zero above), or by lag[base + n - k].  fh_far64_run reads them
// again: they stay as they are until its launches are done.
int fh_far64_weights(fh_ctx *ctx, fh_far64 &f, int K, const double *W, long long row_step, long long ldw, int nrows);
int fh_far64_weights_lag(fh_ctx *ctx, fh_far64 &f, int K, const double *lag, int base, int nrows);
// Result rows S[n] = sum_{k < K} w_n(k) D[k], K a positive multiple of kF64Block.
int fh_far64_run(fh_ctx *ctx, fh_far64 &f, const void *D, long long ldd, int K);
const void *fh_far64_rows(const fh_far64 &f);  // double or float2, row n at n pitch
int fh_far64_check(fh_ctx *ctx, const fh_far64 &f);  // FH_ETIMEOUT once a device wait ran out (synchronises)
int fh_far64_mark(fh_ctx *ctx, const fh_far64 &f, int expired);  // 0 at the start of a solve; 1 as an expired wait does
