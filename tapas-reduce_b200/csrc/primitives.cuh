// Device primitives of libtapas_b200 (scan, radix sort), issued on ctx->stream.
#pragma once
#include "common.cuh"

namespace tb {

// out[i] = sum(in[0..i)); *d_total (device, may be null) = sum(in).  n < 2^31, sums too.
int scan_exclusive(tapas_b200_ctx *ctx, const int32_t *in, int32_t *out, int64_t n,
                   int32_t *d_total);

// The same for two arrays of n values with one set of launches: half the launches
// where the scans are short.  d_max (or an entry of it) may be null; else *d_max[y]
// is raised to array y's largest value.  No output may be another array's input.
int scan_exclusive2(tapas_b200_ctx *ctx, const int32_t *const in[2], int32_t *const out[2],
                    int64_t n, int32_t *const d_total[2], unsigned long long *const d_max[2]);

// Exclusive scan of each row of rows[nrows][ncols] in place; totals[row] = its sum.
int scan_rows(tapas_b200_ctx *ctx, uint32_t *rows, int nrows, int ncols, uint32_t *totals);

// Stable LSD radix sort on key bits [begin_bit, end_bit).  Keys (and values,
// if vals is non-null) are sorted between the two buffers; on return `keys`
// and `vals` point at the sorted data (the pointers are swapped per pass).
int radix_sort(tapas_b200_ctx *ctx, uint64_t *&keys, uint64_t *&keys_alt, uint32_t *&vals,
               uint32_t *&vals_alt, int64_t n, int begin_bit, int end_bit);

// After a radix sort on the bits from low_bits up only: orders every run of keys
// equal there by all bits (stable), except runs of more than max_run, which are listed:
// long_runs[r] = {first element, elements of the listed runs before it}, room for
// n / (max_run + 1) of them; *long_tally (device, 0 before) = {their number, their
// elements} in its high and low 32 bits.
int order_equal_runs(tapas_b200_ctx *ctx, uint64_t *keys, uint32_t *vals, int64_t n, int low_bits,
                     int max_run, int2 *long_runs, unsigned long long *long_tally);

// The listed runs, `total` elements in all, put in order of the bits from begin_bit up
// (stable): their elements are sorted by {run, low bits} in rk and rv (scratch for
// `total` each) and put back.  at (in rv): the places they took.
int order_long_runs(tapas_b200_ctx *ctx, uint64_t *keys, uint32_t *vals, const int2 *runs,
                    int nruns, int64_t total, int begin_bit, int low_bits, uint64_t *const rk[2],
                    uint32_t *const rv[2], const uint32_t *&at);

}  // namespace tb
