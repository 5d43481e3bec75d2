// FP64 direct sum at sampled targets (field form: sum_j q_j / r and
// -sum_j q_j dX / r^3), shared by tapas_b200_direct and tapas_b200_direct_noalloc.
#pragma once
#include "common.cuh"

namespace tb {

constexpr int kDirectThreads = 128;
constexpr int kDirectTargets = 8;  // targets per block
constexpr int kDirectSplits = 64;  // most blocks that share a group's sources

// How many blocks share the sources of each group of eight targets: about twelve
// waves of blocks, at least 16 sources per thread, so up to 28416 + k rows of partial
// sums in all.  1 and 8 targets x 1M bodies: 45 and 47 us; 126 us with 16 splits.
inline int direct_splits(int num_sms, int64_t n, int64_t k) {
  const int64_t nb = (k + kDirectTargets - 1) / kDirectTargets;
  const int64_t waves = ((int64_t)num_sms * 24 + nb - 1) / nb;
  return (int)std::max<int64_t>(
      1, std::min({waves, (int64_t)kDirectSplits, n / (16 * kDirectThreads)}));
}

// Block (b, split): targets 8b .. 8b + 7 over every nsplit-th group of 128
// sources, a thread a source at a time, its eight targets' sums in registers;
// one source load (L2: every block reads all bodies) serves eight pairs.  The
// sums of (target, split) go to part[4 (target * nsplit + split)], in a fixed
// order.  A target index outside [0, n) gives NaN.
//
// Bound: the FP64 pipe, 18 slots per pair with charge_over_distance: 4000 targets x
// 1M bodies 5.06 ms, 76 % of that pipe.  All eight separations are in flight
// at once, which takes 240 registers, so two blocks per SM: 5.44 ms with four and
// three blocks (5.38 against 5.50 ms a call with the bodies out of L2), 5.00 with T = 7
// or 10, 5.15 with sources loaded two steps ahead.  A
// block per target with 1.0 / sqrt(r2) took 13.6 ms.
static __global__ void __launch_bounds__(kDirectThreads, 2) direct_tiles(
    const double *__restrict__ x, const double *__restrict__ y, const double *__restrict__ z,
    const double *__restrict__ q, int64_t n, const int64_t *__restrict__ targets, int64_t k,
    int nsplit, double *__restrict__ part) {
  constexpr int T = kDirectTargets;
  const int64_t t0 = (int64_t)blockIdx.x * T;
  double xi[T], yi[T], zi[T], p[T], ax[T], ay[T], az[T];
#pragma unroll
  for (int r = 0; r < T; r++) {
    const int64_t i = t0 + r < k ? targets[t0 + r] : -1;
    const bool ok = i >= 0 && i < n;
    xi[r] = ok ? x[i] : 0.0;
    yi[r] = ok ? y[i] : 0.0;
    zi[r] = ok ? z[i] : 0.0;
    p[r] = ax[r] = ay[r] = az[r] = 0.0;
  }
  const int64_t step = (int64_t)nsplit * kDirectThreads;
  int64_t j = (int64_t)blockIdx.y * kDirectThreads + threadIdx.x;
  double4 next = make_double4(0, 0, 0, 0);
  if (j < n) next = make_double4(x[j], y[j], z[j], q[j]);
  for (; j < n; j += step) {
    const double4 b = next;
    if (j + step < n)
      next = make_double4(x[j + step], y[j + step], z[j + step], q[j + step]);
    // all T separations in flight
    double dx[T], dy[T], dz[T], R2[T], qj[T], qr[T], inv[T];
#pragma unroll
    for (int i = 0; i < T; i++) {
      dx[i] = xi[i] - b.x;
      dy[i] = yi[i] - b.y;
      dz[i] = zi[i] - b.z;
      R2[i] = dx[i] * dx[i] + dy[i] * dy[i] + dz[i] * dz[i];
      qj[i] = b.w;
    }
    charge_over_distance(R2, qj, qr, inv);
#pragma unroll
    for (int i = 0; i < T; i++) {
      const double s3 = qr[i] * inv[i] * inv[i];
      p[i] += qr[i];
      ax[i] = fma(-dx[i], s3, ax[i]);
      ay[i] = fma(-dy[i], s3, ay[i]);
      az[i] = fma(-dz[i], s3, az[i]);
    }
  }
  __shared__ double red[kDirectThreads / 32][4 * T];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int r = 0; r < T; r++) {
    double v[4] = {p[r], ax[r], ay[r], az[r]};
#pragma unroll
    for (int c = 0; c < 4; c++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
      if (lane == 0) red[w][4 * r + c] = v[c];
    }
  }
  __syncthreads();
  if (threadIdx.x < 4 * T) {
    const int64_t t = t0 + threadIdx.x / 4;
    if (t < k) {
      const int64_t i = targets[t];
      double s = 0;
      for (int m = 0; m < kDirectThreads / 32; m++) s += red[m][threadIdx.x];
      if (i < 0 || i >= n) s = __longlong_as_double(-1);
      part[4 * (t * nsplit + blockIdx.y) + threadIdx.x % 4] = s;
    }
  }
}

// out4[t] = sum over the splits, in split order.
static __global__ void direct_finish(const double *__restrict__ part, int64_t k, int nsplit,
                                     double *__restrict__ out4) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < k * 4;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = i / 4;
    double s = 0;
    for (int sp = 0; sp < nsplit; sp++) s += part[4 * (t * nsplit + sp) + i % 4];
    out4[i] = s;
  }
}

}  // namespace tb
