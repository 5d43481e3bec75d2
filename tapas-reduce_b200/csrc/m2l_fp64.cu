// The plain form's M2L (P >= 4): FP64, batched by offset class on the FP64
// tensor cores, with every target's sum taken in list order.
//
// With M_n scaled by w^-n and L_j by w^(j+1) (w = cell width), the M2L
// (ex/LaplaceSphericalCPU_tapas.h:208-273) of every pair of one offset class
// (level difference and centre offset in half-widths, m2l_tc.cu) is the same
// real K x K map (K = P(P+1)).  The evaluation has two steps:
//  1. products: row e of a buffer is T_class(e) . Mt[source of e], for every
//     list entry e: one launch over the 32-pair tiles of all classes, a warp a
//     tile; the pairs of classes too rare for an operator of their own are
//     translated one warp per pair into the same rows;
//  2. sums: a target's rows are consecutive (the list is sorted by target,
//     then source), so its local expansion is their sum in list order.
// The order of every sum is thus the list's: no atomics, bit-reproducible, and
// independent of how pairs were tiled (a sharded context's targets get the bits
// of a single context's).  The rows cost a write and a read of 8 K bytes per
// pair, which is less time than their multiplication; one launch per class into
// partial sums, which needs no rows, left the GPU idle between its 158 to 1164
// launches of a few tiles each (1M sphere, P = 15: products and sums 1.9 ms
// where the per-class launches took 14.4; 100k cube, P = 10: 0.4 against 6.4).
// A list whose rows would exceed kRowBytes is evaluated in ranges of list
// entries; a target cut by a range boundary goes on from its partial sum, so
// the bits do not depend on the ranges either.
#include <algorithm>

#include "expansions.cuh"
#include "kernels.cuh"
#include "m2l_tc.cuh"
#include "primitives.cuh"

namespace tb {
namespace {

constexpr size_t kRowBytes = (size_t)512 << 20;  // product rows kept at once
constexpr size_t kLeastRowBytes = (size_t)8 << 20;  // the same where memory is short
// Pairs a class needs for an operator of its own: building one and multiplying
// a partly filled tile costs about as much as translating 16 pairs one by one.
constexpr int64_t kMinClassPairs = 16;
constexpr int kGemmWarps = 4;
constexpr int kPairTile = 32;  // pairs (MMA rows) of a warp's tile
constexpr int kOutBlock = 32;  // outputs of one block of the operator
constexpr int kStep = 16;      // sources (MMA K) of one block of the operator

// An output of degree j reads only sources of degree n < P - j, so the block of
// 32 outputs whose lowest degree is j reads the first (P - j)(P - j + 1) real
// sources.  The operator is stored as these 32 x 16 blocks, output blocks in
// order, each with its steps() source blocks.
template <int P>
struct Op64 {
  static constexpr int NT = P * (P + 1) / 2;
  static constexpr int K = 2 * NT;
  static constexpr int KP = (K + kStep - 1) / kStep * kStep;  // row stride of Mt64
  static constexpr int NB = (K + kOutBlock - 1) / kOutBlock;
  static constexpr int degree(int t) {
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= t) j++;
    return j;
  }
  static constexpr int steps(int b) {
    const int j = degree(b * (kOutBlock / 2));
    return ((P - j) * (P - j + 1) + kStep - 1) / kStep;
  }
  static constexpr int blocks(int b) {  // blocks before output block b
    int s = 0;
    for (int i = 0; i < b; i++) s += steps(i);
    return s;
  }
  static constexpr int NBLK = blocks(NB);
  static constexpr size_t DOUBLES = (size_t)NBLK * kOutBlock * kStep;
};

// One block per class: the map's entries from the unit-offset singular
// harmonics (evalLocal, :102-135).  Entry (target (j,k), source (n,m)) collects
// the reference loop's m and -m terms (:229-262) times (w_s / w_t)^n = 2^(delta n).
// Stored in the multiplication's order: per 32 x 16 block, for each 8 outputs f
// and half h of a lane's four sources, the two doubles of each lane.
template <int P>
__global__ void __launch_bounds__(256) build_operators64(const uint64_t *__restrict__ keys,
                                                         double *__restrict__ ops) {
  using O = Op64<P>;
  __shared__ cd Y[P * P];
  __shared__ double scale[P];
  __shared__ unsigned char deg[O::NT], ord[O::NT];
  __shared__ short blk_out[O::NBLK], blk_step[O::NBLK];
  const uint64_t key = keys[blockIdx.x];
  const int delta = (int)((key >> 42) & 63) - 32;
  const double Dx = (double)((long long)(key & 16383) - 8192);
  const double Dy = (double)((long long)((key >> 14) & 16383) - 8192);
  const double Dz = (double)((long long)((key >> 28) & 16383) - 8192);
  const double u = ldexp(1.0, min(delta, 0) - 1);  // half-widths -> target widths
  const Sph sp = sph_of(Dx * u, Dy * u, Dz * u);
  if (threadIdx.x < P) {
    local_column<P>(threadIdx.x, sp.r, sp.x, sp.y, sp.ei, Y);
    scale[threadIdx.x] = ldexp(1.0, delta * (int)threadIdx.x);
  }
  for (int t = threadIdx.x; t < O::NT; t += blockDim.x) {
    int j, k;
    jk_of(t, j, k);
    deg[t] = (unsigned char)j;
    ord[t] = (unsigned char)k;
  }
  if (threadIdx.x < O::NB) {
    int at = 0;
    for (int b = 0; b < (int)threadIdx.x; b++) at += O::steps(b);
    for (int s = 0; s < O::steps(threadIdx.x); s++) {
      blk_out[at + s] = (short)threadIdx.x;
      blk_step[at + s] = (short)s;
    }
  }
  __syncthreads();
  double *op = ops + (size_t)blockIdx.x * O::DOUBLES;
  // one thread per complex (output, source) pair of a block: its real 2 x 2 entries
  constexpr int kPairs = (kOutBlock / 2) * (kStep / 2);
  for (int idx = threadIdx.x; idx < O::NBLK * kPairs; idx += blockDim.x) {
    const int blk = idx / kPairs, in = idx - blk * kPairs;
    const int lo = in >> 3, li = in & 7;  // complex output, source within the block
    const int to = blk_out[blk] * (kOutBlock / 2) + lo, ti = blk_step[blk] * (kStep / 2) + li;
    double v00 = 0, v01 = 0, v10 = 0, v11 = 0;  // [out re/im][in re/im]
    if (to < O::NT && ti < O::NT) {
      const int j = deg[to], k = ord[to], n = deg[ti], ma = ord[ti];
      if (n < P - j) {
        const double Cnm = oddeven(j);
        const int base = (j + n) * (j + n) + j + n - k;
        const double C2 = Cnm * oddeven((k - ma) * (k < ma) + ma);
        const cd Yp = Y[base + ma];
        v00 = C2 * Yp.x;
        v01 = -C2 * Yp.y;
        v10 = C2 * Yp.y;
        v11 = C2 * Yp.x;
        if (ma > 0) {
          const cd Ym = Y[base - ma];
          v00 += Cnm * Ym.x;
          v01 += Cnm * Ym.y;
          v10 += Cnm * Ym.y;
          v11 += -Cnm * Ym.x;
        }
        const double sc = scale[n];
        v00 *= sc; v01 *= sc; v10 *= sc; v11 *= sc;
      }
    }
    // sources 2 li, 2 li + 1 are k = 4t + i of lane t = li / 2, half h = li % 2;
    // outputs 2 lo, 2 lo + 1 are columns g = (2 lo) % 8 (+1) of f = lo / 4
    const int f = lo >> 2, g = (2 * lo) & 7, t = li >> 1, h = li & 1;
    double2 *o = reinterpret_cast<double2 *>(op) +
                 (((size_t)blk * 4 + f) * 2 + h) * 32 + 4 * g + t;
    o[0] = make_double2(v00, v01);
    o[4] = make_double2(v10, v11);
  }
}

// Per cell (one warp each): Mt[c][2t + re/im] = M[c][t] / w^n, rows padded with
// zeros to KP; 0 for an empty cell.
template <int P>
__global__ void __launch_bounds__(256) normalize_M64(int64_t ncells, const int32_t *__restrict__ cnb,
                                                     const double *__restrict__ cmin,
                                                     const double *__restrict__ cmax,
                                                     const double2 *__restrict__ M,
                                                     double2 *__restrict__ Mt) {
  using O = Op64<P>;
  __shared__ double pw[8][P];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int64_t nw = (int64_t)gridDim.x * 8;
  for (int64_t c = (int64_t)blockIdx.x * 8 + wi; c < ncells; c += nw) {
    const bool live = cnb[c] > 0;
    __syncwarp();
    if (live && lane < P) {
      const double iw = 1.0 / (cmax[3 * c] - cmin[3 * c]);
      double p = 1.0;
      for (int k = 0; k < lane; k++) p *= iw;
      pw[wi][lane] = p;
    }
    __syncwarp();
    for (int t = lane; t < O::KP / 2; t += 32) {
      double2 v = make_double2(0.0, 0.0);
      if (live && t < O::NT) {
        int j, k;
        jk_of(t, j, k);
        v = M[c * O::NT + t];
        v.x *= pw[wi][j];
        v.y *= pw[wi][j];
      }
      Mt[c * (O::KP / 2) + t] = v;
    }
  }
}

// Tiles of class r's pairs whose list index lies in range q: pairs of a class
// ascend in list index, so they are a contiguous part of the class.
__global__ void count_tiles64(const int2 *__restrict__ cls_range, int64_t ncls, int64_t nrange,
                              int64_t per_range, const uint32_t *__restrict__ vals,
                              int32_t *__restrict__ cnt, int2 *__restrict__ part) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncls * nrange;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = i / ncls, r = i - q * ncls;
    const int2 cr = cls_range[r];
    int lo = cr.x, hi = cr.x + cr.y;
    if (nrange > 1) {
      auto first_at_least = [&](int64_t e) {
        int a = cr.x, b = cr.x + cr.y;
        while (a < b) {
          const int m = a + ((b - a) >> 1);
          if ((int64_t)vals[m] < e) a = m + 1; else b = m;
        }
        return a;
      };
      lo = first_at_least(q * per_range);
      hi = first_at_least((q + 1) * per_range);
    }
    part[i] = make_int2(lo, hi - lo);
    cnt[i] = (hi - lo + kPairTile - 1) / kPairTile;
  }
}

// One warp per (range, class): its tiles {class, first sorted pair, pairs, 0}.
__global__ void emit_tiles64(int64_t ncls, int64_t nrange, const int32_t *__restrict__ off,
                             const int2 *__restrict__ part, int4 *__restrict__ items) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
       i < ncls * nrange; i += nw) {
    const int2 pr = part[i];
    const int o = off[i], n = (pr.y + kPairTile - 1) / kPairTile;
    for (int k = lane; k < n; k += 32)
      items[o + k] = make_int4((int)(i % ncls), pr.x + k * kPairTile,
                               min(kPairTile, pr.y - k * kPairTile), 0);
  }
}

// The products of the classes' pairs.  A warp takes a tile of 32 pairs; the
// pairs' multipole rows are the MMA's rows (gathered: four lanes read 128
// contiguous bytes of a pair's row), the operator's outputs its columns
// (stored in fragment order, so its loads are coalesced and the four warps of a
// block, on consecutive tiles of mostly one class, share them in L1).  Both
// operands go straight from L2 / L1 to registers: a warp's 32 x 32 tile does
// 8 MMAs (1024 cycles of its scheduler's FP64 pipe) per 16 loads, and three
// warps per scheduler cover the load latency, so staging through shared memory
// would only add work.  Bound: the FP64 pipe.
template <int P>
__global__ void __launch_bounds__(32 * kGemmWarps, 3) product_tiles64(
    const int32_t *__restrict__ tile_off, int64_t first, int64_t last,
    const int4 *__restrict__ items, const uint32_t *__restrict__ vals,
    const uint64_t *__restrict__ list, int shift, int64_t base, const double *__restrict__ ops,
    const double *__restrict__ Mt, double *__restrict__ rows) {
  using O = Op64<P>;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint64_t smask = (1ull << shift) - 1;
  const int i1 = tile_off[last];
  const int nw = (int)gridDim.x * kGemmWarps;
  for (int i = tile_off[first] + (int)blockIdx.x * kGemmWarps + (int)(threadIdx.x >> 5); i < i1;
       i += nw) {
    const int4 it = items[i];
    // lane's pairs: rows g, g + 8, g + 16, g + 24 of the tile (the last pair
    // again beyond the tile's end; those products are not stored)
    const double2 *src[4];
    int64_t dst[4];
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int p = g + 8 * m;
      const uint32_t e = vals[it.y + min(p, it.z - 1)];
      src[m] = reinterpret_cast<const double2 *>(Mt + (int64_t)(list[e] & smask) * O::KP) + 2 * t;
      dst[m] = p < it.z ? ((int64_t)e - base) * O::K : -1;
    }
    const double2 *op =
        reinterpret_cast<const double2 *>(ops + (size_t)it.x * O::DOUBLES) + lane;
    for (int b = 0; b < O::NB; b++) {
      double acc[2][4][4];
#pragma unroll
      for (int m = 0; m < 2; m++)
#pragma unroll
        for (int f = 0; f < 4; f++)
#pragma unroll
          for (int x = 0; x < 4; x++) acc[m][f][x] = 0;
      int j = 0;
      while ((j + 1) * (j + 2) / 2 <= b * (kOutBlock / 2)) j++;
      const int steps = ((P - j) * (P - j + 1) + kStep - 1) / kStep;
      for (int s = 0; s < steps; s++) {
        double a[2][8];
#pragma unroll
        for (int m = 0; m < 4; m++) {
          const double2 u = __ldg(src[m] + 8 * s), v = __ldg(src[m] + 8 * s + 1);
          double *d = a[m >> 1] + (m & 1);
          d[0] = u.x;
          d[2] = u.y;
          d[4] = v.x;
          d[6] = v.y;
        }
#pragma unroll
        for (int f = 0; f < 4; f++) {
          const double2 u = __ldg(op + f * 64), v = __ldg(op + f * 64 + 32);
#pragma unroll
          for (int m = 0; m < 2; m++) dmma_m16n8k16(acc[m][f], a[m], u.x, u.y, v.x, v.y);
        }
        op += 256;
      }
#pragma unroll
      for (int f = 0; f < 4; f++) {
        const int r = b * kOutBlock + 8 * f + 2 * t;
        if (r >= O::K) continue;
#pragma unroll
        for (int m = 0; m < 4; m++)
          if (dst[m] >= 0)
            *reinterpret_cast<double2 *>(rows + dst[m] + r) =
                make_double2(acc[m >> 1][f][2 * (m & 1)], acc[m >> 1][f][2 * (m & 1) + 1]);
      }
    }
  }
}

// The products of the pairs without an operator, one warp per pair, scaled
// into the rows' units (w_t^(j+1)).  The translation is done in units of the power of
// two below w_t, which changes no bit of it and leaves only powers of 1 <= f < 2 to
// multiply by: w_t^16 itself overflows for cells wider than 2^64.
template <int P>
__global__ void __launch_bounds__(128) product_pairs64(
    const uint32_t *__restrict__ pairs, int64_t npairs, int64_t base, int64_t count,
    const uint64_t *__restrict__ list, int shift, const int32_t *__restrict__ cnb,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double *__restrict__ ccen, const double2 *__restrict__ M, double2 *__restrict__ rows) {
  using S = Sizes<P>;
  __shared__ cd Ysm[4][S::NY];
  __shared__ cd Msm[4][S::NT];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  cd *Y = Ysm[wi];
  cd *Mj = Msm[wi];
  int jj[S::R], kk[S::R];
#pragma unroll
  for (int r = 0; r < S::R; r++) jk_of(lane + 32 * r, jj[r], kk[r]);
  const uint64_t src_mask = (1ull << shift) - 1;
  const int64_t nw = (int64_t)gridDim.x * 4;
  for (int64_t p = (int64_t)blockIdx.x * 4 + wi; p < npairs; p += nw) {
    const int64_t e = (int64_t)pairs[p] - base;
    if (e < 0 || e >= count) continue;  // another range's (warp-uniform)
    const uint64_t x = list[e + base];
    const int c = (int)(x >> shift), s = (int)(x & src_mask);
    if (cnb[s] == 0 || cnb[c] == 0) continue;  // not summed either
    const double w = cmax[3 * c] - cmin[3 * c];
    const int ex = ilogb(w);
    const double f = scalbn(w, -ex);
    const Sph sp = sph_of(scalbn(ccen[3 * c] - ccen[3 * s], -ex),
                          scalbn(ccen[3 * c + 1] - ccen[3 * s + 1], -ex),
                          scalbn(ccen[3 * c + 2] - ccen[3 * s + 2], -ex));
    __syncwarp();
    if (lane < P) local_column<P>(lane, sp.r, sp.x, sp.y, sp.ei, Y);
#pragma unroll
    for (int r = 0; r < S::R; r++) {
      const int t = lane + 32 * r;
      if (t >= S::NT) continue;
      const double2 v = M[(int64_t)s * S::NT + t];
      Mj[t] = cd{scalbn(v.x, -ex * jj[r]), scalbn(v.y, -ex * jj[r])};
    }
    __syncwarp();
    cd acc[S::R];
#pragma unroll
    for (int r = 0; r < S::R; r++) acc[r] = cd{0, 0};
    m2l_accumulate<P>(acc, jj, kk, lane, Mj, Y);
#pragma unroll
    for (int r = 0; r < S::R; r++) {
      const int t = lane + 32 * r;
      if (t >= S::NT) continue;
      double sc = f;
      for (int k = 0; k < jj[r]; k++) sc *= f;
      rows[e * S::NT + t] = make_double2(acc[r].x * sc, acc[r].y * sc);
    }
  }
}

// L of the targets with list entries in [base, base + count): a warp per target
// and 32 coefficients, the rows added in list order.  A target that began in
// an earlier range goes on from the partial sum left in L; the range that holds
// its last entry scales the sum by w^-(j+1).
template <int P>
__global__ void __launch_bounds__(256) sum_products64(
    int64_t ncells, const int32_t *__restrict__ off, const uint64_t *__restrict__ list,
    uint64_t src_mask, int64_t base, int64_t count, int skip_empty,
    const int32_t *__restrict__ cnb, const uint8_t *__restrict__ own,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double2 *__restrict__ rows, double2 *__restrict__ L) {
  using O = Op64<P>;
  constexpr int kParts = (O::NT + 31) / 32;
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * 8, total = ncells * kParts;
  for (int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); i < total; i += nw) {
    const int64_t c = i / kParts;
    const int t = (int)(i - c * kParts) * 32 + lane;
    const int64_t s0 = off[c], s1 = off[c + 1];
    const int64_t e0 = max(s0, base), e1 = min(s1, base + count);
    if (e0 >= e1 || cnb[c] == 0) continue;
    if (own && !(own[c] & 1)) continue;  // sharded: another context's target
    if (t >= O::NT) continue;
    double2 acc = s0 < base ? L[c * O::NT + t] : make_double2(0.0, 0.0);
    const double2 *r = rows + (e0 - base) * O::NT + t;
    if (skip_empty) {  // lists with the reference's pairs of empty cells: they have no rows
      for (int64_t e = e0; e < e1; e++, r += O::NT) {
        if (cnb[list[e] & src_mask] == 0) continue;
        const double2 v = *r;
        acc.x += v.x;
        acc.y += v.y;
      }
    } else {
#pragma unroll 8
      for (int64_t e = e0; e < e1; e++, r += O::NT) {
        const double2 v = *r;
        acc.x += v.x;
        acc.y += v.y;
      }
    }
    if (s1 <= base + count) {
      int j, k;
      jk_of(t, j, k);
      const double iw = 1.0 / (cmax[3 * c] - cmin[3 * c]);
      double sc = iw;
      for (int d = 0; d < j; d++) sc *= iw;
      acc.x *= sc;
      acc.y *= sc;
    }
    L[c * O::NT + t] = acc;
  }
}

template <int P>
int m2l_products_P(tapas_b200_ctx *ctx) {
  using O = Op64<P>;
  cudaStream_t s = ctx->stream;
  const int64_t C = ctx->ncells, n = ctx->n_m2l;
  auto &T = ctx->tc;
  TB_CUDA(ctx, ctx->L.ensure((size_t)C * O::NT, s));
  TB_CUDA(ctx, cudaMemsetAsync(ctx->L.p, 0, sizeof(double2) * (size_t)C * O::NT, s));
  ctx->tc_classes = 0;
  if (n == 0) return TAPAS_B200_OK;
  int64_t per_range = std::min<int64_t>(n, (int64_t)(kRowBytes / (sizeof(double) * O::K)));
  int64_t nrange = 1, parts = 0;
  M2LClassInfo ci;
  int64_t max_tiles = 0;
  {
    PhaseTimer t(ctx, &ctx->timings.m2l_setup);
    TB_TRY(m2l_classes(ctx, sizeof(double) * O::DOUBLES, kMinClassPairs, ci));
    if (ci.ntc > 0) {
      TB_CUDA(ctx, T.ops64.ensure(O::DOUBLES * ci.ntc, s));
      TB_CUDA(ctx, T.Mt64.ensure((size_t)C * O::KP, s));
    }
    // the tile tables and the rows, in shorter ranges where memory is too short for the rows
    for (;; per_range = (per_range + 1) / 2) {
      nrange = (n + per_range - 1) / per_range;
      parts = ci.ntc * nrange;
      max_tiles = n / kPairTile + parts;
      auto room = [&]() -> cudaError_t {
        cudaError_t e = T.cnt64.ensure(parts + 1, s);
        if (e == cudaSuccess) e = T.off64.ensure(parts + 1, s);
        if (e == cudaSuccess) e = T.part64.ensure(parts + 1, s);
        if (e == cudaSuccess) e = T.items64.ensure(max_tiles + 1, s);
        return e == cudaSuccess ? T.rows64.ensure((size_t)per_range * O::K, s) : e;
      };
      const cudaError_t e = room();
      if (e == cudaErrorMemoryAllocation &&
          (size_t)per_range * sizeof(double) * O::K > kLeastRowBytes) {
        cudaGetLastError();
        continue;
      }
      TB_CUDA(ctx, e);
      break;
    }
    if (ci.ntc > 0) {
      build_operators64<P><<<(unsigned)ci.ntc, 256, 0, s>>>(T.tc_keys.p, T.ops64.p);
      TB_LAUNCH_CHECK(ctx);
      normalize_M64<P><<<grid_for(C, 8, ctx->num_sms * 8), 256, 0, s>>>(
          C, ctx->cnb.p, ctx->cmin.p, ctx->cmax.p, ctx->M.p,
          reinterpret_cast<double2 *>(T.Mt64.p));
      TB_LAUNCH_CHECK(ctx);
      // tiles, ranges outermost
      count_tiles64<<<grid_for(parts, 256), 256, 0, s>>>(T.cls_range.p, ci.ntc, nrange, per_range,
                                                         T.vals.p, T.cnt64.p, T.part64.p);
      TB_LAUNCH_CHECK(ctx);
      TB_TRY(scan_exclusive(ctx, T.cnt64.p, T.off64.p, parts, T.off64.p + parts));
      emit_tiles64<<<grid_for(parts, 8), 256, 0, s>>>(ci.ntc, nrange, T.off64.p, T.part64.p,
                                                      T.items64.p);
      TB_LAUNCH_CHECK(ctx);
    }
  }
  PhaseTimer t(ctx, &ctx->timings.m2l_fp64);
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  for (int64_t q = 0; q < nrange; q++) {
    const int64_t base = q * per_range, count = std::min(per_range, n - base);
    if (ci.ntc > 0) {
      // three blocks per SM, never more warps than a range can have tiles
      const int64_t most = std::min(max_tiles, count / kPairTile + ci.ntc);
      product_tiles64<P><<<grid_for(most, kGemmWarps, ctx->num_sms * 3), 32 * kGemmWarps, 0, s>>>(
          T.off64.p, q * ci.ntc, (q + 1) * ci.ntc, T.items64.p, T.vals.p, ctx->m2l.p,
          ctx->list_shift, base, T.ops64.p, T.Mt64.p, T.rows64.p);
      TB_LAUNCH_CHECK(ctx);
    }
    if (ci.n64 > 0) {
      product_pairs64<P><<<grid_for(ci.n64, 4, ctx->num_sms * 16), 128, 0, s>>>(
          T.pairs64.p, ci.n64, base, count, ctx->m2l.p, ctx->list_shift, ctx->cnb.p, ctx->cmin.p,
          ctx->cmax.p, ctx->ccen.p, ctx->M.p, reinterpret_cast<double2 *>(T.rows64.p));
      TB_LAUNCH_CHECK(ctx);
    }
    sum_products64<P><<<grid_for(C * ((O::NT + 31) / 32), 8, ctx->num_sms * 16), 256, 0, s>>>(
        C, ctx->m2l_off.p, ctx->m2l.p, mask, base, count, ctx->lists_have_empty ? 1 : 0, ctx->cnb.p,
        owned_cells(ctx), ctx->cmin.p, ctx->cmax.p, reinterpret_cast<const double2 *>(T.rows64.p),
        ctx->L.p);
    TB_LAUNCH_CHECK(ctx);
  }
  ctx->tc_classes = ci.ntc;
  return TAPAS_B200_OK;
}

}  // namespace

int m2l_fp64(tapas_b200_ctx *ctx) {
  switch (ctx->P) {
    case 4: return m2l_products_P<4>(ctx);
    case 5: return m2l_products_P<5>(ctx);
    case 6: return m2l_products_P<6>(ctx);
    case 7: return m2l_products_P<7>(ctx);
    case 8: return m2l_products_P<8>(ctx);
    case 9: return m2l_products_P<9>(ctx);
    case 10: return m2l_products_P<10>(ctx);
    case 11: return m2l_products_P<11>(ctx);
    case 12: return m2l_products_P<12>(ctx);
    case 13: return m2l_products_P<13>(ctx);
    case 14: return m2l_products_P<14>(ctx);
    case 15: return m2l_products_P<15>(ctx);
    case 16: return m2l_products_P<16>(ctx);
    default: return m2l_fp64_cells(ctx);  // P = 2, 3: a warp per target
  }
}

}  // namespace tb
