// Near field (P2P) over the leaf-pair list, replacing the reference's
// vectormap_cuda_pack_kernel2 (cpp/include/tapas/vectormap_cuda.h:219-280)
// with the P2P functor of ex/LaplaceP2PCPU_tapas.h:23-44.
//
// The reference packs target leaves per source leaf and accumulates every
// pair with four CAS-loop atomics on the target attributes.  Here the list is
// grouped by TARGET leaf (CSR) and one warp owns a target leaf at a time:
//  - warps take target leaves from a global queue ordered by decreasing work
//    (nt * sum of source bodies), so long interaction lists start first;
//  - each lane keeps kR targets in registers (kR a template parameter, so no
//    issue slot is spent on unused target slots): the targets take
//    L = ceil(nt/kR) lanes and the warp holds G = 32/L copies of them that split
//    the sources, with kR chosen so that kR/G (time per source) is least;
//  - source bodies are staged in the warp's shared-memory slice and read as
//    broadcasts; each target's sum is written once, without atomics.
//
// FP64 form: the reference's sums (pot += qi qj / r, acc -= qi qj dX/r^3, r == 0
// skipped; the common factor qi at the end), 1/r by charge_over_distance.
//
// Mixed form: FP32 arithmetic with results per unit charge.  Targets and sources
// are taken into the target leaf's frame by an FP64 subtraction (its pipe is idle
// here) and kept as FP32 (hi, lo) parts, so the separation x_i - x_j is formed
// from ~48-bit operands and rounds once.  1/r is the hardware rsqrt (its error is far below
// the near field's summation error, so no Newton step).
// A source leaf whose box is far enough from the target's box skips the lo
// parts.  In the target frame a source coordinate is at most gap + tw/2 + sw
// in magnitude (gap: the boxes' separation along the farthest axis, tw, sw:
// the target and source widths) and every separation is at least gap, so one
// rounding of a coordinate is at most 2^-24 (gap + tw/2 + sw) / gap of the
// separation; with gap >= (tw/2 + sw) / 3 that is <= 4 * 2^-24 ~ 2.4e-7.
// Every 64 source bodies are summed in plain FP32 and the partial is added to the
// target's FP64 sums.
#include <algorithm>
#include <cfloat>

#include "kernels.cuh"
#include "primitives.cuh"

namespace tb {
namespace {

constexpr int kWarps = 4;  // FP64 kernel: 4-warp CTAs, 4 per SM (<= 128 registers)
constexpr int kThreads = 32 * kWarps;
constexpr int kFp64Blocks = 4;
constexpr int kStage = 64;   // mixed: source bodies staged per warp at a time (two per lane)
// mixed kernel: 4-warp CTAs, up to 3 targets per lane (leaves of more than 96
// bodies take two passes)
constexpr int kMixedWarps = 4;
constexpr int kMixedMaxR = 3;
constexpr int kMixedBlocks = 5;     // CTAs per SM (<= 102 registers)
constexpr float kNowhere = 1.25e18f;  // coordinate of a chargeless padding source
constexpr int kMixedThreads = 32 * kMixedWarps;

// ---------------------------------------------------------------------------
// work items: a target leaf with its source list, or a piece of a long list
// ---------------------------------------------------------------------------
// A target leaf with more than piece_pairs body pairs is split into consecutive
// list ranges of about that many, so no single warp carries it alone: with one
// item per leaf the last warps ran on while most of the GPU was idle (1M and
// 300k sphere, FP64: the SMs were busy 60 and 41 % of the kernel's time).  A
// piece writes its partial sums to its own rows of a scratch array;
// split_reduce adds a leaf's pieces in order, so the result does not depend on
// which warp finished first.  piece_pairs is an eighth of a warp's share of all
// pairs (the tail is then at most that), but at least kMinPiecePairs, below
// which a piece's own start and its partial rows cost more than the tail.
constexpr int64_t kMinPiecePairs = 16384;

struct WorkItem {
  int32_t leaf, e0, e1;  // target leaf (cell index) and its list range [e0, e1)
  int32_t pbase;         // -1: writes trg directly; else first row of its partials
};

// Queue key of an item of that many body pairs: decreasing work in steps of an
// eighth of an octave, so that one radix pass orders the queue (exact order took
// four, 12 launches, and shortens the tail by nothing that shows).
__device__ __forceinline__ uint64_t work_key(uint64_t work) {
  if (work == 0) return 255;
  const int e = 63 - __clzll((long long)work);  // work in [2^e, 2^(e+1))
  const int f = (int)((e >= 3 ? work >> (e - 3) : work << (3 - e)) & 7);
  return 255 - min(255, 8 * max(e - 4, 0) + f);
}

// per non-empty leaf w (eight threads): its work key, pieces k (>= 1) and partial
// rows (k * nt when split)
__global__ void __launch_bounds__(256) leaf_pieces(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ off,
    const uint64_t *__restrict__ list, uint64_t src_mask, const int32_t *__restrict__ cnb,
    int64_t piece_pairs, uint8_t *__restrict__ wkey, int32_t *__restrict__ kcnt,
    int32_t *__restrict__ psz, int *__restrict__ counter) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *counter = 0;  // the queue's head
  const int sub = threadIdx.x & 7;
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x) >> 3;
  for (int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31)) >> 3; w0 < nleaves;
       w0 += stride) {  // warp-uniform
    const int64_t w = w0 + ((threadIdx.x & 31) >> 3);
    const bool in = w < nleaves;
    const int c = in ? leaves[w] : 0;
    const int e0 = off[c], e1 = in ? off[c + 1] : e0;
    int64_t ns = 0;
    for (int e = e0 + sub; e < e1; e += 8) ns += cnb[(int)(list[e] & src_mask)];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) ns += __shfl_xor_sync(0xffffffffu, ns, o);
    if (!in || sub != 0) continue;
    const int64_t entries = e1 - e0;
    const int64_t k = max((int64_t)1, min((ns * cnb[c] + piece_pairs - 1) / piece_pairs, entries));
    wkey[w] = (uint8_t)work_key((uint64_t)ns * (uint64_t)cnb[c]);
    kcnt[w] = (int32_t)k;
    psz[w] = k > 1 ? (int32_t)(k * cnb[c]) : 0;
  }
}

// Items of leaf w at koff[w].. (eight threads): its whole list, or its list cut
// after every entry that carries the leaf's running body pairs past a multiple of
// piece_pairs: at most k pieces; slots a large source leaf leaves unused become
// empty pieces with zeroed partials.  Work key = the piece's body pairs, for the
// queue.  (One thread per leaf walked the longest lists alone: 0.12 of 1.9 ms for
// 1M Plummer.)
__global__ void __launch_bounds__(256) emit_items(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ off,
    const uint64_t *__restrict__ list, uint64_t src_mask, const int32_t *__restrict__ cnb,
    int64_t piece_pairs, const uint8_t *__restrict__ wkey, const int32_t *__restrict__ kcnt,
    const int32_t *__restrict__ koff, const int32_t *__restrict__ poff,
    WorkItem *__restrict__ items, uint64_t *__restrict__ keys, uint32_t *__restrict__ vals,
    double *__restrict__ part) {
  const int sub = threadIdx.x & 7, shift = threadIdx.x & 24;  // the group's first lane
  const unsigned group = 0xffu << shift;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; w < nleaves;
       w += ((int64_t)gridDim.x * blockDim.x) >> 3) {
    const int c = leaves[w];
    const int e0 = off[c], e1 = off[c + 1], k = kcnt[w], nt = cnb[c];
    const int base = koff[w];
    auto put = [&](int j, int ea, int ez, uint64_t key) {
      items[base + j] = WorkItem{c, ea, ez, k > 1 ? poff[w] + j * nt : -1};
      keys[base + j] = key;
      vals[base + j] = (uint32_t)(base + j);
    };
    if (k == 1) {  // the whole list (an empty one still writes the leaf's zero sums)
      if (sub == 0) put(0, e0, e1, wkey[w]);
      continue;
    }
    int j = 0, ea = e0;              // next piece and its first entry
    int64_t before = 0, begun = 0;   // bodies before this chunk, before entry ea
    for (int e = e0; e < e1; e += 8) {
      const int64_t ns = e + sub < e1 ? cnb[(int)(list[e + sub] & src_mask)] : 0;
      int64_t upto = ns;
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const int64_t v = __shfl_up_sync(group, upto, o, 8);
        if (sub >= o) upto += v;
      }
      upto += before;
      const bool cut = e + sub < e1 &&
                       (upto * nt / piece_pairs > (upto - ns) * nt / piece_pairs ||
                        e + sub == e1 - 1);
      unsigned cuts = (__ballot_sync(group, cut) >> shift) & 0xffu;
      while (cuts) {
        const int i = __ffs(cuts) - 1;
        cuts &= cuts - 1;
        const int64_t end = __shfl_sync(group, upto, i, 8);
        if (sub == 0) put(j, ea, e + i + 1, work_key((uint64_t)(end - begun) * (uint64_t)nt));
        j++;
        ea = e + i + 1;
        begun = end;
      }
      before = __shfl_sync(group, upto, 7, 8);
    }
    for (; j < k; j++) {  // unused pieces
      if (sub == 0) put(j, e1, e1, work_key(0));
      for (int t = sub; t < 4 * nt; t += 8)
        part[4 * ((int64_t)poff[w] + (int64_t)j * nt) + t] = 0.0;
    }
  }
}

// trg rows of split leaves = sum of their pieces' partial rows, in piece order
// (a warp per leaf, the rows' loads in flight together)
__global__ void split_reduce(const int32_t *__restrict__ leaves, int64_t nleaves,
                             const int32_t *__restrict__ cbeg, const int32_t *__restrict__ cnb,
                             const int32_t *__restrict__ kcnt, const int32_t *__restrict__ poff,
                             const double *__restrict__ part, double *__restrict__ trg) {
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nleaves;
       w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int k = kcnt[w];
    if (k <= 1) continue;
    const int c = leaves[w], nt = cnb[c], b0 = cbeg[c];
    for (int t = threadIdx.x & 31; t < nt; t += 32) {
      double4 acc = make_double4(0, 0, 0, 0);
#pragma unroll 8
      for (int j = 0; j < k; j++) {
        const double4 v =
            reinterpret_cast<const double4 *>(part)[(int64_t)poff[w] + (int64_t)j * nt + t];
        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
      }
      reinterpret_cast<double4 *>(trg)[b0 + t] = acc;
    }
  }
}

// Where a work item's sums go: trg rows of its leaf, or its partial rows.
__device__ __forceinline__ double4 *item_out(const WorkItem &it, int tb0, double *trg,
                                             double *part) {
  return it.pbase < 0 ? reinterpret_cast<double4 *>(trg) + tb0
                      : reinterpret_cast<double4 *>(part) + it.pbase;
}

__device__ __forceinline__ int next_leaf(int *counter, int lane) {
  int w = 0;
  if (lane == 0) w = atomicAdd(counter, 1);
  return __shfl_sync(0xffffffffu, w, 0);
}

// Shape of a tile of nt targets: kR targets per lane, L = ceil(nt/kR) lanes per
// group, G = 32/L groups that split the sources.  Time per source ~ kR / G: the
// least of the kernel's three kR (ties: the larger kR, fewer shared loads and
// more independent chains per lane).  Three, because every variant takes room in
// the instruction cache, where stalls were half as frequent again as issue with
// four.  FP64 uses 4, 3, 1 (89 % of the lanes on leaves of 16 to 64 bodies);
// the mixed kernel 3, 2, 1 (87 %): a fourth target's registers cost it more than
// the lanes (1M Plummer 1.83 against 1.93 ms, 16M sphere 26.4 against 26.7).
template <int kR0, int kR1>
__device__ __forceinline__ void tile_shape(int nt, int &R, int &L, int &G) {
  R = kR0;
  L = (nt + kR0 - 1) / kR0;
  G = 32 / L;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int r = i == 0 ? kR1 : 1;
    const int l = (nt + r - 1) / r;
    if (l > 32) break;
    const int g = 32 / l;
    if (r * G < R * g) {
      R = r;
      L = l;
      G = g;
    }
  }
}

// ---------------------------------------------------------------------------
// FP64
// ---------------------------------------------------------------------------
// Lane (g, l) holds targets l, l + L, ... and takes every G-th staged source;
// the groups' sums are added in group order at the end, so the result is a
// fixed-order sum.  The source bodies of the item's list range are one stream:
// the list is read 32 leaves at a time (lane j: entry j's body range and the
// running count of bodies), and each chunk of 32 consecutive bodies of the
// stream is staged by a lane each, which finds its leaf by a binary search over
// the 32 counts with shuffles, so every chunk but a batch's last is full
// whatever the leaf sizes; the next chunk's loads are issued before the
// current one is computed.
//
// Bound: the FP64 pipe, 18 of its slots per pair (3 separations, 3 for r^2, 5
// for the refined 1/r, 3 for q/r and q/r^3, 4 sums), 3.55 pairs per clock and SM.
template <int kR>
__device__ __forceinline__ void fp64_tile(int lane, int tb0, int nt, int L, int G, int e0, int e1,
                                          const uint64_t *__restrict__ list, uint64_t mask,
                                          const int32_t *__restrict__ cbeg,
                                          const int32_t *__restrict__ cnb,
                                          const double *__restrict__ sx,
                                          const double *__restrict__ sy,
                                          const double *__restrict__ sz,
                                          const double *__restrict__ sq, double4 *src,
                                          double4 *__restrict__ out) {
  const int g = lane / L, tl = lane - g * L;
  const bool active = g < G;
  double xi[kR], yi[kR], zi[kR], pot[kR], ax[kR], ay[kR], az[kR];
#pragma unroll
  for (int r = 0; r < kR; r++) {
    const int i = tl + L * r;
    const bool v = active && i < nt;
    xi[r] = v ? sx[tb0 + i] : 0.0;
    yi[r] = v ? sy[tb0 + i] : 0.0;
    zi[r] = v ? sz[tb0 + i] : 0.0;
    pot[r] = ax[r] = ay[r] = az[r] = 0.0;
  }
  for (int eb = e0; eb < e1; eb += 32) {
    int beg = 0, ns = 0;
    if (eb + lane < e1) {
      const int s = (int)(list[eb + lane] & mask);
      beg = cbeg[s];
      ns = cnb[s];
    }
    int upto = ns;  // bodies of the batch's leaves 0 .. lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    beg -= upto - ns;  // body i of the stream is body beg + i of its leaf's range
    double4 b = make_double4(0, 0, 0, 0);
    auto load = [&](int c0) {
      const int i = c0 + lane;
      int leaf = 0;  // the first leaf with upto > i
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const int v = __shfl_sync(0xffffffffu, upto, leaf + o - 1);
        if (v <= i) leaf += o;
      }
      const int j = __shfl_sync(0xffffffffu, beg, leaf & 31) + i;
      if (i < total) b = make_double4(sx[j], sy[j], sz[j], sq[j]);
    };
    if (total > 0) load(0);
    for (int c0 = 0; c0 < total; c0 += 32) {
      const int cnt = min(32, total - c0);
      __syncwarp();
      src[lane] = b;
      __syncwarp();
      if (c0 + 32 < total) load(c0 + 32);
      if (!active) continue;
      // kU sources at a time: at least three separations in flight per lane
      constexpr int kU = kR == 1 ? 4 : 1, N = kU * kR;
      for (int k = g; k < cnt; k += kU * G) {
        double dx[N], dy[N], dz[N], R2[N], q[N], qr[N], inv[N];
#pragma unroll
        for (int u = 0; u < kU; u++) {
          const bool in = kU == 1 || k + u * G < cnt;
          const double4 s = src[in ? k + u * G : k];
#pragma unroll
          for (int r = 0; r < kR; r++) {
            const int i = u * kR + r;
            dx[i] = xi[r] - s.x;
            dy[i] = yi[r] - s.y;
            dz[i] = zi[r] - s.z;
            R2[i] = dx[i] * dx[i] + dy[i] * dy[i] + dz[i] * dz[i];
            if (!in) R2[i] = 0.0;  // adds nothing
            q[i] = s.w;
          }
        }
        charge_over_distance(R2, q, qr, inv);
#pragma unroll
        for (int i = 0; i < N; i++) {
          const int r = i % kR;
          const double s3 = inv[i] * inv[i] * qr[i];
          pot[r] += qr[i];
          ax[r] = fma(-dx[i], s3, ax[r]);
          ay[r] = fma(-dy[i], s3, ay[r]);
          az[r] = fma(-dz[i], s3, az[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kR; r++) {
    const int i = tl + L * r;
    double4 v = make_double4(pot[r], ax[r], ay[r], az[r]);
    if (G > 1) {
      __syncwarp();
      src[lane] = v;
      __syncwarp();
      if (g == 0) {
        for (int gg = 1; gg < G; gg++) {
          const double4 o = src[tl + gg * L];
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
      }
    }
    if (active && g == 0 && i < nt) {  // the reference's TRG: times the target's charge
      const double qi = sq[tb0 + i];
      out[i] = make_double4(qi * v.x, qi * v.y, qi * v.z, qi * v.w);
    }
  }
  __syncwarp();
}

__global__ void __launch_bounds__(kThreads, kFp64Blocks) p2p_fp64_kernel(
    const uint32_t *__restrict__ order, int64_t nitems, int *__restrict__ counter,
    const WorkItem *__restrict__ items, const uint64_t *__restrict__ list, uint64_t src_mask,
    const int32_t *__restrict__ cbeg, const int32_t *__restrict__ cnb,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, double *__restrict__ trg, double *__restrict__ part) {
  __shared__ double4 src[kWarps][32];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  for (;;) {
    const int w = next_leaf(counter, lane);
    if (w >= nitems) break;
    const WorkItem it = items[order[w]];
    if (it.pbase >= 0 && it.e0 == it.e1) continue;  // unused piece of a split list
    const int c = it.leaf;
    const int tb0 = cbeg[c], nt_all = cnb[c];
    double4 *out = item_out(it, tb0, trg, part);
    for (int tbase = 0; tbase < nt_all; tbase += 128) {
      const int nt = min(nt_all - tbase, 128);
      int R, L, G;
      tile_shape<4, 3>(nt, R, L, G);
#define TB_FP64_TILE(RR)                                                                         \
  fp64_tile<RR>(lane, tb0 + tbase, nt, L, G, it.e0, it.e1, list, src_mask, cbeg, cnb, sx, sy, sz, \
                sq, src[wi], out + tbase)
      if (R == 4) TB_FP64_TILE(4);
      else if (R == 3) TB_FP64_TILE(3);
      else TB_FP64_TILE(1);
#undef TB_FP64_TILE
    }
  }
}

// ---------------------------------------------------------------------------
// mixed
// ---------------------------------------------------------------------------
// 1/sqrt(x) for normal x > 0 from the hardware approximation (relative error
// below 2^-22.9), without the denormal rescaling rsqrtf adds; callers treat
// x < FLT_MIN (a separation below ~1e-19) as coincident bodies.
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// A source leaf of the current batch: body i of the batch's stream of source
// bodies is body b0 + i for the leaf that holds it; far: 1 its box is far enough
// for plain FP32 coordinates (see above), 0 its bodies are tested one by one, -1
// it is the target leaf, whose bodies are near whatever their coordinates: the root
// box can leave bodies outside (they go to the cells at its faces) and be a point,
// and a far body is never compared with itself.
struct __align__(8) LeafMeta {
  int b0, far;
};

// One warp's shared memory.
struct __align__(16) MixedWarp {
  float fx[kStage], fy[kStage], fz[kStage], fq[kStage];  // far: minus coordinates, charge
  float4 near_hi[kStage], near_lo[kStage];               // near: hi parts and charge, lo parts
  LeafMeta meta[32];
  double sum[kMixedMaxR][4][32];   // pot, ax, ay, az per target
  float lo[kMixedMaxR][3][32];     // the targets' lo parts
};

// One tile of a target leaf: lane (g, l) = (lane / L, lane % L) holds targets
// l, l + L, ..., l + (kR-1) L and takes its share of the staged sources.
//
// The source bodies of the target's list are one stream: the list is read 32
// leaves at a time (lane j: entry j's body range and the running body count), and
// 64 consecutive bodies of the stream are staged at a time,
// two per lane; a lane finds its bodies' leaf by a binary search over the 32
// counts with shuffles.  Each body is classed far or near and the far ones are
// stored as coordinate arrays, so that two consecutive sources are one
// load per coordinate and are evaluated per packed FP32 instruction: 13 packed
// operations and 2 MUFU per two pairs.  FP32 additions, multiplications and
// fmas run at the same rate packed or not (measured 112 to 125 lanes per clock
// and SM either way), so the gain is the issue slots: the pair formula alone
// reached 8.1 pairs per clock and SM scalar, 9.05 packed, 9.85 being the pipe.
// With one target per lane the broadcast loads (4 cycles of the shared-memory
// port each) are the bound at 7.8, hence tiles with as many targets per lane
// as splitting the sources over lane groups allows.
template <int kR>
__device__ __forceinline__ void mixed_tile(
    int lane, int c, int tb0, int nt, int L, int G, int e0, int e1, double tcx, double tcy,
    double tcz, double tw, const uint64_t *__restrict__ list, uint64_t mask, const int32_t *__restrict__ cbeg,
    const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, MixedWarp &sm, double4 *__restrict__ out) {
  const int g = lane / L, tl = lane - g * L;
  const bool active = g < G;
  // a source body this far from the target leaf's centre (max norm) is far;
  // the margin covers the FP32 rounding of the test itself
  const float far_body = (float)(tw * (5.0 / 6.0)) * (1.0f + 1e-6f);
  float2 txh[kR], tyh[kR], tzh[kR];  // both halves the target's coordinate
  float2 tp[kR], tx[kR], ty[kR], tz[kR];  // sums of the even and the odd sources
  const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
  for (int r = 0; r < kR; r++) {
    const int t = tl + L * r;
    const bool v = active && t < nt;
    const double dx = v ? sx[tb0 + t] - tcx : 0.0, dy = v ? sy[tb0 + t] - tcy : 0.0,
                 dz = v ? sz[tb0 + t] - tcz : 0.0;
    const float hx = (float)dx, hy = (float)dy, hz = (float)dz;
    txh[r] = make_float2(hx, hx);
    tyh[r] = make_float2(hy, hy);
    tzh[r] = make_float2(hz, hz);
    sm.lo[r][0][lane] = (float)(dx - hx);
    sm.lo[r][1][lane] = (float)(dy - hy);
    sm.lo[r][2][lane] = (float)(dz - hz);
#pragma unroll
    for (int k = 0; k < 4; k++) sm.sum[r][k][lane] = 0.0;
    tp[r] = tx[r] = ty[r] = tz[r] = zero;
  }
  // far bodies: plain FP32 coordinates in the target frame (relative error of a
  // separation <= ~2.4e-7), no r = 0 case
  auto far2 = [&](float2 sx, float2 sy, float2 sz, float2 sq) {
#pragma unroll
    for (int r = 0; r < kR; r++) {
      const float2 dx = __fadd2_rn(txh[r], sx), dy = __fadd2_rn(tyh[r], sy),
                   dz = __fadd2_rn(tzh[r], sz);
      const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
      const float2 ri = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
      const float2 qr = __fmul2_rn(sq, ri);
      const float2 qr3 = __fmul2_rn(__fmul2_rn(qr, ri), ri);
      tp[r] = __fadd2_rn(tp[r], qr);
      tx[r] = __ffma2_rn(dx, qr3, tx[r]);
      ty[r] = __ffma2_rn(dy, qr3, ty[r]);
      tz[r] = __ffma2_rn(dz, qr3, tz[r]);
    }
  };
  for (int eb = e0; eb < e1; eb += 32) {
    __syncwarp();  // the previous batch's table is read
    int ns = 0;
    LeafMeta m{};
    if (eb + lane < e1) {
      const int s = (int)(list[eb + lane] & mask);
      m.b0 = cbeg[s];
      ns = cnb[s];
      const double dcx = ccen[3 * s] - tcx, dcy = ccen[3 * s + 1] - tcy,
                   dcz = ccen[3 * s + 2] - tcz;
      // boxes separated by gap along the farthest axis: every pair is >= gap apart
      const double sw = cmax[3 * s] - cmin[3 * s];
      const double gap = fmax(fabs(dcx), fmax(fabs(dcy), fabs(dcz))) - 0.5 * (tw + sw);
      m.far = s == c ? -1 : 3.0 * gap >= 0.5 * tw + sw ? 1 : 0;
    }
    int upto = ns;  // bodies of the batch's leaves 0 .. lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    m.b0 -= upto - ns;
    sm.meta[lane] = m;
    for (int c0 = 0; c0 < total; c0 += kStage) {
      __syncwarp();  // the table is written; the previous chunk is read
      // Far bodies as single floats, near ones as (hi, lo).  A body is
      // far when its whole leaf is, or when its max-norm distance from the
      // target leaf's centre is at least 5/6 of the leaf width: then every
      // target is >= D - tw/2 away while the coordinates are <= D and tw/2, so
      // one rounding is <= 2^-24 (D + tw/2) / (D - tw/2) <= 4 * 2^-24 of a
      // separation, the leaf rule's bound.
      int nfar = 0, nnear = 0;
#pragma unroll
      for (int h = 0; h < kStage / 32; h++) {
        const int i = c0 + 32 * h + lane;
        if (c0 + 32 * h >= total) break;  // warp-uniform
        int leaf = 0;  // the first leaf with upto > i
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int v = __shfl_sync(0xffffffffu, upto, leaf + o - 1);
          if (v <= i) leaf += o;
        }
        const bool valid = i < total;
        // position in the target leaf's frame: the FP64 difference, rounded once
        double dx = 0.0, dy = 0.0, dz = 0.0;
        float hx = 0.f, hy = 0.f, hz = 0.f, q = 0.f;
        bool farb = false;
        if (valid) {
          const LeafMeta lm = sm.meta[leaf];
          const int j = lm.b0 + i;
          dx = sx[j] - tcx;
          dy = sy[j] - tcy;
          dz = sz[j] - tcz;
          q = (float)sq[j];
          hx = (float)dx;
          hy = (float)dy;
          hz = (float)dz;
          farb = lm.far > 0 || (lm.far == 0 &&
                                fmaxf(fabsf(hx), fmaxf(fabsf(hy), fabsf(hz))) >= far_body);
        }
        const unsigned fm = __ballot_sync(0xffffffffu, farb);
        const unsigned nm = __ballot_sync(0xffffffffu, valid && !farb);
        const unsigned below = (1u << lane) - 1u;
        if (farb) {
          const int k = nfar + __popc(fm & below);
          sm.fx[k] = -hx;
          sm.fy[k] = -hy;
          sm.fz[k] = -hz;
          sm.fq[k] = q;
        } else if (valid) {
          const int k = nnear + __popc(nm & below);
          sm.near_hi[k] = make_float4(hx, hy, hz, q);
          sm.near_lo[k] =
              make_float4((float)(dx - hx), (float)(dy - hy), (float)(dz - hz), 0.f);
        }
        nfar += __popc(fm);
        nnear += __popc(nm);
      }
      // an odd last far body is paired with a chargeless one far away
      if (lane == 0 && (nfar & 1)) {
        sm.fx[nfar] = sm.fy[nfar] = sm.fz[nfar] = kNowhere;
        sm.fq[nfar] = 0.f;
      }
      __syncwarp();
      if (active) {
        // loops short enough for the instruction cache nearest the scheduler: with
        // two or three targets a lane has that many independent chains anyway
#pragma unroll(kR == 1 ? 2 : 1)
        for (int k = 2 * g; k < nfar; k += 2 * G)
          far2(*reinterpret_cast<const float2 *>(sm.fx + k),
               *reinterpret_cast<const float2 *>(sm.fy + k),
               *reinterpret_cast<const float2 *>(sm.fz + k),
               *reinterpret_cast<const float2 *>(sm.fq + k));
        // near bodies: separations from (hi, lo) coordinates
#pragma unroll(kR == 1 ? 2 : 1)
        for (int k = g; k < nnear; k += G) {
          const float4 bh = sm.near_hi[k];
          const float4 bl = sm.near_lo[k];
#pragma unroll
          for (int r = 0; r < kR; r++) {
            const float dx = (txh[r].x - bh.x) + (sm.lo[r][0][lane] - bl.x);
            const float dy = (tyh[r].x - bh.y) + (sm.lo[r][1][lane] - bl.y);
            const float dz = (tzh[r].x - bh.z) + (sm.lo[r][2][lane] - bl.z);
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            const float ri = r2 >= FLT_MIN ? rsqrt_ftz(r2) : 0.f;
            const float qr = bh.w * ri;
            const float qr3 = qr * ri * ri;
            tp[r].x += qr;
            tx[r].x = fmaf(dx, qr3, tx[r].x);
            ty[r].x = fmaf(dy, qr3, ty[r].x);
            tz[r].x = fmaf(dz, qr3, tz[r].x);
          }
        }
      }
      // a chunk is summed in FP32 and added to the target's FP64 sums
#pragma unroll
      for (int r = 0; r < kR; r++) {
        sm.sum[r][0][lane] += (double)(tp[r].x + tp[r].y);
        sm.sum[r][1][lane] += (double)(tx[r].x + tx[r].y);
        sm.sum[r][2][lane] += (double)(ty[r].x + ty[r].y);
        sm.sum[r][3][lane] += (double)(tz[r].x + tz[r].y);
        tp[r] = tx[r] = ty[r] = tz[r] = zero;
      }
    }
  }
  double4 *red = reinterpret_cast<double4 *>(sm.near_hi);  // the sources are done with
#pragma unroll
  for (int r = 0; r < kR; r++) {
    double4 v = make_double4(sm.sum[r][0][lane], -sm.sum[r][1][lane], -sm.sum[r][2][lane],
                             -sm.sum[r][3][lane]);
    if (G > 1) {
      __syncwarp();
      red[lane] = v;
      __syncwarp();
      if (g == 0) {
        for (int gg = 1; gg < G; gg++) {
          const double4 o = red[tl + gg * L];
          v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
        }
      }
    }
    const int t = tl + L * r;
    if (active && g == 0 && t < nt) out[t] = v;
  }
  __syncwarp();  // the next tile reuses the warp's shared memory
}

template <int kBlocks>
__global__ void __launch_bounds__(kMixedThreads, kBlocks) p2p_mixed_kernel(
    const uint32_t *__restrict__ order, int64_t nitems, int *__restrict__ counter,
    const WorkItem *__restrict__ items, const uint64_t *__restrict__ list, uint64_t src_mask,
    const int32_t *__restrict__ cbeg, const int32_t *__restrict__ cnb,
    const double *__restrict__ ccen, const double *__restrict__ cmin,
    const double *__restrict__ cmax, const double *__restrict__ sx,
    const double *__restrict__ sy, const double *__restrict__ sz, const double *__restrict__ sq,
    double *__restrict__ trg, double *__restrict__ part) {
  __shared__ MixedWarp sm[kMixedWarps];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  for (;;) {
    const int w = next_leaf(counter, lane);
    if (w >= nitems) break;
    const WorkItem it = items[order[w]];
    if (it.pbase >= 0 && it.e0 == it.e1) continue;  // unused piece of a split list
    const int c = it.leaf;
    const int tb0 = cbeg[c], nt_all = cnb[c];
    const int e0 = it.e0, e1 = it.e1;
    double4 *out = item_out(it, tb0, trg, part);
    const double tcx = ccen[3 * c], tcy = ccen[3 * c + 1], tcz = ccen[3 * c + 2];
    const double tw = cmax[3 * c] - cmin[3 * c];
    for (int tbase = 0; tbase < nt_all; tbase += 32 * kMixedMaxR) {
      const int nt = min(nt_all - tbase, 32 * kMixedMaxR);
      int R, L, G;
      tile_shape<3, 2>(nt, R, L, G);
#define TB_MIXED_TILE(RR)                                                                        \
  mixed_tile<RR>(lane, c, tb0 + tbase, nt, L, G, e0, e1, tcx, tcy, tcz, tw, list, src_mask, cbeg,  \
                 cnb, ccen, cmin, cmax, sx, sy, sz, sq, sm[wi], out + tbase)
      if (R == 3) TB_MIXED_TILE(3);
      else if (R == 2) TB_MIXED_TILE(2);
      else TB_MIXED_TILE(1);
#undef TB_MIXED_TILE
    }
  }
}

// Pieces of each leaf's list for a grid of warps_per_sm warps, and the read-back
// of their totals.
int count_items(tapas_b200_ctx *ctx, int warps_per_sm) {
  cudaStream_t s = ctx->stream;
  const int64_t piece_pairs = std::max<int64_t>(
      kMinPiecePairs, (int64_t)(ctx->n_p2p_int / ((uint64_t)ctx->num_sms * warps_per_sm * 8)));
  ctx->p2p_piece_pairs = piece_pairs;
  int64_t nl = 0;
  const int32_t *leaves = work_leaves(ctx, nl);  // sharded: owned target leaves
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  TB_CUDA(ctx, ctx->p2p_kcnt.ensure(nl + 1, s));
  TB_CUDA(ctx, ctx->p2p_koff.ensure(nl + 1, s));
  TB_CUDA(ctx, ctx->p2p_psz.ensure(nl + 1, s));
  TB_CUDA(ctx, ctx->p2p_poff.ensure(nl + 1, s));
  TB_CUDA(ctx, ctx->p2p_key.ensure(nl + 1, s));
  TB_CUDA(ctx, ctx->p2p_counter.ensure(4, s));
  leaf_pieces<<<grid_for(8 * nl, 256), 256, 0, s>>>(leaves, nl, ctx->p2p_off.p, ctx->p2p.p, mask,
                                                    ctx->cnb.p, piece_pairs, ctx->p2p_key.p,
                                                    ctx->p2p_kcnt.p, ctx->p2p_psz.p,
                                                    ctx->p2p_counter.p);
  TB_LAUNCH_CHECK(ctx);
  const int32_t *const in[2] = {ctx->p2p_kcnt.p, ctx->p2p_psz.p};
  int32_t *const out[2] = {ctx->p2p_koff.p, ctx->p2p_poff.p};
  int32_t *const tot[2] = {ctx->p2p_counter.p + 1, ctx->p2p_counter.p + 2};
  TB_TRY(scan_exclusive2(ctx, in, out, nl, tot, nullptr));
  TB_CUDA(ctx, ctx->pinned.ensure(tapas_b200_ctx::kPinnedBytes));
  if (!ctx->p2p_counted)
    TB_CUDA(ctx, cudaEventCreateWithFlags(&ctx->p2p_counted, cudaEventDisableTiming));
  TB_CUDA(ctx, cudaMemcpyAsync(ctx->pinned_later(), ctx->p2p_counter.p + 1, 2 * sizeof(int32_t),
                               cudaMemcpyDeviceToHost, s));
  TB_CUDA(ctx, cudaEventRecord(ctx->p2p_counted, s));
  return TAPAS_B200_OK;
}

// Builds the P2P work items that were counted (ctx->p2p_items) and their queue
// order (ctx->p2p_order: items by decreasing work).
int p2p_items(tapas_b200_ctx *ctx) {
  cudaStream_t s = ctx->stream;
  int64_t nl = 0;
  const int32_t *leaves = work_leaves(ctx, nl);
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  const int64_t piece_pairs = ctx->p2p_piece_pairs;
  TB_CUDA(ctx, cudaEventSynchronize(ctx->p2p_counted));
  const int32_t *h = ctx->pinned_later();
  const int64_t ni = h[0], npart = h[1];
  if (ni < nl || npart < 0) {
    set_error(ctx, "p2p: work item count overflow");
    return TAPAS_B200_ERR_CAPACITY;
  }
  ctx->p2p_nitems = ni;
  ctx->p2p_split = npart > 0;
  TB_CUDA(ctx, ctx->p2p_items.ensure((size_t)ni * sizeof(WorkItem) / sizeof(int4) + 1, s));
  TB_CUDA(ctx, ctx->p2p_part.ensure(4 * (size_t)npart + 4, s));
  TB_CUDA(ctx, ctx->p2p_wkey.ensure(ni + 1, s));
  TB_CUDA(ctx, ctx->p2p_wkey_alt.ensure(ni + 1, s));
  TB_CUDA(ctx, ctx->p2p_order.ensure(ni + 1, s));
  TB_CUDA(ctx, ctx->p2p_order_alt.ensure(ni + 1, s));
  emit_items<<<grid_for(8 * nl, 256), 256, 0, s>>>(
      leaves, nl, ctx->p2p_off.p, ctx->p2p.p, mask, ctx->cnb.p, piece_pairs, ctx->p2p_key.p,
      ctx->p2p_kcnt.p, ctx->p2p_koff.p, ctx->p2p_poff.p, reinterpret_cast<WorkItem *>(ctx->p2p_items.p),
      ctx->p2p_wkey.p, ctx->p2p_order.p, ctx->p2p_part.p);
  TB_LAUNCH_CHECK(ctx);
  uint64_t *k = ctx->p2p_wkey.p, *ka = ctx->p2p_wkey_alt.p;
  uint32_t *v = ctx->p2p_order.p, *va = ctx->p2p_order_alt.p;
  TB_TRY(radix_sort(ctx, k, ka, v, va, ni, 0, 8));
  if (v != ctx->p2p_order.p) {
    std::swap(ctx->p2p_order.p, ctx->p2p_order_alt.p);
    std::swap(ctx->p2p_order.cap, ctx->p2p_order_alt.cap);
  }
  if (k != ctx->p2p_wkey.p) {
    std::swap(ctx->p2p_wkey.p, ctx->p2p_wkey_alt.p);
    std::swap(ctx->p2p_wkey.cap, ctx->p2p_wkey_alt.cap);
  }
  return TAPAS_B200_OK;
}

// Adds the pieces of split leaves into trg (after a P2P kernel).
int p2p_finish(tapas_b200_ctx *ctx) {
  if (!ctx->p2p_split) return TAPAS_B200_OK;
  int64_t nl = 0;
  const int32_t *leaves = work_leaves(ctx, nl);
  split_reduce<<<grid_for(32 * nl, 256), 256, 0, ctx->stream>>>(
      leaves, nl, ctx->cbeg.p, ctx->cnb.p, ctx->p2p_kcnt.p, ctx->p2p_poff.p,
      ctx->p2p_part.p, ctx->trg.p);
  TB_LAUNCH_CHECK(ctx);
  return TAPAS_B200_OK;
}

int p2p_grid(tapas_b200_ctx *ctx, int warps_per_block) {
  // persistent: enough warps to fill the GPU, never more than the work items
  const int64_t ni = ctx->p2p_nitems;
  int64_t g = (int64_t)ctx->num_sms * (64 / warps_per_block);
  const int64_t need = (ni + warps_per_block - 1) / warps_per_block;
  return (int)std::max<int64_t>(1, std::min(g, need));
}

}  // namespace

// Sharded: the rows of bodies another context evaluates are exactly zero, so
// the contexts' results add up without changing a bit.
static int zero_results_if_sharded(tapas_b200_ctx *ctx) {
  if (ctx->sharded)
    TB_CUDA(ctx, cudaMemsetAsync(ctx->trg.p, 0, sizeof(double) * 4 * (size_t)ctx->n, ctx->stream));
  return TAPAS_B200_OK;
}

int p2p_begin(tapas_b200_ctx *ctx, int precision) {
  int64_t nl = 0;
  work_leaves(ctx, nl);
  ctx->p2p_begun = true;
  if (nl == 0) return TAPAS_B200_OK;
  const int rc = count_items(ctx, precision == TAPAS_B200_MIXED ? kMixedBlocks * kMixedWarps
                                                                : kFp64Blocks * kWarps);
  ctx->p2p_begun = rc == TAPAS_B200_OK;
  return rc;
}

int p2p_fp64(tapas_b200_ctx *ctx) {
  cudaStream_t s = ctx->stream;
  TB_TRY(zero_results_if_sharded(ctx));
  int64_t nl = 0;
  work_leaves(ctx, nl);
  if (!ctx->p2p_begun) TB_TRY(p2p_begin(ctx, TAPAS_B200_FP64));
  ctx->p2p_begun = false;
  if (nl == 0) return TAPAS_B200_OK;
  TB_TRY(p2p_items(ctx));
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  p2p_fp64_kernel<<<p2p_grid(ctx, kWarps), kThreads, 0, s>>>(
      ctx->p2p_order.p, ctx->p2p_nitems, ctx->p2p_counter.p,
      reinterpret_cast<const WorkItem *>(ctx->p2p_items.p), ctx->p2p.p, mask, ctx->cbeg.p,
      ctx->cnb.p, ctx->sx.p, ctx->sy.p, ctx->sz.p, ctx->sq.p, ctx->trg.p, ctx->p2p_part.p);
  TB_LAUNCH_CHECK(ctx);
  return p2p_finish(ctx);
}

int p2p_mixed(tapas_b200_ctx *ctx) {
  cudaStream_t s = ctx->stream;
  TB_TRY(zero_results_if_sharded(ctx));
  int64_t nl = 0;
  work_leaves(ctx, nl);
  if (!ctx->p2p_begun) TB_TRY(p2p_begin(ctx, TAPAS_B200_MIXED));
  ctx->p2p_begun = false;
  if (nl == 0) return TAPAS_B200_OK;
  TB_TRY(p2p_items(ctx));
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  p2p_mixed_kernel<kMixedBlocks><<<p2p_grid(ctx, kMixedWarps), kMixedThreads, 0, s>>>(
      ctx->p2p_order.p, ctx->p2p_nitems, ctx->p2p_counter.p,
      reinterpret_cast<const WorkItem *>(ctx->p2p_items.p), ctx->p2p.p, mask, ctx->cbeg.p,
      ctx->cnb.p, ctx->ccen.p, ctx->cmin.p, ctx->cmax.p, ctx->sx.p, ctx->sy.p, ctx->sz.p,
      ctx->sq.p, ctx->trg.p, ctx->p2p_part.p);
  TB_LAUNCH_CHECK(ctx);
  return p2p_finish(ctx);
}

}  // namespace tb
