// Dual-tree traversal on the GPU: builds the M2L and P2P work lists.
//
// The reference runs FMM_DTT (sample/exafmm-dev-13274dd4ac68/examples/
// tapas_exafmm.cxx:209-286) recursively from (root, root).  Each visit is a
// pure function of the two cells, so the recursion is replaced by a
// breadth-first frontier of (target, source) pairs: every step classifies all
// pending pairs at once and emits
//   - an M2L pair   if R2 > (Ri + Rj)^2  (R2 = squared centre distance,
//                   geometry.h:81-83; Ri = (max width / 2 * 1.00001) / theta),
//   - a P2P pair    if both are leaves (skipped when either is empty: the
//                   reference's Map over an empty body product is a no-op,
//                   cpp/include/tapas/hot.h:1362-1369),
//   - 8 new pairs   otherwise, splitting by tapas_splitCell (:252-285): split
//                   the non-leaf side, and if both are non-leaves the one with
//                   the larger R, ties -> target.
// With mutual = 1 (the example's -m option) a pair (c, c) of a non-leaf cell
// with itself splits both sides and visits only the 36 child pairs (c_i, c_j),
// i <= j (tapas_splitCell's `mutual && Ci == Cj` branch; the product map's
// AllowMutualInteraction rule, cpp/include/tapas/hot/mapper.h:28-121 and
// iterator.h:98-100,165-167,279-281).  Every unordered cell pair is then
// visited once and acts both ways (M2L both ways, LaplaceSphericalCPU_tapas.h:
// 208-273; P2P both ways, LaplaceP2PCPU_tapas.h:48-74).  Here the unordered
// pairs are expanded into the two directed pairs before the lists are
// ordered, so the evaluation kernels see ordinary (target, source) lists.
// The acceptance test is evaluated with separately rounded FP64 operations so
// every decision matches the reference bit for bit; the lists are therefore
// equal as sets.  They are then sorted by (target, source) so the evaluation
// order, and so every result, is deterministic.
#include <cooperative_groups.h>

#include <algorithm>

#include "coop.cuh"
#include "primitives.cuh"
#include "traverse.cuh"

namespace tb {
namespace {

constexpr int kBlock = 256;

// What one visit reads of a cell, packed so a visit touches two sectors per
// cell: geometry {cx, cy, cz, R} with R = (max width / 2 * 1.00001) / theta,
// and {nb, first child or -1 for a leaf}.
struct TravCells {
  const double4 *geo;
  const int2 *meta;
};

// State of a traversal, in device memory; the host reads it once at the end.
struct TravState {
  // sizes at the start of the step `cur`: frontier (in buffer cur & 1), lists
  unsigned long long nfront, m2l, p2p;
  unsigned long long inter;    // P2P body pairs of the finished steps
  unsigned long long visited;  // pairs classified in them
  int steps;                   // finished steps
  int stop;                    // 1: a buffer was too small for step `steps`
  // what that step reserved, for the host to size the buffers by
  unsigned long long need_front, need_m2l, need_p2p;
  // reservations: step k uses set k % 3 and clears the next step's, whose last
  // readers (step k - 2) are behind the barrier before step k
  unsigned long long cnt[3][4];  // next frontier, M2L, P2P, body pairs
};
constexpr int kTravStateAt = 16;  // in ctx->counters
static_assert(sizeof(TravState) <= (64 - kTravStateAt) * sizeof(unsigned long long), "counters");

// The traversal's cell records for this theta, with the reference's
// operations in its order for R (max over the widths, halve, * 1.00001,
// / theta), computed once per traversal instead of twice per visited pair.
__global__ void trav_cells(int64_t ncells, const double *__restrict__ mn,
                           const double *__restrict__ mx, const double *__restrict__ cen,
                           const int32_t *__restrict__ nb, const int32_t *__restrict__ leaf,
                           const int32_t *__restrict__ child, double theta,
                           double4 *__restrict__ geo, int2 *__restrict__ meta,
                           int2 *__restrict__ front, TravState *__restrict__ st) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {  // the traversal starts with (root, root)
    front[0] = make_int2(0, 0);
    *st = TravState{};
    st->nfront = 1;
  }
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncells;
       i += (int64_t)gridDim.x * blockDim.x) {
    double w = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const double wd = __dsub_rn(mx[3 * i + d], mn[3 * i + d]);
      w = (w < wd) ? wd : w;  // std::max(R, w)
    }
    const double R = __ddiv_rn(__dmul_rn(w / 2, 1.00001), theta);
    geo[i] = make_double4(cen[3 * i + 0], cen[3 * i + 1], cen[3 * i + 2], R);
    meta[i] = make_int2(nb[i], leaf[i] ? -1 : child[i]);
  }
}

// Per-thread output counts packed in one word for the block scan: M2L pairs in
// bits 0-15, P2P pairs in bits 16-31, new frontier pairs (8 per split, 36 for a
// mutual self split) from bit 32.
constexpr int kWarpsPerBlock = kBlock / 32;
constexpr int kPerThread = 4;
constexpr int kSelfSplit = 36;  // child pairs (i, j), i <= j, of a cell with itself
constexpr int kP2pAt = 16, kFrontAt = 32;
constexpr unsigned long long kCountMask = 0xffff;
static_assert(kBlock * kPerThread <= (int)kCountMask, "packed per-block counts");

struct TravBufs {
  int2 *front[2];
  long long front_cap[2];
  uint64_t *m2l, *p2p;
  long long m2l_cap, p2p_cap;
};

constexpr int kMaxSteps = 4 * (kMaxDepth + 2);

// The whole breadth-first traversal in one cooperative launch: every step
// classifies the pairs of the current frontier and appends to the two lists
// and the next frontier, and a grid-wide barrier ends it.  Slots in the three
// outputs are reserved once per block (one atomic per counter per block), the
// block's threads taking consecutive slots.  A step that finds a buffer too
// small ends the kernel without having counted; the host enlarges the buffer
// and starts it again from that step.  (A launch and a host round trip per step
// took about 20 us each, 9 to 25 times.)
__global__ void __launch_bounds__(kBlock) dtt_steps(TravCells c, TravBufs bufs, TravState *st,
                                                    int prune_empty, int mutual) {
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  __shared__ unsigned long long wsum[kWarpsPerBlock];
  __shared__ unsigned long long wint[kWarpsPerBlock];
  __shared__ unsigned long long bbase[3];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t nfront = (int64_t)st->nfront;
  unsigned long long n_m2l = st->m2l, n_p2p = st->p2p, n_int = st->inter, visited = st->visited;
  int step = st->steps;
  while (nfront > 0 && step < kMaxSteps) {
    const int2 *front = bufs.front[step & 1];
    int2 *next = bufs.front[(step & 1) ^ 1];
    const int64_t next_cap = bufs.front_cap[(step & 1) ^ 1];
    unsigned long long *counters = st->cnt[step % 3];
    if (blockIdx.x == 0 && threadIdx.x < 4) st->cnt[(step + 1) % 3][threadIdx.x] = 0;
    // A block takes kPerThread pairs per thread at a time when there are enough for
    // all blocks: the three barriers and the reservations' latency per round were
    // most of the time.
    const int per = nfront > (int64_t)gridDim.x * kBlock ? kPerThread : 1;
    for (int64_t base = (int64_t)blockIdx.x * kBlock * per; base < nfront;
         base += (int64_t)gridDim.x * kBlock * per) {
      int kind[kPerThread];  // 0 none, 1 m2l, 2 p2p, 3 split target, 4 split source, 5 split both
      int2 pair[kPerThread];
      int child[kPerThread];
      unsigned long long mine = 0, inter = 0;
#pragma unroll
      for (int q = 0; q < kPerThread; q++) {
        kind[q] = 0;
        const int64_t i = base + q * kBlock + threadIdx.x;
        if (q >= per || i >= nfront) continue;
        pair[q] = __ldcg(front + i);
        const int t = pair[q].x, s = pair[q].y;
        const int2 mt = c.meta[t], ms = c.meta[s];
        // An empty cell (and so all of its descendants) contributes nothing as a
        // source and receives nothing used later as a target.
        if (prune_empty && (mt.x == 0 || ms.x == 0)) continue;
        const double4 gt = c.geo[t], gs = c.geo[s];
        const double dx = __dsub_rn(gt.x, gs.x);
        const double dy = __dsub_rn(gt.y, gs.y);
        const double dz = __dsub_rn(gt.z, gs.z);
        double R2 = __dadd_rn(0.0, __dmul_rn(dx, dx));
        R2 = __dadd_rn(R2, __dmul_rn(dy, dy));
        R2 = __dadd_rn(R2, __dmul_rn(dz, dz));
        const double Ri = gt.w, Rj = gs.w;
        const double RR = __dadd_rn(Ri, Rj);
        const bool lt = mt.y < 0, ls = ms.y < 0;
        int kd;
        if (R2 > __dmul_rn(RR, RR)) {
          kd = 1;
        } else if (lt && ls) {
          kd = 0;
          if (mt.x > 0 && ms.x > 0) {
            kd = 2;
            // body pairs evaluated: both directions of a mutual pair of two leaves
            inter += (unsigned long long)mt.x * (unsigned long long)ms.x *
                     (mutual && t != s ? 2 : 1);
          }
        } else if (ls) {
          kd = 3;
        } else if (lt) {
          kd = 4;
        } else if (mutual && t == s) {
          kd = 5;
        } else {
          kd = (Ri >= Rj) ? 3 : 4;
        }
        kind[q] = kd;
        child[q] = kd == 3 ? mt.y : ms.y;
        mine += kd == 0   ? 0ull
                : kd == 1 ? 1ull
                : kd == 2 ? 1ull << kP2pAt
                : kd == 5 ? (unsigned long long)kSelfSplit << kFrontAt
                          : 8ull << kFrontAt;
      }
      unsigned long long incl = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) inter += __shfl_xor_sync(0xffffffffu, inter, o);
      if (lane == 31) wsum[warp] = incl;
      if (lane == 0) wint[warp] = inter;
      __syncthreads();
      if (threadIdx.x == 0) {
        unsigned long long run = 0, tot = 0;
#pragma unroll
        for (int k = 0; k < kWarpsPerBlock; k++) {
          const unsigned long long v = wsum[k];
          wsum[k] = run;
          run += v;
          tot += wint[k];
        }
        const unsigned long long n1 = run & kCountMask, n2 = (run >> kP2pAt) & kCountMask,
                                 n3 = run >> kFrontAt;
        bbase[0] = n_m2l + (n1 ? atomicAdd(counters + 1, n1) : 0);
        bbase[1] = n_p2p + (n2 ? atomicAdd(counters + 2, n2) : 0);
        bbase[2] = n3 ? atomicAdd(counters + 0, n3) : 0;
        if (tot) atomicAdd(counters + 3, tot);
      }
      __syncthreads();
      const unsigned long long off = wsum[warp] + incl - mine;
      int64_t at_m2l = (int64_t)(bbase[0] + (off & kCountMask)),
              at_p2p = (int64_t)(bbase[1] + ((off >> kP2pAt) & kCountMask)),
              at_next = (int64_t)(bbase[2] + (off >> kFrontAt));
#pragma unroll
      for (int q = 0; q < kPerThread; q++) {
        if (kind[q] == 0) continue;
        const int t = pair[q].x, s = pair[q].y, ch = child[q];
        const uint64_t packed = ((uint64_t)(uint32_t)t << 32) | (uint32_t)s;
        if (kind[q] == 1) {
          if (at_m2l < bufs.m2l_cap) bufs.m2l[at_m2l] = packed;
          at_m2l++;
        } else if (kind[q] == 2) {
          if (at_p2p < bufs.p2p_cap) bufs.p2p[at_p2p] = packed;
          at_p2p++;
        } else if (kind[q] == 5) {
          if (at_next + kSelfSplit <= next_cap) {
            int2 *o = next + at_next;
            int k = 0;
            for (int a = 0; a < 8; a++)
              for (int b2 = a; b2 < 8; b2++) o[k++] = make_int2(ch + a, ch + b2);
          }
          at_next += kSelfSplit;
        } else {
          if (at_next + 8 <= next_cap) {
            int4 *o4 = reinterpret_cast<int4 *>(next + at_next);  // even: 8 and 36 are
#pragma unroll
            for (int k = 0; k < 8; k += 2)
              o4[k / 2] = kind[q] == 3 ? make_int4(ch + k, s, ch + k + 1, s)
                                       : make_int4(t, ch + k, t, ch + k + 1);
          }
          at_next += 8;
        }
      }
      __syncthreads();  // wsum / bbase are rewritten by the next round
    }
    grid.sync();
    const unsigned long long f = __ldcg(counters + 0), m = n_m2l + __ldcg(counters + 1),
                             p = n_p2p + __ldcg(counters + 2);
    if ((int64_t)f > next_cap || (int64_t)m > bufs.m2l_cap || (int64_t)p > bufs.p2p_cap) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->stop = 1;
        st->need_front = f;
        st->need_m2l = m;
        st->need_p2p = p;
      }
      break;
    }
    n_int += __ldcg(counters + 3);
    visited += (unsigned long long)nfront;
    nfront = (int64_t)f;
    n_m2l = m;
    n_p2p = p;
    step++;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->nfront = (unsigned long long)nfront;
    st->m2l = n_m2l;
    st->p2p = n_p2p;
    st->inter = n_int;
    st->visited = visited;
    st->steps = step;
  }
}

// The directed pairs of a mutual list: (t, s) and (s, t) for t != s, a self
// pair (t, t) once.  Slots are reserved once per warp; the order is set by the
// (target, source) sort that follows.
__global__ void expand_mutual(const uint64_t *__restrict__ in, int64_t n,
                              uint64_t *__restrict__ out, int64_t cap,
                              unsigned long long *__restrict__ cnt) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n;
       base += stride) {
    const int64_t i = base + lane;
    uint64_t x = 0;
    int k = 0;
    if (i < n) {
      x = in[i];
      k = ((x >> 32) != (x & 0xFFFFFFFFull)) ? 2 : 1;
    }
    int incl = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const int tot = __shfl_sync(0xffffffffu, incl, 31);
    unsigned long long b0 = 0;
    if (lane == 0) b0 = atomicAdd(cnt, (unsigned long long)tot);
    b0 = __shfl_sync(0xffffffffu, b0, 0);
    const int64_t dst = (int64_t)b0 + incl - k;
    if (k >= 1 && dst < cap) out[dst] = x;
    if (k == 2 && dst + 1 < cap) out[dst + 1] = (x << 32) | (x >> 32);
  }
}

// Packs (t << 32 | s) into (t << b | s) for a narrower sort key.
__global__ void pack_pairs(uint64_t *__restrict__ v, int64_t n, int b) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t x = v[i];
    v[i] = ((x >> 32) << b) | (x & 0xFFFFFFFFull);
  }
}

// ---------------------------------------------------------------------------
// List ordering.  The traversal emits pairs in an order set by its atomics;
// the lists are put in (target, source) order by a counting sort on the
// target (the counts' scan is the lists' CSR offsets) followed by a bitonic
// sort of each target's sources in shared memory: one warp per segment of up
// to kWarpSegMax pairs, one block per longer segment up to kSegSortMax, and
// the radix sort of the whole list when a segment is longer still.  Every
// (target, source) pair is visited at most once (the split rule is a function
// of the pair, so two visiting paths from (root, root) cannot diverge), so a
// segment's sources are distinct.
// ---------------------------------------------------------------------------
constexpr int kWarpSegMax = 512;
constexpr int kSegSortMax = 8192;
constexpr int kSegWarps = 8;
constexpr int kLongThreads = 1024;

// v0[0, n0) into cnt0, v1[0, n1) into cnt1.
__global__ void target_counts(const uint64_t *__restrict__ v0, int64_t n0,
                              int32_t *__restrict__ cnt0, const uint64_t *__restrict__ v1,
                              int64_t n1, int32_t *__restrict__ cnt1) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n0 + n1;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (i < n0)
      atomicAdd(cnt0 + (v0[i] >> 32), 1);
    else
      atomicAdd(cnt1 + (v1[i - n0] >> 32), 1);
  }
}

// Places each pair's source in its target's segment (order inside it
// arbitrary).  cnt starts as the segments' sizes and counts down to 0.
__global__ void scatter_by_target(const uint64_t *__restrict__ v, int64_t n,
                                  const int32_t *__restrict__ off, int32_t *__restrict__ cnt,
                                  uint32_t *__restrict__ src) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t x = v[i];
    const int64_t t = x >> 32;
    const int32_t o = off[t];
    src[o + atomicSub(cnt + t, 1) - 1] = (uint32_t)x;
  }
}

// Ascending bitonic sort of a[0, np), np a power of two, by threads
// tid = 0 .. nthr-1 of a warp (kBlockLevel false) or of the block.
template <bool kBlockLevel>
__device__ __forceinline__ void bitonic_sort(uint32_t *a, int np, int tid, int nthr) {
  for (int k = 2; k <= np; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int c = tid; c < (np >> 1); c += nthr) {
        const int lo = ((c & ~(j - 1)) << 1) | (c & (j - 1));
        const int hi = lo + j;
        const uint32_t x = a[lo], y = a[hi];
        if ((x > y) == ((lo & k) == 0)) {
          a[lo] = y;
          a[hi] = x;
        }
      }
      if (kBlockLevel) __syncthreads(); else __syncwarp();
    }
  }
}

__device__ __forceinline__ int pow2_at_least(int n) {
  int p = 2;
  while (p < n) p <<= 1;
  return p;
}

// One warp per target segment of at most kWarpSegMax sources; longer segments
// are listed for sort_long_segments.  out[i] = t << b | sorted source.
__global__ void __launch_bounds__(kSegWarps * 32) sort_segments(
    const uint32_t *__restrict__ src, const int32_t *__restrict__ off, int64_t ncells, int b,
    uint64_t *__restrict__ out, int32_t *__restrict__ long_list,
    unsigned long long *__restrict__ long_cnt) {
  __shared__ uint32_t buf[kSegWarps][kWarpSegMax];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *a = buf[warp];
  const int64_t warps = (int64_t)gridDim.x * kSegWarps;
  for (int64_t c = (int64_t)blockIdx.x * kSegWarps + warp; c < ncells; c += warps) {
    const int32_t a0 = off[c], len = off[c + 1] - a0;
    const uint64_t th = (uint64_t)c << b;
    if (len == 0) continue;
    if (len > kWarpSegMax) {
      if (lane == 0) long_list[atomicAdd(long_cnt, 1ull)] = (int32_t)c;
      continue;
    }
    if (len == 1) {
      if (lane == 0) out[a0] = th | src[a0];
      continue;
    }
    const int np = pow2_at_least(len);
    if (np <= 32) {  // in registers, a lane an entry
      uint32_t v = lane < len ? src[a0 + lane] : 0xFFFFFFFFu;
      for (int k = 2; k <= np; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, v, j);
          v = ((lane & j) == 0) == ((lane & k) == 0) ? min(v, o) : max(v, o);
        }
      if (lane < len) out[a0 + lane] = th | v;
      continue;
    }
    for (int i = lane; i < np; i += 32) a[i] = i < len ? src[a0 + i] : 0xFFFFFFFFu;
    __syncwarp();
    bitonic_sort<false>(a, np, lane, 32);
    for (int i = lane; i < len; i += 32) out[a0 + i] = th | a[i];
    __syncwarp();
  }
}

// One block per listed segment of kWarpSegMax < length <= kSegSortMax.
__global__ void __launch_bounds__(kLongThreads) sort_long_segments(
    const uint32_t *__restrict__ src, const int32_t *__restrict__ off, int b,
    uint64_t *__restrict__ out, const int32_t *__restrict__ long_list,
    const unsigned long long *__restrict__ long_cnt) {
  __shared__ uint32_t a[kSegSortMax];
  const int64_t nl = (int64_t)*long_cnt;
  for (int64_t k = blockIdx.x; k < nl; k += gridDim.x) {
    const int32_t c = long_list[k];
    const int32_t a0 = off[c], len = off[c + 1] - a0;
    const uint64_t th = (uint64_t)c << b;
    const int np = pow2_at_least(len);
    for (int i = threadIdx.x; i < np; i += kLongThreads) a[i] = i < len ? src[a0 + i] : 0xFFFFFFFFu;
    __syncthreads();
    bitonic_sort<true>(a, np, threadIdx.x, kLongThreads);
    for (int i = threadIdx.x; i < len; i += kLongThreads) out[a0 + i] = th | a[i];
    __syncthreads();
  }
}

// out[i] = c << b | src[i] over each target segment, sources in the order
// the scatter left them (one warp per target).
__global__ void __launch_bounds__(kSegWarps * 32) pack_segments(
    const uint32_t *__restrict__ src, const int32_t *__restrict__ off, int64_t ncells, int b,
    uint64_t *__restrict__ out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t warps = (int64_t)gridDim.x * kSegWarps;
  for (int64_t c = (int64_t)blockIdx.x * kSegWarps + warp; c < ncells; c += warps) {
    const int32_t a0 = off[c], a1 = off[c + 1];
    const uint64_t th = (uint64_t)c << b;
    for (int32_t i = a0 + lane; i < a1; i += 32) out[i] = th | src[i];
  }
}

__global__ void list_sources(const uint64_t *__restrict__ v, int64_t n, uint64_t mask,
                             uint32_t *__restrict__ src) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    src[i] = (uint32_t)(v[i] & mask);
}

int bits_for(int64_t x) {
  int b = 1;
  while (((int64_t)1 << b) <= x) b++;
  return b;
}

// Sorts each target segment of list w (0: M2L, 1: P2P) by source, given the
// sources in segment order in ctx->list_src and the longest segment.
int sort_segment_sources(tapas_b200_ctx *ctx, int w, unsigned long long longest) {
  cudaStream_t s = ctx->stream;
  const int64_t C = ctx->ncells;
  const int b = ctx->list_shift;
  tb::DBuf<uint64_t> &L = w ? ctx->p2p : ctx->m2l;
  const int32_t *off = w ? ctx->p2p_off.p : ctx->m2l_off.p;
  TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p + 7, 0, sizeof(unsigned long long), s));
  // list 0's counts are spent (list 1's lie after them): their buffer holds the
  // long-segment list
  sort_segments<<<grid_for(C, kSegWarps, ctx->num_sms * 8), kSegWarps * 32, 0, s>>>(
      ctx->list_src.p, off, C, b, L.p, ctx->list_cnt.p, ctx->counters.p + 7);
  TB_LAUNCH_CHECK(ctx);
  if (longest > (unsigned long long)kWarpSegMax) {
    sort_long_segments<<<ctx->num_sms, kLongThreads, 0, s>>>(ctx->list_src.p, off, b, L.p,
                                                              ctx->list_cnt.p,
                                                              ctx->counters.p + 7);
    TB_LAUNCH_CHECK(ctx);
  }
  return TAPAS_B200_OK;
}

}  // namespace

int sort_list_sources(tapas_b200_ctx *ctx, int w) {
  if (!ctx->have_lists || ctx->sources_sorted[w]) return TAPAS_B200_OK;
  const int64_t n = w ? ctx->n_p2p : ctx->n_m2l;
  if (n > 0) {
    cudaStream_t s = ctx->stream;
    TB_CUDA(ctx, ctx->list_src.ensure(n + 1, s));
    TB_CUDA(ctx, ctx->list_cnt.ensure(ctx->ncells + 1, s));
    list_sources<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
        w ? ctx->p2p.p : ctx->m2l.p, n, (1ull << ctx->list_shift) - 1, ctx->list_src.p);
    TB_LAUNCH_CHECK(ctx);
    TB_TRY(sort_segment_sources(ctx, w, ctx->longest_segment[w]));
  }
  ctx->sources_sorted[w] = true;
  return TAPAS_B200_OK;
}

int sort_list_sources(tapas_b200_ctx *ctx) {
  TB_TRY(sort_list_sources(ctx, 0));
  return sort_list_sources(ctx, 1);
}

// build_lists; roomy: with first sizes that hold most trees' lists, and half as much
// again for one that grows, else with no more than each step needs.
static int build_lists_in(tapas_b200_ctx *ctx, double theta, int mutual, bool sort_m2l_sources,
                          bool roomy) {
  if (!ctx->have_tree) {
    set_error(ctx, "build_lists: no tree (call partition first)");
    return TAPAS_B200_ERR_STATE;
  }
  if (!(theta > 0)) {
    set_error(ctx, "build_lists: theta must be > 0");
    return TAPAS_B200_ERR_ARG;
  }
  if (mutual != 0 && mutual != 1) {
    set_error(ctx, "build_lists: mutual must be 0 or 1");
    return TAPAS_B200_ERR_ARG;
  }
  ctx->mutual = mutual;
  ctx->lists_have_empty = ctx->reference_lists;
  cudaStream_t s = ctx->stream;
  ctx->theta = theta;
  ctx->have_lists = false;
  const int64_t C = ctx->ncells;
  TB_CUDA(ctx, ctx->trav_geo.ensure(C + 1, s));
  TB_CUDA(ctx, ctx->trav_meta.ensure(C + 1, s));
  TB_CUDA(ctx, ctx->counters.ensure(64, s));
  ctx->p2p_begun = false;  // counted for other lists
  TB_CUDA(ctx, ctx->pinned.ensure(tapas_b200_ctx::kPinnedBytes));
  // First sizes: a list entry per cell and near or far neighbour of a
  // volume-filling tree for small trees, of a surface for large ones, and the frontier
  // of a step that has both (100k bodies of a cube, ncrit 64, theta 0.4: 667k pairs,
  // 143 per cell); a list that outgrows its buffer is met below, and the buffers
  // stay for the next call.
  auto room = [&](int64_t per_cell, int64_t large, int64_t extra) {
    return (size_t)((roomy ? std::min(per_cell * C, large * C + extra) : 0) + 4096);
  };
  auto grown = [&](unsigned long long need) { return (size_t)(need + (roomy ? need / 2 : 0)); };
  TB_CUDA(ctx, ctx->front_a.ensure(room(160, 16, 2000000), s));
  TB_CUDA(ctx, ctx->front_b.ensure(room(160, 16, 2000000), s));
  TB_CUDA(ctx, ctx->m2l.ensure(room(128, 40, 4000000), s));
  TB_CUDA(ctx, ctx->p2p.ensure(room(64, 24, 2000000), s));
  unsigned long long *hc = reinterpret_cast<unsigned long long *>(ctx->pinned.p);
  TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p, 0, 8 * sizeof(unsigned long long), s));
  TravState *st = reinterpret_cast<TravState *>(ctx->counters.p + kTravStateAt);
  trav_cells<<<grid_for(C, kBlock), kBlock, 0, s>>>(
      C, ctx->cmin.p, ctx->cmax.p, ctx->ccen.p, ctx->cnb.p, ctx->cleaf.p, ctx->cchild.p, theta,
      ctx->trav_geo.p, ctx->trav_meta.p, ctx->front_a.p, st);
  TB_LAUNCH_CHECK(ctx);
  const TravCells cv{ctx->trav_geo.p, ctx->trav_meta.p};
  {
    PhaseTimer tm(ctx, &ctx->timings.traverse);
    if (ctx->trav_blocks == 0) {
      int per_sm = 0;
      TB_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, dtt_steps, kBlock, 0));
      ctx->trav_blocks = std::max(1, per_sm) * ctx->num_sms;
    }
    // few blocks for a small tree: the barrier costs more than their work
    int blocks =
        (int)std::min<int64_t>(ctx->trav_blocks, std::max<int64_t>(32, C * 8 / kBlock));
    TravState *h = reinterpret_cast<TravState *>(hc + 16);
    for (int attempt = 0;; attempt++) {
      TravBufs bufs{{ctx->front_a.p, ctx->front_b.p},
                    {(long long)ctx->front_a.cap, (long long)ctx->front_b.cap},
                    ctx->m2l.p,
                    ctx->p2p.p,
                    (long long)ctx->m2l.cap,
                    (long long)ctx->p2p.cap};
      TravCells cells = cv;
      int prune = ctx->reference_lists ? 0 : 1, mut = mutual;
      TravState *state = st;
      void *args[] = {&cells, &bufs, &state, &prune, &mut};
      const int asked = blocks;
      TB_CUDA(ctx, launch_at_most(blocks, [&](int b) {
                return cudaLaunchCooperativeKernel(reinterpret_cast<void *>(dtt_steps), dim3(b),
                                                   dim3(kBlock), args, 0, s);
              }));
      if (blocks < asked) ctx->trav_blocks = blocks;  // what this stream holds
      count_launch(ctx);
      TB_CUDA(ctx, cudaMemcpyAsync(h, st, sizeof(TravState), cudaMemcpyDeviceToHost, s));
      TB_CUDA(ctx, cudaStreamSynchronize(s));
      if (!h->stop) break;
      if (attempt > 3 * kMaxSteps) {
        set_error(ctx, "traversal: frontier capacity exceeded after resizing");
        return TAPAS_B200_ERR_CAPACITY;
      }
      tb::DBuf<int2> &next = (h->steps & 1) ? ctx->front_a : ctx->front_b;
      if (h->need_front > next.cap)
        TB_CUDA(ctx, next.ensure(grown(h->need_front), s));
      if (h->need_m2l > ctx->m2l.cap)
        TB_CUDA(ctx, ctx->m2l.ensure(grown(h->need_m2l), s, true, h->m2l));
      if (h->need_p2p > ctx->p2p.cap)
        TB_CUDA(ctx, ctx->p2p.ensure(grown(h->need_p2p), s, true, h->p2p));
      h->stop = 0;
      for (auto &set : h->cnt)
        for (auto &v : set) v = 0;
      TB_CUDA(ctx, cudaMemcpyAsync(st, h, sizeof(TravState), cudaMemcpyHostToDevice, s));
    }
    if (h->nfront > 0) {
      set_error(ctx, "traversal did not terminate within its iteration bound");
      return TAPAS_B200_ERR_CAPACITY;
    }
    int64_t n_m2l = (int64_t)h->m2l, n_p2p = (int64_t)h->p2p;
    const unsigned long long n_int = h->inter;
    const int64_t visited = (int64_t)h->visited;
    const int iters = h->steps;
    ctx->n_m2l_visited = n_m2l;
    ctx->n_p2p_visited = n_p2p;
    if (mutual) {
      // unordered pairs -> directed pairs (M2L has no self pairs; P2P has one
      // self pair per non-empty leaf)
      tb::DBuf<uint64_t> *lists[2] = {&ctx->m2l, &ctx->p2p};
      int64_t *counts[2] = {&n_m2l, &n_p2p};
      for (int w = 0; w < 2; w++) {
        const int64_t n = *counts[w];
        if (n == 0) continue;
        TB_CUDA(ctx, ctx->list_alt.ensure(2 * n, s));
        TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p + 5, 0, sizeof(unsigned long long), s));
        expand_mutual<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
            lists[w]->p, n, ctx->list_alt.p, 2 * n, ctx->counters.p + 5);
        TB_LAUNCH_CHECK(ctx);
        TB_CUDA(ctx, cudaMemcpyAsync(hc + 5, ctx->counters.p + 5, sizeof(unsigned long long),
                                     cudaMemcpyDeviceToHost, s));
        TB_CUDA(ctx, cudaStreamSynchronize(s));
        *counts[w] = (int64_t)hc[5];
        std::swap(lists[w]->p, ctx->list_alt.p);
        std::swap(lists[w]->cap, ctx->list_alt.cap);
      }
    }
    ctx->n_m2l = n_m2l;
    ctx->n_p2p = n_p2p;
    ctx->n_p2p_int = n_int;
    ctx->trav_iters = iters;
    ctx->trav_pairs = visited;
    if (!roomy) {
      ctx->front_a.release();
      ctx->front_b.release();
    }
  }
  {
    PhaseTimer tm(ctx, &ctx->timings.list_sort);
    const int b = bits_for(C);
    ctx->list_shift = b;
    TB_CUDA(ctx, ctx->m2l_off.ensure(C + 1, s));
    TB_CUDA(ctx, ctx->p2p_off.ensure(C + 1, s));
    TB_CUDA(ctx, ctx->list_cnt.ensure(2 * (C + 1), s));
    const int64_t nlist[2] = {ctx->n_m2l, ctx->n_p2p};
    tb::DBuf<uint64_t> *lists[2] = {&ctx->m2l, &ctx->p2p};
    tb::DBuf<int32_t> *offs[2] = {&ctx->m2l_off, &ctx->p2p_off};
    int32_t *const cnt[2] = {ctx->list_cnt.p, ctx->list_cnt.p + (C + 1)};
    // 1. per-target counts -> CSR offsets, and the longest segment (counters 5
    // and 6, zero unless the mutual expansion used them)
    if (mutual)
      TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p + 5, 0, 2 * sizeof(unsigned long long), s));
    TB_CUDA(ctx, cudaMemsetAsync(cnt[0], 0, sizeof(int32_t) * 2 * (C + 1), s));
    if (nlist[0] + nlist[1] > 0) {
      target_counts<<<grid_for(nlist[0] + nlist[1], kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
          ctx->m2l.p, nlist[0], cnt[0], ctx->p2p.p, nlist[1], cnt[1]);
      TB_LAUNCH_CHECK(ctx);
    }
    const int32_t *const in[2] = {cnt[0], cnt[1]};
    int32_t *const out[2] = {offs[0]->p, offs[1]->p};
    int32_t *const tot[2] = {offs[0]->p + C, offs[1]->p + C};
    unsigned long long *const longest[2] = {ctx->counters.p + 5, ctx->counters.p + 6};
    TB_TRY(scan_exclusive2(ctx, in, out, C, tot, longest));
    TB_CUDA(ctx, cudaMemcpyAsync(hc + 5, ctx->counters.p + 5, 2 * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost, s));
    TB_CUDA(ctx, cudaStreamSynchronize(s));
    for (int w = 0; w < 2; w++) {
      ctx->longest_segment[w] = hc[5 + w];
      ctx->sources_sorted[w] = true;
    }
    // 2. counting sort by target, then each target's sources
    for (int w = 0; w < 2; w++) {
      tb::DBuf<uint64_t> &L = *lists[w];
      const int64_t n = nlist[w];
      if (n == 0) continue;
      if (hc[5 + w] <= (unsigned long long)kSegSortMax) {
        TB_CUDA(ctx, ctx->list_src.ensure(n + 1, s));
        scatter_by_target<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
            L.p, n, offs[w]->p, cnt[w], ctx->list_src.p);
        TB_LAUNCH_CHECK(ctx);
        if (w == 0 && !sort_m2l_sources) {
          // grouped by target only; sort_list_sources() completes the order
          // when a caller needs it
          pack_segments<<<grid_for(C, kSegWarps, ctx->num_sms * 8), kSegWarps * 32, 0, s>>>(
              ctx->list_src.p, offs[w]->p, C, b, L.p);
          TB_LAUNCH_CHECK(ctx);
          ctx->sources_sorted[w] = false;
        } else {
          TB_TRY(sort_segment_sources(ctx, w, hc[5 + w]));
        }
      } else {
        TB_CUDA(ctx, ctx->list_alt.ensure(n + 1, s));
        pack_pairs<<<grid_for(n, kBlock), kBlock, 0, s>>>(L.p, n, b);
        TB_LAUNCH_CHECK(ctx);
        uint64_t *k = L.p, *ka = ctx->list_alt.p;
        uint32_t *nv = nullptr, *nva = nullptr;
        TB_TRY(radix_sort(ctx, k, ka, nv, nva, n, 0, 2 * b));
        if (k != L.p) {
          std::swap(L.p, ctx->list_alt.p);
          std::swap(L.cap, ctx->list_alt.cap);
        }
      }
    }
  }
  ctx->have_lists = true;
  return TAPAS_B200_OK;
}

int build_lists(tapas_b200_ctx *ctx, double theta, int mutual, bool sort_m2l_sources) {
  const int rc = build_lists_in(ctx, theta, mutual, sort_m2l_sources, true);
  if (rc != TAPAS_B200_ERR_NOMEM) return rc;
  // The GPU's memory does not hold the first sizes (1M sphere, ncrit 128: 122 MB in all,
  // 44 with the least each step needs): give them back and start again.
  ctx->front_a.release();
  ctx->front_b.release();
  for (auto *b : {&ctx->m2l, &ctx->p2p, &ctx->list_alt}) b->release();
  ctx->list_src.release();
  return build_lists_in(ctx, theta, mutual, sort_m2l_sources, false);
}

}  // namespace tb
