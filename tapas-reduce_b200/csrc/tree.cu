// Octree construction on the GPU: bounding cube, Morton keys, key sort, body
// permutation and the cell build.
//
// Follows cpp/include/tapas/hot/buildtree.h (SamplingOctree) on one rank:
//  - bbox_*:        the constructor's box, :72-87, including its scalar
//                   broadcast (the box is a cube; body 0 contributes only z).
//  - keys_kernel:   BodiesToKeys, :505-539, with Morton::CalcFinestKey,
//                   sfc_morton.h:387-402.
//  - radix sort:    SortByKeys, common.h:249-273 (stable here; the reference's
//                   std::sort leaves equal keys in unspecified order).
//  - count_nonleaves, list_nonleaves, build_children: GenerateCell, :388-459: a
//                   cell's bodies are the sorted range [lower_bound(k),
//                   lower_bound(GetNext(k))); it is a leaf iff nb <= ncrit;
//                   non-leaves get all 8 children.  Cells are stored breadth
//                   first, level after level; all levels are built at once.
// Layout in HBM: bodies SoA FP64 (x,y,z,q) in input and sorted order; keys
// u64; cells SoA (key, range, parent, first child, leaf, 3x min/max/center).
#include <algorithm>

#include "primitives.cuh"
#include "tree.cuh"

namespace tb {
namespace {

constexpr int kBlock = 256;

// Exact FP64 operations: the reference is compiled for x86-64 without FMA, so
// every product/sum that decides a key bit or a cell boundary must round
// separately (no contraction).
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// std::max(p, hi) = p < hi ? hi : p ;  std::min(p, lo) = lo < p ? lo : p
__device__ __forceinline__ void mm_update(double p, double &lo, double &hi) {
  hi = (p < hi) ? hi : p;
  lo = (lo < p) ? lo : p;
}

__global__ void __launch_bounds__(kBlock) bbox_partial(const double *__restrict__ x,
                                                       const double *__restrict__ y,
                                                       const double *__restrict__ z, int64_t n,
                                                       double *__restrict__ part) {
  // Initialise from body 0's z (the value the reference's box starts from).
  double lo = z[0], hi = z[0];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x + 1; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    mm_update(x[i], lo, hi);
    mm_update(y[i], lo, hi);
    mm_update(z[i], lo, hi);
  }
  for (int o = 16; o > 0; o >>= 1) {
    double l2 = __shfl_down_sync(0xffffffffu, lo, o);
    double h2 = __shfl_down_sync(0xffffffffu, hi, o);
    lo = fmin(lo, l2);
    hi = fmax(hi, h2);
  }
  __shared__ double sl[kBlock / 32], sh[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { sl[warp] = lo; sh[warp] = hi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBlock / 32; w++) { lo = fmin(lo, sl[w]); hi = fmax(hi, sh[w]); }
    part[2 * blockIdx.x] = lo;
    part[2 * blockIdx.x + 1] = hi;
  }
}

// The box over the blocks' boxes, one block (a single thread's chain of loads
// took 28 us for 400 boxes).
__global__ void __launch_bounds__(kBlock) bbox_final(const double *__restrict__ part, int nparts,
                                                     double *__restrict__ out) {
  double lo = part[0], hi = part[1];
  for (int i = threadIdx.x; i < nparts; i += kBlock) {
    lo = fmin(lo, part[2 * i]);
    hi = fmax(hi, part[2 * i + 1]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  __shared__ double sl[kBlock / 32], sh[kBlock / 32];
  if ((threadIdx.x & 31) == 0) {
    sl[threadIdx.x >> 5] = lo;
    sh[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kBlock / 32; w++) { lo = fmin(lo, sl[w]); hi = fmax(hi, sh[w]); }
    out[0] = lo;
    out[1] = hi;
  }
}

// Keys of the bodies, and each body packed as one 32-byte record (x, y, z, q)
// so the gather into key order reads one sector per body; with q null the
// charge is packed later (pack_charges).
__global__ void __launch_bounds__(kBlock) keys_kernel(const double *__restrict__ x,
                                                      const double *__restrict__ y,
                                                      const double *__restrict__ z,
                                                      const double *__restrict__ q, int64_t n,
                                                      const double *__restrict__ box,
                                                      uint64_t *__restrict__ keys,
                                                      uint32_t *__restrict__ idx,
                                                      double4 *__restrict__ packed) {
  const double lo = box[0], hi = box[1];
  const int nfc = 1 << kMaxDepth;
  const double pitch = ddiv(dsub(hi, lo), (double)nfc);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    int a[3];
    const double p[3] = {x[i], y[i], z[i]};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      double o = ddiv(dsub(p[d], lo), pitch);
      a[d] = to_int_x86(o);
      if (a[d] == nfc) a[d]--;
    }
    keys[i] = finest_key(a[0], a[1], a[2]);
    idx[i] = (uint32_t)i;
    packed[i] = make_double4(p[0], p[1], p[2], q ? q[i] : 0.0);
  }
}

__global__ void pack_charges(const double *__restrict__ q, int64_t n,
                             double4 *__restrict__ packed) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    packed[i].w = q[i];
}

__global__ void __launch_bounds__(kBlock) gather_bodies(
    const double4 *__restrict__ packed, const uint32_t *__restrict__ idx, int64_t n,
    double *__restrict__ sx, double *__restrict__ sy, double *__restrict__ sz,
    double *__restrict__ sq) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double4 b = packed[idx[i]];
    sx[i] = b.x;
    sy[i] = b.y;
    sz[i] = b.z;
    sq[i] = b.w;
  }
}

// The same for the bodies in m places only.
__global__ void __launch_bounds__(kBlock) gather_places(
    const double4 *__restrict__ packed, const uint32_t *__restrict__ idx,
    const uint32_t *__restrict__ at, int64_t m, double *__restrict__ sx, double *__restrict__ sy,
    double *__restrict__ sz, double *__restrict__ sq) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t p = at[i];
    const double4 b = packed[idx[p]];
    sx[p] = b.x;
    sy[p] = b.y;
    sz[p] = b.z;
    sq[p] = b.w;
  }
}

__global__ void init_root(int64_t n, int ncrit, const double *__restrict__ box,
                          uint64_t *ckey, int32_t *cbeg, int32_t *cnb, int32_t *cparent,
                          int32_t *cchild, int32_t *cleaf, int32_t *clevel, double *cmin,
                          double *cmax, double *ccen) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  ckey[0] = 0;
  cbeg[0] = 0;
  cnb[0] = (int32_t)n;
  cparent[0] = -1;
  cchild[0] = -1;
  cleaf[0] = n <= ncrit ? 1 : 0;
  clevel[0] = 0;
  for (int d = 0; d < 3; d++) {
    cmin[d] = box[0];
    cmax[d] = box[1];
    ccen[d] = dadd(box[1], box[0]) / 2;  // (max + min) / 2, hot.h:232-238
  }
}

// ---------------------------------------------------------------------------
// Cells of all levels at once.  With the keys sorted, body i begins a cell of
// every level below the one it shares with body i - 1, and that cell holds more
// than ncrit bodies iff body i + ncrit is still in it, so the non-leaf cells
// body i begins are those of levels a + 1 .. b, a and b being the levels i
// shares with i - 1 and with i + ncrit (at most kMaxDepth - 1: cells of the
// deepest level are leaves).  Counting them per level and tile of bodies, a
// scan and one read-back give every level's size; each non-leaf cell's rank in
// its level is its order by first body, and its eight children are the cells
// 1 + 8q .. 8 + 8q for its rank q over all levels, level after level.  (Level by
// level, every level cost six launches and a host round trip: 20k bodies at
// ncrit 1, 18 levels, 0.67 ms.)
// ---------------------------------------------------------------------------
// The body sort takes the 40 highest of the 57 key bits (13 of 19 levels; five radix
// passes instead of eight) and orders the few bodies that agree there by
// insertion.  More than kMaxRun of them in one place (1 in 10^4 of the root's
// width: the core of a Plummer sphere from some 5M bodies on, or clusters) are listed,
// and only they are sorted on, by their low bits, once the read-back of the level sizes
// has told of them: six launches more up to 4096 such bodies.  Tree build of 16M Plummer
// 3.15 ms, of an 8M cube without and with 40 coincident bodies 1.31 and 1.38 ms; 5.17 and
// 2.52 ms when all bodies were sorted again on all bits.
constexpr int kSortLow = kDepthBits + 3 * kMaxDepth - 40;
constexpr int kMaxRun = 32;

constexpr int kTreeSteps = 8;                       // bodies per thread
constexpr int kTreeTile = kBlock * kTreeSteps;      // bodies per block
constexpr int kTreeLevels = kMaxDepth;              // levels that can have non-leaf cells

// Levels two body keys share: 0 (the root only) .. kMaxDepth (equal keys).
__device__ __forceinline__ int shared_levels(uint64_t x, uint64_t y) {
  const uint64_t v = (x ^ y) >> kDepthBits;
  if (v == 0) return kMaxDepth;
  return (3 * kMaxDepth - 1 - (63 - __clzll((long long)v))) / 3;
}

// Levels (a, b] of the non-leaf cells that body i begins (none if a >= b).
__device__ __forceinline__ void begun_levels(const uint64_t *__restrict__ keys, int64_t n,
                                             int ncrit, int64_t i, int &a, int &b) {
  a = 0;
  b = -1;
  if (i >= n || i + ncrit >= n) return;
  const uint64_t k = keys[i];
  b = min(shared_levels(k, keys[i + ncrit]), kMaxDepth - 1);
  a = i == 0 ? -1 : shared_levels(keys[i - 1], k);
}

// Calls f(level, lanes that begin a non-leaf cell there) for the levels any of
// the warp's 32 bodies begins one at.
template <class F>
__device__ __forceinline__ void each_begun_level(int a, int b, F f) {
  if (!__any_sync(0xffffffffu, a < b)) return;
  const int lo = __reduce_min_sync(0xffffffffu, a < b ? a + 1 : kMaxDepth),
            hi = __reduce_max_sync(0xffffffffu, a < b ? b : -1);
  for (int l = lo; l <= hi; l++) f(l, __ballot_sync(0xffffffffu, a < l && l <= b));
}

// Non-leaf cells begun per level (row) and tile (column).
__global__ void __launch_bounds__(kBlock) count_nonleaves(const uint64_t *__restrict__ keys,
                                                          int64_t n, int ncrit, int ntiles,
                                                          uint32_t *__restrict__ cnt) {
  __shared__ uint32_t tot[kTreeLevels];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < kTreeLevels) tot[threadIdx.x] = 0;
  __syncthreads();
  uint32_t mine = 0;  // lane l: level l's
  const int64_t base = (int64_t)blockIdx.x * kTreeTile + (threadIdx.x >> 5) * (32 * kTreeSteps);
  for (int s = 0; s < kTreeSteps; s++) {
    int a, b;
    begun_levels(keys, n, ncrit, base + 32 * s + lane, a, b);
    each_begun_level(a, b, [&](int l, unsigned m) {
      if (lane == l) mine += __popc(m);
    });
  }
  if (lane < kTreeLevels && mine) atomicAdd(&tot[lane], mine);
  __syncthreads();
  if (threadIdx.x < kTreeLevels) cnt[(size_t)threadIdx.x * ntiles + blockIdx.x] = tot[threadIdx.x];
}

// First rank (over all levels) of the non-leaf cells of each level.
struct LevelRanks {
  int32_t first[kTreeLevels + 1];
};

// node[q] = {first body, cell} of the non-leaf cell of rank q.
__global__ void __launch_bounds__(kBlock) list_nonleaves(const uint64_t *__restrict__ keys,
                                                         int64_t n, int ncrit, int ntiles,
                                                         const uint32_t *__restrict__ before,
                                                         LevelRanks ranks,
                                                         int2 *__restrict__ node) {
  __shared__ uint32_t warp_cnt[kBlock / 32][kTreeLevels];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kTreeTile + wi * (32 * kTreeSteps);
  int a[kTreeSteps], b[kTreeSteps];
  uint32_t mine = 0;
#pragma unroll
  for (int s = 0; s < kTreeSteps; s++) {
    begun_levels(keys, n, ncrit, base + 32 * s + lane, a[s], b[s]);
    each_begun_level(a[s], b[s], [&](int l, unsigned m) {
      if (lane == l) mine += __popc(m);
    });
  }
  if (lane < kTreeLevels) warp_cnt[wi][lane] = mine;
  __syncthreads();
  // lane l: non-leaf cells of level l begun before this warp's next body
  uint32_t run = 0;
  if (lane < kTreeLevels) {
    run = before[(size_t)lane * ntiles + blockIdx.x];
    for (int w = 0; w < wi; w++) run += warp_cnt[w][lane];
  }
#pragma unroll
  for (int s = 0; s < kTreeSteps; s++) {
    const int64_t i = base + 32 * s + lane;
    // upto: cells of the level above begun by bodies 0 .. i
    int upto = 0, prev = -2;
    each_begun_level(a[s], b[s], [&](int l, unsigned m) {
      if (l != prev + 1 && l > 0) upto = (int)__shfl_sync(0xffffffffu, run, l - 1);
      prev = l;
      const int incl = (int)__shfl_sync(0xffffffffu, run, l) + __popc(m & ((2u << lane) - 1));
      if ((m >> lane) & 1u) {
        int cell = 0;
        if (l > 0) {
          const int oct = (int)(keys[i] >> (kDepthBits + 3 * (kMaxDepth - l))) & 7;
          cell = 1 + 8 * (ranks.first[l - 1] + upto - 1) + oct;
        }
        node[ranks.first[l] + incl - 1] = make_int2((int)i, cell);
      }
      upto = incl;
      if (lane == l) run += __popc(m);
    });
  }
}

__device__ __forceinline__ int64_t lower_bound_u64(const uint64_t *__restrict__ a, int64_t lo,
                                                   int64_t hi, uint64_t v) {
  while (lo < hi) {
    int64_t mid = lo + ((hi - lo) >> 1);
    if (a[mid] < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// One thread per child of the non-leaf cells (rank q, octant o: cell 1 + 8q + o).
__global__ void __launch_bounds__(kBlock) build_children(
    int64_t nnode, LevelRanks ranks, const int2 *__restrict__ node,
    const uint64_t *__restrict__ keys, int64_t n, int ncrit, const double *__restrict__ box,
    uint64_t *__restrict__ ckey, int32_t *__restrict__ cbeg, int32_t *__restrict__ cnb,
    int32_t *__restrict__ cparent, int32_t *__restrict__ cchild, int32_t *__restrict__ cleaf,
    int32_t *__restrict__ clevel, double *__restrict__ cmin, double *__restrict__ cmax,
    double *__restrict__ ccen) {
  const int64_t total = 8 * nnode, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t t0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); t0 < total;
       t0 += stride) {  // warp-uniform: the lanes of a node exchange their bounds
    const int64_t t = t0 + (threadIdx.x & 31);
    const bool in = t < total;
    const int64_t q = in ? t >> 3 : 0;
    const int o = (int)(t & 7);
    const int2 nd = node[q];
    int level = 0;  // of the parent
    while (q >= ranks.first[level + 1]) level++;
    const int shift = kDepthBits + 3 * (kMaxDepth - level);
    const uint64_t pk = (keys[nd.x] >> shift << shift) | (uint64_t)level;
    const uint64_t k = key_child(pk, o);
    // this child's end: the first body of the next one, or beyond the parent
    const uint64_t next = o < 7 ? key_child(pk, o + 1) : key_next(pk);
    int64_t lo = nd.x, hi = lo + ncrit + 1;  // the parent holds more than ncrit bodies
    while (hi < n && keys[hi] < next) {
      const int64_t w = hi - lo;
      lo = hi;
      hi += 2 * w;
    }
    const int64_t re = lower_bound_u64(keys, lo, min(hi, n), next);
    const int64_t rprev = __shfl_up_sync(0xffffffffu, re, 1, 8);
    const int64_t rb = o == 0 ? nd.x : rprev;
    if (!in) continue;
    const int64_t c = 1 + t;
    if (o == 0) cchild[nd.y] = (int32_t)c;
    const int nb = (int)(re - rb), depth = level + 1;
    // Leaf iff nb <= ncrit.  Cells at the deepest key level are leaves too:
    // the reference's child-key shift is undefined there.
    const bool leaf = nb <= ncrit || depth >= kMaxDepth;
    ckey[c] = k;
    cbeg[c] = (int32_t)rb;
    cnb[c] = nb;
    cparent[c] = nd.y;
    if (leaf) cchild[c] = -1;  // else its own children's thread writes it
    cleaf[c] = leaf ? 1 : 0;
    clevel[c] = depth;
    // Region: the root's box halved once per level (CalcRegion, sfc_morton.h:536-557).
    double mn[3] = {box[0], box[0], box[0]}, mx[3] = {box[1], box[1], box[1]};
    for (int l = 1; l <= depth; l++) {
      const int ci = (int)(k >> (kDepthBits + 3 * (kMaxDepth - l))) & 7;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const double mid = dadd(mx[d], mn[d]) / 2;
        if ((ci >> d) & 1) mn[d] = mid; else mx[d] = mid;
      }
    }
#pragma unroll
    for (int d = 0; d < 3; d++) {
      cmin[3 * c + d] = mn[d];
      cmax[3 * c + d] = mx[d];
      ccen[3 * c + d] = dadd(mx[d], mn[d]) / 2;
    }
  }
}

__global__ void collect_leaves(const int32_t *__restrict__ cleaf, const int32_t *__restrict__ cnb,
                               int64_t ncells, int32_t *__restrict__ flag) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ncells;
       i += (int64_t)gridDim.x * blockDim.x)
    flag[i] = (cleaf[i] && cnb[i] > 0) ? 1 : 0;
}

__global__ void compact_indices(const int32_t *__restrict__ flag,
                                const int32_t *__restrict__ scan, int64_t n,
                                int32_t *__restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    if (flag[i]) out[scan[i]] = (int32_t)i;
}

__global__ void leaf_depth_hist(const int32_t *__restrict__ leaves, int64_t nleaves,
                                const int32_t *__restrict__ clevel, const int32_t *__restrict__ cnb,
                                int nbins, unsigned long long *__restrict__ hist) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < nleaves;
       w += (int64_t)gridDim.x * blockDim.x) {
    const int c = leaves[w];
    const int d = min(clevel[c], nbins - 1);
    atomicAdd(hist + d, (unsigned long long)cnb[c]);
  }
}

}  // namespace

int leaf_depth_histogram(tapas_b200_ctx *ctx, int nbins, int64_t *out) {
  if (!ctx->have_tree) {
    set_error(ctx, "leaf_depth_histogram: no tree");
    return TAPAS_B200_ERR_STATE;
  }
  if (nbins < 1 || nbins > 64 || !out) {
    set_error(ctx, "leaf_depth_histogram: nbins must be 1..64");
    return TAPAS_B200_ERR_ARG;
  }
  cudaStream_t s = ctx->stream;
  TB_CUDA(ctx, ctx->counters.ensure(64, s));
  TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p, 0, 64 * sizeof(unsigned long long), s));
  const int64_t nl = ctx->n_nonempty_leaves;
  if (nl > 0) {
    leaf_depth_hist<<<grid_for(nl, kBlock), kBlock, 0, s>>>(ctx->leaf_list.p, nl, ctx->clevel.p,
                                                             ctx->cnb.p, nbins, ctx->counters.p);
    TB_LAUNCH_CHECK(ctx);
  }
  TB_CUDA(ctx, cudaMemcpyAsync(out, ctx->counters.p, nbins * sizeof(unsigned long long),
                               cudaMemcpyDeviceToHost, s));
  TB_CUDA(ctx, cudaStreamSynchronize(s));
  return TAPAS_B200_OK;
}

static int ensure_cells(tapas_b200_ctx *ctx, int64_t need) {
  cudaStream_t s = ctx->stream;
  TB_CUDA(ctx, ctx->ckey.ensure(need, s));
  TB_CUDA(ctx, ctx->cbeg.ensure(need, s));
  TB_CUDA(ctx, ctx->cnb.ensure(need, s));
  TB_CUDA(ctx, ctx->cparent.ensure(need, s));
  TB_CUDA(ctx, ctx->cchild.ensure(need, s));
  TB_CUDA(ctx, ctx->cleaf.ensure(need, s));
  TB_CUDA(ctx, ctx->clevel.ensure(need, s));
  TB_CUDA(ctx, ctx->cmin.ensure(3 * need, s));
  TB_CUDA(ctx, ctx->cmax.ensure(3 * need, s));
  TB_CUDA(ctx, ctx->ccen.ensure(3 * need, s));
  return TAPAS_B200_OK;
}

int build_tree(tapas_b200_ctx *ctx, int ncrit) {
  cudaStream_t s = ctx->stream;
  const int64_t n = ctx->n;
  if (n <= 0) {
    set_error(ctx, "partition: no bodies");
    return TAPAS_B200_ERR_ARG;
  }
  ctx->have_tree = ctx->have_lists = ctx->have_M = ctx->have_L = false;
  ctx->level_ops_P = 0;  // translation operators belong to the previous tree
  ctx->ncrit = ncrit;
  TB_CUDA(ctx, ctx->keys.ensure(n, s));
  TB_CUDA(ctx, ctx->keys_alt.ensure(n, s));
  TB_CUDA(ctx, ctx->idx.ensure(n, s));
  TB_CUDA(ctx, ctx->idx_alt.ensure(n, s));
  TB_CUDA(ctx, ctx->sx.ensure(n, s));
  TB_CUDA(ctx, ctx->sy.ensure(n, s));
  TB_CUDA(ctx, ctx->sz.ensure(n, s));
  TB_CUDA(ctx, ctx->sq.ensure(n, s));
  TB_CUDA(ctx, ctx->body_pack.ensure(n, s));
  TB_CUDA(ctx, ctx->trg.ensure(4 * n, s));
  TB_CUDA(ctx, ctx->bbox.ensure(2, s));

  {
    PhaseTimer t(ctx, &ctx->timings.bbox_keys);
    const int nparts = grid_for(n, kBlock, ctx->num_sms * 4);
    TB_CUDA(ctx, ctx->scratch_d.ensure(2 * nparts + 2, s));
    bbox_partial<<<nparts, kBlock, 0, s>>>(ctx->x.p, ctx->y.p, ctx->z.p, n, ctx->scratch_d.p);
    TB_LAUNCH_CHECK(ctx);
    bbox_final<<<1, kBlock, 0, s>>>(ctx->scratch_d.p, nparts, ctx->bbox.p);
    TB_LAUNCH_CHECK(ctx);
    keys_kernel<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
        ctx->x.p, ctx->y.p, ctx->z.p, ctx->q_pending ? nullptr : ctx->q.p, n, ctx->bbox.p,
        ctx->keys.p, ctx->idx.p, ctx->body_pack.p);
    TB_LAUNCH_CHECK(ctx);
  }
  const int ntiles = (int)((n + kTreeTile - 1) / kTreeTile);
  // tally of the long unordered runs, level totals, counts per level and tile
  constexpr int kTotals = 2 + kTreeLevels;
  TB_CUDA(ctx, ctx->tree_cnt.ensure(kTotals + (size_t)kTreeLevels * ntiles, s));
  unsigned long long *d_tally = reinterpret_cast<unsigned long long *>(ctx->tree_cnt.p);
  uint32_t *d_total = ctx->tree_cnt.p + 2, *cnt = ctx->tree_cnt.p + kTotals;
  // the long runs and the sort of their bodies live in the results' rows, which
  // nothing holds yet: 24 n bytes of keys and values, then at most n / 33 runs
  uint64_t *const rk[2] = {reinterpret_cast<uint64_t *>(ctx->trg.p),
                           reinterpret_cast<uint64_t *>(ctx->trg.p) + n};
  uint32_t *const rv[2] = {reinterpret_cast<uint32_t *>(rk[1] + n),
                           reinterpret_cast<uint32_t *>(rk[1] + n) + n};
  int2 *const runs = reinterpret_cast<int2 *>(rk[1] + 2 * n);
  {
    PhaseTimer t(ctx, &ctx->timings.sort);
    // bits 4..0, the depth, are 19 for every body
    uint64_t *k = ctx->keys.p, *ka = ctx->keys_alt.p;
    uint32_t *v = ctx->idx.p, *va = ctx->idx_alt.p;
    TB_TRY(radix_sort(ctx, k, ka, v, va, n, kSortLow, kDepthBits + 3 * kMaxDepth));
    if (k != ctx->keys.p) { std::swap(ctx->keys.p, ctx->keys_alt.p); std::swap(ctx->keys.cap, ctx->keys_alt.cap); }
    if (v != ctx->idx.p) { std::swap(ctx->idx.p, ctx->idx_alt.p); std::swap(ctx->idx.cap, ctx->idx_alt.cap); }
    TB_CUDA(ctx, cudaMemsetAsync(d_tally, 0, sizeof *d_tally, s));
    TB_TRY(order_equal_runs(ctx, ctx->keys.p, ctx->idx.p, n, kSortLow, kMaxRun, runs, d_tally));
    if (ctx->q_pending) {  // the charges' copy ran alongside the keys and the sort
      TB_CUDA(ctx, cudaStreamWaitEvent(s, ctx->q_ready, 0));
      pack_charges<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(ctx->q.p, n,
                                                                            ctx->body_pack.p);
      TB_LAUNCH_CHECK(ctx);
      ctx->q_pending = false;
    }
    gather_bodies<<<grid_for(n, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
        ctx->body_pack.p, ctx->idx.p, n, ctx->sx.p, ctx->sy.p, ctx->sz.p, ctx->sq.p);
    TB_LAUNCH_CHECK(ctx);
  }
  TB_CUDA(ctx, ctx->pinned.ensure(tapas_b200_ctx::kPinnedBytes));
  const unsigned long long *h_tally = reinterpret_cast<unsigned long long *>(ctx->pinned.p);
  const uint32_t *h_total = reinterpret_cast<uint32_t *>(ctx->pinned.p) + 2;
  auto count_levels = [&]() -> int {
    PhaseTimer t(ctx, &ctx->timings.tree, true);
    count_nonleaves<<<ntiles, kBlock, 0, s>>>(ctx->keys.p, n, ncrit, ntiles, cnt);
    TB_LAUNCH_CHECK(ctx);
    TB_TRY(scan_rows(ctx, cnt, kTreeLevels, ntiles, d_total));
    TB_CUDA(ctx, cudaMemcpyAsync(ctx->pinned.p, d_tally, kTotals * sizeof(uint32_t),
                                 cudaMemcpyDeviceToHost, s));
    TB_CUDA(ctx, cudaStreamSynchronize(s));
    return TAPAS_B200_OK;
  };
  TB_TRY(count_levels());
  if (*h_tally) {
    {
      PhaseTimer t(ctx, &ctx->timings.sort, true);
      const int64_t total = (int64_t)(*h_tally & 0xFFFFFFFFull);
      const uint32_t *at = nullptr;
      TB_TRY(order_long_runs(ctx, ctx->keys.p, ctx->idx.p, runs, (int)(*h_tally >> 32), total,
                             kDepthBits, kSortLow, rk, rv, at));
      gather_places<<<grid_for(total, kBlock, ctx->num_sms * 16), kBlock, 0, s>>>(
          ctx->body_pack.p, ctx->idx.p, at, total, ctx->sx.p, ctx->sy.p, ctx->sz.p, ctx->sq.p);
      TB_LAUNCH_CHECK(ctx);
    }
    TB_TRY(count_levels());
  }
  PhaseTimer t(ctx, &ctx->timings.tree, true);
  LevelRanks ranks;
  int64_t nnode = 0;
  int depth = 0;
  ctx->level_off.assign(1, 0);
  ctx->level_off.push_back(1);
  for (int l = 0; l < kTreeLevels; l++) {
    ranks.first[l] = (int32_t)nnode;
    nnode += h_total[l];
    if (nnode > (int64_t)0x0FFFFFFF) {
      set_error(ctx, "tree build: more than 2^31 cells");
      return TAPAS_B200_ERR_CAPACITY;
    }
    if (h_total[l]) {
      depth = l + 1;
      ctx->level_off.push_back(1 + 8 * nnode);
    }
  }
  ranks.first[kTreeLevels] = (int32_t)nnode;
  ctx->ncells = 1 + 8 * nnode;
  ctx->max_depth = depth;
  TB_TRY(ensure_cells(ctx, ctx->ncells));
  init_root<<<1, 32, 0, s>>>(n, ncrit, ctx->bbox.p, ctx->ckey.p, ctx->cbeg.p, ctx->cnb.p,
                             ctx->cparent.p, ctx->cchild.p, ctx->cleaf.p, ctx->clevel.p,
                             ctx->cmin.p, ctx->cmax.p, ctx->ccen.p);
  TB_LAUNCH_CHECK(ctx);
  if (nnode > 0) {
    TB_CUDA(ctx, ctx->tree_nodes.ensure(nnode, s));
    list_nonleaves<<<ntiles, kBlock, 0, s>>>(ctx->keys.p, n, ncrit, ntiles, cnt, ranks,
                                             ctx->tree_nodes.p);
    TB_LAUNCH_CHECK(ctx);
    build_children<<<grid_for(8 * nnode, kBlock, ctx->num_sms * 32), kBlock, 0, s>>>(
        nnode, ranks, ctx->tree_nodes.p, ctx->keys.p, n, ncrit, ctx->bbox.p, ctx->ckey.p,
        ctx->cbeg.p, ctx->cnb.p, ctx->cparent.p, ctx->cchild.p, ctx->cleaf.p, ctx->clevel.p,
        ctx->cmin.p, ctx->cmax.p, ctx->ccen.p);
    TB_LAUNCH_CHECK(ctx);
  }
  // Non-empty leaves (the P2M / L2P / P2P work units).
  const int64_t C = ctx->ncells;
  TB_CUDA(ctx, ctx->flag.ensure(C + 1, s));
  TB_CUDA(ctx, ctx->flag_scan.ensure(C + 1, s));
  TB_CUDA(ctx, ctx->leaf_list.ensure(C + 1, s));
  collect_leaves<<<grid_for(C, kBlock), kBlock, 0, s>>>(ctx->cleaf.p, ctx->cnb.p, C, ctx->flag.p);
  TB_LAUNCH_CHECK(ctx);
  TB_TRY(scan_exclusive(ctx, ctx->flag.p, ctx->flag_scan.p, C, ctx->flag_scan.p + C));
  compact_indices<<<grid_for(C, kBlock), kBlock, 0, s>>>(ctx->flag.p, ctx->flag_scan.p, C,
                                                         ctx->leaf_list.p);
  TB_LAUNCH_CHECK(ctx);
  double *hb = reinterpret_cast<double *>(ctx->pinned.p);
  TB_CUDA(ctx, cudaMemcpyAsync(hb, ctx->bbox.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
  TB_CUDA(ctx, cudaMemcpyAsync(reinterpret_cast<int32_t *>(hb + 2), ctx->flag_scan.p + C,
                               sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  TB_CUDA(ctx, cudaStreamSynchronize(s));
  ctx->box_lo = hb[0];
  ctx->box_hi = hb[1];
  ctx->n_nonempty_leaves = *reinterpret_cast<int32_t *>(hb + 2);
  ctx->have_tree = true;
  return TAPAS_B200_OK;
}

}  // namespace tb
