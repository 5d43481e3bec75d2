// Barnes-Hut path of the reference's sample (sample/barnes-hut/bh.cc) on the
// same octree (tree.cu), body mass in the charge slot.
//
//  bh_upward_level  Approximate (bh.cc:155-190), one launch per level from the
//                   deepest: an empty leaf is zero, a one-body leaf is that
//                   body, a non-leaf the mass and mass-weighted centre of its 8
//                   children summed in index order (leaves with more bodies,
//                   ncrit > 1, use the same formula over their bodies).
//  bh_walk64, bh_walk32   interact + ComputeForce (bh.cc:135-153, 192-224): each
//                   body walks the tree depth first from the root, children
//                   visited 0..7 like the sample's recursion; a warp's 32
//                   bodies (consecutive in Morton order) share one bounded
//                   stack of the union of their walks (below).  A cell is
//                   accepted when width / |centre - body| < theta; a leaf is
//                   summed body by body (the body itself included, as in the
//                   sample).
// The FP64 form rounds as the sample does, operation by operation in the
// sample's order, so it reproduces the sample bit for bit; the FP32 form
// ("mixed") takes the same decisions and sums FP32 terms of FP32 positions and
// FP32 copies of the FP64 cell moments.
#include <cfloat>

#include "common.cuh"
#include "primitives.cuh"

namespace tb {
namespace {

constexpr int kStack = 192;  // > 7 pending siblings x 19 levels + 1

__global__ void bh_upward_level(int64_t a, int64_t cnt, const int32_t *__restrict__ cleaf,
                                const int32_t *__restrict__ cnb, const int32_t *__restrict__ cbeg,
                                const int32_t *__restrict__ cchild, const double *__restrict__ sx,
                                const double *__restrict__ sy, const double *__restrict__ sz,
                                const double *__restrict__ sm, double4 *__restrict__ attr) {
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < cnt;
       w += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = a + w;
    double4 r;
    if (cleaf[c]) {
      const int nb = cnb[c], b0 = cbeg[c];
      if (nb == 0) {
        r = make_double4(0, 0, 0, 0);
      } else if (nb == 1) {
        r = make_double4(sx[b0], sy[b0], sz[b0], sm[b0]);
      } else {
        double W = 0, X = 0, Y = 0, Z = 0;
        for (int i = 0; i < nb; i++) {
          const int b = b0 + i;
          W = __dadd_rn(W, sm[b]);
          X = __dadd_rn(X, __dmul_rn(sx[b], sm[b]));
          Y = __dadd_rn(Y, __dmul_rn(sy[b], sm[b]));
          Z = __dadd_rn(Z, __dmul_rn(sz[b], sm[b]));
        }
        r = make_double4(__ddiv_rn(X, W), __ddiv_rn(Y, W), __ddiv_rn(Z, W), W);
      }
    } else {
      double W = 0, X = 0, Y = 0, Z = 0;
      const int ch = cchild[c];
      for (int i = 0; i < 8; i++) {
        const double4 s = attr[ch + i];
        W = __dadd_rn(W, s.w);
        X = __dadd_rn(X, __dmul_rn(s.x, s.w));
        Y = __dadd_rn(Y, __dmul_rn(s.y, s.w));
        Z = __dadd_rn(Z, __dmul_rn(s.z, s.w));
      }
      r = make_double4(__ddiv_rn(X, W), __ddiv_rn(Y, W), __ddiv_rn(Z, W), W);
    }
    attr[c] = r;
  }
}

// What the walks read of a cell, packed per walk: centre and squared width, and
// {first child, -1}, or for a leaf {its bodies, their number}: the first body
// of the FP64 walk, the first pair of the FP32 walk's body pairs.
struct BhCells {
  const double4 *geo;
  const int2 *meta;
  const double *cmin, *cmax, *ccen;  // the acceptance test inside its band
};

// 1/x of the rounded sqrt(r2), each correctly rounded, as the sample computes it
// (bh.cc:148-149), from the hardware's approximation: refined to about an ulp
// (the series of charge_over_distance), then one residual step each for the square
// root and the reciprocal (Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990).  The residuals are exact in an fma, so
// before its rounding the root is off by less than 2^-103, relative, and the
// reciprocal (its step taken to second order, e + e^2: y is up to an ulp off 1/s) by at
// most 2^-106.  The roots that lie so close to the middle of two numbers, squares of odd
// 54-bit integers within 128 of a multiple of 2^54 or 2^55, were enumerated: all round
// right whatever the approximation's error (below 2^-20).  The one reciprocal within
// 2^-106 of a middle that does not is that of an s with all mantissa bits set (r2 just
// below a power of four, as for a unit step of a lattice summed up from tenths),
// which is tested for.  11 FP64 operations (y is halved in its
// exponent) where the two library sequences take about 57 slots of the FP64 pipe.
// kN at once, with one branch for all: a branch each would keep their chains
// from overlapping.
template <int kN>
__device__ __forceinline__ void rounded_inv_sqrt(const double (&r2)[kN], double (&inv)[kN]) {
  // outside 2^-767 .. 2^768 the residuals could underflow; s has all mantissa bits set for
  // the two numbers below a power of four only
  auto library = [](double r2) {
    return (unsigned)__double2hiint(r2) - 0x10000000u >= 0x60000000u ||
           (unsigned)__double2loint(r2) >= 0xfffffffeu;
  };
  bool odd = false;
#pragma unroll
  for (int i = 0; i < kN; i++) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2[i]));
    double e = fma(-(r2[i] * y), y, 1.0);
    y = fma(y, e * fma(e, 0.375, 0.5), y);
    const double g = r2[i] * y;
    const double half_y = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    const double s = fma(fma(-g, g, r2[i]), half_y, g);
    e = fma(-s, y, 1.0);
    inv[i] = fma(y, fma(e, e, e), y);
    odd |= library(r2[i]);
  }
  if (odd) {
#pragma unroll
    for (int i = 0; i < kN; i++)
      if (library(r2[i])) inv[i] = __ddiv_rn(1.0, __dsqrt_rn(r2[i]));
  }
}

// The sample's acceptance test fl(width / fl(|centre - body|)) < theta.  That
// quotient is width / distance within ~2.3 ulp and d below is s^2 - theta^2 R
// within ~5 ulp of s^2, so outside a relative band of 2^-42 (2.3e-13) the sign
// of d decides the same way without the square root and the division; inside
// it (and for d not finite) the sample's own operations decide.  The band is
// tested on the high words: 8 slots of the FP64 pipe per test.
__device__ __forceinline__ bool bh_accept(const BhCells &T, int c, const double4 &g, double px,
                                          double py, double pz, double theta, double theta2) {
  const double dx = px - g.x, dy = py - g.y, dz = pz - g.z;
  const double R = fma(dz, dz, fma(dy, dy, dx * dx));
  const double d = fma(-theta2, R, g.w);
  const int hd = __double2hiint(d);
  const int lo = max(__double2hiint(g.w) - (42 << 20), 0);
  if ((unsigned)((hd & 0x7fffffff) - lo) < (unsigned)(0x7ff00000 - lo)) return hd < 0;
  const double ex = __dsub_rn(px, T.ccen[3 * c]), ey = __dsub_rn(py, T.ccen[3 * c + 1]),
               ez = __dsub_rn(pz, T.ccen[3 * c + 2]);
  double R2 = __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey));
  R2 = __dadd_rn(R2, __dmul_rn(ez, ez));
  const double s = __dsub_rn(T.cmax[3 * c], T.cmin[3 * c]);
  return __ddiv_rn(s, __dsqrt_rn(R2)) < theta;
}

// What the acceptance test gives for all bodies of a warp at once, from their
// bounding box: 1 every body accepts the cell, 2 every body opens it, 0 neither is
// certain.  The nearest and farthest squared distances of the box to the centre
// bound the bodies' own; the margin of 1e-12 is far above the rounding on
// either side and the exact test's band, so a certain answer is every body's.
struct BodyBox {
  double lo[3], hi[3];
};
__device__ __forceinline__ BodyBox body_box(bool valid, double px, double py, double pz) {
  BodyBox b;
  const double p[3] = {px, py, pz}, inf = __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    b.lo[d] = valid ? p[d] : inf;
    b.hi[d] = valid ? p[d] : -inf;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      b.lo[d] = fmin(b.lo[d], __shfl_xor_sync(0xffffffffu, b.lo[d], o));
      b.hi[d] = fmax(b.hi[d], __shfl_xor_sync(0xffffffffu, b.hi[d], o));
    }
  }
  return b;
}
__device__ __forceinline__ int box_accept(const BodyBox &b, const double4 &g, double theta2) {
  const double c[3] = {g.x, g.y, g.z};
  double near2 = 0, far2 = 0;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double u = b.lo[d] - c[d], v = c[d] - b.hi[d];  // > 0: the box is beyond c
    const double n = fmax(fmax(u, v), 0.0), f = fmax(-u, -v);
    near2 = fma(n, n, near2);
    far2 = fma(f, f, far2);
  }
  if (g.w < theta2 * near2 * (1.0 - 1e-12)) return 1;
  if (g.w > theta2 * far2 * (1.0 + 1e-12)) return 2;
  return 0;
}

__device__ __forceinline__ void add_counts(int lane, unsigned long long napprox,
                                           unsigned long long ndirect, bool overflow,
                                           unsigned long long *__restrict__ counters) {
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    napprox += __shfl_xor_sync(0xffffffffu, napprox, s);
    ndirect += __shfl_xor_sync(0xffffffffu, ndirect, s);
  }
  if (lane == 0) {
    if (napprox) atomicAdd(counters + 0, napprox);
    if (ndirect) atomicAdd(counters + 1, ndirect);
    if (overflow) atomicOr(counters + 2, 1ull);
  }
}

// Opens a cell for the lanes `reach`: its eight children (from ch on) are classed
// by eight lanes with the bodies' box, the uncertain ones tested body by body, and
// each is pushed, child 7 first, with the lanes that accept it and the lanes that
// open it (a leaf with `reach`; empty leaves are left out).  Returns the new
// stack height; the warp is converged before and after.
__device__ __forceinline__ int push_children(const BhCells &T, int ch, unsigned reach,
                                             const BodyBox &box, int lane, double px, double py,
                                             double pz, double theta, double theta2, int4 *stack,
                                             int sp) {
  const int c = ch + (lane & 7);
  const int2 m = T.meta[c];
  const double4 g = T.geo[c];
  const int kind = m.y < 0 ? box_accept(box, g, theta2) : 3;  // 3: a leaf
  // this lane's child (lanes 0..7): accepting and opening lanes
  unsigned am = kind == 1 ? reach : 0u, om = kind == 2 ? reach : 0u;
  unsigned todo = __ballot_sync(0xffffffffu, kind == 0) & 0xffu;
  while (todo) {
    const int i = __ffs(todo) - 1;
    todo &= todo - 1;
    double4 gi;
    gi.x = __shfl_sync(0xffffffffu, g.x, i);
    gi.y = __shfl_sync(0xffffffffu, g.y, i);
    gi.z = __shfl_sync(0xffffffffu, g.z, i);
    gi.w = __shfl_sync(0xffffffffu, g.w, i);
    const bool acc = bh_accept(T, ch + i, gi, px, py, pz, theta, theta2);
    const unsigned a = __ballot_sync(0xffffffffu, acc) & reach;
    if (lane == i) {
      am = a;
      om = reach & ~a;
    }
  }
  // every lane has read the popped entries (the ballots); child 7 at the bottom
  const bool push = lane < 8 && m.y != 0;  // not an empty leaf
  const unsigned pushes = __ballot_sync(0xffffffffu, push);
  if (push)
    stack[sp + __popc(pushes >> (lane + 1))] =
        m.y > 0 ? make_int4(m.x, m.y, (int)reach, 0) : make_int4(c, -m.x, (int)am, (int)om);
  __syncwarp();
  return sp + __popc(pushes);
}

// A warp's walk: the stack, and the accepted cells and leaves in walk order.
struct __align__(16) Walk {
  // {cell, -first child, accepting lanes, opening lanes} or, a leaf, {first body
  // or pair, bodies, lanes, 0}
  int4 stack[kStack];
  int2 list[64];  // {first body or pair, bodies} or {~cell, -1}
  unsigned list_lanes[64];
};

// One step of a warp's walk: pops the entries from the top down to the first that
// opens, appends the accepted cells and the leaves among them to the list (at
// most 31 long before), and opens that one.  False: the stack would overflow.
// napprox and ndirect count the interactions of the entries this lane popped.
__device__ __forceinline__ bool walk_step(const BhCells &T, Walk &S, const BodyBox &box, int lane,
                                          double px, double py, double pz, double theta,
                                          double theta2, int &sp, int &count,
                                          unsigned long long &napprox,
                                          unsigned long long &ndirect) {
  int4 e = make_int4(0, 0, 0, 0);
  if (lane < sp) e = S.stack[sp - 1 - lane];
  const bool leaf = e.y >= 0;
  const unsigned opens = __ballot_sync(0xffffffffu, !leaf && e.w != 0);
  const int top = opens ? __ffs(opens) : min(sp, 32);
  const bool add = lane < top && e.z != 0;
  const unsigned adds = __ballot_sync(0xffffffffu, add);
  if (add) {
    const int k = count + __popc(adds & ((1u << lane) - 1));
    S.list[k] = leaf ? make_int2(e.x, e.y) : make_int2(~e.x, -1);
    S.list_lanes[k] = (unsigned)e.z;
    if (leaf) ndirect += (unsigned long long)e.y * __popc(e.z);
    else napprox += __popc(e.z);
  }
  count += __popc(adds);
  sp -= top;
  __syncwarp();
  if (opens) {
    const int ch = -__shfl_sync(0xffffffffu, e.y, top - 1);
    const unsigned reach = __shfl_sync(0xffffffffu, e.w, top - 1);
    if (sp + 8 > kStack) return false;
    sp = push_children(T, ch, reach, box, lane, px, py, pz, theta, theta2, S.stack, sp);
  }
  return true;
}

// Puts the root on a walk's empty stack.
__device__ __forceinline__ void walk_start(const BhCells &T, Walk &S, int lane, unsigned lanes,
                                           double px, double py, double pz, double theta,
                                           double theta2) {
  const int2 m = T.meta[0];
  int4 e = make_int4(m.x, m.y, (int)lanes, 0);
  if (m.y < 0) {
    const bool acc = (lanes >> lane & 1) && bh_accept(T, 0, T.geo[0], px, py, pz, theta, theta2);
    const unsigned am = __ballot_sync(0xffffffffu, acc);
    e = make_int4(0, -m.x, (int)am, (int)(lanes & ~am));
  }
  if (lane == 0) S.stack[0] = e;
  __syncwarp();
}

// Drops the list's first 32 entries.
__device__ __forceinline__ void walk_shift(Walk &S, int lane, int &count) {
  count -= 32;
  if (lane < count) {
    S.list[lane] = S.list[lane + 32];
    S.list_lanes[lane] = S.list_lanes[lane + 32];
  }
  __syncwarp();
}

// The inclusive sums of v over the lanes, and the first lane whose sum is above i.
__device__ __forceinline__ int lane_sums(int lane, int v) {
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, s);
    if (lane >= s) v += u;
  }
  return v;
}
__device__ __forceinline__ int lane_above(int sums, int i) {
  int k = 0;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1)
    if (__shfl_sync(0xffffffffu, sums, k + s - 1) <= i) k += s;
  return k;
}

// FP64: one walk per warp over the union of its 32 bodies' walks.  Opening a
// cell classes its eight children by eight lanes with the bodies' box, tests
// the uncertain ones body by body, and pushes each child with the lanes that
// accept it and the lanes that open it (leaves with the lanes that reach them).
// Popped depth first, children 0..7, the accepted cells and the leaves form a
// list; 32 entries at a time, their moments and bodies are loaded by a lane each
// and every lane adds the terms of its own entries in list order.  A lane's
// entries in the list are its own walk's, in its own walk's order, so it takes
// the sample's decisions and sums the sample's terms in the sample's order, bit
// for bit.
//
// Why so: 32 bodies' union walk is long and small sets have few warps (20k
// bodies: 625, one per scheduler), so the time is one warp's chain of dependent
// loads and FP64 sequences; here a chain step serves up to 32 popped entries,
// eight opened cells, 32 loads or four terms instead of one.  One warp per block,
// so that few warps spread evenly over the SMs.  20k bodies, ncrit 1: 0.67 ms (4M, ncrit 32:
// 128 ms; 125 with the reciprocal's step to first order, which a few s round wrong by);
// 0.81 ms with one entry popped at a time, 2.39 ms with one cell and one term at
// a time, 1.68 ms without the box's tests.
__global__ void __launch_bounds__(32) bh_walk64(
    BhCells T, int64_t n, const double *__restrict__ sx, const double *__restrict__ sy,
    const double *__restrict__ sz, const double *__restrict__ sm,
    const double4 *__restrict__ attr, double theta, double eps2, double *__restrict__ out,
    unsigned long long *__restrict__ counters) {
  __shared__ Walk S;
  __shared__ double4 data[32];
  __shared__ unsigned data_lanes[32];
  const int lane = threadIdx.x;
  const double theta2 = __dmul_rn(theta, theta);
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = b < n;
  const double px = valid ? sx[b] : 0.0, py = valid ? sy[b] : 0.0, pz = valid ? sz[b] : 0.0;
  double4 o = make_double4(0, 0, 0, 0);
  unsigned long long napprox = 0, ndirect = 0;
  bool overflow = false;
  const unsigned lanes = __ballot_sync(0xffffffffu, valid);
  if (lanes == 0) return;

  const BodyBox box = body_box(valid, px, py, pz);

  // Adds the terms of the first `count` (<= 32) list entries.
  auto flush = [&](int count) {
    int2 r = make_int2(0, 0);
    unsigned rm = 0;
    if (lane < count) {
      r = S.list[lane];
      rm = S.list_lanes[lane];
    }
    const int terms = r.y >= 0 ? r.y : 1;
    const int upto = lane_sums(lane, terms);
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    for (int c0 = 0; c0 < total; c0 += 32) {
      const int i = c0 + lane, k = lane_above(upto, i);
      const int p = __shfl_sync(0xffffffffu, r.x, k);
      const int p0 = __shfl_sync(0xffffffffu, upto - terms, k);
      const unsigned m = __shfl_sync(0xffffffffu, rm, k);
      double4 v = make_double4(0, 0, 0, 0);
      if (i < total) {
        const int j = p + (i - p0);
        v = p >= 0 ? make_double4(sx[j], sy[j], sz[j], sm[j]) : attr[~p];
      }
      data[lane] = v;
      data_lanes[lane] = i < total ? m : 0u;
      __syncwarp();
      const int end = min(32, total - c0);
#pragma unroll 1
      for (int q = 0; q < end; q += 4) {
        // ComputeForce (bh.cc:135-153), the sample's rounding order
        double dx[4], dy[4], dz[4], w[4], R2[4], inv[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const double4 a = data[q + i];
          dx[i] = __dsub_rn(a.x, px);
          dy[i] = __dsub_rn(a.y, py);
          dz[i] = __dsub_rn(a.z, pz);
          w[i] = a.w;
          R2[i] = __dadd_rn(__dmul_rn(dx[i], dx[i]), __dmul_rn(dy[i], dy[i]));
          R2[i] = __dadd_rn(__dadd_rn(R2[i], __dmul_rn(dz[i], dz[i])), eps2);
        }
        rounded_inv_sqrt(R2, inv);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const double inv3 = __dmul_rn(__dmul_rn(inv[i], inv[i]), inv[i]);
          const double tx = __dmul_rn(__dmul_rn(dx[i], inv3), w[i]),
                       ty = __dmul_rn(__dmul_rn(dy[i], inv3), w[i]),
                       tz = __dmul_rn(__dmul_rn(dz[i], inv3), w[i]), tw = __dmul_rn(inv[i], w[i]);
          if (data_lanes[q + i] >> lane & 1u) {
            o.x = __dadd_rn(o.x, tx);
            o.y = __dadd_rn(o.y, ty);
            o.z = __dadd_rn(o.z, tz);
            o.w = __dadd_rn(o.w, tw);
          }
        }
      }
      __syncwarp();
    }
  };

  int sp = 1, count = 0;
  walk_start(T, S, lane, lanes, px, py, pz, theta, theta2);
  while (sp > 0) {
    if (!walk_step(T, S, box, lane, px, py, pz, theta, theta2, sp, count, napprox, ndirect)) {
      overflow = true;
      break;
    }
    if (count >= 32) {
      flush(32);
      walk_shift(S, lane, count);
    }
  }
  if (!overflow) flush(count);
  if (valid) reinterpret_cast<double4 *>(out)[b] = o;
  add_counts(lane, napprox, ndirect, overflow, counters);
}

// 1/sqrt(x): the hardware approximation for x >= FLT_MIN (kNormal), else rsqrtf.
template <bool kNormal>
__device__ __forceinline__ float inv_sqrt32(float x) {
  if (!kNormal) return rsqrtf(x);
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// FP32: the same union walk, decisions and order (the acceptance test stays
// FP64).  Accepted cells and leaves form one list in walk order, appended for all
// the stack's top entries down to the first that opens at once.  32 entries are
// evaluated as one stream of slots, a slot a pair of leaf bodies or of cells: 32
// slots at a time are loaded by a lane each, whatever entry they belong to, into
// shared memory with the lanes that add each half, then evaluated by all lanes.
// Leaf bodies are stored as pairs {x0,x1,y0,y1},{z0,z1,m0,m1}, each leaf starting
// a pair (an odd leaf's last one is padded with a copy of its first body that no
// lane adds).  A slot's terms are evaluated by packed FP32 instructions, then added one
// after the other: an FP32 sum of 10^4 terms of one sign is rounded by 3e-5
// somewhere, and only the walk's own order rounds it where this form always has.
// Bound: issue slots and FP32 pipe; the union holds 1.37 times the bodies' own leaf
// bodies (a simulated 400k Plummer sphere: 73 % of the lanes add a listed body).
// 4M Plummer, ncrit 32: 41.4 ms; 66.5 ms with a cell or a body at a time; 43.7 ms as
// four warps to a block, whose slowest holds the others' places; 57.2 ms with one
// entry popped and evaluated at a time.
// kNormal: eps2 is a normal FP32 number, so no squared distance is below it.
constexpr int kSlots = 4;  // slots evaluated at once: 41.4 ms; 2: 42.5 ms

template <bool kNormal>
__global__ void __launch_bounds__(32, 32) bh_walk32(
    BhCells T, int64_t n, const double *__restrict__ sx, const double *__restrict__ sy,
    const double *__restrict__ sz, const float4 *__restrict__ attr32,
    const float4 *__restrict__ pairs, double theta, float eps2, double *__restrict__ out,
    unsigned long long *__restrict__ counters) {
  __shared__ Walk S;
  __shared__ BodyBox box;  // kept here: the registers are needed
  // staged slots {x0,x1,y0,y1}, {z0,z1,m0,m1} and the lanes that add their halves
  __shared__ float4 slot_a[32], slot_b[32];
  __shared__ uint2 slot_lanes[32];
  const int lane = threadIdx.x;
  const unsigned me = 1u << lane;
  const double theta2 = __dmul_rn(theta, theta);
  const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = b < n;
  const double px = valid ? sx[b] : 0.0, py = valid ? sy[b] : 0.0, pz = valid ? sz[b] : 0.0;
  const float fx = -(float)px, fy = -(float)py, fz = -(float)pz;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  unsigned long long napprox = 0, ndirect = 0;
  bool overflow = false;
  const unsigned lanes = __ballot_sync(0xffffffffu, valid);
  if (lanes == 0) return;
  {
    const BodyBox bx = body_box(valid, px, py, pz);
    if (lane == 0) box = bx;
    __syncwarp();
  }

  // Evaluates the first `count` (<= 32) list entries.
  auto flush = [&](int count) {
    int2 r = make_int2(0, 0);
    unsigned rm = 0;
    if (lane < count) {
      r = S.list[lane];
      rm = S.list_lanes[lane];
    }
    // a run of cells is taken in pairs: the second one's slot is the first one's
    const unsigned cells = __ballot_sync(0xffffffffu, r.y < 0);
    const int before = lane ? __clz(~(cells << (32 - lane))) : 0;  // cells just below
    const int slots = r.y >= 0 ? (r.y + 1) >> 1 : (before & 1) ^ 1;
    const int upto = lane_sums(lane, slots);
    const int total = __shfl_sync(0xffffffffu, upto, 31);
    for (int c0 = 0; c0 < total; c0 += 32) {
      const int i = c0 + lane, k = lane_above(upto, i);
      const int p = __shfl_sync(0xffffffffu, r.x, k);
      const int p0 = __shfl_sync(0xffffffffu, upto - slots, k);
      const int nb = __shfl_sync(0xffffffffu, r.y, k);
      const unsigned m0 = __shfl_sync(0xffffffffu, rm, k);
      const int pn = __shfl_sync(0xffffffffu, r.x, (k + 1) & 31);
      const unsigned mn = __shfl_sync(0xffffffffu, rm, (k + 1) & 31);
      if (i < total) {
        if (p >= 0) {
          const float4 *src = pairs + 2 * ((int64_t)p + (i - p0));
          slot_a[lane] = __ldg(src);
          slot_b[lane] = __ldg(src + 1);
          // no lane adds an odd leaf's padding: with eps2 = 0 its term is 0 * inf
          slot_lanes[lane] = make_uint2(m0, 2 * (i - p0) + 1 < nb ? m0 : 0u);
        } else {
          const bool two = k < 31 && (cells >> (k + 1) & 1);
          const float4 u = __ldg(attr32 + ~p);
          const float4 v = two ? __ldg(attr32 + ~pn) : u;
          slot_a[lane] = make_float4(u.x, v.x, u.y, v.y);
          slot_b[lane] = make_float4(u.z, v.z, u.w, v.w);
          slot_lanes[lane] = make_uint2(m0, two ? mn : 0u);
        }
      } else {
        slot_lanes[lane] = make_uint2(0u, 0u);  // whatever the slot holds
      }
      __syncwarp();
      const int end = min(32, total - c0);
#pragma unroll 1
      for (int q0 = 0; q0 < end; q0 += kSlots)
#pragma unroll
      for (int q = q0; q < q0 + kSlots; q++) {
        const float4 u = slot_a[q], v = slot_b[q];
        const uint2 m = slot_lanes[q];
        const float2 dx = __fadd2_rn(make_float2(u.x, u.y), make_float2(fx, fx)),
                     dy = __fadd2_rn(make_float2(u.z, u.w), make_float2(fy, fy)),
                     dz = __fadd2_rn(make_float2(v.x, v.y), make_float2(fz, fz));
        const float2 R2 = __ffma2_rn(
            dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, make_float2(eps2, eps2))));
        const float2 inv = make_float2(inv_sqrt32<kNormal>(R2.x), inv_sqrt32<kNormal>(R2.y));
        const float2 wr = __fmul2_rn(make_float2(v.z, v.w), inv);
        const float2 wr3 = __fmul2_rn(__fmul2_rn(wr, inv), inv);
        if (m.x & me) {
          o.x = fmaf(dx.x, wr3.x, o.x);
          o.y = fmaf(dy.x, wr3.x, o.y);
          o.z = fmaf(dz.x, wr3.x, o.z);
          o.w = __fadd_rn(o.w, wr.x);
        }
        if (m.y & me) {
          o.x = fmaf(dx.y, wr3.y, o.x);
          o.y = fmaf(dy.y, wr3.y, o.y);
          o.z = fmaf(dz.y, wr3.y, o.z);
          o.w = __fadd_rn(o.w, wr.y);
        }
      }
      __syncwarp();
    }
  };

  int sp = 1, count = 0;
  walk_start(T, S, lane, lanes, px, py, pz, theta, theta2);
  while (sp > 0) {
    if (!walk_step(T, S, box, lane, px, py, pz, theta, theta2, sp, count, napprox, ndirect)) {
      overflow = true;
      break;
    }
    if (count >= 32) {
      flush(32);
      walk_shift(S, lane, count);
    }
  }
  if (!overflow) flush(count);
  if (valid)
    reinterpret_cast<double4 *>(out)[b] =
        make_double4((double)o.x, (double)o.y, (double)o.z, (double)o.w);
  add_counts(lane, napprox, ndirect, overflow, counters);
}

// Body pairs of a leaf (0 for other cells), for the FP32 walk's pair offsets.
__global__ void bh_pair_counts(int64_t ncells, const int32_t *__restrict__ cleaf,
                               const int32_t *__restrict__ cnb, int32_t *__restrict__ cnt) {
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < ncells;
       c += (int64_t)gridDim.x * blockDim.x)
    cnt[c] = cleaf[c] ? (cnb[c] + 1) >> 1 : 0;
}

// The walk's cell records; with pair_off (FP32 walk) also the FP32 moments and
// the leaves' body pairs, eight threads per cell.
__global__ void __launch_bounds__(256) bh_pack(
    int64_t ncells, const int32_t *__restrict__ cleaf, const int32_t *__restrict__ cnb,
    const int32_t *__restrict__ cbeg, const int32_t *__restrict__ cchild,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double *__restrict__ ccen, const double4 *__restrict__ attr,
    const int32_t *__restrict__ pair_off, const double *__restrict__ sx,
    const double *__restrict__ sy, const double *__restrict__ sz, const double *__restrict__ sm,
    double4 *__restrict__ geo, int2 *__restrict__ meta, float4 *__restrict__ attr32,
    float4 *__restrict__ pairs) {
  const int sub = threadIdx.x & 7;
  for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3; c < ncells;
       c += ((int64_t)gridDim.x * blockDim.x) >> 3) {
    const bool is_leaf = cleaf[c] != 0;
    const int nb = cnb[c], b0 = cbeg[c];
    if (sub == 0) {
      const double s = __dsub_rn(cmax[3 * c], cmin[3 * c]);
      geo[c] = make_double4(ccen[3 * c], ccen[3 * c + 1], ccen[3 * c + 2], __dmul_rn(s, s));
      meta[c] = is_leaf ? make_int2(pair_off ? pair_off[c] : b0, nb) : make_int2(cchild[c], -1);
      if (pair_off) {
        const double4 a = attr[c];
        attr32[c] = make_float4((float)a.x, (float)a.y, (float)a.z, (float)a.w);
      }
    }
    if (!pair_off || !is_leaf) continue;
    for (int k = sub; k < (nb + 1) >> 1; k += 8) {
      const int i = b0 + 2 * k;
      const int j = 2 * k + 1 < nb ? i + 1 : b0;
      float4 *o = pairs + 2 * ((int64_t)pair_off[c] + k);
      o[0] = make_float4((float)sx[i], (float)sx[j], (float)sy[i], (float)sy[j]);
      o[1] = make_float4((float)sz[i], (float)sz[j], (float)sm[i], (float)sm[j]);
    }
  }
}

}  // namespace

int bh_upward(tapas_b200_ctx *ctx) {
  if (!ctx->have_tree) {
    set_error(ctx, "bh_upward: no tree (call partition first)");
    return TAPAS_B200_ERR_STATE;
  }
  cudaStream_t s = ctx->stream;
  TB_CUDA(ctx, ctx->bh_attr.ensure(ctx->ncells + 1, s));
  PhaseTimer t(ctx, &ctx->timings.upward);
  for (int lev = (int)ctx->level_off.size() - 2; lev >= 0; lev--) {
    const int64_t a = ctx->level_off[lev], cnt = ctx->level_off[lev + 1] - a;
    if (cnt <= 0) continue;
    bh_upward_level<<<grid_for(cnt, 256), 256, 0, s>>>(
        a, cnt, ctx->cleaf.p, ctx->cnb.p, ctx->cbeg.p, ctx->cchild.p, ctx->sx.p, ctx->sy.p,
        ctx->sz.p, ctx->sq.p, ctx->bh_attr.p);
    TB_LAUNCH_CHECK(ctx);
  }
  ctx->have_bh_attr = true;
  return TAPAS_B200_OK;
}

int bh_interact(tapas_b200_ctx *ctx, double theta, double eps2, int precision) {
  if (!ctx->have_bh_attr) {
    set_error(ctx, "bh_interact: call bh_upward first");
    return TAPAS_B200_ERR_STATE;
  }
  if (!(theta > 0) || !(eps2 >= 0)) {
    set_error(ctx, "bh_interact: need theta > 0 and eps2 >= 0");
    return TAPAS_B200_ERR_ARG;
  }
  cudaStream_t s = ctx->stream;
  const int64_t n = ctx->n, C = ctx->ncells;
  TB_CUDA(ctx, ctx->counters.ensure(8, s));
  TB_CUDA(ctx, cudaMemsetAsync(ctx->counters.p, 0, 8 * sizeof(unsigned long long), s));
  const bool fp64 = precision == TAPAS_B200_FP64;
  TB_CUDA(ctx, ctx->trav_geo.ensure(C + 1, s));
  TB_CUDA(ctx, ctx->trav_meta.ensure(C + 1, s));
  PhaseTimer t(ctx, &ctx->timings.p2p);
  const int32_t *pair_off = nullptr;
  if (!fp64) {
    TB_CUDA(ctx, ctx->flag.ensure(C + 1, s));
    TB_CUDA(ctx, ctx->flag_scan.ensure(C + 1, s));
    TB_CUDA(ctx, ctx->bh_attr32.ensure(C + 1, s));
    TB_CUDA(ctx, ctx->bh_pairs.ensure(n + C + 2, s));  // two per pair, at most (n + leaves) / 2 pairs
    bh_pair_counts<<<grid_for(C, 256), 256, 0, s>>>(C, ctx->cleaf.p, ctx->cnb.p, ctx->flag.p);
    TB_LAUNCH_CHECK(ctx);
    TB_TRY(scan_exclusive(ctx, ctx->flag.p, ctx->flag_scan.p, C, nullptr));
    pair_off = ctx->flag_scan.p;
  }
  bh_pack<<<grid_for(8 * C, 256), 256, 0, s>>>(
      C, ctx->cleaf.p, ctx->cnb.p, ctx->cbeg.p, ctx->cchild.p, ctx->cmin.p, ctx->cmax.p,
      ctx->ccen.p, ctx->bh_attr.p, pair_off, ctx->sx.p, ctx->sy.p, ctx->sz.p, ctx->sq.p,
      ctx->trav_geo.p, ctx->trav_meta.p, ctx->bh_attr32.p, ctx->bh_pairs.p);
  TB_LAUNCH_CHECK(ctx);
  const BhCells T{ctx->trav_geo.p, ctx->trav_meta.p, ctx->cmin.p, ctx->cmax.p, ctx->ccen.p};
  if (fp64) {
    bh_walk64<<<(unsigned)((n + 31) / 32), 32, 0, s>>>(T, n, ctx->sx.p, ctx->sy.p, ctx->sz.p,
                                                       ctx->sq.p, ctx->bh_attr.p, theta, eps2,
                                                       ctx->trg.p, ctx->counters.p);
  } else {
    auto walk = (float)eps2 >= FLT_MIN ? bh_walk32<true> : bh_walk32<false>;
    walk<<<(unsigned)((n + 31) / 32), 32, 0, s>>>(T, n, ctx->sx.p, ctx->sy.p, ctx->sz.p,
                                                  ctx->bh_attr32.p, ctx->bh_pairs.p, theta,
                                                  (float)eps2, ctx->trg.p, ctx->counters.p);
  }
  TB_LAUNCH_CHECK(ctx);
  unsigned long long *h = reinterpret_cast<unsigned long long *>(ctx->pinned.p);
  TB_CUDA(ctx, ctx->pinned.ensure(tapas_b200_ctx::kPinnedBytes));
  h = reinterpret_cast<unsigned long long *>(ctx->pinned.p);
  TB_CUDA(ctx, cudaMemcpyAsync(h, ctx->counters.p, 3 * sizeof(unsigned long long),
                               cudaMemcpyDeviceToHost, s));
  TB_CUDA(ctx, cudaStreamSynchronize(s));
  ctx->bh_napprox = h[0];
  ctx->bh_ndirect = h[1];
  if (h[2]) {
    set_error(ctx, "bh_interact: a walk exceeded its stack bound");
    return TAPAS_B200_ERR_CAPACITY;
  }
  return TAPAS_B200_OK;
}

}  // namespace tb
