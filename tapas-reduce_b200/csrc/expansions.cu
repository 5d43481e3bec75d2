// Expansion kernels: P2M, M2M, M2L, L2L, L2P (ExaFMM Laplace spherical
// harmonics, ex/LaplaceSphericalCPU_tapas.h), templated on the order P.
//
// Work mapping:
//   P2M  - warp per non-empty leaf; lanes own bodies; 8 coefficients at a time
//          are summed over the warp by one reduce-scatter.
//   M2M  - per level, one FP64 GEMM of the level's precomputed translation
//          operator with the stacked multipoles of the children (below).
//   M2L  - P = 2, 3 only (m2l_fp64.cu and m2l_tc.cu have the others): warp per
//          target cell over its CSR list of sources; the harmonics table of
//          each translation is built by P lanes, one Legendre column per lane,
//          into the warp's shared-memory slice.
//   L2L  - per level, one FP64 GEMM as M2M, parents to stacked children.
//   L2P  - warp per non-empty leaf; lane per body, harmonics streamed in
//          registers (no table), L of the leaf staged in shared memory.
// Mixed form only: m2l_pair_kernel (the FP64 M2L of the pairs the tensor cores
// leave, one warp per pair) and l2p32_prep/l2p32_bodies (L2P in FP32, in units
// of the leaf width, one thread per body).
#include "expansions.cuh"
#include "kernels.cuh"
#include "m2l_tc.cuh"

namespace tb {
namespace {

constexpr int kWarps = 4;  // warps per block
constexpr int kThreads = 32 * kWarps;

// ---------------------------------------------------------------------------
// P2M (:138-163): M[n,m] = sum_b q_b * conj(Y_n^m(x_b - center))
// ---------------------------------------------------------------------------
// Coefficient index t = n(n+1)/2 + m of position s in P2M's term order
// (m = 0..P-1, then n = m..P-1).
template <int P>
__device__ __forceinline__ int p2m_term_index(int s) {
  int m = 0;
  while (s >= P - m) {
    s -= P - m;
    m++;
  }
  const int n = m + s;
  return n * (n + 1) / 2 + m;
}

// Sums buf[0..15] of every lane over the warp, leaving lane l (and l ^ 1) with
// the total of buf[(l >> 1) & 15]: four halving exchanges (each lane keeps the
// half its lane bit selects and sends the other), then one pairwise add.
// 16 + 8 + 4 + 2 values are exchanged instead of 16 separate 5-step sums.
__device__ __forceinline__ double warp_reduce_scatter16(double (&buf)[16], int lane) {
#pragma unroll
  for (int o = 16, h = 8; o >= 2; o >>= 1, h >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; i++) {
      const double keep = up ? buf[i + h] : buf[i];
      const double send = up ? buf[i] : buf[i + h];
      buf[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return buf[0] + __shfl_xor_sync(0xffffffffu, buf[0], 1);
}

template <int P>
__global__ void __launch_bounds__(kThreads) p2m_kernel(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ cbeg,
    const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, double2 *__restrict__ M) {
  using S = Sizes<P>;
  constexpr int kGroups = (S::NT + 7) / 8;  // 8 complex terms per reduction
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (w >= nleaves) return;
  const int c = leaves[w];
  const int b0 = cbeg[c], nb = cnb[c];
  const double cx = ccen[3 * c], cy = ccen[3 * c + 1], cz = ccen[3 * c + 2];
  // acc[g]: this lane's share of group g's sums, component (lane >> 1) & 15
  double acc[kGroups];
#pragma unroll
  for (int g = 0; g < kGroups; g++) acc[g] = 0;
  for (int base = 0; base < nb; base += 32) {
    const int b = base + lane;
    const bool valid = b < nb;
    double q = 0, dx = 0, dy = 0, dz = 0;
    if (valid) {
      q = sq[b0 + b];
      dx = sx[b0 + b] - cx;
      dy = sy[b0 + b] - cy;
      dz = sz[b0 + b] - cz;
    }
    // cart2sph (:43-47) then cos/sin of the angles, formed directly
    const Sph sp = sph_of(dx, dy, dz);
    const double rho = sp.r, x = sp.x, y = sp.y;
    const cd ei = sp.ei;
    // Streamed evalMultipole (:63-99): this body's q*conj(Y_n^m) terms, 8 at a
    // time, summed over the warp's bodies by one reduce-scatter.
    double buf[16];
    int s = 0;
    double fact = 1, pn = 1, rhom = 1;
    cd eim{1.0, 0.0};
#pragma unroll
    for (int m = 0; m < P; m++) {
      double p = pn, p1 = pn;
      double rhon = rhom;
#pragma unroll
      for (int n = m; n < P; n++) {
        if (n > m) rhon *= 1.0 / -(n + m);  // constants after unrolling
        const double sc = q * rhon * p;
        buf[2 * (s & 7)] = sc * eim.x;
        buf[2 * (s & 7) + 1] = -sc * eim.y;
        if ((s & 7) == 7 || s == S::NT - 1) {
#pragma unroll
          for (int i = 2 * (s & 7) + 2; i < 16; i++) buf[i] = 0;
          acc[s >> 3] += warp_reduce_scatter16(buf, lane);
        }
        s++;
        if (n == m) {
          p = x * (2 * m + 1) * p1;
          rhon = rhom * rho;
        } else {
          const double p2 = p1;
          p1 = p;
          p = (x * (2 * n + 1) * p1 - (n + m) * p2) * (1.0 / (n - m + 1));
          rhon *= rho;
        }
      }
      rhom = rhom * rho * (1.0 / (double)(-(2 * m + 2) * (2 * m + 1)));
      pn = -pn * fact * y;
      fact += 2;
      eim = cmul(eim, ei);
    }
  }
  double *Mc = reinterpret_cast<double *>(M + (int64_t)c * S::NT);
  const int d = (lane >> 1) & 15;
  if ((lane & 1) == 0) {
#pragma unroll
    for (int g = 0; g < kGroups; g++) {
      const int sp = 8 * g + (d >> 1);
      if (sp < S::NT) Mc[2 * p2m_term_index<P>(sp) + (d & 1)] = acc[g];
    }
  }
}

// warp_reduce_scatter16 for FP32 values (half the shuffles of the FP64 one).
__device__ __forceinline__ float warp_reduce_scatter16f(float (&buf)[16], int lane) {
#pragma unroll
  for (int o = 16, h = 8; o >= 2; o >>= 1, h >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < h; i++) {
      const float keep = up ? buf[i + h] : buf[i];
      const float send = up ? buf[i] : buf[i + h];
      buf[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return buf[0] + __shfl_xor_sync(0xffffffffu, buf[0], 1);
}

// The unit of a leaf's expansions in the mixed form: its width, or 1 where it has none
// (the root of a single body is a point, and the body beside it).
__device__ __forceinline__ double unit_of(double width) { return width > 0 ? width : 1.0; }

// P2M of the mixed form: each body's terms in FP32, in units of the leaf width
// w (rho' = rho / w <= ~0.87, so rho'^n stays in range at every n; M_n = w^n
// times the sum), 8 complex terms at a time summed over the warp by one
// FP32 reduce-scatter, the sums over body chunks and the output in FP64.  A
// term's rounding is ~6e-8 of itself and the warp's tree sum adds ~5 such
// roundings, so M's error stays near 1e-7 of the cell's multipoles of |q|
// (measured below 1e-6 of them per cell); where zero-mean charges cancel, that
// is more than 1e-7 of M itself (up to ~2e-5 of it measured), which the final
// potential does not feel (it sums the same terms the cancellation removed).
template <int P>
__global__ void __launch_bounds__(kThreads, 6) p2m32_kernel(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ cbeg,
    const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, double2 *__restrict__ M) {
  using S = Sizes<P>;
  constexpr int kGroups = (S::NT + 7) / 8;  // 8 complex terms per reduction
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (w >= nleaves) return;
  const int c = leaves[w];
  const int b0 = cbeg[c], nb = cnb[c];
  const double cx = ccen[3 * c], cy = ccen[3 * c + 1], cz = ccen[3 * c + 2];
  const double width = unit_of(cmax[3 * c] - cmin[3 * c]), iw = 1.0 / width;
  double acc[kGroups];  // lane l: component of slot (l >> 1) & 15 of group g
#pragma unroll
  for (int g = 0; g < kGroups; g++) acc[g] = 0;
  for (int base = 0; base < nb; base += 32) {
    const int b = base + lane;
    float q = 0.f, dx = 0.f, dy = 0.f, dz = 0.f;
    if (b < nb) {
      q = (float)sq[b0 + b];
      dx = (float)((sx[b0 + b] - cx) * iw);
      dy = (float)((sy[b0 + b] - cy) * iw);
      dz = (float)((sz[b0 + b] - cz) * iw);
    }
    // cart2sph (:43-47): rho', cos/sin of alpha and e^{i beta} from the offset
    const float rxy2 = dx * dx + dy * dy;
    const float rho = sqrtf(rxy2 + dz * dz);
    float x = 1.f, y = 0.f, eix = 1.f, eiy = 0.f;
    if (rho > 0.f) {
      const float rxy = sqrtf(rxy2);
      x = dz / rho;
      y = rxy / rho;
      if (rxy > 0.f) {
        eix = dx / rxy;
        eiy = dy / rxy;
      }
    }
    float buf[16];
    int s = 0;
    float fact = 1.f, pn = 1.f, rhom = 1.f;
    float emx = 1.f, emy = 0.f;  // e^{i m beta}
#pragma unroll
    for (int m = 0; m < P; m++) {
      float p = pn, p1 = pn;
      float rhon = rhom;
#pragma unroll
      for (int n = m; n < P; n++) {
        if (n > m) rhon *= 1.f / (float)(-(n + m));  // constants after unrolling
        const float sc = q * rhon * p;
        buf[2 * (s & 7)] = sc * emx;
        buf[2 * (s & 7) + 1] = -sc * emy;
        if ((s & 7) == 7 || s == S::NT - 1) {
#pragma unroll
          for (int i = 2 * (s & 7) + 2; i < 16; i++) buf[i] = 0.f;
          acc[s >> 3] += (double)warp_reduce_scatter16f(buf, lane);
        }
        s++;
        if (n == m) {
          p = x * (float)(2 * m + 1) * p1;
          rhon = rhom * rho;
        } else {
          const float p2 = p1;
          p1 = p;
          p = (x * (float)(2 * n + 1) * p1 - (float)(n + m) * p2) * (1.f / (float)(n - m + 1));
          rhon *= rho;
        }
      }
      rhom = rhom * rho * (1.f / (float)(-(2 * m + 2) * (2 * m + 1)));
      pn = -pn * fact * y;
      fact += 2.f;
      const float ex = emx * eix - emy * eiy;
      emy = emx * eiy + emy * eix;
      emx = ex;
    }
  }
  double *Mc = reinterpret_cast<double *>(M + (int64_t)c * S::NT);
  const int d = (lane >> 1) & 15;
  if ((lane & 1) == 0) {
#pragma unroll
    for (int g = 0; g < kGroups; g++) {
      const int sp = 8 * g + (d >> 1);
      if (sp < S::NT) {
        const int t = p2m_term_index<P>(sp);
        int n, m;
        jk_of(t, n, m);
        double wn = 1.0;
        for (int k = 0; k < n; k++) wn *= width;
        Mc[2 * t + (d & 1)] = acc[g] * wn;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// M2L (:208-273, mutual = 0): L[t] = sum over sources s of T(c_t - c_s) M[s]
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(kThreads) m2l_kernel(
    int64_t ncells, const int32_t *__restrict__ off, const uint64_t *__restrict__ list,
    uint64_t src_mask, const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double2 *__restrict__ M, double2 *__restrict__ L, const uint8_t *__restrict__ own) {
  using S = Sizes<P>;
  __shared__ cd Ysm[kWarps][S::NY];
  __shared__ cd Msm[kWarps][S::NT];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * kWarps + wi;
  if (c >= ncells) return;
  const int e0 = off[c], e1 = off[c + 1];
  if (e1 == e0 || cnb[c] == 0) return;
  if (own && !(own[c] & 1)) return;  // sharded: another context's target
  cd *Y = Ysm[wi];
  cd *Mj = Msm[wi];
  cd acc[S::R];
  int jj[S::R], kk[S::R];
#pragma unroll
  for (int r = 0; r < S::R; r++) {
    acc[r] = cd{0, 0};
    jk_of(lane + 32 * r, jj[r], kk[r]);
  }
  const double tx = ccen[3 * c], ty = ccen[3 * c + 1], tz = ccen[3 * c + 2];
  for (int e = e0; e < e1; e++) {
    const int s = (int)(list[e] & src_mask);
    if (cnb[s] == 0) continue;  // M of an empty cell is exactly zero
    const Sph sp = sph_of(tx - ccen[3 * s], ty - ccen[3 * s + 1], tz - ccen[3 * s + 2]);
    __syncwarp();
    if (lane < P) local_column<P>(lane, sp.r, sp.x, sp.y, sp.ei, Y);
    for (int t = lane; t < S::NT; t += 32) {
      double2 v = M[(int64_t)s * S::NT + t];
      Mj[t] = cd{v.x, v.y};
    }
    __syncwarp();
    m2l_accumulate<P>(acc, jj, kk, lane, Mj, Y);
  }
#pragma unroll
  for (int r = 0; r < S::R; r++) {
    const int t = lane + 32 * r;
    if (t < S::NT) L[c * S::NT + t] = make_double2(acc[r].x, acc[r].y);
  }
}

// The mixed form's FP64 remainder: one warp per listed pair (list index),
// added into L[target] with atomics, so a target with many such pairs does
// not hold one warp alone.
template <int P>
__global__ void __launch_bounds__(kThreads) m2l_pair_kernel(
    const uint32_t *__restrict__ pairs, int64_t npairs, const uint64_t *__restrict__ list,
    int shift, const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double2 *__restrict__ M, double2 *__restrict__ L) {
  using S = Sizes<P>;
  __shared__ cd Ysm[kWarps][S::NY];
  __shared__ cd Msm[kWarps][S::NT];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  cd *Y = Ysm[wi];
  cd *Mj = Msm[wi];
  int jj[S::R], kk[S::R];
#pragma unroll
  for (int r = 0; r < S::R; r++) jk_of(lane + 32 * r, jj[r], kk[r]);
  const uint64_t src_mask = (1ull << shift) - 1;
  const int64_t nw = (int64_t)gridDim.x * kWarps;
  for (int64_t p = (int64_t)blockIdx.x * kWarps + wi; p < npairs; p += nw) {
    const uint64_t x = list[pairs[p]];
    const int c = (int)(x >> shift), s = (int)(x & src_mask);
    if (cnb[s] == 0 || cnb[c] == 0) continue;
    const Sph sp = sph_of(ccen[3 * c] - ccen[3 * s], ccen[3 * c + 1] - ccen[3 * s + 1],
                          ccen[3 * c + 2] - ccen[3 * s + 2]);
    __syncwarp();
    if (lane < P) local_column<P>(lane, sp.r, sp.x, sp.y, sp.ei, Y);
    for (int t = lane; t < S::NT; t += 32) {
      double2 v = M[(int64_t)s * S::NT + t];
      Mj[t] = cd{v.x, v.y};
    }
    __syncwarp();
    cd acc[S::R];
#pragma unroll
    for (int r = 0; r < S::R; r++) acc[r] = cd{0, 0};
    m2l_accumulate<P>(acc, jj, kk, lane, Mj, Y);
    double *Lc = reinterpret_cast<double *>(L + (int64_t)c * S::NT);
#pragma unroll
    for (int r = 0; r < S::R; r++) {
      const int t = lane + 32 * r;
      if (t < S::NT) {
        atomicAdd(Lc + 2 * t, acc[r].x);
        atomicAdd(Lc + 2 * t + 1, acc[r].y);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// L2P (:275-307): per body, trg /= q, then add the local expansion's
// potential and gradient (spherical components -> Cartesian, sph2cart :50-60).
// ---------------------------------------------------------------------------
template <int P>
__global__ void __launch_bounds__(kThreads) l2p_kernel(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ cbeg,
    const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double *__restrict__ sx, const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, const double2 *__restrict__ L, double *__restrict__ trg,
    int near_has_q) {
  using S = Sizes<P>;
  __shared__ cd Lsm[kWarps][S::NT];
  const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5;
  const int64_t w = (int64_t)blockIdx.x * kWarps + wi;
  if (w >= nleaves) return;
  const int c = leaves[w];
  const int b0 = cbeg[c], nb = cnb[c];
  cd *Lc = Lsm[wi];
  for (int t = lane; t < S::NT; t += 32) {
    double2 v = L[(int64_t)c * S::NT + t];
    Lc[t] = cd{v.x, v.y};
  }
  __syncwarp();
  const double cx = ccen[3 * c], cy = ccen[3 * c + 1], cz = ccen[3 * c + 2];
  for (int b = lane; b < nb; b += 32) {
    const int64_t bi = b0 + b;
    double r, theta, phi;
    cart2sph(sx[bi] - cx, sy[bi] - cy, sz[bi] - cz, r, theta, phi);
    const double x = cos(theta), y = sin(theta);
    const double inv_y = 1.0 / y, inv_r = 1.0 / r;
    double sp, cp;
    sincos(phi, &sp, &cp);
    const cd ei{cp, sp};
    double pot = 0, s0 = 0, s1 = 0, s2 = 0;
    double fact = 1, pn = 1, rhom = 1;
    cd eim{1.0, 0.0};
    // For each m the sums over n are taken before the common factor e^{im phi}:
    //   sa = sum ys L, sb = sum n ys L, sc = sum (yts / inv_y) L,
    // where Y_n^m = ys e^{im phi} and dY_n^m/dtheta = yts e^{im phi}.
#pragma unroll
    for (int m = 0; m < P; m++) {
      double p = pn, p1 = pn;
      double rhon = rhom;
      cd sa{0, 0}, sb{0, 0}, sc{0, 0};
#pragma unroll
      for (int n = m; n < P; n++) {
        double ys, yt;
        const double t1 = x * p1;
        if (n == m) {
          const double pnew = (2 * m + 1) * t1;
          ys = rhom * p;
          yt = rhom * (pnew - (m + 1) * t1);
          p = pnew;
          rhon = rhom * r;
        } else {
          rhon *= 1.0 / -(n + m);  // constants after unrolling
          ys = rhon * p;
          const double p2 = p1;
          p1 = p;
          const double tn = x * p1;
          p = ((2 * n + 1) * tn - (n + m) * p2) * (1.0 / (n - m + 1));
          yt = rhon * ((n - m + 1) * p - (n + 1) * tn);
          rhon *= r;
        }
        const cd Lv = Lc[n * (n + 1) / 2 + m];
        sa.x = fma(ys, Lv.x, sa.x);
        sa.y = fma(ys, Lv.y, sa.y);
        const double nys = n * ys;
        sb.x = fma(nys, Lv.x, sb.x);
        sb.y = fma(nys, Lv.y, sb.y);
        sc.x = fma(yt, Lv.x, sc.x);
        sc.y = fma(yt, Lv.y, sc.y);
      }
      const double f = (m == 0) ? 1.0 : 2.0;
      const cd za = cmul(sa, eim);
      pot += f * za.x;
      s0 += f * inv_r * (sb.x * eim.x - sb.y * eim.y);
      s1 += f * inv_y * (sc.x * eim.x - sc.y * eim.y);
      if (m > 0) s2 += 2 * (-za.y) * m;  // real(L*Y*i) = -imag(L*Y)
      rhom = rhom * r * (1.0 / (double)(-(2 * m + 2) * (2 * m + 1)));
      pn = -pn * fact * y;
      fact += 2;
      eim = cmul(eim, ei);
    }
    double *o = trg + 4 * bi;
    // The FP64 near field holds q_i * sum(q_j / r) (the reference's TRG before
    // its `ba /= b.SRC`); the mixed near field is already per unit charge.
    const double iq = near_has_q ? 1.0 / sq[bi] : 1.0;
    const double st = y, ct = x;
    const double c0 = st * cp * s0 + ct * cp * inv_r * s1 - sp * inv_r * inv_y * s2;
    const double c1 = st * sp * s0 + ct * sp * inv_r * s1 + cp * inv_r * inv_y * s2;
    const double c2 = ct * s0 - st * inv_r * s1;
    o[0] = o[0] * iq + pot;
    o[1] = o[1] * iq + c0;
    o[2] = o[2] * iq + c1;
    o[3] = o[3] * iq + c2;
  }
}

// L2P of the mixed form in FP32: the local expansion's terms fall off
// geometrically inside the leaf, so one FP32 evaluation of them is accurate
// to ~1e-7 of the far-field potential; the result is added into the FP64
// totals.  The evaluation runs in units of the leaf width w (L'_n = L_n w^n,
// r' = r / w: every term L Y_n^m(r) is unchanged, the gradient is scaled by
// 1/w at the end), which keeps every FP32 quantity bounded; L_n itself grows
// like 1/R^(n+1) and leaves the FP32 range at high n in small cells.
//
// One thread per body: a warp per leaf would leave 23% of its lanes idle on a
// surface tree (leaves of ~57 bodies take 2.3 passes of 32), so the leaves are
// prepared first (l2p32_prep: the width-scaled FP32 local expansion and the
// geometry, indexed by the leaf's ordinal, and each of its bodies' ordinal),
// then l2p32_bodies evaluates every body, reading its leaf's coefficients
// through L1 (the lanes of a warp share one to three leaves).
template <int P>
__global__ void __launch_bounds__(256) l2p32_prep(
    const int32_t *__restrict__ leaves, int64_t nleaves, const int32_t *__restrict__ cbeg,
    const int32_t *__restrict__ cnb, const double *__restrict__ ccen,
    const double *__restrict__ cmin, const double *__restrict__ cmax,
    const double2 *__restrict__ L, float2 *__restrict__ Lf, double4 *__restrict__ geo,
    int32_t *__restrict__ body_leaf) {
  using S = Sizes<P>;
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  if (w >= nleaves) return;
  const int c = leaves[w];
  const double width = unit_of(cmax[3 * c] - cmin[3 * c]);
  for (int t = lane; t < S::NT; t += 32) {
    int n, m;
    jk_of(t, n, m);
    double wn = 1.0;
    for (int k = 0; k < n; k++) wn *= width;
    const double2 v = L[(int64_t)c * S::NT + t];
    Lf[w * S::NT + t] = make_float2((float)(v.x * wn), (float)(v.y * wn));
  }
  if (lane == 0) geo[w] = make_double4(ccen[3 * c], ccen[3 * c + 1], ccen[3 * c + 2], width);
  const int b0 = cbeg[c], nb = cnb[c];
  for (int b = lane; b < nb; b += 32) body_leaf[b0 + b] = (int32_t)w;
}

template <int P>
__global__ void __launch_bounds__(kThreads) l2p32_bodies(
    int64_t n, const int32_t *__restrict__ body_leaf, const double4 *__restrict__ geo,
    const float2 *__restrict__ Lf, const double *__restrict__ sx,
    const double *__restrict__ sy, const double *__restrict__ sz,
    const double *__restrict__ sq, double *__restrict__ trg, int near_has_q) {
  using S = Sizes<P>;
  for (int64_t bi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; bi < n;
       bi += (int64_t)gridDim.x * blockDim.x) {
    const int w = body_leaf[bi];
    if (w < 0) continue;  // a body another context evaluates
    const double4 g = geo[w];
    const double iw = 1.0 / g.w;
    const float2 *__restrict__ Lc = Lf + (int64_t)w * S::NT;
    const float dx = (float)((sx[bi] - g.x) * iw), dy = (float)((sy[bi] - g.y) * iw),
                dz = (float)((sz[bi] - g.z) * iw);
    const float rxy2 = dx * dx + dy * dy;
    const float r = sqrtf(rxy2 + dz * dz);
    float x = 1.f, y = 0.f, cp = 1.f, sp = 0.f;
    if (r > 0.f) {
      const float rxy = sqrtf(rxy2);
      x = dz / r;
      y = rxy / r;
      if (rxy > 0.f) {
        cp = dx / rxy;
        sp = dy / rxy;
      } else if (dz < 0.f) {
        y = 1.2246468e-16f;  // sin(acos(-1)) in FP64, as the FP64 form gets it
      }
    }
    const float inv_y = 1.f / y, inv_r = 1.f / r;
    float pot = 0, s0 = 0, s1 = 0, s2 = 0;
    float fact = 1, pn = 1, rhom = 1;
    float2 eim = make_float2(1.f, 0.f);
#pragma unroll
    for (int m = 0; m < P; m++) {
      // keeps the compiler from hoisting every column's loads of the
      // coefficients ahead of the loop (register pressure)
      asm volatile("" ::: "memory");
      float p = pn, p1 = pn;
      float rhon = rhom;
      float2 sa = make_float2(0.f, 0.f), sb = sa, sc = sa;
#pragma unroll
      for (int nn = m; nn < P; nn++) {
        float ys, yt;
        const float t1 = x * p1;
        if (nn == m) {
          const float pnew = (float)(2 * m + 1) * t1;
          ys = rhom * p;
          yt = rhom * (pnew - (float)(m + 1) * t1);
          p = pnew;
          rhon = rhom * r;
        } else {
          rhon *= 1.f / (float)(-(nn + m));
          ys = rhon * p;
          const float p2 = p1;
          p1 = p;
          const float tn = x * p1;
          p = ((float)(2 * nn + 1) * tn - (float)(nn + m) * p2) * (1.f / (float)(nn - m + 1));
          yt = rhon * ((float)(nn - m + 1) * p - (float)(nn + 1) * tn);
          rhon *= r;
        }
        const float2 Lv = __ldg(Lc + nn * (nn + 1) / 2 + m);
        sa.x = fmaf(ys, Lv.x, sa.x);
        sa.y = fmaf(ys, Lv.y, sa.y);
        const float nys = (float)nn * ys;
        sb.x = fmaf(nys, Lv.x, sb.x);
        sb.y = fmaf(nys, Lv.y, sb.y);
        sc.x = fmaf(yt, Lv.x, sc.x);
        sc.y = fmaf(yt, Lv.y, sc.y);
      }
      const float f = (m == 0) ? 1.f : 2.f;
      const float zax = sa.x * eim.x - sa.y * eim.y, zay = sa.x * eim.y + sa.y * eim.x;
      pot += f * zax;
      s0 += f * inv_r * (sb.x * eim.x - sb.y * eim.y);
      s1 += f * inv_y * (sc.x * eim.x - sc.y * eim.y);
      if (m > 0) s2 += 2.f * (-zay) * (float)m;
      rhom = rhom * r * (1.f / (float)(-(2 * m + 2) * (2 * m + 1)));
      pn = -pn * fact * y;
      fact += 2.f;
      eim = make_float2(eim.x * cp - eim.y * sp, eim.x * sp + eim.y * cp);
    }
    const float st = y, ct = x;
    const float c0 = st * cp * s0 + ct * cp * inv_r * s1 - sp * inv_r * inv_y * s2;
    const float c1 = st * sp * s0 + ct * sp * inv_r * s1 + cp * inv_r * inv_y * s2;
    const float c2 = ct * s0 - st * inv_r * s1;
    double *o = trg + 4 * bi;
    const double iq = near_has_q ? 1.0 / sq[bi] : 1.0;
    o[0] = o[0] * iq + (double)pot;
    o[1] = o[1] * iq + (double)c0 * iw;
    o[2] = o[2] * iq + (double)c1 * iw;
    o[3] = o[3] * iq + (double)c2 * iw;
  }
}

// ---------------------------------------------------------------------------
// Level-batched M2M and L2L.
//
// Every cell of a level has the same width (the root cube halved per level),
// so a child's offset from its parent is one of eight per level and the
// translation of M2M (:165-206) or L2L (:309-345) is one fixed real-linear
// map per (level, octant), acting on (Re, Im) pairs.  The eight children of
// the non-leaf cells of a level are stored consecutively in parent order, so
//   M2M:  M[parent_i]          = Tup_l (2NT x 16NT) . M[children_i] (16NT)
//   L2L:  L[children_i] (16NT) += Tdn_l (16NT x 2NT) . L[parent_i]
// are one FP64 GEMM per level over the level's non-leaf cells i.  The
// operators are built from one representative parent of the level with the
// reference's formulas, one thread per (target, source) pair; M2M rows of
// degree j read only source degrees <= j and L2L rows of degree j only source
// degrees >= j, and the operators are stored without the zero ranges this leaves.
// ---------------------------------------------------------------------------
constexpr int kMaxLevels = kMaxDepth + 1;
struct LevelFirstChild {
  int64_t c0[kMaxLevels];  // first cell of level l + 1 (child 0 of the level's first parent)
};

constexpr int kOutBlock = 32;  // outputs of one block of an operator
constexpr int kStep = 16;      // sources of one block of an operator

// A level operator: per octant the blocks of 32 outputs in order, each with its
// source blocks of 16 from first(b) on, stored in the multiplication's order
// (dmma_m16n8k16): for each 8 outputs f and half h of a lane's four sources, the
// two doubles of each lane.
template <int P, bool kUp>
struct LevelOp {
  static constexpr int NT = P * (P + 1) / 2;
  static constexpr int K = 2 * NT;
  static constexpr int NB = (K + kOutBlock - 1) / kOutBlock;
  __host__ __device__ static constexpr int degree(int t) {
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= t) j++;
    return j;
  }
  __host__ __device__ static constexpr int first(int b) {
    if (kUp) return 0;
    const int j = degree(b * (kOutBlock / 2));
    return j * (j + 1) / kStep;
  }
  __host__ __device__ static constexpr int steps(int b) {
    if (!kUp) return (K + kStep - 1) / kStep - first(b);
    const int last = (b + 1) * (kOutBlock / 2) - 1;
    const int j = degree(last < NT ? last : NT - 1);
    return ((j + 1) * (j + 2) + kStep - 1) / kStep;
  }
  __host__ __device__ static constexpr int blocks(int b) {  // blocks before output block b
    int s = 0;
    for (int i = 0; i < b; i++) s += steps(i);
    return s;
  }
  static constexpr int NBLK = blocks(NB);                          // per octant
  static constexpr size_t OCTANT = (size_t)NBLK * kOutBlock * kStep;  // doubles
};

// One block of the grid (levels with children, 8 octants, parts): its share of
// one (level, octant) operator.  Entry (target (j,k), source (j',k')) collects
// the terms of the reference's loops that read that source: M2M (:165-206) with
// n = j - j' and m = k - k' (source as is) or m = k + k' (conjugated); L2L
// (:309-345) with n = j' and m = k' (as is) or m = -k' (conjugated).  The real
// 2 x 2 block of out = a * src + b * conj(src):
//   [Re out]   [a.x + b.x   b.y - a.y] [Re src]
//   [Im out] = [a.y + b.y   a.x - b.x] [Im src]
template <int P, bool kUp>
__global__ void __launch_bounds__(256) build_level_op(LevelFirstChild lf,
                                                      const int32_t *__restrict__ cparent,
                                                      const double *__restrict__ ccen,
                                                      double *__restrict__ ops) {
  using S = Sizes<P>;
  using O = LevelOp<P, kUp>;
  __shared__ cd Y[S::NY];
  __shared__ short blk_out[O::NBLK], blk_step[O::NBLK];
  const int l = blockIdx.x, o = blockIdx.y;
  const int64_t cj = lf.c0[l] + o;
  const int p = cparent[cj];
  const double dx = ccen[3 * p] - ccen[3 * cj], dy = ccen[3 * p + 1] - ccen[3 * cj + 1],
               dz = ccen[3 * p + 2] - ccen[3 * cj + 2];
  // M2M translates by parent - child, L2L by child - parent
  const Sph sp = kUp ? sph_of(dx, dy, dz) : sph_of(-dx, -dy, -dz);
  if (threadIdx.x < P) multipole_column<P>(threadIdx.x, sp.r, sp.x, sp.y, sp.ei, Y);
  if (threadIdx.x >= 32 && threadIdx.x < 32 + O::NB) {
    const int b = threadIdx.x - 32;
    const int at = O::blocks(b);
    for (int i = 0; i < O::steps(b); i++) {
      blk_out[at + i] = (short)b;
      blk_step[at + i] = (short)(O::first(b) + i);
    }
  }
  __syncthreads();
  double2 *op = reinterpret_cast<double2 *>(ops + ((size_t)l * 8 + o) * O::OCTANT);
  constexpr int kPairs = (kOutBlock / 2) * (kStep / 2);
  for (int idx = blockIdx.z * blockDim.x + threadIdx.x; idx < O::NBLK * kPairs;
       idx += gridDim.z * blockDim.x) {
    const int blk = idx / kPairs, in = idx - blk * kPairs;
    const int lo = in >> 3, li = in & 7;  // complex target, source within the block
    const int t = blk_out[blk] * (kOutBlock / 2) + lo, u = blk_step[blk] * (kStep / 2) + li;
    cd a{0, 0}, b{0, 0};
    if (t < S::NT && u < S::NT) {
      int j, k, jp, kp;
      jk_of(t, j, k);
      jk_of(u, jp, kp);
      if (kUp) {
        const int n = j - jp;
        if (n >= 0) {
          if (kp >= 1) {
            const int m = k - kp;
            if (m >= -n && m <= n) {
              const double sgn = ((m >= 0) ? 1.0 : oddeven(m)) * oddeven(n);
              a = scal(sgn, Y[n * n + n - m]);
            }
          }
          const int m = k + kp;
          if (m <= n) b = scal(oddeven(k + n + m), Y[n * n + n - m]);
        }
      } else {
        const int n = jp;
        if (n >= j) {
          const int base = (n - j) * (n - j) + n - j - k;
          if (kp >= 1 && kp <= n - j - k) b = scal(oddeven(k), Y[base - kp]);
          if (n - j >= abs(kp - k)) a = scal(oddeven((kp - k) * (kp < k)), Y[base + kp]);
        }
      }
    }
    const int f = lo >> 2, g = (2 * lo) & 7;
    double2 *dst = op + (((size_t)blk * 4 + f) * 2 + (li & 1)) * 32 + 4 * g + (li >> 1);
    dst[0] = make_double2(a.x + b.x, b.y - a.y);
    dst[4] = make_double2(a.y + b.y, a.x - b.x);
  }
}

// One level's translation GEMM on the FP64 tensor cores.  A block takes 32 of
// the level's non-leaf cells (c0 + 8i .. c0 + 8i + 7 are cell i's children) and
// one block of 32 outputs, a warp per octant: 32 x 32 x 16 steps with both
// operands read from L2 / L1 straight into MMA fragments (four lanes read 128
// contiguous bytes of a cell's row; the operator is stored in fragment order).
// L2L: each warp adds into its octant's child.  M2M: the eight octants'
// products are added in octant order through shared memory.  Every output is a
// fixed-order sum, so the result does not depend on the grid.  Bound: the FP64
// pipe; small levels by the chain of a few steps and the launch.
template <int P, bool kUp>
__global__ void __launch_bounds__(kUp ? 256 : 64, kUp ? 1 : 6) level_gemm(const double *__restrict__ ops, int64_t c0,
                                                     int64_t ncols,
                                                     const int32_t *__restrict__ cparent,
                                                     double *__restrict__ X) {
  using O = LevelOp<P, kUp>;
  extern __shared__ __align__(16) double red[];  // M2M: [octant][cell][output]
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int o = blockIdx.z * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t i0 = (int64_t)blockIdx.x * 32;
  const int b = blockIdx.y;
  const double2 *src[4];
#pragma unroll
  for (int m = 0; m < 4; m++) {  // the last cell again beyond the level's end
    const int64_t child0 = c0 + 8 * min(i0 + g + 8 * m, ncols - 1);
    const int64_t cell = kUp ? child0 + o : (int64_t)cparent[child0];
    src[m] = reinterpret_cast<const double2 *>(X + cell * O::K) + 2 * t;
  }
  int at = 0;
  for (int i = 0; i < b; i++) at += O::steps(i);
  const double2 *op =
      reinterpret_cast<const double2 *>(ops + (size_t)o * O::OCTANT) + (size_t)at * 256 + lane;
  double acc[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int f = 0; f < 4; f++)
#pragma unroll
      for (int x = 0; x < 4; x++) acc[m][f][x] = 0;
  const int s1 = O::first(b) + O::steps(b);
  for (int s = O::first(b); s < s1; s++) {
    double a[2][8];
    // rows hold K = P(P+1) doubles: the last step's pairs beyond them are zero
    const bool in0 = s * kStep + 4 * t < O::K, in1 = s * kStep + 4 * t + 2 < O::K;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const double2 zero = make_double2(0.0, 0.0);
      const double2 u = in0 ? src[m][8 * s] : zero, v = in1 ? src[m][8 * s + 1] : zero;
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
  if (kUp) {
#pragma unroll
    for (int f = 0; f < 4; f++)
#pragma unroll
      for (int m = 0; m < 4; m++)
        *reinterpret_cast<double2 *>(red + ((o * 32 + g + 8 * m) * 32 + 8 * f + 2 * t)) =
            make_double2(acc[m >> 1][f][2 * (m & 1)], acc[m >> 1][f][2 * (m & 1) + 1]);
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * 16; e += 256) {
      const int row = e >> 4, col = 2 * (e & 15);
      if (i0 + row >= ncols || b * kOutBlock + col >= O::K) continue;
      double2 v = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        const double2 w = *reinterpret_cast<const double2 *>(red + (q * 32 + row) * 32 + col);
        v.x += w.x;
        v.y += w.y;
      }
      *reinterpret_cast<double2 *>(X + (int64_t)cparent[c0 + 8 * (i0 + row)] * O::K +
                                   b * kOutBlock + col) = v;
    }
  } else {
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const int64_t i = i0 + g + 8 * m;
      if (i >= ncols) continue;
      double *dst = X + (c0 + 8 * i + o) * O::K + b * kOutBlock + 2 * t;
#pragma unroll
      for (int f = 0; f < 4; f++) {
        if (b * kOutBlock + 8 * f + 2 * t >= O::K) continue;
        double2 *d = reinterpret_cast<double2 *>(dst + 8 * f);
        const double2 w = *d;
        *d = make_double2(w.x + acc[m >> 1][f][2 * (m & 1)],
                          w.y + acc[m >> 1][f][2 * (m & 1) + 1]);
      }
    }
  }
}

// Builds this tree's per-level operators for order P (levels 0 .. nlev-1 have
// children).
template <int P>
int build_level_ops(tapas_b200_ctx *ctx, int &nlev, LevelFirstChild &lf) {
  cudaStream_t s = ctx->stream;
  nlev = 0;
  for (int l = 0; l + 2 < (int)ctx->level_off.size() && l < kMaxLevels; l++) {
    if (ctx->level_off[l + 2] <= ctx->level_off[l + 1]) break;
    lf.c0[l] = ctx->level_off[l + 1];
    nlev = l + 1;
  }
  if (nlev == 0) return TAPAS_B200_OK;
  using Up = LevelOp<P, true>;
  using Dn = LevelOp<P, false>;
  TB_CUDA(ctx, ctx->op_m2m.ensure(8 * Up::OCTANT * nlev, s));
  TB_CUDA(ctx, ctx->op_l2l.ensure(8 * Dn::OCTANT * nlev, s));
  // enough blocks to fill the GPU, each building its harmonics table again
  const dim3 grid(nlev, 8, std::max(1, 2 * ctx->num_sms / (8 * nlev)));
  build_level_op<P, true><<<grid, 256, 0, s>>>(lf, ctx->cparent.p, ctx->ccen.p, ctx->op_m2m.p);
  TB_LAUNCH_CHECK(ctx);
  build_level_op<P, false><<<grid, 256, 0, s>>>(lf, ctx->cparent.p, ctx->ccen.p, ctx->op_l2l.p);
  TB_LAUNCH_CHECK(ctx);
  return TAPAS_B200_OK;
}

template <int P, bool kUp>
int level_translate(tapas_b200_ctx *ctx, int l, const LevelFirstChild &lf) {
  using O = LevelOp<P, kUp>;
  const int64_t ncols = (ctx->level_off[l + 2] - ctx->level_off[l + 1]) / 8;
  if (ncols <= 0) return TAPAS_B200_OK;
  const dim3 grid((unsigned)((ncols + 31) / 32), O::NB, kUp ? 1 : 4);
  const int smem = kUp ? 8 * 32 * 32 * (int)sizeof(double) : 0;
  if (kUp)
    TB_CUDA(ctx, cudaFuncSetAttribute(level_gemm<P, kUp>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  level_gemm<P, kUp><<<grid, kUp ? 256 : 64, smem, ctx->stream>>>(
      (kUp ? ctx->op_m2m.p : ctx->op_l2l.p) + 8 * O::OCTANT * l, lf.c0[l], ncols, ctx->cparent.p,
      reinterpret_cast<double *>(kUp ? ctx->M.p : ctx->L.p));
  TB_LAUNCH_CHECK(ctx);
  return TAPAS_B200_OK;
}

template <int P>
int p2m_P(tapas_b200_ctx *ctx, bool p2m_f32) {
  using S = Sizes<P>;
  cudaStream_t s = ctx->stream;
  const int64_t C = ctx->ncells;
  TB_CUDA(ctx, ctx->M.ensure((size_t)C * S::NT, s));
  TB_CUDA(ctx, cudaMemsetAsync(ctx->M.p, 0, sizeof(double2) * (size_t)C * S::NT, s));
  PhaseTimer t(ctx, &ctx->timings.p2m);
  int64_t nl = 0;
  const int32_t *leaves = work_leaves(ctx, nl);  // sharded: owned leaves only
  if (nl > 0 && p2m_f32) {
    p2m32_kernel<P><<<(unsigned)((nl + kWarps - 1) / kWarps), kThreads, 0, s>>>(
        leaves, nl, ctx->cbeg.p, ctx->cnb.p, ctx->ccen.p, ctx->cmin.p, ctx->cmax.p, ctx->sx.p,
        ctx->sy.p, ctx->sz.p, ctx->sq.p, ctx->M.p);
    TB_LAUNCH_CHECK(ctx);
  } else if (nl > 0) {
    p2m_kernel<P><<<(unsigned)((nl + kWarps - 1) / kWarps), kThreads, 0, s>>>(
        leaves, nl, ctx->cbeg.p, ctx->cnb.p, ctx->ccen.p, ctx->sx.p, ctx->sy.p, ctx->sz.p,
        ctx->sq.p, ctx->M.p);
    TB_LAUNCH_CHECK(ctx);
  }
  return TAPAS_B200_OK;
}

template <int P>
int m2m_P(tapas_b200_ctx *ctx) {
  PhaseTimer t(ctx, &ctx->timings.m2m);
  int nlev = 0;
  LevelFirstChild lf;
  TB_TRY(build_level_ops<P>(ctx, nlev, lf));
  ctx->level_ops_P = P;
  for (int lev = nlev - 1; lev >= 0; lev--) TB_TRY((level_translate<P, true>(ctx, lev, lf)));
  return TAPAS_B200_OK;
}

// FP64 M2M level GEMMs of the parent levels max_levels - 1 .. 0 only.
template <int P>
int fp64_m2m_levels_P(tapas_b200_ctx *ctx, int max_levels) {
  int nlev = 0;
  LevelFirstChild lf;
  TB_TRY(build_level_ops<P>(ctx, nlev, lf));  // the upward pass builds them for this tree
  ctx->level_ops_P = P;
  for (int lev = std::min(nlev, max_levels) - 1; lev >= 0; lev--)
    TB_TRY((level_translate<P, true>(ctx, lev, lf)));
  return TAPAS_B200_OK;
}

template <int P>
int upward_P(tapas_b200_ctx *ctx, bool p2m_f32) {
  TB_TRY(p2m_P<P>(ctx, p2m_f32));
  return m2m_P<P>(ctx);
}

template <int P>
int m2l_P(tapas_b200_ctx *ctx) {
  using S = Sizes<P>;
  cudaStream_t s = ctx->stream;
  const int64_t C = ctx->ncells;
  TB_CUDA(ctx, ctx->L.ensure((size_t)C * S::NT, s));
  TB_CUDA(ctx, cudaMemsetAsync(ctx->L.p, 0, sizeof(double2) * (size_t)C * S::NT, s));
  PhaseTimer t(ctx, &ctx->timings.m2l_fp64);
  const uint64_t mask = (1ull << ctx->list_shift) - 1;
  m2l_kernel<P><<<(unsigned)((C + kWarps - 1) / kWarps), kThreads, 0, s>>>(
      C, ctx->m2l_off.p, ctx->m2l.p, mask, ctx->cnb.p, ctx->ccen.p, ctx->M.p, ctx->L.p,
      owned_cells(ctx));
  TB_LAUNCH_CHECK(ctx);
  return TAPAS_B200_OK;
}

template <int P>
int m2l_pairs_P(tapas_b200_ctx *ctx) {
  cudaStream_t s = ctx->stream;
  PhaseTimer t(ctx, &ctx->timings.m2l_fp64);
  const int64_t np = ctx->m2l_npairs;
  if (np > 0) {
    m2l_pair_kernel<P><<<grid_for(np, kWarps, ctx->num_sms * 16), kThreads, 0, s>>>(
        ctx->m2l_pairs, np, ctx->m2l.p, ctx->list_shift, ctx->cnb.p, ctx->ccen.p, ctx->M.p,
        ctx->L.p);
    TB_LAUNCH_CHECK(ctx);
  }
  return TAPAS_B200_OK;
}

template <int P>
int downward_P(tapas_b200_ctx *ctx, bool l2p_f32) {
  cudaStream_t s = ctx->stream;
  {
    PhaseTimer t(ctx, &ctx->timings.l2l);
    int nlev = 0;
    LevelFirstChild lf;
    if (ctx->level_ops_P != P) {  // the operators of the upward pass are reused
      TB_TRY(build_level_ops<P>(ctx, nlev, lf));
      ctx->level_ops_P = P;
    } else {
      for (int l = 0; l + 2 < (int)ctx->level_off.size() && l < kMaxLevels; l++) {
        if (ctx->level_off[l + 2] <= ctx->level_off[l + 1]) break;
        lf.c0[l] = ctx->level_off[l + 1];
        nlev = l + 1;
      }
    }
    for (int lev = 0; lev < nlev; lev++) TB_TRY((level_translate<P, false>(ctx, lev, lf)));
  }
  PhaseTimer t(ctx, &ctx->timings.l2p);
  int64_t nl = 0;
  const int32_t *leaves = work_leaves(ctx, nl);  // sharded: owned leaves only
  if (nl > 0 && l2p_f32) {
    TB_CUDA(ctx, ctx->l2p_lf.ensure((size_t)nl * Sizes<P>::NT, s));
    TB_CUDA(ctx, ctx->l2p_geo.ensure((size_t)nl, s));
    TB_CUDA(ctx, ctx->l2p_body_leaf.ensure((size_t)ctx->n, s));
    if (ctx->sharded)  // bodies of other contexts' leaves: -1
      TB_CUDA(ctx, cudaMemsetAsync(ctx->l2p_body_leaf.p, 0xff, sizeof(int32_t) * ctx->n, s));
    l2p32_prep<P><<<(unsigned)((nl + kWarps - 1) / kWarps), kThreads, 0, s>>>(
        leaves, nl, ctx->cbeg.p, ctx->cnb.p, ctx->ccen.p, ctx->cmin.p, ctx->cmax.p, ctx->L.p,
        ctx->l2p_lf.p, ctx->l2p_geo.p, ctx->l2p_body_leaf.p);
    TB_LAUNCH_CHECK(ctx);
    l2p32_bodies<P><<<grid_for(ctx->n, kThreads, ctx->num_sms * 8), kThreads, 0, s>>>(
        ctx->n, ctx->l2p_body_leaf.p, ctx->l2p_geo.p, ctx->l2p_lf.p, ctx->sx.p, ctx->sy.p,
        ctx->sz.p, ctx->sq.p, ctx->trg.p, ctx->near_precision == TAPAS_B200_FP64 ? 1 : 0);
    TB_LAUNCH_CHECK(ctx);
  } else if (nl > 0) {
    l2p_kernel<P><<<(unsigned)((nl + kWarps - 1) / kWarps), kThreads, 0, s>>>(
        leaves, nl, ctx->cbeg.p, ctx->cnb.p, ctx->ccen.p, ctx->sx.p, ctx->sy.p,
        ctx->sz.p, ctx->sq.p, ctx->L.p, ctx->trg.p, ctx->near_precision == TAPAS_B200_FP64 ? 1 : 0);
    TB_LAUNCH_CHECK(ctx);
  }
  return TAPAS_B200_OK;
}

}  // namespace

#define TB_DISPATCH_P(P, FN)                                                         \
  switch (P) {                                                                       \
    case 2: return FN<2>(ctx);   case 3: return FN<3>(ctx);   case 4: return FN<4>(ctx);   \
    case 5: return FN<5>(ctx);   case 6: return FN<6>(ctx);   case 7: return FN<7>(ctx);   \
    case 8: return FN<8>(ctx);   case 9: return FN<9>(ctx);   case 10: return FN<10>(ctx); \
    case 11: return FN<11>(ctx); case 12: return FN<12>(ctx); case 13: return FN<13>(ctx); \
    case 14: return FN<14>(ctx); case 15: return FN<15>(ctx); case 16: return FN<16>(ctx); \
    default: break;                                                                  \
  }                                                                                  \
  set_error(ctx, "expansion order P=%d outside %d..%d", (P), kMinP, kMaxP);          \
  return TAPAS_B200_ERR_UNSUPPORTED;

template <int P>
int upward_fp64_P(tapas_b200_ctx *ctx) { return upward_P<P>(ctx, false); }
template <int P>
int upward_f32leaf_P(tapas_b200_ctx *ctx) { return upward_P<P>(ctx, true); }
int upward_fp64(tapas_b200_ctx *ctx, int P) { TB_DISPATCH_P(P, upward_fp64_P) }
int upward_fp32_p2m(tapas_b200_ctx *ctx, int P) { TB_DISPATCH_P(P, upward_f32leaf_P) }
template <int P>
int p2m_fp64_P(tapas_b200_ctx *ctx) { return p2m_P<P>(ctx, false); }
template <int P>
int p2m_f32leaf_P(tapas_b200_ctx *ctx) { return p2m_P<P>(ctx, true); }
int p2m_only(tapas_b200_ctx *ctx, int P, bool fp32) {
  if (fp32) { TB_DISPATCH_P(P, p2m_f32leaf_P) }
  TB_DISPATCH_P(P, p2m_fp64_P)
}
int m2m_only(tapas_b200_ctx *ctx) { TB_DISPATCH_P(ctx->P, m2m_P) }

int fp64_m2m_levels(tapas_b200_ctx *ctx, int max_levels) {
  switch (ctx->P) {
    case 2: return fp64_m2m_levels_P<2>(ctx, max_levels);
    case 3: return fp64_m2m_levels_P<3>(ctx, max_levels);
    case 4: return fp64_m2m_levels_P<4>(ctx, max_levels);
    case 5: return fp64_m2m_levels_P<5>(ctx, max_levels);
    case 6: return fp64_m2m_levels_P<6>(ctx, max_levels);
    case 7: return fp64_m2m_levels_P<7>(ctx, max_levels);
    case 8: return fp64_m2m_levels_P<8>(ctx, max_levels);
    case 9: return fp64_m2m_levels_P<9>(ctx, max_levels);
    case 10: return fp64_m2m_levels_P<10>(ctx, max_levels);
    case 11: return fp64_m2m_levels_P<11>(ctx, max_levels);
    case 12: return fp64_m2m_levels_P<12>(ctx, max_levels);
    case 13: return fp64_m2m_levels_P<13>(ctx, max_levels);
    case 14: return fp64_m2m_levels_P<14>(ctx, max_levels);
    case 15: return fp64_m2m_levels_P<15>(ctx, max_levels);
    case 16: return fp64_m2m_levels_P<16>(ctx, max_levels);
    default: break;
  }
  set_error(ctx, "expansion order P=%d outside %d..%d", ctx->P, kMinP, kMaxP);
  return TAPAS_B200_ERR_UNSUPPORTED;
}
int m2l_fp64_cells(tapas_b200_ctx *ctx) { return ctx->P == 2 ? m2l_P<2>(ctx) : m2l_P<3>(ctx); }

static int m2l_pairs_dispatch(tapas_b200_ctx *ctx) { TB_DISPATCH_P(ctx->P, m2l_pairs_P) }

int m2l_fp64_pairs(tapas_b200_ctx *ctx, const uint32_t *pairs, int64_t npairs) {
  ctx->m2l_pairs = pairs;
  ctx->m2l_npairs = npairs;
  const int rc = m2l_pairs_dispatch(ctx);
  ctx->m2l_pairs = nullptr;
  ctx->m2l_npairs = 0;
  return rc;
}
template <int P>
int downward_fp64_P(tapas_b200_ctx *ctx) { return downward_P<P>(ctx, false); }
template <int P>
int downward_f32leaf_P(tapas_b200_ctx *ctx) { return downward_P<P>(ctx, true); }
int downward_fp64(tapas_b200_ctx *ctx) { TB_DISPATCH_P(ctx->P, downward_fp64_P) }
int downward_fp32_l2p(tapas_b200_ctx *ctx) { TB_DISPATCH_P(ctx->P, downward_f32leaf_P) }

}  // namespace tb
