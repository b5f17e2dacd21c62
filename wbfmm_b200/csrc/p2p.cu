// Near field (P2P): the sources of the 27 neighbour boxes of each target leaf
// box (src/indexing.c:250-286).
#include <cuda_runtime.h>

#include <type_traits>

#include "engine.h"
#include "expand.cuh"
#include "f32x2.cuh"
#include "kernels.h"
#include "translate.cuh"

namespace wbfmm {

// ------------------------------------------------------------------- P2P
// One CTA per target leaf box.  The sources of the 27 neighbour boxes (a
// virtual list, box by box) are staged through shared memory in tiles of NT
// (the CTA's thread count: 128, or 32 for trees whose leaves hold a few
// points each, so that more boxes are resident per SM).  The box's targets
// are taken NT at a time, the m of a pass spread over all NT threads (NT/m
// or NT/m + 1 consecutive threads per target, so that no thread idles
// whatever m is): thread gl of a target's g takes tile entries gl, gl + g,
// ..., accumulating in FP64 registers in a fixed order, and the target's
// first thread adds its threads' sums in thread order.  The FP32
// form computes pair terms in FP32 from separations that keep FP64 accuracy
// (coordinates as float pairs hi + lo, the hi parts of neighbouring points
// subtracting exactly), sums each run of 8 of a thread's terms in FP32 and
// adds that into the FP64 sums.  Pair kernels and the r > 1e-6 cutoff follow
// src/local.c:32-262 and src/local-laplace.c:400-523, 1091-1227.
constexpr int kP2PRun = 8;     // FP32 terms summed before each FP64 add

template <typename T, bool HELM, int NT>
struct P2PTile {
  double x[NT], y[NT], z[NT];   // FP32 form: float hi[NT], lo[NT] in each
  T q[NT * (HELM ? 2 : 1)];
  T d[NT * (HELM ? 2 : 1)];
  T nx[NT], ny[NT], nz[NT];
};

// sin and cos of x >= 0 in FP32 for the near field: x = n pi/2 + r with
// |r| <= pi/4 by the two-constant reduction of Cody and Waite (FMA), the
// Taylor series of sin r to r^9 and of cos r to r^10 (truncation below 2e-9
// at |r| = pi/4), then the quadrant's swap and signs.  A few ulp for x up to
// about 1e4; the near field's k r stays far below that.
__device__ __forceinline__ void sincos_near(float x, float* sp, float* cp) {
  const float q = rintf(x * 0.636619772367581343f);            // 2/pi
  float r = fmaf(-q, 1.57079637050628662109375f, x);          // fl(pi/2)
  r = fmaf(-q, -4.37113900018624283e-8f, r);                  // pi/2 - fl(pi/2)
  const float r2 = r * r;
  float ps = fmaf(r2, 2.75573192239858907e-6f, -1.98412698412698413e-4f);
  ps = fmaf(r2, ps, 8.33333333333333333e-3f);
  ps = fmaf(r2, ps, -1.66666666666666667e-1f);
  const float sn = fmaf(r * r2, ps, r);
  float pc = fmaf(r2, -2.75573192239858907e-7f, 2.48015873015873016e-5f);
  pc = fmaf(r2, pc, -1.38888888888888889e-3f);
  pc = fmaf(r2, pc, 4.16666666666666667e-2f);
  pc = fmaf(r2, pc, -0.5f);
  const float cn = fmaf(r2, pc, 1.0f);
  const int n = (int)q;
  float so = (n & 1) ? cn : sn, co = (n & 1) ? sn : cn;
  if (n & 2) so = -so;
  if ((n + 1) & 2) co = -co;
  *sp = so;
  *cp = co;
}

// sin and cos in FP64 for the near field, the same reduction (its constants
// pi/2 and pi/2 - fl(pi/2) in FP64; up to 1e5 the first step is exact) and the
// Taylor series to r^17 and r^18 (truncation below 1e-19 at |r| = pi/4): about
// 40 instructions, within 5e-16 of the library's sincos (2 ulp of its own),
// which serves larger arguments.
__device__ __forceinline__ void sincos_near(double x, double* sp, double* cp) {
  if (fabs(x) > 1e5) {
    sincos(x, sp, cp);
    return;
  }
  const double q = rint(x * 0.63661977236758134308);
  double r = fma(-q, 1.57079632679489655800, x);
  r = fma(-q, 6.12323399573676603587e-17, r);
  const double r2 = r * r;
  double ps = 1.0 / 355687428096000.0;                      // 1/17!
  ps = fma(r2, ps, -1.0 / 1307674368000.0);
  ps = fma(r2, ps, 1.0 / 6227020800.0);
  ps = fma(r2, ps, -1.0 / 39916800.0);
  ps = fma(r2, ps, 1.0 / 362880.0);
  ps = fma(r2, ps, -1.0 / 5040.0);
  ps = fma(r2, ps, 1.0 / 120.0);
  ps = fma(r2, ps, -1.0 / 6.0);
  const double sn = fma(r * r2, ps, r);
  double pc = -1.0 / 6402373705728000.0;                    // 1/18!
  pc = fma(r2, pc, 1.0 / 20922789888000.0);
  pc = fma(r2, pc, -1.0 / 87178291200.0);
  pc = fma(r2, pc, 1.0 / 479001600.0);
  pc = fma(r2, pc, -1.0 / 3628800.0);
  pc = fma(r2, pc, 1.0 / 40320.0);
  pc = fma(r2, pc, -1.0 / 720.0);
  pc = fma(r2, pc, 1.0 / 24.0);
  pc = fma(r2, pc, -0.5);
  const double cn = fma(r2, pc, 1.0);
  const int n = (int)q;
  const double so = (n & 1) ? cn : sn, co = (n & 1) ? sn : cn;
  *sp = (n & 2) ? -so : so;
  *cp = ((n + 1) & 2) ? -co : co;
}

// The terms of one (target, source) pair at separation r = (rx, ry, rz)
// (|r|^2 = r2) added to acc[0..] (Helmholtz: pot re, im, then grad x re,
// x im, y, z; Laplace: pot, grad x, y, z), without the kernels' constant
// factors, which the caller applies once per target (p2p_scale): 1/(4 pi)
// on the potential, -k/(4 pi) (Helmholtz) and 1/(4 pi) (Laplace) on the
// gradient.
// MASKED: a pair within the cutoff (r2 <= rc2) takes 1/r = 0, which makes
// each of its terms an exact zero, instead of being branched around (the
// pairs of a run then interleave without divergence)
// 1/sqrt(x) of a pair: in FP32 the MUFU approximation alone
// (rsqrt.approx.ftz: no subnormal handling, which a squared distance above
// the cutoff, at least 1e-12, never needs; for such normal arguments it is
// the approximation rsqrtf returns)
__device__ __forceinline__ float pair_rsqrt(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ double pair_rsqrt(double x) { return rsqrt(x); }

template <typename T, bool HELM, int NT, bool want_pot, bool want_grad, bool MASKED = false>
__device__ __forceinline__ void p2p_pair(const P2PTile<T, HELM, NT>& tl, int j, T rx, T ry, T rz,
                                         T r2, T k, T kinv, bool hd, T* acc, T rc2 = T(0)) {
  const T ir = MASKED ? (r2 > rc2 ? pair_rsqrt(r2) : T(0)) : pair_rsqrt(r2);
  if (HELM) {
    const T r = r2 * ir;
    const T kr = k * r, ikr = ir * kinv;
    T sn, cs;
    sincos_near(kr, &sn, &cs);
    // h0 = e^{ikr} / (i k r), h1 = h0 / (i k r) - ... (the first-order
    // spherical Hankel function), so that grad h0(kr) = -k h1 r / r
    const T h0r = sn * ikr, h0i = -cs * ikr;
    const T h1r = fma(h0r, ikr, h0i), h1i = fma(h0i, ikr, -h0r);
    const T qr = tl.q[2 * j], qi = tl.q[2 * j + 1];
    if (want_pot) {
      if (sizeof(T) == 8) {
        // the products first: one rounding of the sum per term (two, a product
        // at a time: 8.5e-16 against 6.2e-16 on 401 sources)
        acc[0] += fma(h0r, qr, -h0i * qi);
        acc[1] += fma(h0i, qr, h0r * qi);
      } else {
        acc[0] = fma(h0r, qr, fma(-h0i, qi, acc[0]));
        acc[1] = fma(h0i, qr, fma(h0r, qi, acc[1]));
      }
      if (hd) {
        const T nr = (rx * tl.nx[j] + ry * tl.ny[j] + rz * tl.nz[j]) * ir;
        const T dr = tl.d[2 * j] * nr, di = tl.d[2 * j + 1] * nr;
        acc[0] -= k * (h1r * dr - h1i * di);
        acc[1] -= k * (h1r * di + h1i * dr);
      }
    }
    if (want_grad) {
      const T ar = (h1r * qr - h1i * qi) * ir, ai = (h1r * qi + h1i * qr) * ir;
      acc[2] = fma(ar, rx, acc[2]); acc[3] = fma(ai, rx, acc[3]);
      acc[4] = fma(ar, ry, acc[4]); acc[5] = fma(ai, ry, acc[5]);
      acc[6] = fma(ar, rz, acc[6]); acc[7] = fma(ai, rz, acc[7]);
      if (hd) {
        const T nxs = tl.nx[j], nys = tl.ny[j], nzs = tl.nz[j];
        const T nr = rx * nxs + ry * nys + rz * nzs;
        const T dpr = h0r - T(2) * h1r * ikr, dpi = h0i - T(2) * h1i * ikr;
        const T dr = tl.d[2 * j], di = tl.d[2 * j + 1];
        const T rv[3] = {rx, ry, rz}, nv[3] = {nxs, nys, nzs};
        const T ir2 = ir * ir;
        for (int c = 0; c < 3; c++) {
          T ur = dpr * k * nr * rv[c] * ir2 + h1r * (nv[c] * ir - nr * rv[c] * ir2 * ir);
          T ui = dpi * k * nr * rv[c] * ir2 + h1i * (nv[c] * ir - nr * rv[c] * ir2 * ir);
          acc[2 + 2 * c] += ur * dr - ui * di;
          acc[3 + 2 * c] += ur * di + ui * dr;
        }
      }
    }
  } else {
    const T q = tl.q[j];
    const T ir2 = ir * ir;
    if (want_pot) {
      T v = q;
      if (hd) v += tl.d[j] * (rx * tl.nx[j] + ry * tl.ny[j] + rz * tl.nz[j]) * ir2;
      acc[0] = fma(v, ir, acc[0]);
    }
    if (want_grad) {
      const T ir3 = ir * ir2;
      const T gq = -q * ir3;
      acc[1] = fma(gq, rx, acc[1]); acc[2] = fma(gq, ry, acc[2]); acc[3] = fma(gq, rz, acc[3]);
      if (hd) {
        const T nxs = tl.nx[j], nys = tl.ny[j], nzs = tl.nz[j];
        const T nr = rx * nxs + ry * nys + rz * nzs;
        const T ad = tl.d[j] * ir3;
        acc[1] += ad * (nxs - T(3) * nr * rx * ir2);
        acc[2] += ad * (nys - T(3) * nr * ry * ir2);
        acc[3] += ad * (nzs - T(3) * nr * rz * ir2);
      }
    }
  }
}

// sincos_near of both numbers of a pair: sin and cos of r packed (the same
// reduction, the quadrant from adding 1.5 x 2^23, the same series), the
// quadrant's swap and signs one by one
__device__ __forceinline__ void sincos_near(f32x2 x, f32x2* sp, f32x2* cp) {
  const f32x2 t = fma2(x, both(0.636619772367581343f), both(12582912.0f));
  const f32x2 q = add2(t, both(-12582912.0f));
  f32x2 r = fma2(q, both(-1.57079637050628662109375f), x);
  r = fma2(q, both(4.37113900018624283e-8f), r);
  const f32x2 r2 = mul2(r, r);
  f32x2 ps = fma2(r2, both(2.75573192239858907e-6f), both(-1.98412698412698413e-4f));
  ps = fma2(r2, ps, both(8.33333333333333333e-3f));
  ps = fma2(r2, ps, both(-1.66666666666666667e-1f));
  const float2 sn = pair(fma2(mul2(r, r2), ps, r));
  f32x2 pc = fma2(r2, both(-2.75573192239858907e-7f), both(2.48015873015873016e-5f));
  pc = fma2(r2, pc, both(-1.38888888888888889e-3f));
  pc = fma2(r2, pc, both(4.16666666666666667e-2f));
  pc = fma2(r2, pc, both(-0.5f));
  const float2 cn = pair(fma2(r2, pc, both(1.0f)));
  const float2 tf = pair(t);
  auto turn = [](float tq, float s, float c, float* so, float* co) {
    const int n = __float_as_int(tq);        // low bits: the quadrant
    const float a = (n & 1) ? c : s, b = (n & 1) ? s : c;
    *so = __int_as_float(__float_as_int(a) ^ ((n & 2) << 30));
    *co = __int_as_float(__float_as_int(b) ^ (((n + 1) & 2) << 30));
  };
  float2 so, co;
  turn(tf.x, sn.x, cn.x, &so.x, &co.x);
  turn(tf.y, sn.y, cn.y, &so.y, &co.y);
  *sp = packed(so);
  *cp = packed(co);
}

// p2p_pair (monopoles, cutoff masked) of tile entries j0 and j1, the terms
// two at a time in packed arithmetic (f32x2.cuh) and then added one after
// the other: the operations and the order of sums of two calls of p2p_pair.
// second: false for a lone entry j0, whose partner counts nothing: 1/r and
// strength zero (1/r alone would not do: 0 x Inf of an infinite strength).
// t: the target's coordinates, each hi and lo
template <bool HELM, int NT, bool POT, bool GRAD>
__device__ __forceinline__ void p2p_two(const P2PTile<float, HELM, NT>& tl, int j0, int j1,
                                        bool second, const f32x2 (&t)[3], float rc2, f32x2 k,
                                        f32x2 kinv, float* acc) {
  const f32x2 m1 = both(-1.0f);
  auto sep = [&](const double* a, f32x2 tc) {
    const f32x2* c = reinterpret_cast<const f32x2*>(a);
    const float2 d0 = pair(fma2(c[j0], m1, tc)), d1 = pair(fma2(c[j1], m1, tc));
    return packed(make_float2(d0.x + d0.y, d1.x + d1.y));
  };
  const f32x2 rx = sep(tl.x, t[0]), ry = sep(tl.y, t[1]), rz = sep(tl.z, t[2]);
  const f32x2 r2 = fma2(rz, rz, fma2(rx, rx, mul2(ry, ry)));
  const float2 s2 = pair(r2);
  const f32x2 ir = packed(make_float2(s2.x > rc2 ? pair_rsqrt(s2.x) : 0.0f,
                                      second && s2.y > rc2 ? pair_rsqrt(s2.y) : 0.0f));
  const float2 x = pair(rx), y = pair(ry), z = pair(rz);
  if constexpr (HELM) {
    const f32x2 kr = mul2(k, mul2(r2, ir)), ikr = mul2(ir, kinv);
    f32x2 sn, cs;
    sincos_near(kr, &sn, &cs);
    // h0 = a - i b, h1 = c - i d
    const f32x2 a = mul2(sn, ikr), b = mul2(cs, ikr);
    const float2 q0 = reinterpret_cast<const float2*>(tl.q)[j0],
                 q1 = second ? reinterpret_cast<const float2*>(tl.q)[j1] : make_float2(0.0f, 0.0f);
    const f32x2 qr = packed(make_float2(q0.x, q1.x)), qi = packed(make_float2(q0.y, q1.y));
    if (POT) {
      const float2 a2 = pair(a), b2 = pair(b);
      acc[0] = fmaf(a2.x, q0.x, fmaf(b2.x, q0.y, acc[0]));
      acc[1] = fmaf(-b2.x, q0.x, fmaf(a2.x, q0.y, acc[1]));
      acc[0] = fmaf(a2.y, q1.x, fmaf(b2.y, q1.y, acc[0]));
      acc[1] = fmaf(-b2.y, q1.x, fmaf(a2.y, q1.y, acc[1]));
    }
    if (GRAD) {
      const f32x2 c = fma2(a, ikr, mul2(b, m1)), d = fma2(b, ikr, a);
      const float2 ar = pair(mul2(fma2(c, qr, mul2(d, qi)), ir));
      const float2 ai = pair(mul2(fma2(c, qi, mul2(d, mul2(qr, m1))), ir));
      acc[2] = fmaf(ar.x, x.x, acc[2]); acc[3] = fmaf(ai.x, x.x, acc[3]);
      acc[4] = fmaf(ar.x, y.x, acc[4]); acc[5] = fmaf(ai.x, y.x, acc[5]);
      acc[6] = fmaf(ar.x, z.x, acc[6]); acc[7] = fmaf(ai.x, z.x, acc[7]);
      acc[2] = fmaf(ar.y, x.y, acc[2]); acc[3] = fmaf(ai.y, x.y, acc[3]);
      acc[4] = fmaf(ar.y, y.y, acc[4]); acc[5] = fmaf(ai.y, y.y, acc[5]);
      acc[6] = fmaf(ar.y, z.y, acc[6]); acc[7] = fmaf(ai.y, z.y, acc[7]);
    }
  } else {
    const f32x2 q = packed(make_float2(tl.q[j0], second ? tl.q[j1] : 0.0f));
    if (POT) {
      const float2 q2 = pair(q), i2 = pair(ir);
      acc[0] = fmaf(q2.y, i2.y, fmaf(q2.x, i2.x, acc[0]));
    }
    if (GRAD) {
      const float2 g = pair(mul2(q, mul2(ir, mul2(ir, ir))));
      acc[1] = fmaf(-g.y, x.y, fmaf(-g.x, x.x, acc[1]));
      acc[2] = fmaf(-g.y, y.y, fmaf(-g.x, y.x, acc[2]));
      acc[3] = fmaf(-g.y, z.y, fmaf(-g.x, z.x, acc[3]));
    }
  }
}

// the constant factor of accumulator c of p2p_pair (see there)
template <bool HELM>
__device__ __forceinline__ double p2p_scale(int c, double k) {
  const double f4pi = 0.25 / kPi;
  return HELM ? (c < 2 ? f4pi : -k * f4pi) : f4pi;
}

// POT / GRAD: the fields computed, fixed at compile time (dipoles at run time).
// 128-thread CTAs are held to 4 (Helmholtz) / 5 (Laplace) resident per SM:
// with the masked runs the compiler's own choice took 149 registers; the
// caps measured best (FP32 Helmholtz pot+grad evaluation of 2e5 points:
// 1.152 ms before the masking, 1.130 ms masked, 1.046 ms with 4 CTAs, 1.093
// with 5; Laplace 0.615 / 0.564 / 0.566 / 0.544 ms)
// DIP: dipole sources (p.dip set), fixed at compile time so that the
// monopole kernels carry no dipole code (a smaller loop body: fewer
// instruction-fetch stalls)
// SHARE (FP32 form): several CTAs per box.  A lane takes whole runs of terms,
// those that a CTA with all the box's targets would sum, so that the sums do
// not depend on the shares; its entries are then 8 apart, and the tile holds
// entry j at tile_at(j), where lanes of neighbouring runs read neighbours
template <int NT, bool SHARE>
__device__ __forceinline__ int tile_at(int j) {
  return SHARE ? (j & (kP2PRun - 1)) * (NT / kP2PRun) + j / kP2PRun : j;
}

template <typename T, bool HELM, int NT, bool POT, bool GRAD, bool DIP, bool SHARE = false>
__global__ void __launch_bounds__(NT, NT == 32 ? 20 : (HELM ? 4 : 5))
k_p2p(EvalParams<T> p) {
  constexpr bool F32 = sizeof(T) == 4;
  constexpr int NA = HELM ? 8 : 4;
  // packed terms, except for Helmholtz potential and gradient in CTAs of 128
  // that share no box, where they are slower (ms one by one / packed: 49 points
  // per leaf 0.741 / 0.759, 10 per leaf 0.074 / 0.078; in CTAs of 32, 8 per leaf,
  // 0.324 / 0.284; 64 shared leaves of 625 points 3.60 / 3.02; the potential
  // alone, 49 per leaf, 0.547 / 0.510; Laplace, 49 per leaf, potential and
  // gradient 0.333 / 0.314, the potential alone 0.261 / 0.251)
  constexpr bool PACK = F32 && !DIP && !(HELM && POT && GRAD && NT == 128 && !SHARE);
  __shared__ P2PTile<T, HELM, NT> tl;
  __shared__ uint32_t s_st[27], s_pref[28];
  __shared__ double s_red[NA][NT];     // each lane's sums, for its target's group
  const int64_t b = blockIdx.x;
  // this CTA's share of the box's targets (gridDim.y CTAs per box)
  const uint64_t all = p.tcount[b];
  const uint32_t tc0 = (uint32_t)(all * blockIdx.y / gridDim.y),
                 tc = (uint32_t)(all * (blockIdx.y + 1) / gridDim.y);
  if (tc == tc0) return;
  const int tid = threadIdx.x;
  if (tid < 32) {
    uint32_t bi, bj, bk;
    demorton((uint64_t)b, &bi, &bj, &bk);
    const int nside = 1 << p.level;
    uint32_t cnt = 0, st = 0;
    if (tid < 27) {
      int ii = (int)bi + tid / 9 - 1, jj = (int)bj + (tid / 3) % 3 - 1,
          kk = (int)bk + tid % 3 - 1;
      if (ii >= 0 && jj >= 0 && kk >= 0 && ii < nside && jj < nside && kk < nside) {
        uint64_t nb = morton((uint32_t)ii, (uint32_t)jj, (uint32_t)kk);
        cnt = p.box_n[nb];
        st = p.box_i[nb];
      }
    }
    uint32_t incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (tid >= o) incl += v;
    }
    if (tid < 27) { s_st[tid] = st; s_pref[tid] = incl - cnt; }
    if (tid == 26) s_pref[27] = incl;
  }
  __syncthreads();
  const uint32_t total = s_pref[27];
  if (total == 0) return;   // no sources near: the whole CTA, before any other barrier
  const T rc2 = T(kCutoffRadius * kCutoffRadius);
  const T k = p.k;
  const T kinv = HELM ? T(1) / k : T(0);
  const bool hq = p.q != nullptr;
  constexpr bool hd = DIP, want_pot = POT, want_grad = GRAD;
  // FP32 form: source coordinates as float pairs (hi, lo) in the FP64 arrays' bytes
  float2* xp = (float2*)tl.x;
  float2* yp = (float2*)tl.y;
  float2* zp = (float2*)tl.z;
  // Each pass takes m = min(NT, targets left) targets and spreads them over
  // all NT lanes: NT / m lanes per target, one more for the first
  // NT mod m targets, the lanes of a target consecutive; lane gl of a
  // target's g lanes takes tile entries gl, gl + g, ... (every lane busy
  // whatever the box's target count)
  for (uint32_t t0 = tc0; t0 < tc; t0 += NT) {
    const int m = (int)min((uint32_t)NT, tc - t0);
    const int glo = NT / m, extra = NT - glo * m, split = extra * (glo + 1);
    const int ti = tid < split ? tid / (glo + 1) : extra + (tid - split) / glo;
    const int g = tid < split ? glo + 1 : glo;
    const int gl = tid < split ? tid % (glo + 1) : (tid - split) % glo;
    const uint32_t jt = p.tstart[b] + t0 + ti;
    // gv: the lanes that a CTA with all the box's targets gives this target
    // (FP32 form: they name its runs of terms, which are then the same
    // whatever the shares)
    int gv = g;
    if constexpr (SHARE) {
      const uint32_t t = t0 + ti, f = t / NT * NT;
      const int mv = (int)min((uint64_t)NT, all - f);
      gv = NT / mv + ((int)(t - f) < NT % mv ? 1 : 0);
    }
    const double x = p.tx[jt], y = p.ty[jt], z = p.tz[jt];
    const float txh = (float)x, tyh = (float)y, tzh = (float)z;
    const float txl = (float)(x - (double)txh), tyl = (float)(y - (double)tyh),
                tzl = (float)(z - (double)tzh);
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    [[maybe_unused]] const f32x2 tt[3] = {packed(make_float2(txh, txl)),
                                          packed(make_float2(tyh, tyl)),
                                          packed(make_float2(tzh, tzl))};
    for (uint32_t f0 = 0; f0 < total; f0 += NT) {
      const uint32_t f = f0 + tid;
      __syncthreads();
      if (f < total) {
        int l = 0;
        while (l < 26 && s_pref[l + 1] <= f) l++;
        const uint32_t s = s_st[l] + (f - s_pref[l]);
        const double sx = p.x[s], sy = p.y[s], sz = p.z[s];
        const int at = tile_at<NT, SHARE>(tid);
        if constexpr (F32) {
          const float hx = (float)sx, hy = (float)sy, hz = (float)sz;
          xp[at] = make_float2(hx, (float)(sx - (double)hx));
          yp[at] = make_float2(hy, (float)(sy - (double)hy));
          zp[at] = make_float2(hz, (float)(sz - (double)hz));
        } else {
          tl.x[at] = sx; tl.y[at] = sy; tl.z[at] = sz;
        }
        if (HELM) {
          tl.q[2 * at] = hq ? p.q[2 * s] : T(0);
          tl.q[2 * at + 1] = hq ? p.q[2 * s + 1] : T(0);
          if (hd) { tl.d[2 * at] = p.dip[2 * s]; tl.d[2 * at + 1] = p.dip[2 * s + 1]; }
        } else {
          tl.q[at] = hq ? p.q[s] : T(0);
          if (hd) tl.d[at] = p.dip[s];
        }
        if (hd) { tl.nx[at] = p.nx[s]; tl.ny[at] = p.ny[s]; tl.nz[at] = p.nz[s]; }
      }
      __syncthreads();
      const int nt = (int)min((uint32_t)NT, total - f0);
      if constexpr (PACK) {
        // runs of kP2PRun pairs, two at a time: a full run without bounds
        // checks, the tile's last run with them
        const f32x2 kk = both(k), ki = both(kinv);
        auto two = [&](int j0, int j1, bool second, float* acc) {
          p2p_two<HELM, NT, POT, GRAD>(tl, tile_at<NT, SHARE>(j0), tile_at<NT, SHARE>(j1), second,
                                       tt, rc2, kk, ki, acc);
        };
        for (int w = gl;; w += g) {
          const int j0 = SHARE ? w % gv + w / gv * (kP2PRun * gv) : gl + (w - gl) * kP2PRun;
          if (j0 >= nt) {
            if (!SHARE || w / gv * (kP2PRun * gv) >= nt) break;
            continue;
          }
          float acc[NA];
#pragma unroll
          for (int c = 0; c < NA; c++) acc[c] = 0.0f;
          if (j0 + (kP2PRun - 1) * gv < nt) {
#pragma unroll
            for (int u = 0; u < kP2PRun; u += 2) two(j0 + u * gv, j0 + (u + 1) * gv, true, acc);
          } else {
#pragma unroll 1
            for (int u = 0; u < kP2PRun && j0 + u * gv < nt; u += 2) {
              const int j = j0 + u * gv;
              two(j, j + gv < nt ? j + gv : j, j + gv < nt, acc);
            }
          }
#pragma unroll
          for (int c = 0; c < NA; c++) a[c] += (double)acc[c];
        }
      } else if constexpr (F32) {
        // runs of kP2PRun pairs: a full run without bounds checks, the
        // tile's last run with them; the cutoff by masking (p2p_pair)
        auto pair_at = [&](int entry, T* acc) {
          const int j = tile_at<NT, SHARE>(entry);
          const float2 cx = xp[j], cy = yp[j], cz = zp[j];
          const T rx = (T)((txh - cx.x) + (txl - cx.y));
          const T ry = (T)((tyh - cy.x) + (tyl - cy.y));
          const T rz = (T)((tzh - cz.x) + (tzl - cz.y));
          const T r2 = rx * rx + ry * ry + rz * rz;
          p2p_pair<T, HELM, NT, POT, GRAD, true>(tl, j, rx, ry, rz, r2, k, kinv, hd, acc, rc2);
        };
        for (int w = gl;; w += g) {
          const int j0 = SHARE ? w % gv + w / gv * (kP2PRun * gv) : gl + (w - gl) * kP2PRun;
          if (j0 >= nt) {
            if (!SHARE || w / gv * (kP2PRun * gv) >= nt) break;
            continue;
          }
          T acc[NA];
          for (int c = 0; c < NA; c++) acc[c] = T(0);
          if (j0 + (kP2PRun - 1) * gv < nt) {
#pragma unroll
            for (int u = 0; u < kP2PRun; u++) pair_at(j0 + u * gv, acc);
          } else {
#pragma unroll
            for (int u = 0; u < kP2PRun; u++)
              if (j0 + u * gv < nt) pair_at(j0 + u * gv, acc);
          }
          for (int c = 0; c < NA; c++) a[c] += (double)acc[c];
        }
      } else {
        // the terms straight into the sums
        for (int j = gl; j < nt; j += g) {
          const T rx = (T)(x - tl.x[j]), ry = (T)(y - tl.y[j]), rz = (T)(z - tl.z[j]);
          const T r2 = rx * rx + ry * ry + rz * rz;
          if (!(r2 > rc2)) continue;
          p2p_pair<T, HELM, NT, POT, GRAD>(tl, j, rx, ry, rz, r2, k, kinv, hd, (T*)a);
        }
      }
    }
    // the sums of a target's lanes, in lane order, by its first lane (the
    // next pass writes s_red only after its first tile barrier)
    for (int c = 0; c < NA; c++) s_red[c][tid] = a[c];
    __syncthreads();
    if (gl != 0) continue;
    double v[8];
    for (int c = 0; c < NA; c++) {
      double sum = s_red[c][tid];
      for (int i = 1; i < g; i++) sum += s_red[c][tid + i];
      v[c] = sum * p2p_scale<HELM>(c, (double)p.k);
    }
    const uint32_t o = p.tperm[jt];
    if (HELM) {
      if (want_pot) {
        p.pot[2 * (size_t)o] = (T)((double)p.pot[2 * (size_t)o] + v[0]);
        p.pot[2 * (size_t)o + 1] = (T)((double)p.pot[2 * (size_t)o + 1] + v[1]);
      }
      if (want_grad)
        for (int c = 0; c < 6; c++)
          p.grad[6 * (size_t)o + c] = (T)((double)p.grad[6 * (size_t)o + c] + v[2 + c]);
    } else {
      if (want_pot) p.pot[o] = (T)((double)p.pot[o] + v[0]);
      if (want_grad)
        for (int c = 0; c < 3; c++)
          p.grad[3 * (size_t)o + c] = (T)((double)p.grad[3 * (size_t)o + c] + v[1 + c]);
    }
  }
}

template <typename T, bool HELM>
int launch_p2p(const EvalParams<T>& p, cudaStream_t s) {
  if (p.nbox <= 0 || p.ntgt <= 0) return 0;
  auto go = [&](auto pot, auto grad, auto dip) {
    constexpr bool P = decltype(pot)::value, G = decltype(grad)::value;
    constexpr bool D = decltype(dip)::value;
    // a tree with fewer leaves than two per SM (depth 2 at most): several
    // CTAs share a box's targets, in shares of 64, 32, 16 or 8 on average,
    // the largest that give four CTAs per SM (1e4 FP32 Laplace points in 64
    // leaves: 218 us with a CTA per leaf, on 64 of 148 SMs, about 125 so)
    int64_t y = 1;
    if (p.nbox < 2 * 148)
      for (int64_t share = 64; share >= 8 && p.nbox * y < 4 * 148; share /= 2)
        y = (p.ntgt + p.nbox * share - 1) / (p.nbox * share);
    if (y > 65535) y = 65535;
    const dim3 grid((unsigned)p.nbox, (unsigned)(y < 1 ? 1 : y));
    if (p.ntgt <= 8 * p.nbox)   // a few targets per leaf on average
      k_p2p<T, HELM, 32, P, G, D><<<grid, 32, 0, s>>>(p);   // (y is 1)
    else if (sizeof(T) == 4 && grid.y > 1)
      k_p2p<T, HELM, 128, P, G, D, sizeof(T) == 4><<<grid, 128, 0, s>>>(p);
    else
      k_p2p<T, HELM, 128, P, G, D><<<grid, 128, 0, s>>>(p);
  };
  auto fields = [&](auto dip) {
    if (p.pot && p.grad) go(std::true_type(), std::true_type(), dip);
    else if (p.pot) go(std::true_type(), std::false_type(), dip);
    else if (p.grad) go(std::false_type(), std::true_type(), dip);
  };
  if (p.dip) fields(std::true_type());
  else fields(std::false_type());
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// dst[i] = (float)src[i]; dst[i] += src[i] (FP64 solvers' FP32 near field)
__global__ void k_narrow(const double* __restrict__ src, float* __restrict__ dst, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = (float)src[i];
}
__global__ void k_add_widened(double* __restrict__ dst, const float* __restrict__ src, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dst[i] += (double)src[i];
}
int launch_narrow(const double* src, float* dst, int64_t n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_narrow<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, dst, n);
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}
int launch_add_widened(double* dst, const float* src, int64_t n, cudaStream_t s) {
  if (n <= 0) return 0;
  k_add_widened<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(dst, src, n);
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// largest |sin| and |cos| errors of sincos_near and of sincosf against the
// FP64 values at the same FP32 arguments x_i = i * xmax / n (one block;
// err[0] ours, err[1] sincosf)
__global__ void k_sincos_check(double xmax, int n, double* err) {
  __shared__ double m[2][256];
  double e0 = 0, e1 = 0;
  for (int i = threadIdx.x; i <= n; i += blockDim.x) {
    const float x = (float)(xmax * i / n);
    float s, c, s1, c1;
    f32x2 sp, cp;
    sincos_near(both(x), &sp, &cp);
    float s0, c0;
    sincos_near(x, &s0, &c0);
    s = pair(sp).x; c = pair(cp).y;
    sincosf(x, &s1, &c1);
    const double sd = sin((double)x), cd = cos((double)x);
    e0 = fmax(e0, fmax(fabs(s - sd), fabs(c - cd)));
    e0 = fmax(e0, fmax(fabs(s0 - sd), fabs(c0 - cd)));
    e1 = fmax(e1, fmax(fabs(s1 - sd), fabs(c1 - cd)));
  }
  m[0][threadIdx.x] = e0; m[1][threadIdx.x] = e1;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int t = 1; t < blockDim.x; t++) { e0 = fmax(e0, m[0][t]); e1 = fmax(e1, m[1][t]); }
    err[0] = e0; err[1] = e1;
  }
}

// largest difference between the FP64 sincos_near and CUDA's sincos at
// +-i xmax / n and at the two FP64 neighbours of each multiple of pi/2 up to
// xmax (one block)
__global__ void k_sincos64_check(double xmax, int n, double* err) {
  __shared__ double m[256];
  double e = 0;
  auto check = [&](double x) {
    double s, c, s1, c1;
    sincos_near(x, &s, &c);
    sincos(x, &s1, &c1);
    const double d = fmax(fabs(s - s1), fabs(c - c1));
    if (!(d <= e)) e = d;                     // (a NaN stays)
  };
  for (int i = threadIdx.x; i <= n; i += blockDim.x) {
    check(xmax * i / n);
    check(-xmax * i / n);
  }
  const double h = 1.57079632679489661923;
  for (int i = threadIdx.x; i * h <= xmax; i += blockDim.x) {
    const double x = i * h;
    check(x);
    check(nextafter(x, x + 1.0));
  }
  m[threadIdx.x] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int t = 1; t < blockDim.x; t++)
      if (!(m[t] <= e)) e = m[t];
    *err = e;
  }
}

int sincos_near64_error(double xmax, int n, double* host_err) {
  double* d = nullptr;
  WBFMM_CUDA(cudaMalloc(&d, sizeof(double)));
  k_sincos64_check<<<1, 256>>>(xmax, n, d);
  cudaError_t e = cudaMemcpy(host_err, d, sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  WBFMM_CUDA(e);
  return 0;
}

int sincos_near_errors(double xmax, int n, double* host_err) {
  double* d = nullptr;
  WBFMM_CUDA(cudaMalloc(&d, 2 * sizeof(double)));
  k_sincos_check<<<1, 256>>>(xmax, n, d);
  cudaError_t e = cudaMemcpy(host_err, d, 2 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  WBFMM_CUDA(e);
  return 0;
}

// ------------------------------------------------------ instantiations
#define WBFMM_INST(T, H) template int launch_p2p<T, H>(const EvalParams<T>&, cudaStream_t);
WBFMM_INST(double, true)
WBFMM_INST(double, false)
WBFMM_INST(float, true)
WBFMM_INST(float, false)

}  // namespace wbfmm
