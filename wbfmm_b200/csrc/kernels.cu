// Leaf kernels: P2M and L2P.
//
//  P2M  a group of 32 or 8 lanes per leaf box; lanes take the box's sources
//       and every coefficient contribution is reduced across the group in a
//       fixed order (deterministic), accumulating in shared memory.
//  L2P  one thread per target.
#include <cuda_runtime.h>

#include <type_traits>

#include "engine.h"
#include "expand.cuh"
#include "kernels.h"
#include "translate.cuh"

namespace wbfmm {

// Sums over the groups of G lanes of a warp of several values at once, by
// transposing while reducing: after the exchanges across lanes G/2 (and G/4)
// apart, each half (quarter) of a group carries one value, whose sum the
// remaining steps form.  Two values: the first half of the group holds the
// sum of a, the second of b; four: the quarters those of a, b, c, d (G = 32:
// 6 shuffles instead of 20).
template <int G, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <int G, typename T>
__device__ __forceinline__ T group_sum2(T a, T b, int lane) {
  const bool hi = lane & (G / 2);
  T w = (hi ? b : a) + __shfl_xor_sync(0xffffffffu, hi ? a : b, G / 2);
#pragma unroll
  for (int o = G / 4; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  return w;
}
template <int G, typename T>
__device__ __forceinline__ T group_sum4(T a, T b, T c, T d, int lane) {
  const bool hi = lane & (G / 2), q = lane & (G / 4);
  const T u = (hi ? c : a) + __shfl_xor_sync(0xffffffffu, hi ? a : c, G / 2);
  const T v = (hi ? d : b) + __shfl_xor_sync(0xffffffffu, hi ? b : d, G / 2);
  T w = (q ? v : u) + __shfl_xor_sync(0xffffffffu, q ? u : v, G / 4);
#pragma unroll
  for (int o = G / 8; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
  return w;
}

// the P2M kernel's emitters: each emission summed over the group's points
// (one per lane) into the group's accumulator in shared memory; values that
// come together are reduced together, their sums added by one lane of each
// half / quarter
template <typename T, int G>
struct P2MEmitHelm {
  T* acc;
  int lane;
  __device__ __forceinline__ void operator()(int idx, T re, T im) const {
    const T w = group_sum2<G>(re, im, lane);
    if ((lane & (G / 2 - 1)) == 0) acc[2 * idx + ((lane & (G / 2)) ? 1 : 0)] += w;
  }
  __device__ __forceinline__ void pair(int i1, T r1, T m1, int i2, T r2, T m2) const {
    const T w = group_sum4<G>(r1, m1, r2, m2, lane);
    if ((lane & (G / 4 - 1)) == 0)
      acc[2 * ((lane & (G / 2)) ? i2 : i1) + ((lane & (G / 4)) ? 1 : 0)] += w;
  }
};
template <typename T, int G>
struct P2MEmitLap {
  T* acc;
  int lane;
  __device__ __forceinline__ void operator()(int idx, T v) const {
    v = group_sum<G>(v);
    if ((lane & (G - 1)) == 0) acc[idx] += v;
  }
  __device__ __forceinline__ void pair(int i1, T v1, int i2, T v2) const {
    const T w = group_sum2<G>(v1, v2, lane);
    if ((lane & (G / 2 - 1)) == 0) acc[(lane & (G / 2)) ? i2 : i1] += w;
  }
};

// box centre exactly as wbfmm_tree_box_centre (src/util.c:290-330)
__device__ __forceinline__ void box_centre(int64_t b, double x0, double y0,
                                           double z0, double wb, double* c) {
  uint32_t i, j, k;
  demorton((uint64_t)b, &i, &j, &k);
  c[0] = x0 + wb * i; c[1] = y0 + wb * j; c[2] = z0 + wb * k;
  c[0] += 0.5 * wb; c[1] += 0.5 * wb; c[2] += 0.5 * wb;
}

// ------------------------------------------------------------------- P2M
// shared-memory bytes of the Legendre constants of degrees <= N + 2
// (LegTab), or 0 where they would take more than 40 KB (then computed)
template <typename T>
static size_t leg_table_bytes(int N) {
  const size_t b = 4 * sizeof(T) * (size_t)(N + 3) * (N + 3);
  return b <= 40 * 1024 ? b : 0;
}

// shared-memory bytes of the per-thread recursion rows (expand.cuh) of a
// CTA of `threads` threads
template <typename T>
static size_t p2m_row_bytes(int N, int threads) {
  return sizeof(T) * (size_t)p2m_rows() * (N + kRowPad) * threads;
}
template <typename T>
static size_t l2p_row_bytes(int N, bool helm, bool grad, int threads) {
  return sizeof(T) * (size_t)l2p_rows(helm, grad) * (N + kRowPad) * threads;
}
// rows in shared memory up to this many bytes per CTA; above it (high
// orders, FP64) the rows stay in per-thread local arrays, where occupancy
// is worth more than the shorter latency
constexpr size_t kRowSmemMax = 48 * 1024;
constexpr int kP2MWarps = 4;     // per CTA
constexpr int kL2PBoxes = 4;     // leaf boxes whose expansions an L2P CTA stages
constexpr int kFixedOrder = 14;   // P2M / L2P order with a compile-time instantiation
#define WBFMM_TRY_K(call)          \
  do {                             \
    const int rc_ = (call);        \
    if (rc_) return rc_;           \
  } while (0)

// SROWS: recursion rows in shared memory (else per-thread local arrays);
// NC > 0: the expansion order fixed at compile time (p.N == NC), the rows
// in a per-thread array whose every index the unrolled recursion knows, so
// that they stay in registers.
// A warp takes 32 / G boxes, G lanes each: with a few points per leaf a whole
// warp per box leaves most lanes idle (2.5e5 points in 32768 leaves, FP64
// Helmholtz p = 8: 0.54 ms with a warp per box, 0.28 with 8 lanes).  At G = 32
// each warp has one box and the SMs take the CTAs as they get free, so that
// full boxes hold up no others; at G = 8, whose boxes hold 32 points at most,
// the grid is what the SMs hold, each warp walking over the boxes, and the
// recursion constants (square roots and divisions) are formed once per CTA.
// share (G = 32): the warps of a CTA share a box and their sums are added in
// warp order, for trees of fewer boxes than the SMs have warps.
// p.stat: of two launches, with G = 8 and with G = 32, one runs (p2m_few).
// (The block size named to the compiler: without it, it took 64 registers for
// FP32 Laplace, with it 117: 0.057 -> 0.054 ms on 60000 points in 32768 leaves
// at order 8, 0.109 -> 0.099 at order 14.)
template <typename T, bool HELM, bool SROWS, int NC, int G>
__global__ void __launch_bounds__(kP2MWarps * 32) k_p2m(P2MParams<T> p, int legt, int share) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int NG = 32 / G;
  if (p.stat && p2m_few(p.stat) != (G == 8)) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gl = lane & (G - 1);
  const int nw = blockDim.x >> 5;
  int64_t c0 = share ? (int64_t)blockIdx.x : ((int64_t)blockIdx.x * nw + warp) * NG;
  // the box's storage index, and (sparse storage) its Morton index
  int64_t cb, b;
  uint32_t cnt, start;
  bool in;
  auto box = [&]() {
    cb = c0 + lane / G;
    in = cb < p.nbox;
    b = !in ? 0 : p.glist ? (((int64_t)p.glist[cb >> 3] << 3) | (cb & 7)) : cb;
    cnt = in ? p.box_n[b] : 0;
    start = in ? p.box_i[b] : 0;
  };
  box();
  // Legendre recursion constants of degrees <= N + 2, once per CTA (not where
  // its boxes are empty)
  const int LW = (NC > 0 ? NC : p.N) + 3;
  T* lt = (T*)smraw;
  if (legt) {
    if (G == 8 || __syncthreads_or(cnt > 0)) leg_table_fill(lt, LW - 1, threadIdx.x, blockDim.x);
    __syncthreads();
  }
  const int N = NC > 0 ? NC : p.N;
  const int nc = ncoef(N);
  const int w = HELM ? 2 : 1;
  const int RL = N + kRowPad;
  T* rows = (T*)smraw + (legt ? 4 * LW * LW : 0);
  T loc[NC > 0 ? 2 * (NC + kRowPad) : (SROWS ? 1 : 2 * kPtMax)];
  const Scratch<T> sc = SROWS && NC == 0 ? Scratch<T>{rows + threadIdx.x, RL, (int)blockDim.x}
                                         : Scratch<T>{loc, RL, 1};
  T* acc = rows + (SROWS && NC == 0 ? p2m_rows() * RL * blockDim.x : 0) +
           (size_t)(warp * NG + lane / G) * nc * w;
#pragma unroll 1
  while (c0 < p.nbox) {
    const uint32_t most = NG == 1 ? cnt : __reduce_max_sync(0xffffffffu, cnt);
    if (most > 0) {
      for (int c = gl; c < nc * w; c += G) acc[c] = T(0);
      __syncwarp();
      // the points of box b, W lanes at a time
      auto points = [&](auto lanes, int64_t b, uint32_t cnt, uint32_t start, uint32_t most, T* acc) {
        constexpr int W = decltype(lanes)::value;
        double cd[3];
        box_centre(b, p.x0, p.y0, p.z0, p.wb, cd);
        // source position relative to the box centre, formed in FP64
        const T xc[3] = {T(0), T(0), T(0)};
        for (uint32_t base = share ? warp * W : 0; base < most; base += share ? nw * W : W) {
          const uint32_t t = base + (lane & (W - 1));
          const bool act = t < cnt;
          const uint32_t s = act ? start + t : 0;
          T xs[3] = {act ? (T)(p.x[s] - cd[0]) : T(0),
                     act ? (T)(p.y[s] - cd[1]) : T(0),
                     act ? (T)(p.z[s] - cd[2]) : T(0)};
          auto expand = [&](const auto& leg) {
            if (HELM) {
              const P2MEmitHelm<T, W> emit{acc, lane};
              if (p.q) {
                T qr = act ? p.q[2 * s] : T(0), qi = act ? p.q[2 * s + 1] : T(0);
                p2m_helmholtz<T>(N, p.k, xc, xs, qr, qi, emit, leg, sc);
              }
              if (p.dip) {
                T dr = act ? p.dip[2 * s] : T(0), di = act ? p.dip[2 * s + 1] : T(0);
                T nrm[3] = {act ? p.nx[s] : T(0), act ? p.ny[s] : T(0),
                            act ? p.nz[s] : T(1)};
                p2m_helmholtz_dipole<T>(N, p.k, xc, xs, nrm, dr, di, emit, leg, sc);
              }
            } else {
              const P2MEmitLap<T, W> emit{acc, lane};
              if (p.q) {
                T qv = act ? p.q[s] : T(0);
                p2m_laplace<T>(N, xc, xs, qv, emit, leg, sc);
              }
              if (p.dip) {
                T dv = act ? p.dip[s] : T(0);
                T nrm[3] = {act ? p.nx[s] : T(0), act ? p.ny[s] : T(0),
                            act ? p.nz[s] : T(1)};
                p2m_laplace_dipole<T>(N, xc, xs, nrm, dv, emit, leg, sc);
              }
            }
          };
          if (legt) expand(LegTab<T>{lt, LW});
          else expand(LegDirect<T>());
        }
      };
      // boxes of very unequal counts one after the other, a warp each, where
      // that takes fewer rounds
      if (NG > 1 && __reduce_add_sync(0xffffffffu, gl == 0 ? (cnt + 31) / 32 : 0) <
                        (most + G - 1) / G) {
#pragma unroll 1
        for (int i = 0; i < NG; i++) {
          const uint32_t ci = __shfl_sync(0xffffffffu, cnt, i * G);
          const uint32_t si = __shfl_sync(0xffffffffu, start, i * G);
          const int64_t bi = __shfl_sync(0xffffffffu, (long long)b, i * G);
          points(std::integral_constant<int, 32>(), bi, ci, si, ci,
                 acc + (size_t)(i - lane / G) * nc * w);
        }
      } else {
        points(std::integral_constant<int, G>(), b, cnt, start, most, acc);
      }
      __syncwarp();
    }
    if (share) {             // (the CTA's only box)
      if (most > 0) __syncthreads();
      if (warp) return;
      if (most > 0)
        for (int c = lane; c < nc * w; c += 32)
          for (int u = 1; u < nw; u++) acc[c] += acc[c + u * nc * w];
      __syncwarp();
    }
    // (a box without points beside one with points holds zeros)
    for (int c = gl; in && c < nc; c += G) {
      const int64_t o = layout_off(cb, c, nc);
      for (int u = 0; u < w; u++) {
        const T v = most > 0 ? acc[w * c + u] : T(0);
        if (p.accumulate) p.mps[w * o + u] += v;
        else p.mps[w * o + u] = v;
      }
    }
    if (G == 32) break;
    __syncwarp();
    c0 += (int64_t)gridDim.x * nw * NG;
    box();
  }
}

// lanes per leaf box: 8, 32 or (the warps of a CTA sharing it) 128
template <typename T, bool HELM>
int p2m_lanes(int N, int64_t nbox, int64_t npts) {
  const size_t leg = leg_table_bytes<T>(N);
  const size_t rows = p2m_row_bytes<T>(N, kP2MWarps * 32);
  const size_t one = sizeof(T) * (size_t)kP2MWarps * ncoef(N) * (HELM ? 2 : 1);   // a box per warp
  // leaves of up to 12 points on average, 96 per SM, or of up to 6, 24 per SM
  // (not at order 14, whose form with a warp per box is unrolled): four boxes
  // per warp, while their accumulators leave room for a second CTA (the rows
  // counted wherever they are) and the leaves' counts allow (p2m_few).  FP64
  // Laplace p = 8, ms with a warp per box / 8 lanes: 32768 uniform leaves of 7.6
  // points 0.23 / 0.15, 4096 of 2 0.043 / 0.036, 4096 of 11 0.045 / 0.047; of
  // clustered points, 8 lanes throughout: 4096 leaves of 11 0.28 / 0.82
  const bool many = nbox >= 4 * 148 * 24, fixed = N == kFixedOrder && !(HELM && sizeof(T) == 8);
  if (nbox >= 148 * 24 && (many || !fixed) && npts <= (many ? 12 : 6) * nbox &&
      leg + rows + 4 * one <= 100 * 1024)
    return 8;
  return nbox <= 148 * 8 && npts > 48 * nbox ? 128 : 32;
}

template <typename T, bool HELM>
int launch_p2m(const P2MParams<T>& p, cudaStream_t s) {
  if (p.nbox <= 0) return 0;
  const int nw = kP2MWarps;
  const size_t leg = leg_table_bytes<T>(p.N);
  const size_t rows = p2m_row_bytes<T>(p.N, nw * 32);
  const size_t one = sizeof(T) * (size_t)nw * ncoef(p.N) * (HELM ? 2 : 1);
  const int lanes = p2m_lanes<T, HELM>(p.N, p.nbox, p.npts);
  const bool few = lanes == 8, share = lanes == 128;
  auto go = [&](auto srows, auto nc, auto group) -> int {
    constexpr bool SR = decltype(srows)::value;
    constexpr int NC = decltype(nc)::value, G = decltype(group)::value;
    const size_t smem = leg + (SR ? rows : 0) + one * (32 / G);
    if (smem > 48 * 1024) WBFMM_SMEM(smem, k_p2m<T, HELM, SR, NC, G>);
    P2MParams<T> a = p;
    if (!few) a.stat = nullptr;
    // G = 8: at most 8 CTAs per SM, about what registers and shared memory hold
    const int64_t need = share ? p.nbox : (p.nbox + nw * (32 / G) - 1) / (nw * (32 / G));
    const unsigned grid = (unsigned)(G == 32 || need < 148 * 8 ? need : 148 * 8);
    k_p2m<T, HELM, SR, NC, G><<<grid, nw * 32, smem, s>>>(a, leg ? 1 : 0, share ? 1 : 0);
    return 0;
  };
  const std::integral_constant<int, 0> any;
  const std::integral_constant<int, 32> whole;
  const std::integral_constant<int, 8> eighth;
  const std::true_type yes;
  const std::false_type no;
  // the serving orders' leaf expansions: rows in registers (not for FP64
  // Helmholtz, whose unrolled recursion exceeds the register file)
  constexpr bool kFixedOk = !(HELM && sizeof(T) == 8);
  if (few) WBFMM_TRY_K(rows <= kRowSmemMax ? go(yes, any, eighth) : go(no, any, eighth));
  if (kFixedOk && p.N == kFixedOrder) {
    if constexpr (kFixedOk) WBFMM_TRY_K(go(no, std::integral_constant<int, kFixedOrder>(), whole));
  } else {
    WBFMM_TRY_K(rows <= kRowSmemMax ? go(yes, any, whole) : go(no, any, whole));
  }
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------------- L2P
// recursion constants of the L2P gradients from shared-memory tables filled
// once per CTA (rows n = -1..N+1, columns m + M0)
template <typename T>
struct RecTab {
  const T* ta;   // rec_a(n, m): row n + 1, column m
  const T* tb;   // rec_b(n, m): row n, column m + M0
  int W, M0;
  __device__ T a(int n, int m) const { return ta[(n + 1) * W + (m < 0 ? -m : m)]; }
  __device__ T b(int n, int m) const { return tb[n * W + m + M0]; }
};
template <typename T>
struct LapRecTab {
  const T* t;    // (am, a0, ap) at ((n (N+1) + m) * 3
  int N1;
  __device__ void c(int n, int m, T* am, T* a0, T* ap) const {
    const T* e = t + (n * N1 + m) * 3;
    *am = e[0]; *a0 = e[1]; *ap = e[2];
  }
};

// shared-memory bytes of the L2P tables at order N (0: computed on the fly)
template <typename T, bool HELM>
__host__ __device__ inline size_t l2p_table_bytes(int N) {
  const size_t b = HELM ? 2 * (size_t)(N + 3) * (2 * N + 3) * sizeof(T)
                        : 3 * (size_t)(N + 1) * (N + 1) * sizeof(T);
  return b <= 40 * 1024 ? b : 0;
}

// one thread per target (sorted by box); potential and gradient in one sweep
// SROWS: recursion rows in shared memory, after the tables (else
// per-thread local arrays)
// stage: the CTA's leaf expansions copied to shared memory when its targets
// fall in at most kL2PBoxes leaf boxes (targets are sorted by box)
// NC > 0: the expansion order fixed at compile time (p.N == NC), the rows
// in a per-thread array whose every index the unrolled recursion knows
template <typename T, bool HELM, bool SROWS, bool STAGE, int NC = 0>
__global__ void k_l2p(EvalParams<T> p, int tab, int legt) {
  const int stage = STAGE ? 1 : 0;
  extern __shared__ __align__(16) unsigned char l2p_sm[];
  __shared__ unsigned s_bal[32];
  __shared__ int64_t s_box[kL2PBoxes];
  T* st = (T*)l2p_sm;
  const int N = NC > 0 ? NC : p.N;
  const int W = 2 * N + 3, M0 = N + 1;
  // Legendre constants (degrees <= N + 2) after the recursion tables
  const int LW = N + 3;
  T* lt = st + (tab ? l2p_table_bytes<T, HELM>(N) / sizeof(T) : 0);
  T* rows = lt + (legt ? 4 * LW * LW : 0);
  constexpr bool SR = SROWS && NC == 0;
  T* cst = rows + (SR ? (size_t)l2p_rows(HELM, p.grad != nullptr) * (N + kRowPad) * blockDim.x : 0);
  T loc[NC > 0 ? 3 * (NC + kRowPad) : (SROWS ? 1 : 3 * kPtMax)];
  const Scratch<T> sc = SR ? Scratch<T>{rows + threadIdx.x, N + kRowPad, (int)blockDim.x}
                           : Scratch<T>{loc, N + kRowPad, 1};
  if (legt) leg_table_fill(lt, N + 2, threadIdx.x, blockDim.x);
  if (tab) {
    if (HELM) {
      T* ta = st;
      T* tb = st + (N + 3) * W;
      for (int i = threadIdx.x; i < (N + 3) * W; i += blockDim.x) {
        const int row = i / W, col = i - row * W;
        ta[i] = rec_a<T>(row - 1, col);
        tb[i] = rec_b<T>(row, col - M0);
      }
    } else {
      const int N1 = N + 1;
      for (int i = threadIdx.x; i < N1 * N1; i += blockDim.x) {
        const int n = i / N1, m = i - n * N1;
        T* e = st + 3 * i;
        if (n >= 1 && m <= n) LapRecDirect<T>().c(n, m, &e[0], &e[1], &e[2]);
        else e[0] = e[1] = e[2] = T(0);
      }
    }
  }
  const int jt = blockIdx.x * blockDim.x + threadIdx.x;
  const int nc = ncoef(N), wc = HELM ? 2 : 1;
  int slot = -1;
  if (stage) {
    const int j0 = blockIdx.x * blockDim.x;
    const bool in = jt < p.ntgt;
    const bool first = in && (jt == j0 || p.tbox[jt] != p.tbox[jt - 1]);
    const int nb = __syncthreads_count(first);
    if (nb <= kL2PBoxes) {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const unsigned bal = __ballot_sync(0xffffffffu, first);
      if (lane == 0) s_bal[warp] = bal;
      __syncthreads();
      int before = __popc(bal & ((1u << lane) - 1u));
      for (int w = 0; w < warp; w++) before += __popc(s_bal[w]);
      slot = before + (first ? 1 : 0) - 1;
      if (first) s_box[slot] = compact_box(p.gmap, (int64_t)p.tbox[jt]);
      __syncthreads();
      for (int i = threadIdx.x; i < nb * nc; i += blockDim.x) {
        const int k = i / nc, c = i - k * nc;
        if (s_box[k] < 0) {   // (targets lie in stored groups)
          for (int u = 0; u < wc; u++) cst[(size_t)i * wc + u] = T(0);
          continue;
        }
        const int64_t o = layout_off(s_box[k], c, nc);
        for (int u = 0; u < wc; u++) cst[(size_t)i * wc + u] = p.mpr[wc * o + u];
      }
      if (!in) slot = -1;
    }
  }
  if (tab || legt || stage) __syncthreads();
  if (jt >= p.ntgt) return;
  const int64_t b = p.tbox[jt];
  const int64_t cb = compact_box(p.gmap, b);   // storage index
  if (cb < 0) return;   // (targets lie in stored groups) no barriers below
  double cd[3];
  box_centre(b, p.x0, p.y0, p.z0, p.wb, cd);
  // target position relative to the box centre, formed in FP64
  const T xc[3] = {T(0), T(0), T(0)};
  const T xf[3] = {(T)(p.tx[jt] - cd[0]), (T)(p.ty[jt] - cd[1]),
                   (T)(p.tz[jt] - cd[2])};
  const uint32_t o = p.tperm[jt];
  // the staged copy, or (a CTA whose targets span more boxes) null
  const T* mine = STAGE && slot >= 0 ? cst + (size_t)slot * nc * wc : nullptr;
  if (HELM) {
    auto coef = [&](int idx, T* re, T* im) {
      if (STAGE && mine) { *re = mine[2 * idx]; *im = mine[2 * idx + 1]; return; }
      int64_t off = layout_off(cb, idx, nc);
      *re = p.mpr[2 * off]; *im = p.mpr[2 * off + 1];
    };
    auto eval = [&](const auto& leg) {
      if (p.grad) {
        T g[6] = {T(0), T(0), T(0), T(0), T(0), T(0)}, f[2] = {T(0), T(0)};
        T* fp = p.pot ? f : nullptr;
        if (tab) {
          RecTab<T> rt{st, st + (N + 3) * W, W, M0};
          l2p_helmholtz_grad<T>(N, p.k, xc, xf, coef, g, fp, rt, leg, sc);
        } else {
          l2p_helmholtz_grad<T>(N, p.k, xc, xf, coef, g, fp, RecDirect<T>(), leg, sc);
        }
        for (int c = 0; c < 6; c++) p.grad[6 * (size_t)o + c] = g[c];
        if (p.pot) { p.pot[2 * (size_t)o] = f[0]; p.pot[2 * (size_t)o + 1] = f[1]; }
      } else if (p.pot) {
        T fr = T(0), fi = T(0);
        l2p_helmholtz<T>(N, p.k, xc, xf, coef, &fr, &fi, leg, sc);
        p.pot[2 * (size_t)o] = fr; p.pot[2 * (size_t)o + 1] = fi;
      }
    };
    if (legt) eval(LegTab<T>{lt, LW}); else eval(LegDirect<T>());
  } else {
    auto coef = [&](int idx) -> T {
      return STAGE && mine ? mine[idx] : p.mpr[layout_off(cb, idx, nc)];
    };
    auto eval = [&](const auto& leg) {
      if (p.grad) {
        T g[3] = {T(0), T(0), T(0)}, f = T(0);
        T* fp = p.pot ? &f : nullptr;
        if (tab) {
          LapRecTab<T> rt{st, N + 1};
          l2p_laplace_grad<T>(N, xc, xf, coef, g, fp, rt, leg, sc);
        } else {
          l2p_laplace_grad<T>(N, xc, xf, coef, g, fp, LapRecDirect<T>(), leg, sc);
        }
        for (int c = 0; c < 3; c++) p.grad[3 * (size_t)o + c] = g[c];
        if (p.pot) p.pot[o] = f;
      } else if (p.pot) {
        p.pot[o] = l2p_laplace<T>(N, xc, xf, coef, leg, sc);
      }
    };
    if (legt) eval(LegTab<T>{lt, LW}); else eval(LegDirect<T>());
  }
}

template <typename T, bool HELM>
int launch_l2p(const EvalParams<T>& p, cudaStream_t s) {
  if (p.ntgt <= 0) return 0;
  const size_t sm = l2p_table_bytes<T, HELM>(p.N);
  const size_t lg = leg_table_bytes<T>(p.N);
  const size_t rows = l2p_row_bytes<T>(p.N, HELM, p.grad != nullptr, 128);
  const unsigned grid = (unsigned)((p.ntgt + 127) / 128);
  // staged leaf expansions: up to kL2PBoxes per CTA within 32 KB
  const size_t cb = (size_t)kL2PBoxes * ncoef(p.N) * (HELM ? 2 : 1) * sizeof(T);
  const int stage = cb <= 32 * 1024 ? 1 : 0;
  auto go = [&](auto srows, auto stg) -> int {
    constexpr bool SR = decltype(srows)::value, ST = decltype(stg)::value;
    const size_t bytes = sm + lg + (SR ? rows : 0) + (ST ? cb : 0);
    if (bytes > 48 * 1024) WBFMM_SMEM(bytes, k_l2p<T, HELM, SR, ST>);
    k_l2p<T, HELM, SR, ST><<<grid, 128, bytes, s>>>(p, sm ? 1 : 0, lg ? 1 : 0);
    return 0;
  };
  // the serving orders' Laplace leaf evaluation: rows in registers (the
  // Helmholtz one, unrolled, needs 170-255 registers and runs slower)
  constexpr bool kFixedOk = !HELM;
  if (kFixedOk && p.N == kFixedOrder) {
    if constexpr (kFixedOk) {
      auto fixed = [&](auto stg) -> int {
        constexpr bool ST = decltype(stg)::value;
        const size_t bytes = sm + lg + (ST ? cb : 0);
        if (bytes > 48 * 1024) WBFMM_SMEM(bytes, k_l2p<T, HELM, false, ST, kFixedOrder>);
        k_l2p<T, HELM, false, ST, kFixedOrder><<<grid, 128, bytes, s>>>(p, sm ? 1 : 0, lg ? 1 : 0);
        return 0;
      };
      WBFMM_TRY_K(stage ? fixed(std::true_type()) : fixed(std::false_type()));
    }
  } else if (rows <= kRowSmemMax) {
    WBFMM_TRY_K(stage ? go(std::true_type(), std::true_type()) : go(std::true_type(), std::false_type()));
  } else {
    WBFMM_TRY_K(stage ? go(std::false_type(), std::true_type()) : go(std::false_type(), std::false_type()));
  }
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------ instantiations
#define WBFMM_INST(T, H)                                                      \
  template int p2m_lanes<T, H>(int, int64_t, int64_t);                       \
  template int launch_p2m<T, H>(const P2MParams<T>&, cudaStream_t);          \
  template int launch_l2p<T, H>(const EvalParams<T>&, cudaStream_t);
WBFMM_INST(double, true)
WBFMM_INST(double, false)
WBFMM_INST(float, true)
WBFMM_INST(float, false)

}  // namespace wbfmm
