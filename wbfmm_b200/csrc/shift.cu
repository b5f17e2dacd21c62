// Warp translation kernels: M2M, L2L and the warp-per-source M2L.
//
//  M2M  one CTA per parent; warps take the eight children.
//  M2L  one CTA per target box (optionally split over several CTAs); warps
//       take the list-4 sources (src/indexing.c:330-377) and run the
//       rotate / coaxial / rotate-back sequence in shared memory,
//       accumulating per warp; the warps' partial sums are added in a
//       fixed order.
//  L2L  one CTA per parent; one warp per child.
#include <cuda_runtime.h>

#include <type_traits>

#include "engine.h"
#include "expand.cuh"
#include "kernels.h"
#include "translate.cuh"

namespace wbfmm {

// |d|^2 of the 15 list-4 distances (src/shift.c:709-723), device copy
__constant__ int c_list_dist2[15] = {4, 5, 6, 8, 9, 10, 11, 12, 13, 14,
                                     17, 18, 19, 22, 27};

// ----------------------------------------------------- translation core
// vector length (complex entries) for order N
template <bool HELM>
__host__ __device__ __forceinline__ int vlen(int N) {
  return HELM ? (N + 1) * (N + 1) : nhalf(N);
}

// load a Layout-L box vector into a shared complex vector
template <typename T, bool HELM>
__device__ __forceinline__ void load_vec(T* v, const T* arr, int64_t b, int N,
                                         int nc, int lane) {
  if (HELM) {
    for (int c = lane; c < (N + 1) * (N + 1); c += 32) {
      int64_t o = layout_off(b, c, nc);
      v[2 * c] = arr[2 * o]; v[2 * c + 1] = arr[2 * o + 1];
    }
  } else {
    for (int c = lane; c < nhalf(N); c += 32) {
      int n = half_degree(c), m = c - n * (n + 1) / 2;
      if (m == 0) {
        v[2 * c] = arr[layout_off(b, n * n, nc)];
        v[2 * c + 1] = T(0);
      } else {
        int id = lidx(n, m);
        v[2 * c] = arr[layout_off(b, id, nc)];
        v[2 * c + 1] = arr[layout_off(b, id + 1, nc)];
      }
    }
  }
}

// out[b] (+)= v  (Layout L), all lanes of the caller cooperate
template <typename T, bool HELM, bool ACC>
__device__ __forceinline__ void store_vec(T* arr, int64_t b, int N, int nc,
                                          const T* v, int tid, int nt) {
  if (HELM) {
    for (int c = tid; c < (N + 1) * (N + 1); c += nt) {
      int64_t o = layout_off(b, c, nc);
      if (ACC) { arr[2 * o] += v[2 * c]; arr[2 * o + 1] += v[2 * c + 1]; }
      else { arr[2 * o] = v[2 * c]; arr[2 * o + 1] = v[2 * c + 1]; }
    }
  } else {
    for (int c = tid; c < nhalf(N); c += nt) {
      int n = half_degree(c), m = c - n * (n + 1) / 2;
      if (m == 0) {
        int64_t o = layout_off(b, n * n, nc);
        if (ACC) arr[o] += v[2 * c]; else arr[o] = v[2 * c];
      } else {
        int id = lidx(n, m);
        int64_t o0 = layout_off(b, id, nc), o1 = layout_off(b, id + 1, nc);
        if (ACC) { arr[o0] += v[2 * c]; arr[o1] += v[2 * c + 1]; }
        else { arr[o0] = v[2 * c]; arr[o1] = v[2 * c + 1]; }
      }
    }
  }
}

// A holds the input vector (order Nin).  Runs rotate -> coaxial -> rotate
// back for shift operator `op`; result added to (ACC) or written into out.
// kind: Laplace coaxial kind (0 S|R, 1 S|S, 2 R|R); Helmholtz: CPLX table
// for M2L (S|R), real for M2M/L2L.
template <typename T, bool HELM, bool CPLX, bool ACC>
__device__ void shift_vec(T* A, T* B, T* out, int Nin, int Nout, int op,
                          const OpTables<T>& t, const T* coax, const T* tp,
                          int kind, int lane) {
  const T* H = t.H + (int64_t)t.op_ith[op] * t.hstride;
  const T* eph = t.ph + (size_t)op * (t.lmax + 1) * 2;
  const T* ech = t.ch + (size_t)op * (t.lmax + 1) * 2;
  if (HELM) {
    phase_full(A, Nin, ech, lane, 32);
    __syncwarp();
    hsum_full<T, T, false>(B, A, Nin, H, eph, lane, 32);
    __syncwarp();
    coax_full<T, T, CPLX>(A, B, Nout, Nin, coax, lane, 32);
    __syncwarp();
    phase_full(A, Nout, eph, lane, 32);
    __syncwarp();
    hsum_full<T, T, ACC>(out, A, Nout, H, ech, lane, 32);
    __syncwarp();
  } else {
    phase_half(A, Nin, ech, lane, 32);
    __syncwarp();
    hsum_half<T, T, false>(B, A, Nin, H, eph, lane, 32);
    __syncwarp();
    coax_half<T, T>(A, B, Nout, Nin,
                    kind == 0 ? t.lapSR : (kind == 1 ? t.lapSS : t.lapRR),
                    t.lt, tp, kind, lane, 32);
    __syncwarp();
    phase_half(A, Nout, eph, lane, 32);
    __syncwarp();
    hsum_half<T, T, ACC>(out, A, Nout, H, ech, lane, 32);
    __syncwarp();
  }
}

// shared memory per warp: three vectors of the larger order
template <bool HELM>
static size_t warp_smem_bytes(int Nmax, size_t tsize) {
  return tsize * 2 * 3 * (size_t)vlen<HELM>(Nmax);
}

// ------------------------------------------------------------------- M2L
template <typename T, bool HELM>
__global__ void k_m2l(XlateParams<T> p, OpTables<T> t) {
  extern __shared__ unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const int Ns = p.Nin, Nr = p.Nout, Lm = Ns > Nr ? Ns : Nr;
  const int V = vlen<HELM>(Lm);
  T* A = (T*)smraw + (size_t)warp * 6 * V;
  T* B = A + 2 * V;
  T* acc = B + 2 * V;
  T* tpow = (T*)smraw + (size_t)nw * 6 * V;   // Laplace: [15][Ns+Nr+2] of (2^e t)^j
  const int tpn = Ns + Nr + 2;
  const int64_t tb = blockIdx.x / p.nsplit;
  const int split = blockIdx.x % p.nsplit;
  const int outlen = vlen<HELM>(Nr);
  for (int c = lane; c < 2 * outlen; c += 32) acc[c] = T(0);
  if (!HELM) {
    for (int di = threadIdx.x; di < 15; di += blockDim.x) {
      // sources enter scaled by 2^(e l) and results leave scaled by
      // 2^(e (n+1)), so S|R / (2^e t)^(n+l+1) stays in range
      T r = scale2(p.width * (T)sqrt((double)c_list_dist2[di]), p.lap_e);
      T* tp = tpow + di * tpn;
      tp[0] = T(1);
      for (int j = 1; j < tpn; j++) tp[j] = r * tp[j - 1];
    }
  }
  __syncthreads();
  const bool active = !(p.tmask && !p.tmask[tb]);
  if (active) {
    uint32_t i, j, k;
    demorton((uint64_t)tb, &i, &j, &k);
    const int nside = 1 << p.level;
    int i0 = (int)(i - i % 2), j0 = (int)(j - j % 2), k0 = (int)(k - k % 2);
    int i1 = min(i0 + 3, nside - 1), j1 = min(j0 + 3, nside - 1),
        k1 = min(k0 + 3, nside - 1);
    if (i0 > 0) i0 -= 2;
    if (j0 > 0) j0 -= 2;
    if (k0 > 0) k0 -= 2;
    const int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
    const int total = ni * nj * nk;
    const int ncs = ncoef(Ns);
    for (int e = split * nw + warp; e < total; e += p.nsplit * nw) {
      int ii = i0 + e / (nj * nk), jj = j0 + (e / nk) % nj, kk = k0 + e % nk;
      int dx = ii - (int)i, dy = jj - (int)j, dz = kk - (int)k;
      if (dx >= -1 && dx <= 1 && dy >= -1 && dy <= 1 && dz >= -1 && dz <= 1)
        continue;
      uint64_t s = morton((uint32_t)ii, (uint32_t)jj, (uint32_t)kk);
      if (p.src_n && p.src_n[s] == 0) continue;
      const int op = (dx + 3) * 49 + (dy + 3) * 7 + dz + 3;
      const int di = t.op_dist[op];
      load_vec<T, HELM>(A, p.cin, (int64_t)s, Ns, ncs, lane);
      if (!HELM) {
        for (int c = lane; c < nhalf(Ns); c += 32) {
          const int n = half_degree(c);
          A[2 * c] = scale2(A[2 * c], p.lap_e * n);
          A[2 * c + 1] = scale2(A[2 * c + 1], p.lap_e * n);
        }
      }
      __syncwarp();
      shift_vec<T, HELM, true, true>(A, B, acc, Ns, Nr, op, t,
                                     HELM ? p.coax + di * p.coax_stride : nullptr,
                                     HELM ? nullptr : tpow + di * tpn, 0, lane);
    }
  }
  __syncthreads();
  // fixed-order sum of the warps' partial results
  const T* acc0 = (T*)smraw + 4 * V;
  const int ncr = ncoef(Nr);
  if (p.nsplit == 1) {
    if (!active) return;
    T* red = A;   // reuse warp 0's first vector as the reduction buffer
    __syncthreads();
    for (int c = threadIdx.x; c < 2 * outlen; c += blockDim.x) {
      T v = acc0[c];
      for (int w = 1; w < nw; w++) v += acc0[(size_t)w * 6 * V + c];
      if (!HELM) v = scale2(v, p.lap_e * (half_degree(c >> 1) + 1));
      ((T*)smraw)[c] = v;
    }
    __syncthreads();
    store_vec<T, HELM, true>(p.cout, tb, Nr, ncr, (T*)smraw, threadIdx.x,
                             blockDim.x);
    (void)red;
  } else {
    T* part = p.partial + ((size_t)split * p.nbox + tb) * 2 * outlen;
    for (int c = threadIdx.x; c < 2 * outlen; c += blockDim.x) {
      T v = acc0[c];
      for (int w = 1; w < nw; w++) v += acc0[(size_t)w * 6 * V + c];
      if (!HELM) v = scale2(v, p.lap_e * (half_degree(c >> 1) + 1));
      part[c] = v;
    }
  }
}

// adds the split partial sums, in split order, into cout
template <typename T, bool HELM>
__global__ void k_m2l_reduce(XlateParams<T> p) {
  const int64_t tb = blockIdx.x;
  if (p.tmask && !p.tmask[tb]) return;
  extern __shared__ unsigned char smraw[];
  T* v = (T*)smraw;
  const int Nr = p.Nout, outlen = vlen<HELM>(Nr);
  for (int c = threadIdx.x; c < 2 * outlen; c += blockDim.x) {
    T s = T(0);
    for (int sp = 0; sp < p.nsplit; sp++)
      s += p.partial[((size_t)sp * p.nbox + tb) * 2 * outlen + c];
    v[c] = s;
  }
  __syncthreads();
  store_vec<T, HELM, true>(p.cout, tb, Nr, ncoef(Nr), v, threadIdx.x,
                           blockDim.x);
}

static int pick_warps(size_t per_warp, size_t extra, int want) {
  const size_t cap = 200 * 1024;
  int nw = want;
  while (nw > 1 && per_warp * nw + extra > cap) nw--;
  return nw;
}

template <typename T, bool HELM>
int launch_m2l(const XlateParams<T>& p, const OpTables<T>& t, cudaStream_t s) {
  const int Lm = p.Nin > p.Nout ? p.Nin : p.Nout;
  const size_t per = warp_smem_bytes<HELM>(Lm, sizeof(T));
  const size_t extra = HELM ? 0 : sizeof(T) * 15 * (p.Nin + p.Nout + 2);
  const int nw = pick_warps(per, extra, 4);
  const size_t smem = per * nw + extra;
  if (smem > 227 * 1024) return set_error(-3, "M2L: expansion order too large for shared memory");
  WBFMM_SMEM(smem, k_m2l<T, HELM>);
  unsigned grid = (unsigned)(p.nbox * p.nsplit);
  k_m2l<T, HELM><<<grid, nw * 32, smem, s>>>(p, t);
  WBFMM_CUDA(cudaGetLastError());
  if (p.nsplit > 1) {
    size_t rs = sizeof(T) * 2 * vlen<HELM>(p.Nout);
    if (rs > 48 * 1024)
      WBFMM_SMEM(rs, k_m2l_reduce<T, HELM>);
    k_m2l_reduce<T, HELM><<<(unsigned)p.nbox, 256, rs, s>>>(p);
    WBFMM_CUDA(cudaGetLastError());
  }
  return 0;
}

// ------------------------------------------------------------------- M2M
// parents at `level-1` receive the shifted expansions of their children at
// `level`; p.nbox = number of parents, p.width = child box width
template <typename T, bool HELM>
__global__ void k_m2m(XlateParams<T> p, OpTables<T> t) {
  extern __shared__ unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const int Nc = p.Nin, Np = p.Nout, Lm = Nc > Np ? Nc : Np;
  const int V = vlen<HELM>(Lm);
  T* A = (T*)smraw + (size_t)warp * 6 * V;
  T* B = A + 2 * V;
  T* acc = B + 2 * V;
  T* tp = (T*)smraw + (size_t)nw * 6 * V;
  const int tpn = Nc + Np + 2;
  // the children's group (dense: the parent box); the parent's storage index
  const int64_t P = blockIdx.x;
  const int64_t Pout = p.glist ? compact_box(p.gmap, (int64_t)p.glist[P]) : P;
  if (Pout < 0) return;   // (a stored group's parent is stored) whole CTA, before any barrier
  const int outlen = vlen<HELM>(Np);
  if (p.src_n && p.src_n[p.glist ? (int64_t)p.glist[P] : P] == 0) {
    // no sources below: zeros (whole CTA, before any barrier)
    for (int c = threadIdx.x; c < 2 * outlen; c += blockDim.x) ((T*)smraw)[c] = T(0);
    __syncthreads();
    store_vec<T, HELM, false>(p.cout, Pout, Np, ncoef(Np), (T*)smraw, threadIdx.x, blockDim.x);
    return;
  }
  for (int c = lane; c < 2 * outlen; c += 32) acc[c] = T(0);
  if (!HELM && threadIdx.x == 0) {
    T r = p.width * (T)t.op_r[kOpM2M];
    tp[0] = T(1);
    for (int j = 1; j < tpn; j++) tp[j] = r * tp[j - 1];
  }
  __syncthreads();
  const int ncc = ncoef(Nc);
  for (int ch = warp; ch < 8; ch += nw) {
    int64_t c = 8 * P + ch;
    load_vec<T, HELM>(A, p.cin, c, Nc, ncc, lane);
    __syncwarp();
    shift_vec<T, HELM, false, true>(A, B, acc, Nc, Np, kOpM2M + ch, t, p.coax,
                                    tp, 1, lane);
  }
  __syncthreads();
  const T* acc0 = (T*)smraw + 4 * V;
  T* red = (T*)smraw;
  for (int c = threadIdx.x; c < 2 * outlen; c += blockDim.x) {
    T v = acc0[c];
    for (int w = 1; w < nw; w++) v += acc0[(size_t)w * 6 * V + c];
    red[c] = v;   // entries c of warp 0's A are read only by this thread
  }
  __syncthreads();
  store_vec<T, HELM, false>(p.cout, Pout, Np, ncoef(Np), red, threadIdx.x,
                            blockDim.x);
}

template <typename T, bool HELM>
int launch_m2m(const XlateParams<T>& p, const OpTables<T>& t, cudaStream_t s) {
  const int Lm = p.Nin > p.Nout ? p.Nin : p.Nout;
  const size_t per = warp_smem_bytes<HELM>(Lm, sizeof(T));
  const size_t extra = sizeof(T) * (p.Nin + p.Nout + 2);
  const int nw = pick_warps(per, extra, 8);
  const size_t smem = per * nw + extra;
  if (smem > 227 * 1024) return set_error(-3, "M2M: expansion order too large for shared memory");
  WBFMM_SMEM(smem, k_m2m<T, HELM>);
  k_m2m<T, HELM><<<(unsigned)p.nbox, nw * 32, smem, s>>>(p, t);
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------------- L2L
// children at `level+1` receive (overwrite) the shifted expansion of their
// parent at `level`; p.nbox = number of parents, p.width = child width
template <typename T, bool HELM>
__global__ void k_l2l(XlateParams<T> p, OpTables<T> t) {
  extern __shared__ unsigned char smraw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = blockDim.x >> 5;
  const int Np = p.Nin, Nc = p.Nout, Lm = Nc > Np ? Nc : Np;
  const int V = vlen<HELM>(Lm);
  T* A = (T*)smraw + (size_t)warp * 6 * V;
  T* B = A + 2 * V;
  T* out = B + 2 * V;
  T* tp = (T*)smraw + (size_t)nw * 6 * V;
  const int tpn = Nc + Np + 2;
  // the children's group (dense: the parent box); the parent's storage index
  const int64_t P = blockIdx.x;
  const int64_t Pin = p.glist ? compact_box(p.gmap, (int64_t)p.glist[P]) : P;
  if (Pin < 0) return;    // (a stored group's parent is stored) whole CTA, before any barrier
  if (p.tmask && !p.tmask[p.glist ? (int64_t)p.glist[P] : P]) {
    // no targets below: zeros (whole CTA, before any barrier)
    const int64_t len = (int64_t)8 * ncoef(Nc) * (HELM ? 2 : 1);
    for (int64_t c = threadIdx.x; c < len; c += blockDim.x) p.cout[P * len + c] = T(0);
    return;
  }
  if (!HELM && threadIdx.x == 0) {
    T r = p.width * (T)t.op_r[kOpL2L];
    tp[0] = T(1);
    for (int j = 1; j < tpn; j++) tp[j] = r * tp[j - 1];
  }
  __syncthreads();
  const int ncp = ncoef(Np), ncc = ncoef(Nc);
  for (int ch = warp; ch < 8; ch += nw) {
    load_vec<T, HELM>(A, p.cin, Pin, Np, ncp, lane);
    __syncwarp();
    shift_vec<T, HELM, false, false>(A, B, out, Np, Nc, kOpL2L + ch, t, p.coax,
                                     tp, 2, lane);
    store_vec<T, HELM, false>(p.cout, 8 * P + ch, Nc, ncc, out, lane, 32);
    __syncwarp();
  }
}

template <typename T, bool HELM>
int launch_l2l(const XlateParams<T>& p, const OpTables<T>& t, cudaStream_t s) {
  const int Lm = p.Nin > p.Nout ? p.Nin : p.Nout;
  const size_t per = warp_smem_bytes<HELM>(Lm, sizeof(T));
  const size_t extra = sizeof(T) * (p.Nin + p.Nout + 2);
  const int nw = pick_warps(per, extra, 8);
  const size_t smem = per * nw + extra;
  if (smem > 227 * 1024) return set_error(-3, "L2L: expansion order too large for shared memory");
  WBFMM_SMEM(smem, k_l2l<T, HELM>);
  k_l2l<T, HELM><<<(unsigned)p.nbox, nw * 32, smem, s>>>(p, t);
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------ instantiations
#define WBFMM_INST(T, H)                                                      \
  template int launch_m2m<T, H>(const XlateParams<T>&, const OpTables<T>&,   \
                                cudaStream_t);                               \
  template int launch_m2l<T, H>(const XlateParams<T>&, const OpTables<T>&,   \
                                cudaStream_t);                               \
  template int launch_l2l<T, H>(const XlateParams<T>&, const OpTables<T>&,   \
                                cudaStream_t);
WBFMM_INST(double, true)
WBFMM_INST(double, false)
WBFMM_INST(float, true)
WBFMM_INST(float, false)

}  // namespace wbfmm
