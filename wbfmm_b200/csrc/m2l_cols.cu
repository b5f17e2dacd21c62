// M2L for orders up to kColsMaxOrder: register-blocked matrix products on
// columns of target boxes.
//
// As in the tile kernel (m2l_tiles.cu), the list-4 interactions of a level
// are regrouped by target child type, so that a CTA's target boxes (the
// children of one type of consecutive parents) see the same 189 offsets,
// each with one rotate / coaxial / rotate-back operator (src/pass.c:56-105).
// What differs is the basis the vectors are kept in, and the blocking.
//
// Basis.  Write H for the rotation block of a degree, H(nu, -m) = H(-nu, m),
// and X_m for the phased source e^{i m ch} S_m.  In the even and odd parts
//   E_m = (X_m + X_-m) / 2 (E_0 = X_0),   O_m = (X_m - X_-m) / 2,  m >= 0,
// the rotation splits into two real blocks over m, nu >= 0,
//   E'_nu = H(nu,0) E_0 + sum_{m>0} (H(nu,m) + H(nu,-m)) E_m
//   O'_nu =               sum_{m>0} (H(nu,m) - H(nu,-m)) O_m,
// half the products of the full block.  The coaxial translation depends on
// |m| only, so it acts on E and O alike, and the phases e^{-i nu ph} after
// the forward rotation and e^{i m ph} before the back rotation cancel (the
// translation is diagonal in m): no phase is applied between the rotations.
// The source phase e^{i m ch} and the target phase e^{-i nu ch} mix E and O;
// with O'' = -i O in O's place (and S'' = -i S-, S+- the even and odd parts of
// the source, formed once per level by k_cols_planes) they do so with real
// factors,
//   E = c S+ - s S'',  O'' = c S'' + s S+   and   T+ += c E + s O'', T'' += c O'' - s E,
// T+ and T'' the sums over the offsets, turned into (nu, -nu) once at the end.
// Laplace's half vectors have this form with E the real and O'' the imaginary
// parts.
//
// Blocking.  A column is a pair of numbers: a Helmholtz target's complex
// value, or the real values of two Laplace targets.  Each of the (P+1)^2
// rows (E: m = 0..n, O: m = 1..n of every degree) holds the CTA's NC columns.
// All three stages are products of a real table (rows x k) with such rows,
// cut into tiles of up to 16 rows that are dealt to the warps in order of
// cost, forwards and backwards in turn.  The Helmholtz coaxial table is
// complex: its real and imaginary parts are two tables whose products are
// combined at the end.
//   FP64: tensor cores (mma.m8n8k4 f64, IEEE arithmetic), tables stored in
// fragment order.  A warp tile is 1 or 2 x 8 rows by 8 or 16 columns; an mma
// is one issued instruction for 8 multiply-adds per lane, 36.8 TFLOP/s from
// one warp per scheduler on (scalar FP64: 33.1 with 16 warps per SM, and it
// reads 96 bytes of shared memory per lane for 16 multiply-adds, the mma tile
// 48 for 64).
//   FP32: packed multiply-adds (fma.rn.f32x2), the lanes as 4 x 8 with R rows
// x CPL columns each in registers, so that one step over k reads R table
// values and CPL columns for 2 R CPL multiply-adds.
//
// Pipeline.  Two row buffers and the sums: the rotation reads buffer a and
// writes b, the coaxial stage reads b and writes a, the back rotation reads
// a and adds to the sums; during it the next offset's source rows (cp.async)
// and coaxial table arrive in b's place.  The offsets are taken in the order
// of rotation angle and distance, so that consecutive ones share tables.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "f32x2.cuh"
#include "kernels.h"
#include "m2l_lanes.h"
#include "tables.h"
#include "translate.cuh"

namespace wbfmm {

namespace {

template <typename T> struct P2;
template <> struct P2<float> { typedef float2 t; };
template <> struct P2<double> { typedef double2 t; };

HD int pad4(int n) { return (n + 3) & ~3; }
// Table rows in warp tiles of 16: the rows rl, rl + 4, ... of the lanes of row
// group rl, R = 1..4 of them (from the tile's row count), in one aligned word
// of 1, 2, 4 or 4 values.  Slots of `rows` rows, and the slot of row r
HD int tile_R(int rows) { return rows >= 16 ? 4 : (rows + 3) / 4; }
HD int word(int R) { return R == 3 ? 4 : R; }
HD int slots(int rows) { return (rows & ~15) + 4 * word(tile_R(rows & 15)); }
HD int slot(int rows, int r) {
  const int R = tile_R(rows - (r & ~15)), i = r & 15;
  return (r & ~15) + (i & 3) * word(R) + (i >> 2);
}
HD int ksteps(int K) { return (K + 3) / 4; }
// values of a rows x K table, and the place of (r, k) in it: FP32 k-major in
// slots (storing every value twice, as the packed multiply-adds take it, saved
// their moves but read more shared memory: 1.62 -> 1.76 ms on 4096 boxes of
// order 14); FP64 fragments of 8 rows x 4 k (lane 4 (r & 7) + (k & 3)), the k
// steps of 8 rows in turn
template <typename T>
HD int tab_size(int rows, int K) {
  return sizeof(T) == 4 ? K * slots(rows) : (rows + 7) / 8 * ksteps(K) * 32;
}
template <typename T>
HD int tab_at(int rows, int K, int r, int k) {
  return sizeof(T) == 4 ? k * slots(rows) + slot(rows, r)
                        : ((r >> 3) * ksteps(K) + (k >> 2)) * 32 + (r & 7) * 4 + (k & 3);
}
// first value of the tile at row r0 (a multiple of 16)
template <typename T>
HD int tab_tile(int K, int r0) { return sizeof(T) == 4 ? r0 : r0 / 8 * ksteps(K) * 32; }
// rows of the even / odd parts of (n, m)
HD int e_row(int n, int m) { return n * (n + 1) / 2 + m; }
HD int o_base(int P) { return (P + 1) * (P + 2) / 2; }
HD int o_row(int P, int n, int m) { return o_base(P) + n * (n - 1) / 2 + m - 1; }   // m >= 1
// rotation tables: per degree the even block (k = m = 0..n) then the odd one
// (k = m - 1), rows nu = 0..n; offset of degree n
template <typename T>
HD int he_off(int n) {
  int s = 0;
  for (int i = 0; i < n; i++) s += tab_size<T>(i + 1, i + 1) + tab_size<T>(i + 1, i);
  return s;
}
// coaxial tables: per order m, k = l - m, rows n - m (Helmholtz: the real
// parts then the imaginary ones); offset of order m
template <typename T, bool HELM>
HD int cx_off(int P, int m) {
  int s = 0;
  for (int i = 0; i < m; i++) s += tab_size<T>(P + 1 - i, P + 1 - i) * (HELM ? 2 : 1);
  return s;
}

// one warp tile of a stage
struct __align__(16) ColsTask {
  int h, x, K, rh;      // table offset, first input row, steps, rows | (n + m) & 3 of
                        // the first input << 8 and output row << 10 | column share << 12
  int y, lo, step, ld;  // output row, first valid row / degree, input row step, table slots
};

struct ColsPlan {
  int P, V, ncol, nhe, ncx, nB, nC, nD;
  size_t buf, total;
};

// shares that a stage's tiles cut the columns into: FP64 16 columns each, FP32
// all; half of that in the back rotation, whose tiles hold the even and odd
// sums at once
template <typename T>
HD int col_parts(int ncol, int stage) {
  if (ncol <= 8) return 1;
  return (stage == 2 ? 2 : 1) * (sizeof(T) == 8 ? ncol / 16 : 1);
}

// the tiles of a stage (0 rotation, 1 coaxial, 2 back rotation) in the order
// of enumeration: the number of them, or (e >= 0) task e into *t and its cost
template <typename T, bool HELM>
HD int cols_tasks(int P, int stage, int ncol, int e, ColsTask* t, int* cost) {
  const int parts = col_parts<T>(ncol, stage);
  int c = 0;
  if (stage == 1) {
    for (int m = 0; m <= P; m++) {
      const int len = P + 1 - m;
      for (int v = 0; v < (m > 0 ? 2 : 1) * parts; v++)
        for (int r0 = 0; r0 < len; r0 += 16, c++) {
          if (c != e) continue;
          const int odd = v / parts;
          const int rows = len - r0 < 16 ? len - r0 : 16;
          t->h = cx_off<T, HELM>(P, m) + tab_tile<T>(len, r0);
          t->x = odd ? o_row(P, m, m) : e_row(m, m);
          t->K = len;
          t->rh = rows | (2 * m & 3) << 8 | (2 * m & 3) << 10 | v % parts << 12;
          t->y = odd ? o_base(P) + m - 1 : m;    // + n (n +- 1) / 2
          t->lo = (m + r0) | odd << 16;
          t->step = odd ? m : m + 1;             // row(l + 1, m) - row(l, m) at l = m
          t->ld = sizeof(T) == 4 ? slots(len) : tab_size<T>(len, len);
          *cost = len * ((rows + 3) / 4);
        }
    }
    return c;
  }
  for (int n = P; n >= 0; n--) {
    for (int v = 0; v < (stage == 2 || n == 0 ? 1 : 2) * parts; v++)
      for (int r0 = 0; r0 <= n; r0 += 16, c++) {
        if (c != e) continue;
        const int rows = n + 1 - r0 < 16 ? n + 1 - r0 : 16;
        const int odd = v / parts;
        t->K = odd ? n : n + 1;
        t->h = he_off<T>(n) + (odd ? tab_size<T>(n + 1, n + 1) : 0) + tab_tile<T>(t->K, r0);
        t->x = odd ? o_row(P, n, 1) : e_row(n, 0);
        t->rh = rows | ((n + odd) & 3) << 8 | (n & 3) << 10 | v % parts << 12;
        t->y = odd ? o_row(P, n, 1) + r0 - 1 : e_row(n, r0);
        t->ld = slots(n + 1);                    // (FP32)
        if (stage == 0) {
          t->lo = odd && r0 == 0 ? 1 : 0;
          t->step = 1;
        } else {
          // the odd table of the same rows, from the even one's tile
          t->ld = sizeof(T) == 4 ? slots(n + 1)
                                 : tab_size<T>(n + 1, n + 1) - tab_tile<T>(n + 1, r0) + tab_tile<T>(n, r0);
          t->lo = r0;
          t->step = o_row(P, n, 1);              // the odd rows
        }
        *cost = t->K * ((rows + 3) / 4);
      }
  }
  return c;
}

template <typename T, bool HELM>
ColsPlan cols_plan(int P, int ncol) {
  ColsPlan q;
  q.P = P;
  q.V = (P + 1) * (P + 1);
  q.ncol = ncol;
  q.nhe = he_off<T>(P + 1);
  q.ncx = cx_off<T, HELM>(P, P + 1);
  q.nB = cols_tasks<T, HELM>(P, 0, ncol, -1, nullptr, nullptr);
  q.nC = cols_tasks<T, HELM>(P, 1, ncol, -1, nullptr, nullptr);
  q.nD = cols_tasks<T, HELM>(P, 2, ncol, -1, nullptr, nullptr);
  q.buf = (size_t)q.V * ncol;
  const size_t NE = (size_t)o_base(P);
  q.total = 3 * q.buf * 2 * sizeof(T) + sizeof(T) * ((size_t)q.nhe + q.ncx + 4 * pad4(P + 1)) +
            sizeof(ColsTask) * (q.nB + q.nC + q.nD) + 8 * 192 + 2 * 192 + 2 * 4 * 64 +
            2 * ((NE + 7) & ~(size_t)7) + 16;
  return q;
}

constexpr size_t kColsSmemCap = 227 * 1024;

// columns per lane: the most whose rows fit (fewer table reads per product).
// ms on 4096 boxes with them and with half of them, which two CTAs per SM may
// then hold: FP32 Helmholtz p = 8 0.63 / 0.81, p = 14 1.60 / 2.17, Laplace
// p = 10 0.44 / 0.54, p = 14 0.85 / 0.91; FP64 Helmholtz p = 8 1.25 / 1.30,
// p = 10 1.77 / 1.94, Laplace p = 10 0.90 / 0.94; half are faster at FP64 p = 7
// (1.04 / 0.93), p = 12 (2.71 / 2.40) and Laplace p = 9 (0.75 / 0.69) only.
// Level 2 has 8 targets of a type, which 8 columns hold (Laplace FP32 order 14:
// 0.155 ms with 32 columns, 28 of them idle)
template <typename T, bool HELM>
int cols_cpl(int P, int level) {
  if (P < 2 || P > kColsMaxOrder) return 0;
  for (int c = level <= 2 ? 1 : 4; c >= 1; c /= 2)
    if (cols_plan<T, HELM>(P, 8 * c).total <= kColsSmemCap) return c;
  return 0;
}

// CTAs per SM that a launch is compiled for: 2 (8 warps each, 128 registers
// per thread) where two share an SM's shared memory, else 1 (12 warps, 168)
int cols_ctas(size_t smem) { return 2 * (smem + 1024) <= 228 * 1024 ? 2 : 1; }

// per target type: the 189 offsets ordered by rotation angle, then distance:
// the packed code of build_offset_table | distance index << 18 | angle << 22
__constant__ int c_cols_offsets[8][189];
DeviceOnce g_cols_offsets;

int ensure_cols_offsets() {
  return g_cols_offsets.run([] {
    int tab[8 * 189];
    build_offset_table(tab);
    ShiftGeometry g;
    build_shift_geometry(&g);
    for (int tau = 0; tau < 8; tau++) {
      int* o = tab + tau * 189;
      for (int j = 0; j < 189; j++) {
        const ShiftAngles& a = g.offset[o[j] & 511];
        o[j] |= list_dist_index(a.idist) << 18 | a.ith << 22;
      }
      std::stable_sort(o, o + 189, [](int a, int b) { return (a >> 18) < (b >> 18); });
      std::stable_sort(o, o + 189, [](int a, int b) { return (a >> 22) < (b >> 22); });
    }
    WBFMM_CUDA(cudaMemcpyToSymbol(c_cols_offsets, tab, sizeof(tab)));
    return 0;
  });
}

__constant__ int c_cols_dist2[15] = {4, 5, 6, 8, 9, 10, 11, 12, 13, 14, 17, 18, 19, 22, 27};

// Per level: the 15 distances' coaxial tables (block x = distance, y = order)
// and, in block (15, 0), the stages' tiles sorted by falling cost.
template <typename T, bool HELM>
__global__ void k_cols_prep(LanesParams<T> p, OpTables<T> t, int nB, int nC, int nD, int ncx, int ncol,
                            T* __restrict__ cx, ColsTask* __restrict__ tasks) {
  const int P = p.N;
  if (blockIdx.x == 15) {
    if (blockIdx.y) return;
    __shared__ int s_cost[256];
    const int cnt[3] = {nB, nC, nD};
    int base = 0;
    for (int st = 0; st < 3; st++) {
      ColsTask tk;
      int cost = 0;
      const int e = threadIdx.x;
      if (e < cnt[st]) {
        cols_tasks<T, HELM>(P, st, ncol, e, &tk, &cost);
        s_cost[e] = cost;
      }
      __syncthreads();
      if (e < cnt[st]) {
        int rank = 0;
        for (int i = 0; i < cnt[st]; i++)
          if (s_cost[i] > cost || (s_cost[i] == cost && i < e)) rank++;
        tasks[base + rank] = tk;
      }
      __syncthreads();
      base += cnt[st];
    }
    return;
  }
  const int d = blockIdx.x, m = blockIdx.y, len = P + 1 - m, sz = tab_size<T>(len, len);
  T* o = cx + (int64_t)d * ncx + cx_off<T, HELM>(P, m);
  for (int e = threadIdx.x; e < sz * (HELM ? 2 : 1); e += blockDim.x) o[e] = T(0);
  __syncthreads();
  for (int e = threadIdx.x; e < len * len; e += blockDim.x) {
    const int k = e / len, i = e - k * len, at = tab_at<T>(len, len, i, k), l = m + k, n = m + i;
    if (HELM) {
      const T* c = p.coax + (int64_t)d * p.coax_stride;
      const int ic = l >= n ? coax_idx(l, m, n) : coax_idx(n, m, l);
      const T sg = (l >= n || ((n + l) & 1) == 0) ? T(1) : T(-1);
      o[at] = sg * c[2 * ic];
      o[sz + at] = sg * c[2 * ic + 1];
    } else {
      // S|R(n, l, m) / (r^(n+1) (2^e r)^l) on sources scaled by 2^(e l)
      const T r = p.width * (T)sqrt((double)c_cols_dist2[d]);
      const T rinv = T(1) / r, qinv = T(1) / scale2(r, p.lap_e);
      T sc = rinv, q = T(1);
      for (int j = 0; j < n; j++) sc *= rinv;
      for (int j = 0; j < l; j++) q *= qinv;
      const int D = t.lt + 1;
      o[at] = (t.lapSR[((int64_t)n * D + l) * D + m] * q) * sc;
    }
  }
}

// rotation tables in even / odd blocks: block (angle, degree)
template <typename T>
__global__ void k_cols_rotations(const double* __restrict__ H, int64_t hstride,
                                 T* __restrict__ he, int64_t hestride) {
  const int n = blockIdx.y, se = tab_size<T>(n + 1, n + 1), so = tab_size<T>(n + 1, n);
  const double* h = H + (int64_t)blockIdx.x * hstride;
  T* o = he + (int64_t)blockIdx.x * hestride + he_off<T>(n);
  for (int e = threadIdx.x; e < se + so; e += blockDim.x) o[e] = T(0);
  __syncthreads();
  for (int e = threadIdx.x; e < (2 * n + 1) * (n + 1); e += blockDim.x) {
    const int k = e / (n + 1), nu = e - k * (n + 1), m = k <= n ? k : k - n;
    const double a = h[rot_idx(nu, m, n)], b = h[rot_idx(-nu, m, n)];
    if (k <= n) o[tab_at<T>(n + 1, n + 1, nu, k)] = (T)(m ? a + b : a);
    else o[se + tab_at<T>(n + 1, n, nu, k - n - 1)] = (T)(nu ? a - b : 0.0);
  }
}

// Layout L level array -> rows lin[tau][row][column], S+ and S'' (Laplace:
// the real and imaginary parts) of degree n scaled by 2^(scale_e n).
// Columns: the padded parent grid (zeros on the padding), or with sparse
// storage the stored groups and a zero column (groups >= 0).  A thread takes
// one (n, m >= 0) of one parent: its eight children are consecutive values.
template <typename T, bool HELM>
__global__ void k_cols_planes(const T* __restrict__ arr, int level, int N, int scale_e,
                              int64_t groups, int64_t ncols, bool boxmajor,
                              const uint32_t* __restrict__ src_n, T* __restrict__ lin) {
  typedef typename P2<T>::t T2;
  const int64_t pp = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pp >= ncols) return;
  const int pr = blockIdx.y, n = half_degree(pr), m = pr - n * (n + 1) / 2;
  const int V = (N + 1) * (N + 1), nc = V;
  bool in;
  int64_t P;
  if (groups >= 0) {
    in = pp < groups;
    P = pp;
  } else {
    const int nx = 1 << (level - 1), npx = nx + 2;
    const int px = (int)(pp % npx) - 1, py = (int)((pp / npx) % npx) - 1,
              pz = (int)(pp / ((int64_t)npx * npx)) - 1;
    in = px >= 0 && px < nx && py >= 0 && py < nx && pz >= 0 && pz < nx;
    P = in ? (int64_t)morton(px, py, pz) : 0;
  }
  const int er = e_row(n, m), orow = m ? o_row(N, n, m) : 0;
  const int se = scale_e * n;
  // row and column steps of lin, and the type's start
  const int64_t rs = boxmajor ? 1 : ncols, first = boxmajor ? pp * V : pp;
#pragma unroll
  for (int tau = 0; tau < 8; tau++) {
    if (src_n && !(in && src_n[(P << 3) | tau])) continue;   // never read
    if (HELM) {
      T2 a, b;
      a.x = a.y = b.x = b.y = T(0);
      if (in) {
        const T* u = arr + 2 * ((P * nc + cidx(n, m)) * 8 + tau);
        a.x = u[0]; a.y = u[1];
        if (m) {
          u = arr + 2 * ((P * nc + cidx(n, -m)) * 8 + tau);
          b.x = u[0]; b.y = u[1];
        }
      }
      const T h = m ? T(0.5) : T(1);
      T2* o = (T2*)lin + (int64_t)tau * V * ncols + first;
      T2 s;
      s.x = scale2(h * (a.x + b.x), se); s.y = scale2(h * (a.y + b.y), se);
      o[er * rs] = s;
      if (m) {
        // -i (a - b) / 2
        s.x = scale2(h * (a.y - b.y), se); s.y = -scale2(h * (a.x - b.x), se);
        o[orow * rs] = s;
      }
    } else {
      T a = T(0), b = T(0);
      if (in) {
        a = arr[(P * nc + (m ? lidx(n, m) : n * n)) * 8 + tau];
        if (m) b = arr[(P * nc + lidx(n, m) + 1) * 8 + tau];
      }
      T* o = lin + (int64_t)tau * V * ncols + first;
      o[er * rs] = scale2(a, se);
      if (m) o[orow * rs] = scale2(b, se);
    }
  }
}

// ------------------------------------------------------ shared-memory access
// asynchronous global -> shared copy of B bytes (zeros when !on)
template <int B>
__device__ __forceinline__ void cpa(void* dst, const void* src, bool on) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = on ? B : 0;
  if constexpr (B == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n));
  else if constexpr (B == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(n));
}
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// A column value as the multiply-adds take it: FP32 pairs packed in 64 bits
// (fma.rn.f32x2: both numbers in one instruction, halving the issue slots
// the products take), FP64 pairs as double2.
template <typename T> struct Col;
template <> struct Col<float> { typedef f32x2 t; };
template <> struct Col<double> { typedef double2 t; };
using wbfmm::both;
__device__ __forceinline__ double both(double h) { return h; }
__device__ __forceinline__ void mac(f32x2& a, f32x2 h, f32x2 x) { a = fma2(h, x, a); }
__device__ __forceinline__ void mac(double2& a, double h, const double2& x) {
  a.x = fma(h, x.x, a.x);
  a.y = fma(h, x.y, a.y);
}
__device__ __forceinline__ f32x2 mul(f32x2 h, f32x2 x) { return mul2(h, x); }
__device__ __forceinline__ double2 mul(double h, const double2& x) {
  return make_double2(h * x.x, h * x.y);
}
// where column col of a row with (n + m) & 3 = g stands in the row's NC:
// FP32 rows of odd g hold their 64-byte halves exchanged, FP64 rows their
// 32-byte quarters in the order j ^ g and, for odd g, each quarter's two
// columns exchanged, so that neighbouring rows (n, m),
// (n, m + 1) or (n, m), (n + 1, m) read or written by one access do not meet
// in the same banks
template <typename T2, int NC>
__device__ __forceinline__ int swz(int col, int g) {
  if constexpr (sizeof(T2) == 16) return col ^ ((g & 3) << 1 | (g & 1));
  else if constexpr (NC >= 16) return col ^ ((g & 1) << 3);
  return col;
}

// FP32 lanes: row group rl = bits 0 and 4, column group cl = bits 1..3.  A
// warp's 16-byte shared load takes 2 cycles where every two neighbouring
// lanes read the same word or every second lane does, 4 where four neighbours
// differ (measured: words indexed by lane bits 1..3 or by bits 0 and 4: 2.00
// cycles, by bits 0..2: 4.00): so both the column and the table reads take 2.
// A row's first column of the lane (c0: first of the tile's share); its CPL
// columns: two neighbours (and two 16 further)
template <int CPL, int NC>
__device__ __forceinline__ int lane_col(int cl, int c0, int g) {
  return swz<float2, NC>(c0 + (CPL > 1 ? 2 : 1) * cl, g);
}
template <int CPL>
__device__ __forceinline__ void ldx(const float2* x, f32x2 (&v)[CPL]) {
  if constexpr (CPL == 1) {
    v[0] = *reinterpret_cast<const f32x2*>(x);
  } else {
#pragma unroll
    for (int c = 0; c < CPL; c += 2) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(x + 8 * c);
      v[c] = a.x;
      v[c + 1] = a.y;
    }
  }
}
template <int CPL>
__device__ __forceinline__ void stx(float2* x, const f32x2 (&v)[CPL]) {
  if constexpr (CPL == 1) {
    *reinterpret_cast<f32x2*>(x) = v[0];
  } else {
#pragma unroll
    for (int c = 0; c < CPL; c += 2)
      *reinterpret_cast<ulonglong2*>(x + 8 * c) = make_ulonglong2(v[c], v[c + 1]);
  }
}
// table values of the lane's R rows (one aligned word, h the lane's)
template <int R>
__device__ __forceinline__ void ldh(const float* h, f32x2 (&v)[R]) {
  if constexpr (R >= 3) {
    const float4 a = *reinterpret_cast<const float4*>(h);
    v[0] = both(a.x); v[1] = both(a.y); v[2] = both(a.z);
    if constexpr (R == 4) v[3] = both(a.w);
  } else if constexpr (R == 2) {
    const float2 a = *reinterpret_cast<const float2*>(h);
    v[0] = both(a.x); v[1] = both(a.y);
  } else {
    v[0] = both(h[0]);
  }
}

// acc[j][i][c] += sum_k h_jk[row i] x_k[column c]; consecutive k: table step
// ld, input rows step + k dstep columns apart, their columns at o0 and o1 in
// turn (lane_col); tables j = 0..N-1, hn apart
template <int N, int R, int CPL>
__device__ __forceinline__ void mm(f32x2 (&acc)[N][R][CPL], const float* h, int hn, int ld,
                                   const float2* x, int step, int dstep, int K, int o0, int o1) {
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int c = 0; c < CPL; c++) acc[j][i][c] = 0;
  auto one = [&](int o) {
    f32x2 hv[N][R], xv[CPL];
    ldx<CPL>(x + o, xv);
#pragma unroll
    for (int j = 0; j < N; j++) ldh<R>(h + j * hn, hv[j]);
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int i = 0; i < R; i++)
#pragma unroll
        for (int c = 0; c < CPL; c++) mac(acc[j][i][c], hv[j][i], xv[c]);
    h += ld;
    x += step;
    step += dstep;
  };
#pragma unroll 1
  for (int k = 1; k < K; k += 2) {
    one(o0);
    one(o1);
  }
  if (K & 1) one(o0);
}

// T+ += c E + s O'', T'' += c O'' - s E
template <typename C, typename H>
__device__ __forceinline__ void turn(C& w, const C& u, const C& v, H c, H s) {
  mac(w, c, u);
  mac(w, s, v);
}

template <int R, int CPL>
__device__ __forceinline__ void rotate_tile(const ColsTask& k, const float* sH, const float2* in,
                                            float2* out, int rl, int cl) {
  constexpr int NC = 8 * CPL;
  f32x2 acc[1][R][CPL];
  const int g = k.rh >> 8, gy = k.rh >> 10, hi = k.rh & 255;
  mm(acc, sH + k.h + rl * word(R), 0, k.ld, in + k.x * NC, NC, 0, k.K, lane_col<CPL, NC>(cl, 0, g),
     lane_col<CPL, NC>(cl, 0, g ^ 1));
  // the lane's rows 4 i + rl are of one parity
  float2* o = out + (k.y + rl) * NC + lane_col<CPL, NC>(cl, 0, gy + rl);
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int r = 4 * i + rl;
    if (r >= k.lo && r < hi) stx<CPL>(o + 4 * i * NC, acc[0][i]);
  }
}

template <int R, int CPL, bool HELM>
__device__ __forceinline__ void coaxial_tile(const ColsTask& k, const float* sC, const float2* in,
                                             float2* out, int rl, int cl) {
  constexpr int NC = 8 * CPL, N = HELM ? 2 : 1;
  f32x2 acc[N][R][CPL];
  mm(acc, sC + k.h + rl * word(R), k.K * k.ld, k.ld, in + k.x * NC, k.step * NC, NC, k.K,
     lane_col<CPL, NC>(cl, 0, 0), lane_col<CPL, NC>(cl, 0, 1));
  if constexpr (HELM) {       // (re + i im) x
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
      for (int c = 0; c < CPL; c++) {
        float2 u = pair(acc[0][i][c]);
        const float2 v = pair(acc[1][i][c]);
        u.x -= v.y;
        u.y += v.x;
        acc[0][i][c] = packed(u);
      }
  }
  const int hi = k.rh & 255, n0 = k.lo & 0xffff, s = k.lo >> 16 ? -1 : 1;
  float2* o = out + lane_col<CPL, NC>(cl, 0, rl);
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int r = 4 * i + rl, n = n0 + r;
    if (r < hi) stx<CPL>(o + (k.y + n * (n + s) / 2) * NC, acc[0][i]);
  }
}

// CPL: the columns per lane of this tile's share of the NC columns
template <int R, int CPL, int NC>
__device__ __forceinline__ void back_tile(const ColsTask& k, const float* sH, const float* ech,
                                          const float2* in, float2* A, int rl, int cl) {
  f32x2 e[1][R][CPL], o[1][R][CPL];
  const int c0 = (k.rh >> 12) * 8 * CPL, r0 = k.lo, hi = k.rh & 255;
  const int g = k.rh >> 8, gy = k.rh >> 10;
  const int oe = lane_col<CPL, NC>(cl, c0, g), oo = lane_col<CPL, NC>(cl, c0, g ^ 1);
  const float* h = sH + k.h + rl * word(R);
  mm(e, h, 0, k.ld, in + k.x * NC, NC, 0, k.K, oe, oo);
  mm(o, h + k.K * k.ld, 0, k.ld, in + k.step * NC, NC, 0, k.K - 1, oo, oe);
  float2* a0 = A + lane_col<CPL, NC>(cl, c0, gy + rl);
#pragma unroll
  for (int i = 0; i < R; i++) {
    const int r = 4 * i + rl, nu = r0 + r;
    if (r >= hi) continue;
    const f32x2 c = both(ech[2 * nu]), s = both(ech[2 * nu + 1]), ms = both(-ech[2 * nu + 1]);
    float2* ae = a0 + (k.y + r) * NC;
    float2* ao = a0 + (k.step + nu - 1) * NC;
    f32x2 a[CPL];
    ldx<CPL>(ae, a);
#pragma unroll
    for (int j = 0; j < CPL; j++) turn(a[j], e[0][i][j], o[0][i][j], c, s);
    stx<CPL>(ae, a);
    if (nu == 0) continue;
    ldx<CPL>(ao, a);
#pragma unroll
    for (int j = 0; j < CPL; j++) turn(a[j], o[0][i][j], e[0][i][j], c, ms);
    stx<CPL>(ao, a);
  }
}

// FP64 warp tile: MT x 8 rows by CB x 8 columns.  Lane: k = lane & 3 and
// column (or table row) lane >> 2 of the operands; an mma takes the first or
// second numbers of eight columns, so that its results, row lane >> 2 and
// columns 2 (lane & 3), + 1, make whole columns: acc[j][mt][cb][first /
// second][column].
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
// Input rows: that of k < K is x0 + k (step 0), or row0 + k l + k (k + s) / 2
// for the coaxial stage's rows (l + k, m), l = m; a lane advances by 4 of them
// per step, its place within the row unchanged, and the last step's padding
// (zeros of the table) reads row K - 1.
template <int N, int MT, int CB, int NC, bool COAX>
__device__ __forceinline__ void mmd(double (&acc)[N][MT][CB][2][2], const double* h, int hn,
                                    const double2* in, int c0, int g0, int x0, int m, int s, int K,
                                    int lane) {
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int t = 0; t < MT; t++)
#pragma unroll
      for (int b = 0; b < CB; b++)
#pragma unroll
        for (int e = 0; e < 2; e++) acc[j][t][b][e][0] = acc[j][t][b][e][1] = 0.0;
  const int ks = ksteps(K), q = lane & 3;
  // row of k relative to the first
  auto at = [&](int k) { return COAX ? k * m + (k * (k + s) >> 1) : k; };
  const int kl = 4 * (ks - 1) + q < K ? 4 * (ks - 1) + q : K - 1;
  const int col = c0 + (lane >> 2);
  const double2* x = in + (x0 + at(q)) * NC + swz<double2, NC>(col, g0 + q);
  const double2* xl = in + (x0 + at(kl)) * NC + swz<double2, NC>(col, g0 + kl);
  int hop = COAX ? (4 * (m + q) + 8 + 2 * s) * NC : 4 * NC;
  h += lane;
  auto step = [&](const double2* xp) {
    double2 xv[CB];
    double hv[N][MT];
#pragma unroll
    for (int b = 0; b < CB; b++) xv[b] = xp[8 * b];
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int t = 0; t < MT; t++) hv[j][t] = h[j * hn + t * ks * 32];
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int t = 0; t < MT; t++)
#pragma unroll
        for (int b = 0; b < CB; b++) {
          dmma(acc[j][t][b][0], hv[j][t], xv[b].x);
          dmma(acc[j][t][b][1], hv[j][t], xv[b].y);
        }
    h += 32;
  };
  for (int i = 1; i < ks; i++) {
    step(x);
    x += hop;
    if (COAX) hop += 16 * NC;
  }
  if (ks > 0) step(xl);
}

// the lane's column v (0, 1) of 8-column block b as (first, second)
template <int CB>
__device__ __forceinline__ double2 result(const double (&a)[CB][2][2], int b, int v) {
  return make_double2(a[b][0][v], a[b][1][v]);
}

// CB x 8 columns: the tile's share of the NC
template <int MT, int CB, int NC>
__device__ __forceinline__ void rotate_tile_d(const ColsTask& k, const double* sH,
                                              const double2* in, double2* out, int lane) {
  double acc[1][MT][CB][2][2];
  const int c0 = (k.rh >> 12) * 8 * CB;
  mmd<1, MT, CB, NC, false>(acc, sH + k.h, 0, in, c0, k.rh >> 8, k.x, 0, 0, k.K, lane);
  const int hi = k.rh & 255;
#pragma unroll
  for (int t = 0; t < MT; t++) {
    const int r = 8 * t + (lane >> 2);
    if (r < k.lo || r >= hi) continue;
    const int col = swz<double2, NC>(c0 + 2 * (lane & 3), (k.rh >> 10) + r);
    double2* o = out + (k.y + r) * NC;
#pragma unroll
    for (int b = 0; b < CB; b++)
#pragma unroll
      for (int v = 0; v < 2; v++) o[8 * b + (col ^ v)] = result(acc[0][t], b, v);
  }
}

template <int MT, int CB, int NC, bool HELM>
__device__ __forceinline__ void coaxial_tile_d(const ColsTask& k, int P, const double* sC,
                                               const double2* in, double2* out, int lane) {
  constexpr int N = HELM ? 2 : 1;
  double acc[N][MT][CB][2][2];
  const int c0 = (k.rh >> 12) * 8 * CB, s = k.lo >> 16 ? -1 : 1, m = P + 1 - k.K;
  mmd<N, MT, CB, NC, true>(acc, sC + k.h, k.ld, in, c0, k.rh >> 8, k.x, m, s, k.K, lane);
  const int hi = k.rh & 255, n0 = k.lo & 0xffff;
#pragma unroll
  for (int t = 0; t < MT; t++) {
    const int r = 8 * t + (lane >> 2), n = n0 + r;
    if (r >= hi) continue;
    const int col = swz<double2, NC>(c0 + 2 * (lane & 3), (k.rh >> 10) + r);
    double2* o = out + (k.y + n * (n + s) / 2) * NC;
#pragma unroll
    for (int b = 0; b < CB; b++)
#pragma unroll
      for (int v = 0; v < 2; v++) {
        double2 w = result(acc[0][t], b, v);
        if constexpr (HELM) {   // (re + i im) x
          const double2 z = result(acc[1][t], b, v);
          w.x -= z.y;
          w.y += z.x;
        }
        o[8 * b + (col ^ v)] = w;
      }
  }
}

template <int MT, int CB, int NC>
__device__ __forceinline__ void back_tile_d(const ColsTask& k, const double* sH, const double* ech,
                                            const double2* in, double2* A, int lane) {
  double e[1][MT][CB][2][2], o[1][MT][CB][2][2];
  const int c0 = (k.rh >> 12) * 8 * CB, r0 = k.lo, hi = k.rh & 255;
  const double* h = sH + k.h;
  mmd<1, MT, CB, NC, false>(e, h, 0, in, c0, k.rh >> 8, k.x, 0, 0, k.K, lane);
  mmd<1, MT, CB, NC, false>(o, h + k.ld, 0, in, c0, (k.rh >> 8) + 1, k.step, 0, 0, k.K - 1, lane);
#pragma unroll
  for (int t = 0; t < MT; t++) {
    const int r = 8 * t + (lane >> 2), nu = r0 + r;
    if (r >= hi) continue;
    const double c = ech[2 * nu], s = ech[2 * nu + 1];
    const int col = swz<double2, NC>(c0 + 2 * (lane & 3), (k.rh >> 10) + r);
    double2* ae = A + (k.y + r) * NC;
    double2* ao = A + (k.step + nu - 1) * NC;
#pragma unroll
    for (int b = 0; b < CB; b++)
#pragma unroll
      for (int v = 0; v < 2; v++) {
        const double2 x = result(e[0][t], b, v), y = result(o[0][t], b, v);
        const int at = 8 * b + (col ^ v);
        double2 w = ae[at];
        turn(w, x, y, c, s);
        ae[at] = w;
        if (nu == 0) continue;
        w = ao[at];
        turn(w, y, x, c, -s);
        ao[at] = w;
      }
  }
}

// ------------------------------------------------------------------ kernel
template <typename T, bool HELM, int CPL, int NTHR, int MINB>
__global__ void __launch_bounds__(NTHR, MINB)
k_m2l_cols(LanesParams<T> p, OpTables<T> t, ColsPlan q, const T* __restrict__ cx,
           const ColsTask* __restrict__ tasks) {
  typedef typename P2<T>::t T2;
  constexpr int NC = 8 * CPL, TG = HELM ? NC : 2 * NC;   // columns, targets
  constexpr int DC = CPL > 1 ? CPL / 2 : 1;   // FP32: columns per lane in the back rotation
  constexpr int CB = NC >= 16 ? 2 : 1;        // FP64: 8-column blocks of a tile's share
  extern __shared__ __align__(16) unsigned char smraw[];
  const int P = q.P, V = q.V, NE = o_base(P);
  T2* buf0 = (T2*)smraw;
  T2* A = buf0 + 2 * q.buf;
  T* sH = (T*)(A + q.buf);
  T* sC = sH + q.nhe;
  T* sE = sC + q.ncx;                         // phases of the offset and the next
  const int eb = 2 * pad4(P + 1);
  ColsTask* sT = (ColsTask*)(sE + 2 * eb);
  unsigned long long* s_mask = (unsigned long long*)(sT + q.nB + q.nC + q.nD);
  int* s_pp = (int*)(s_mask + 192);           // padded-grid index of each target's parent
  int* s_act = s_pp + 64;                     // 1 + parent linear index, 0: no target
  unsigned short* s_list = (unsigned short*)(s_act + 64);
  unsigned short* s_om = s_list + 192;        // (n, m) of each odd row
  int* s_cnt = (int*)(s_om + ((NE + 7) & ~7));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int nth = NTHR, W = NTHR / 32;
  const int rl = (lane & 1) | (lane >> 4) << 1, cl = (lane >> 1) & 7;

  const int tau = blockIdx.x & 7, split = blockIdx.z;
  const int nx = 1 << (p.level - 1), npx = nx + 2;
  const int64_t npp = (int64_t)npx * npx * npx;
  const int64_t np = (int64_t)nx * nx * nx;
  const int64_t lstride = p.pmap ? p.lin_stride : npp;
  const int64_t base = (int64_t)(blockIdx.x >> 3) * TG;
  const int64_t nlist = p.act ? (int64_t)p.act_n[tau] : np;
  if (base >= nlist) return;                  // the whole CTA, before any barrier

  for (int i = tid; i < TG; i += nth) {
    int64_t plin = base + i;
    int act = plin < nlist;
    int pp = 0;
    if (act) {
      if (p.act) plin = p.act[(int64_t)tau * np + plin];
      const int px = (int)(plin % nx), py = (int)((plin / nx) % nx), pz = (int)(plin / ((int64_t)nx * nx));
      pp = (px + 1) + npx * ((py + 1) + npx * (pz + 1));
      if (!p.act && p.tmask && !p.tmask[((int64_t)morton(px, py, pz) << 3) | tau]) act = 0;
    }
    s_pp[i] = pp;
    s_act[i] = act ? (int)plin + 1 : 0;
  }
  for (int i = tid; i < q.nB + q.nC + q.nD; i += nth) sT[i] = tasks[i];
  for (int i = tid; i < V - NE; i += nth) {
    const int n = half_degree(i) + 1;         // i = n (n - 1) / 2 + m - 1
    s_om[i] = (unsigned short)(n | (i - n * (n - 1) / 2 + 1) << 8);
  }
  for (int i = tid; i < (int)q.buf; i += nth) { T2 z; z.x = z.y = T(0); A[i] = z; }
  __syncthreads();
  // this CTA's offsets, and which of its targets have a source there
  const int j0 = split * 189 / p.nsplit, j1 = (split + 1) * 189 / p.nsplit;
  auto parent_off = [&](int code) {
    const int ddx = ((code >> 12) & 3) - 1, ddy = ((code >> 14) & 3) - 1, ddz = ((code >> 16) & 3) - 1;
    return ddx + npx * (ddy + npx * ddz);
  };
  for (int j = j0 + warp; j < j1; j += W) {
    const int code = c_cols_offsets[tau][j], sg = (code >> 9) & 7;
    const int ddx = ((code >> 12) & 3) - 1, ddy = ((code >> 14) & 3) - 1, ddz = ((code >> 16) & 3) - 1;
    unsigned long long mask = 0;
#pragma unroll
    for (int h = 0; h < (TG + 31) / 32; h++) {
      const int i = h * 32 + lane;
      int f = 0;
      if (i < TG && s_act[i]) {
        const int pp = s_pp[i];
        if (p.smask) {
          f = p.smask[(int64_t)sg * npp + pp + parent_off(code)];
        } else {
          const int sx = pp % npx + ddx, sy = (pp / npx) % npx + ddy, sz = pp / (npx * npx) + ddz;
          f = sx >= 1 && sx <= nx && sy >= 1 && sy <= nx && sz >= 1 && sz <= nx;
        }
      }
      mask |= (unsigned long long)__ballot_sync(0xffffffffu, f) << (32 * h);
    }
    if (lane == 0) s_mask[j - j0] = mask;
  }
  __syncthreads();
  if (warp == 0) {
    int cnt = 0;
    for (int b = 0; b < j1 - j0; b += 32) {
      const int j = b + lane;
      const bool on = j < j1 - j0 && s_mask[j] != 0;
      const unsigned bal = __ballot_sync(0xffffffffu, on);
      if (on) s_list[cnt + __popc(bal & ((1u << lane) - 1u))] = (unsigned short)j;
      cnt += __popc(bal);
    }
    if (lane == 0) *s_cnt = cnt;
  }
  __syncthreads();
  const int cnt = *s_cnt;

  // the thread's share of the source rows: column mycol of rows row0,
  // row0 + rstep, ...
  const int mycol = tid & (NC - 1), row0 = tid / NC, rstep = nth / NC;
  unsigned long long gbits = 0;               // (n + m) & 3 of those rows (at most 32)
  for (int r = row0, b = 0; r < V; r += rstep, b += 2) {
    int g;
    if (r < NE) {
      const int n = half_degree(r);
      g = n + r - n * (n + 1) / 2;
    } else {
      const int i = r - NE, n = half_degree(i) + 1;
      g = n + i - n * (n - 1) / 2 + 1;
    }
    gbits |= (unsigned long long)(g & 3) << b;
  }
  auto gather = [&](int j, T2* dst, T* ech) {
    const int code = c_cols_offsets[tau][j0 + j], sg = (code >> 9) & 7, op = code & 511;
    const unsigned long long mask = s_mask[j];
    const int doff = parent_off(code);
    const T* ph = t.ch + (size_t)op * (t.lmax + 1) * 2;
    for (int i = tid; i < 2 * (P + 1); i += nth) cpa<sizeof(T)>(ech + i, ph + i, true);
    auto column = [&](int i) -> int64_t {
      const int64_t c = (int64_t)s_pp[i] + doff;
      return p.pmap ? (int64_t)p.pmap[c] : c;
    };
    const int64_t hop = (int64_t)rstep * lstride;
    T2* d = dst + row0 * NC;
    unsigned long long gb = gbits;
    if (HELM) {
      const bool on = (mask >> mycol) & 1;
      const T2* s0 = (const T2*)p.lin_raw + ((int64_t)sg * V + row0) * lstride + (on ? column(mycol) : 0);
#pragma unroll 4
      for (int r = row0; r < V; r += rstep, d += rstep * NC, s0 += hop, gb >>= 2)
        cpa<2 * sizeof(T)>(d + swz<T2, NC>(mycol, (int)gb & 3), s0, on);
    } else {
      const bool on0 = (mask >> mycol) & 1, on1 = (mask >> (mycol + NC)) & 1;
      const T* s = (const T*)p.lin_raw + ((int64_t)sg * V + row0) * lstride;
      const T* s0 = s + (on0 ? column(mycol) : 0);
      const T* s1 = s + (on1 ? column(mycol + NC) : 0);
#pragma unroll 4
      for (int r = row0; r < V; r += rstep, d += rstep * NC, s0 += hop, s1 += hop, gb >>= 2) {
        T* w = (T*)(d + swz<T2, NC>(mycol, (int)gb & 3));
        cpa<sizeof(T)>(w, s0, on0);
        cpa<sizeof(T)>(w + 1, s1, on1);
      }
    }
  };
  auto stage_h = [&](int th) {
    const T* h = t.HE + (int64_t)th * t.hestride;
    constexpr int E = 16 / sizeof(T);
    for (int i = tid * E; i < q.nhe; i += nth * E) cpa<16>(sH + i, h + i, true);
  };
  auto stage_c = [&](int d) {
    const T* c = cx + (int64_t)d * q.ncx;
    constexpr int E = 16 / sizeof(T);
    for (int i = tid * E; i < q.ncx; i += nth * E) cpa<16>(sC + i, c + i, true);
  };
  // the i-th tile of this warp
  auto deal = [&](int i) { return i * W + ((i & 1) ? W - 1 - warp : warp); };

  int th = -1, ds = -1;
  if (cnt > 0) {
    const int code = c_cols_offsets[tau][j0 + s_list[0]];
    th = code >> 22;
    ds = (code >> 18) & 15;
    stage_h(th);
    stage_c(ds);
    gather(s_list[0], buf0, sE);
  }
#pragma unroll 1
  for (int a = 0; a < cnt; a++) {
    T2* in = buf0 + (a & 1) * q.buf;
    T2* out = buf0 + ((a & 1) ^ 1) * q.buf;
    const T* ech = sE + (a & 1) * eb;
    cpa_wait();
    __syncthreads();      // the phases and tables of every thread's copies
    // source phases on the pairs (n, m), (n, -m) of odd row NE + j, four at
    // a time
    for (int j = row0; j < V - NE; j += 4 * rstep) {
      typedef typename Col<T>::t C;
      C *pe[4], *po[4], e[4], o[4];
      T c[4], s[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = j + u * rstep;
        if (k >= V - NE) break;
        const int nm = s_om[k], n = nm & 255, m = nm >> 8;
        const int col = swz<T2, NC>(mycol, n + m);
        pe[u] = (C*)(in + (k + n + 1) * NC + col);
        po[u] = (C*)(in + (NE + k) * NC + col);
        e[u] = *pe[u];
        o[u] = *po[u];
        c[u] = ech[2 * m]; s[u] = ech[2 * m + 1];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int k = j + u * rstep;
        if (k >= V - NE) break;
        C x = mul(both(c[u]), e[u]), y = mul(both(c[u]), o[u]);
        mac(x, both(-s[u]), o[u]);
        mac(y, both(s[u]), e[u]);
        *pe[u] = x;
        *po[u] = y;
      }
    }
    __syncthreads();
    for (int i = 0, k = deal(0); k < q.nB; k = deal(++i)) {
      const ColsTask tk = sT[k];
      const int rows = tk.rh & 255;
      if constexpr (sizeof(T) == 8) {
        if (rows <= 8) rotate_tile_d<1, CB, NC>(tk, sH, in, out, lane);
        else rotate_tile_d<2, CB, NC>(tk, sH, in, out, lane);
      } else if (rows <= 4) rotate_tile<1, CPL>(tk, sH, in, out, rl, cl);
      else if (rows <= 8) rotate_tile<2, CPL>(tk, sH, in, out, rl, cl);
      else if (rows <= 12) rotate_tile<3, CPL>(tk, sH, in, out, rl, cl);
      else rotate_tile<4, CPL>(tk, sH, in, out, rl, cl);
    }
    __syncthreads();
    for (int i = 0, k = deal(0); k < q.nC; k = deal(++i)) {
      const ColsTask tk = sT[q.nB + k];
      const int rows = tk.rh & 255;
      if constexpr (sizeof(T) == 8) {
        if (rows <= 8) coaxial_tile_d<1, CB, NC, HELM>(tk, P, sC, out, in, lane);
        else coaxial_tile_d<2, CB, NC, HELM>(tk, P, sC, out, in, lane);
      } else if (rows <= 4) coaxial_tile<1, CPL, HELM>(tk, sC, out, in, rl, cl);
      else if (rows <= 8) coaxial_tile<2, CPL, HELM>(tk, sC, out, in, rl, cl);
      else if (rows <= 12) coaxial_tile<3, CPL, HELM>(tk, sC, out, in, rl, cl);
      else coaxial_tile<4, CPL, HELM>(tk, sC, out, in, rl, cl);
    }
    __syncthreads();
    // the next offset's rows and coaxial table, behind the back rotation
    int next_th = th;
    if (a + 1 < cnt) {
      const int code = c_cols_offsets[tau][j0 + s_list[a + 1]];
      const int nd = (code >> 18) & 15;
      next_th = code >> 22;
      if (nd != ds) stage_c(nd);
      ds = nd;
      gather(s_list[a + 1], out, sE + ((a & 1) ^ 1) * eb);
    }
    for (int i = 0, k = deal(0); k < q.nD; k = deal(++i)) {
      const ColsTask tk = sT[q.nB + q.nC + k];
      const int rows = tk.rh & 255;
      if constexpr (sizeof(T) == 8) {
        if (rows <= 8) back_tile_d<1, 1, NC>(tk, sH, ech, in, A, lane);
        else back_tile_d<2, 1, NC>(tk, sH, ech, in, A, lane);
      } else if (rows <= 4) back_tile<1, DC, NC>(tk, sH, ech, in, A, rl, cl);
      else if (rows <= 8) back_tile<2, DC, NC>(tk, sH, ech, in, A, rl, cl);
      else if (rows <= 12) back_tile<3, DC, NC>(tk, sH, ech, in, A, rl, cl);
      else back_tile<4, DC, NC>(tk, sH, ech, in, A, rl, cl);
    }
    if (next_th != th) {
      __syncthreads();    // the rotation table is free
      stage_h(next_th);
      th = next_th;
    }
  }
  __syncthreads();
  // results: (n, m) and (n, -m) from the even and odd sums, added into the
  // level array or written to the split partials
  const int nc = (P + 1) * (P + 1);
  const int VP = HELM ? V : NE;               // complex values of a partial
  for (int i = tid; i < NE * TG; i += nth) {
    const int pr = i / TG, tt = i - pr * TG;
    if (!s_act[tt]) continue;
    const int64_t plin = s_act[tt] - 1;
    const int n = half_degree(pr), m = pr - n * (n + 1) / 2;
    T2 u, v;
    u.x = u.y = v.x = v.y = T(0);
    const int col = swz<T2, NC>(tt & (NC - 1), n + m);
    const T2 e = A[pr * NC + col];
    T2 o;
    o.x = o.y = T(0);
    if (m) o = A[(NE + pr - n - 1) * NC + col];
    if (HELM) {
      u.x = e.x - o.y; u.y = e.y + o.x;       // T+ +- i T''
      v.x = e.x + o.y; v.y = e.y - o.x;
      if (p.helm_e) {
        u.x = scale2(u.x, p.helm_e * n); u.y = scale2(u.y, p.helm_e * n);
        v.x = scale2(v.x, p.helm_e * n); v.y = scale2(v.y, p.helm_e * n);
      }
    } else {
      u.x = tt < NC ? e.x : e.y;
      u.y = tt < NC ? o.x : o.y;
    }
    if (p.nsplit > 1) {
      T2* w = (T2*)p.partial_raw + ((int64_t)split * 8 + tau) * VP * np + plin;
      if (HELM) {
        w[(int64_t)cidx(n, m) * np] = u;
        if (m) w[(int64_t)cidx(n, -m) * np] = v;
      } else {
        w[(int64_t)pr * np] = u;
      }
      continue;
    }
    const int px = (int)(plin % nx), py = (int)((plin / nx) % nx), pz = (int)(plin / ((int64_t)nx * nx));
    const int64_t g0 = compact_box(p.gmap, (int64_t)morton(px, py, pz) << 3);
    if (g0 < 0) continue;   // (targets lie in stored groups)
    const int64_t b = g0 | tau;
    if (HELM) {
      T* o = p.cout + 2 * layout_off(b, cidx(n, m), nc);
      o[0] += u.x; o[1] += u.y;
      if (m) {
        o = p.cout + 2 * layout_off(b, cidx(n, -m), nc);
        o[0] += v.x; o[1] += v.y;
      }
    } else if (m == 0) {
      p.cout[layout_off(b, n * n, nc)] += u.x;
    } else {
      p.cout[layout_off(b, lidx(n, m), nc)] += u.x;
      p.cout[layout_off(b, lidx(n, m) + 1, nc)] += u.y;
    }
  }
}

template <typename T, bool HELM, int CPL>
int launch_cols(const LanesParams<T>& p, const OpTables<T>& t, const ColsPlan& q, const T* cx,
                const ColsTask* tasks, cudaStream_t s) {
  const int TG = (HELM ? 1 : 2) * q.ncol;
  const int64_t np = (int64_t)1 << (3 * (p.level - 1));
  dim3 grid((unsigned)(8 * ((np + TG - 1) / TG)), 1, p.nsplit);
  if (cols_ctas(q.total) == 2) {
    WBFMM_SMEM(q.total, k_m2l_cols<T, HELM, CPL, 256, 2>);
    k_m2l_cols<T, HELM, CPL, 256, 2><<<grid, 256, q.total, s>>>(p, t, q, cx, tasks);
  } else {
    WBFMM_SMEM(q.total, k_m2l_cols<T, HELM, CPL, 384, 1>);
    k_m2l_cols<T, HELM, CPL, 384, 1><<<grid, 384, q.total, s>>>(p, t, q, cx, tasks);
  }
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace

template <typename T>
int64_t cols_rotation_stride(int L) { return he_off<T>(std::min(L, kColsMaxOrder) + 1); }
template int64_t cols_rotation_stride<float>(int);
template int64_t cols_rotation_stride<double>(int);

template <typename T>
int build_cols_rotations(const double* H, int64_t hstride, int nth, int L, T* he, cudaStream_t s) {
  const int Lc = std::min(L, kColsMaxOrder);
  k_cols_rotations<T><<<dim3(nth, Lc + 1), 128, 0, s>>>(H, hstride, he, cols_rotation_stride<T>(L));
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}
template int build_cols_rotations<float>(const double*, int64_t, int, int, float*, cudaStream_t);
template int build_cols_rotations<double>(const double*, int64_t, int, int, double*, cudaStream_t);

template <typename T, bool HELM>
bool cols_supported(int Ns, int Nr) {
  return Ns == Nr && cols_cpl<T, HELM>(Ns, 2) > 0;
}

template <typename T, bool HELM>
ColsWork cols_work(int P, int level) {
  const int cpl = cols_cpl<T, HELM>(P, level);
  const ColsPlan q = cols_plan<T, HELM>(P, 8 * cpl);
  ColsWork w;
  w.table = (size_t)15 * q.ncx;
  w.tasks = sizeof(ColsTask) * (q.nB + q.nC + q.nD);
  // CTAs per target tile: the offsets split so that the CTAs fill whole
  // rounds of the SMs, each CTA's start and end costing about two offsets
  const int64_t np = (int64_t)1 << (3 * (level - 1)), tg = (HELM ? 1 : 2) * q.ncol;
  const int64_t ctas = 8 * ((np + tg - 1) / tg);
  const int64_t slots = 148 * cols_ctas(q.total);
  w.nsplit = 1;
  int64_t best = -1;
  for (int ns = 1; ns <= 37 && ctas * (ns - 1) < 8 * slots; ns++) {
    const int64_t c = ((ctas * ns + slots - 1) / slots) * ((189 + ns - 1) / ns + 2);
    if (best < 0 || c < best) { best = c; w.nsplit = ns; }
  }
  return w;
}

template <typename T, bool HELM>
int cols_planes(const T* arr, int level, int N, int scale_e, int64_t groups, void* lin,
                cudaStream_t s, bool boxmajor, const uint32_t* src_n) {
  const int64_t npx = (1 << (level - 1)) + 2;
  const int64_t ncols = groups >= 0 ? groups + 1 : npx * npx * npx;
  k_cols_planes<T, HELM><<<dim3((unsigned)((ncols + 127) / 128), o_base(N)), 128, 0, s>>>(
      arr, level, N, scale_e, groups, ncols, boxmajor, src_n, (T*)lin);
  WBFMM_CUDA(cudaGetLastError());
  return 0;
}

template <typename T, bool HELM>
int launch_m2l_cols(const LanesParams<T>& p, const OpTables<T>& t, T* table, void* tasks,
                    cudaStream_t s) {
  {
    const int rc = ensure_cols_offsets();
    if (rc) return rc;
  }
  const int cpl = cols_cpl<T, HELM>(p.N, p.level);
  if (!cpl || !t.HE) return set_error(-3, "M2L columns: expansion order not supported");
  const ColsPlan q = cols_plan<T, HELM>(p.N, 8 * cpl);
  k_cols_prep<T, HELM><<<dim3(16, p.N + 1), 256, 0, s>>>(p, t, q.nB, q.nC, q.nD, q.ncx,
                                                         q.ncol, table,
                                                         (ColsTask*)tasks);
  WBFMM_CUDA(cudaGetLastError());
  const ColsTask* tk = (const ColsTask*)tasks;
  int rc;
  rc = cpl == 4 ? launch_cols<T, HELM, 4>(p, t, q, table, tk, s)
       : cpl == 2 ? launch_cols<T, HELM, 2>(p, t, q, table, tk, s)
                  : launch_cols<T, HELM, 1>(p, t, q, table, tk, s);
  if (rc) return rc;
  return p.nsplit > 1 ? launch_lanes_reduce<T, HELM>(p, s) : 0;
}

#define WBFMM_COLS_INST(T, H)                                                              \
  template bool cols_supported<T, H>(int, int);                                            \
  template ColsWork cols_work<T, H>(int, int);                                             \
  template int cols_planes<T, H>(const T*, int, int, int, int64_t, void*, cudaStream_t, bool, \
                                 const uint32_t*);                                         \
  template int launch_m2l_cols<T, H>(const LanesParams<T>&, const OpTables<T>&, T*, void*, \
                                     cudaStream_t);
WBFMM_COLS_INST(double, true)
WBFMM_COLS_INST(double, false)
WBFMM_COLS_INST(float, true)
WBFMM_COLS_INST(float, false)

}  // namespace wbfmm
