// Batched factor + solve of many independent systems of uneven order in one
// persistent launch (no reference counterpart: charmlu factors one
// distributed matrix).  Each system is LU with partial pivoting followed by
// forward/backward substitution, the same algorithm as the single-matrix
// path (strict '>' pivot search with the lowest row on ties, true division,
// swaps of whole rows and of b).
//
// Scheduling: a small prep kernel orders the systems by decreasing order
// (counting sort on n) and builds the workspace offsets; the persistent
// kernel's CTAs (one per SM, 512 threads) take systems from an atomic
// queue in that order, so the big systems start first and the small ones
// fill the tail (longest-processing-time-first balance).
//
// Per system (one CTA):
//   n <= small threshold  the whole matrix in shared memory (factor_small)
//   otherwise             two-level blocked LU in global memory (factor_system)
//   then                  blocked forward / backward substitution
// What bounds it: an SM works on one system, phase after phase, so every
// phase's latency counts as much as its arithmetic.  Panels keep their rows in
// registers and rename rows instead of moving them (panel_regs); a panel of an
// outer block is brought up to date as it is loaded; interchanges, U rows and
// trailing update of an outer block go over the matrix together.
// B200, 4096 systems of order 32 .. 1024 (log-uniform): FP64 64.5 -> 39.7 ms,
// FP32 with refinement 71.9 -> 39.6 ms; one system of order 1024 on every SM:
// FP64 14.3 -> 9.4 ms (trailing update 4.6, panels 1.2 + 0.9 for loading and
// storing them, U rows of the outer blocks 1.0, substitution 0.8).  Results are
// bit for bit those of the right-looking form with plain fmas that it
// replaced: every element sees the same fmas and sums in the same order.
//
// LU_PREC_FP32: the FP32 copy of each matrix (workspace) is factored, then
// FP64 refinement (r = b - A x against the FP64 A, FP32 correction solve,
// FP64 update) until the system's scaled residual r_hpl < 16, at most 10
// steps.  One step is not enough at these orders: after one step r_hpl is
// ~1e4 for a uniform n = 109 system (the remaining error lies along the
// small singular directions); two steps bring it to O(1).
#include <climits>
#include <mutex>

#include "argmax.cuh"
#include "common.cuh"
#include "kernels.h"

namespace lub {
namespace {

constexpr int BT = 512;                    // threads per CTA
constexpr int NWARP = BT / 32;
constexpr int kBatchMaxN = 2048;
constexpr size_t kBatchSmem = 200 * 1024;  // dynamic shared memory per CTA
constexpr int kBatchRefineMax = 10;        // FP64 refinement steps at most (FP32 mode)

struct Tuning {
  int n_max, nb, small;
};
__constant__ Tuning c_tuning[16];
__constant__ int c_tuning_n;

struct BatchArgs {
  int count;
  const int* n;
  const int64_t* a_off;
  const int64_t* b_off;
  double* A;
  double* b;
  int* info;
  int precision;  // LU_PREC_FP64 or LU_PREC_FP32
  unsigned char* work;
};

// Workspace header written by the prep kernel (offsets in bytes from work).
constexpr int kRefineHistBins = kBatchRefineMax + 2;  // steps 0 .. 10, then "not converged"
struct WorkHeader {
  unsigned queue;
  int bad;          // nonzero: an order outside [1, kBatchMaxN] or workspace too small
  long long s1, s2; // sum n, sum n^2
  long long order, offA32, offV, A32, r64, total;
  // FP32 mode: systems that reached r_hpl < 16 after s FP64 refinement
  // steps (s = 0 .. 10), and in the last bin those that did not
  int refine_hist[kRefineHistBins];
};
static_assert(sizeof(WorkHeader) <= 256, "workspace header exceeds its 256 bytes");

// Outer block width of the two-level blocking: the inner panels (nb columns)
// are brought up to date inside the outer block as they come up; the rest of
// the trailing matrix gets one update of depth outer_block per outer block.
template <typename T>
constexpr int outer_block() { return sizeof(T) == 8 ? 64 : 128; }

// Dynamic shared memory of factor_system at the panel of columns k0 .. k0 + kw,
// in elements of T: U rows of the outer block's earlier panels from 0 (pitch
// up), the panel (kw columns of pitch mp) at lb, then the panel kernel's rows.
// Before the panel takes its place, L of the earlier panels lies at lb; while it
// is loaded, FP32 stages stage_rows rows of L (pitch kStagePitch) behind it.
// Every pointer of factor_system comes from here, and end is the last element
// that any of them reaches.
constexpr int kStagePitch = 33, kStageMin = 64;
template <typename T>
struct PanelLayout {
  int Kp, kw, m, mp, up, W, lb, rowbuf, urow, zero, stage, stage_rows, end;
  __host__ __device__ PanelLayout(int n, int nb, int k0) {
    constexpr bool f64 = sizeof(T) == 8;
    Kp = k0 % outer_block<T>();
    m = n - k0;
    kw = nb < m ? nb : m;
    mp = m | 1;
    up = f64 ? kw + 2 : kw;
    W = kw <= 8 && f64 ? 8 : (kw <= 16 ? 16 : 32);
    lb = (Kp * up + 3) & ~3;
    rowbuf = lb + ((kw * mp + 3) & ~3);
    urow = rowbuf + (f64 ? 0 : 2 * NWARP * W);
    zero = urow + W * W;
    end = zero + W;
    stage = rowbuf;
    stage_rows = 0;
    if (Kp > 0) {
      const int lt = lb + Kp * (Kp + 4);
      if (lt > end) end = lt;
      if (!f64) {
        // 256 rows, or as many as there is room for
        stage_rows = ((int)(kBatchSmem / sizeof(T)) - stage) / kStagePitch;
        if (stage_rows > 256) stage_rows = 256;
        if (stage_rows < kStageMin) stage_rows = kStageMin;
        if (stage + stage_rows * kStagePitch > end) end = stage + stage_rows * kStagePitch;
      }
    }
  }
};

// Panel width for order n, at most nb.  The first sum sets the orders at which
// the width halves (a panel and 128 columns of it; another line would change the
// order of the sums, and with it the last bits).  The second is what a panel
// needs at least, an upper bound of PanelLayout::end with kStageMin staged rows.
template <typename T>
__host__ __device__ inline int panel_width(int n, int nb) {
  constexpr int NB = outer_block<T>();
  constexpr int cap = (int)(kBatchSmem / sizeof(T));
  while (nb > 4) {
    const int W = nb <= 16 ? 16 : 32, rows = 2 * NWARP * W + W * W + W;
    const int tail = sizeof(T) == 4 && rows < kStageMin * kStagePitch ? kStageMin * kStagePitch : rows;
    if (n * (nb + 1) + nb * 128 <= cap && 2 * NB + nb * (n + 1) + 8 + tail <= cap) break;
    nb >>= 1;
  }
  return nb;
}

template <typename T>
__device__ __forceinline__ void tuning_for(int n, int& nb, int& small) {
  constexpr int esize = (int)sizeof(T);
  nb = esize == 8 ? 16 : 32;
  small = esize == 8 ? 128 : 192;
  for (int i = 0; i < c_tuning_n; i++) {
    if (n <= c_tuning[i].n_max) {
      nb = c_tuning[i].nb;
      small = c_tuning[i].small;
      break;
    }
  }
  // the small path holds n x (n | 1) elements
  const int small_cap = (int)(sqrtf((float)(kBatchSmem / esize)) - 1.f);
  if (small > small_cap) small = small_cap;
  nb = panel_width<T>(n, nb);
}

// Element copy global -> shared through the async copy unit; pred false
// zero-fills the destination (src-size 0: nothing is read).
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* sdst, const void* gsrc, bool pred) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(sdst)), "l"(gsrc), "n"(BYTES),
               "r"(pred ? BYTES : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Shared memory beside the dynamic part.  Row numbers of one system fit 16 bits.
template <typename T>
struct BShared {
  T key[2][NWARP];
  int pos[2][NWARP];
  int mv_n;
  int info;
  unsigned short src[kBatchMaxN];   // panel: row that now stands at each position
  unsigned short ob[kBatchMaxN];    // the same since the outer block began
  unsigned short perm[kBatchMaxN];  // the same since the system began
  unsigned short mv_dst[256], mv_src[256];
  unsigned short to[256];           // outer block: where each row of its old top block stands
  T acc[32];
  alignas(16) T diag[32][33];
};

// mma.sync.m16n8k4.f64 is bit for bit the chain of four fmas in k order
// (checked against the host's fma), so sums over it are those of a scalar loop
__device__ __forceinline__ void dmma_k4(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// LU with partial pivoting of an m x kw panel at lb (column c of row r at
// lb[c * mp + r]), kw <= W, m <= RPT * BT: as the single-matrix leaf, each
// thread holds RPT whole rows in registers and rotates them, an interchange
// renames two rows, the CTA's candidate takes one barrier per column.  On
// return lb holds the multipliers by original row, urow[j][i] = U(j, j + i),
// sh.src[d] = the original row at position d.  Returns the 1-based first
// column without a usable pivot (0: none).  rowbuf: [2][NWARP][W] (FP32 only).
template <typename T, int W, int RPT>
__device__ __noinline__ int panel_regs(T* lb, int mp, int m, int kw, T* rowbuf, T* urow, T* zero, BShared<T>& sh) {
  constexpr int V = 16 / (int)sizeof(T);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  T v[RPT][W];
  int pos[RPT];
#pragma unroll
  for (int u = 0; u < RPT; u++) {
    const int r = tid + u * BT;
    pos[u] = r < m ? r : INT_MIN;
#pragma unroll
    for (int i = 0; i < W; i++) v[u][i] = (r < m && i < kw) ? lb[i * mp + r] : T(0);
  }
  if (tid < W) zero[tid] = T(0);
  int info = 0;
  const int steps = min(kw, m);
#pragma unroll 1
  for (int j = 0; j < steps; j++) {
    const int buf = j & 1;
    T* rows = rowbuf + buf * NWARP * W;
    T bv = 0;
    int bp = -1, bu = 0;
#pragma unroll
    for (int u = 0; u < RPT; u++) {
      const T x = fabs(v[u][0]);
      if (pos[u] >= 0 && (x > bv || (x == bv && bp >= 0 && pos[u] < bp))) {
        bv = x;
        bp = pos[u];
        bu = u;
      }
    }
    const int wl = warp_best(bv, bp >= 0, bp);
    // One lane stores 4 bytes a cycle.  FP64: sixteen candidates' rows would take
    // longer than a second barrier, so only the best row is written, once it
    // is known (4096 systems 41.5 -> 39.7 ms); FP32 rows are half as long and
    // are written ahead (39.6 ms, 40.8 the other way)
    constexpr bool kAheadRows = sizeof(T) == 4;
    auto put_row = [&](T* dst) {
#pragma unroll
      for (int u = 0; u < RPT; u++)
        if (RPT == 1 || bu == u) {
#pragma unroll
          for (int i = 0; i < W; i += V) {
            if (kAheadRows || i < W - j) {
              int4 q;
              memcpy(&q, &v[u][i], 16);
              *reinterpret_cast<int4*>(dst + i) = q;
            }
          }
        }
    };
    if (lane == max(wl, 0)) {
      sh.key[buf][warp] = bv;
      sh.pos[buf][warp] = wl < 0 ? -1 : bp;
      if (kAheadRows) put_row(rows + warp * W);
    }
    __syncthreads();
    const T ck = lane < NWARP ? sh.key[buf][lane] : T(0);
    const int cp = lane < NWARP ? sh.pos[buf][lane] : -1;
    const int cw = warp_best(ck, cp >= 0, cp);
    const bool none = cw < 0;
    const int p = none ? j : sh.pos[buf][max(cw, 0)];
    if (!kAheadRows) {
      if (warp == cw && lane == wl) put_row(urow + j * W);
      __syncthreads();
    }
    const T* pr = none ? zero : (kAheadRows ? rows + max(cw, 0) * W : urow + j * W);
    if (none) {
      if (info == 0) info = j + 1;
#pragma unroll
      for (int u = 0; u < RPT; u++)
        if (pos[u] == j) {
#pragma unroll
          for (int i = 0; i < W; i++) urow[j * W + i] = v[u][i];
        }
    } else if (kAheadRows && warp == (j & (NWARP - 1))) {
      for (int k = lane; k < W; k += 32) urow[j * W + k] = pr[k];
    }
    const T piv = pr[0];
    T mu[RPT];
#pragma unroll
    for (int u = 0; u < RPT; u++) {
      if (pos[u] == p) pos[u] = ~j;
      else if (pos[u] == j) pos[u] = p;
      // rows that are done or absent divide the pivot by itself: a zero
      // numerator leaves the division's fast path, and its warp with it
      const T l = none ? v[u][0] : (pos[u] >= 0 ? v[u][0] : piv) / piv;
      const int r = tid + u * BT;
      if (r < m) lb[j * mp + r] = l;
      mu[u] = none ? T(0) : l;
    }
#pragma unroll
    for (int c = 0; c < W; c += V) {
      T pv[V];
      const int4 q = *reinterpret_cast<const int4*>(pr + c);
      memcpy(pv, &q, 16);
#pragma unroll
      for (int e = 0; e < V; e++) {
        if (c + e == 0) continue;
#pragma unroll
        for (int u = 0; u < RPT; u++) v[u][c + e - 1] = fma(-mu[u], pv[e], v[u][c + e]);
      }
    }
#pragma unroll
    for (int u = 0; u < RPT; u++) v[u][W - 1] = T(0);
  }
#pragma unroll
  for (int u = 0; u < RPT; u++)
    if (pos[u] != INT_MIN) sh.src[pos[u] >= 0 ? pos[u] : ~pos[u]] = (unsigned short)(tid + u * BT);
  __syncthreads();
  return info;
}

template <typename T, int W>
__device__ __forceinline__ int panel_any(T* lb, int mp, int m, int kw, T* rowbuf, T* urow, T* zero, BShared<T>& sh) {
  if (m <= BT) return panel_regs<T, W, 1>(lb, mp, m, kw, rowbuf, urow, zero, sh);
  if (m <= 2 * BT) return panel_regs<T, W, 2>(lb, mp, m, kw, rowbuf, urow, zero, sh);
  if constexpr (W * sizeof(T) <= 128) {
    if (m <= 3 * BT) return panel_regs<T, W, 3>(lb, mp, m, kw, rowbuf, urow, zero, sh);
  }
  if constexpr (W * sizeof(T) <= 64) return panel_regs<T, W, 4>(lb, mp, m, kw, rowbuf, urow, zero, sh);
  return -1;
}

// Value of the factored panel at (position d, column c); W: urow's pitch
template <typename T>
__device__ __forceinline__ T panel_value(const T* lb, int mp, const T* urow, int W, const unsigned short* src, int d,
                                         int c) {
  return c < d ? lb[c * mp + src[d]] : urow[d * W + c - d];
}

// Positions whose row changed (map[d] != d, d < m) as moves mv_dst <- mv_src,
// both offset by base; call between barriers, sh.mv_n = 0 before.
template <typename T>
__device__ __forceinline__ void list_moves(BShared<T>& sh, const unsigned short* map, int m, int base) {
  for (int d = threadIdx.x; d < m; d += BT) {
    const int s = map[d];
    if (s != d) {
      const int o = atomicAdd(&sh.mv_n, 1);
      sh.mv_dst[o] = (unsigned short)(base + d);
      sh.mv_src[o] = (unsigned short)(base + s);
    }
  }
}

// map <- map after the moves (rows base + ..): map[dst] = old map[src]
template <typename T>
__device__ __forceinline__ void compose_map(BShared<T>& sh, unsigned short* map, int base) {
  const int tid = threadIdx.x;
  unsigned short t = 0;
  if (tid < sh.mv_n) t = map[sh.mv_src[tid] - base];
  __syncthreads();
  if (tid < sh.mv_n) map[sh.mv_dst[tid] - base] = t;
}

// The listed row moves on columns [ca, cb) minus [xa, xb): per pass every
// source of up to E x BT elements is read before any destination is written.
// sr, sc: the strides of a row and of a column of A.
template <typename T, int E>
__device__ __forceinline__ void apply_moves(T* A, int64_t sr, int64_t sc, const BShared<T>& sh, int ca, int xa, int xb,
                                            int cb) {
  const int tid = threadIdx.x, mm = sh.mv_n;
  const int nl = xa - ca, ncols = nl + cb - xb;
  if (mm == 0 || ncols <= 0) return;
  const int lg = 31 - __clz(max(1, E * BT / mm)), CW = 1 << lg;  // columns per pass, a power of two
  for (int c0 = 0; c0 < ncols; c0 += CW) {
    T v[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int idx = tid + e * BT, q = idx >> lg, k = c0 + (idx & (CW - 1));
      if (q < mm && k < ncols) v[e] = A[sh.mv_src[q] * sr + (k < nl ? ca + k : xb + k - nl) * sc];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int idx = tid + e * BT, q = idx >> lg, k = c0 + (idx & (CW - 1));
      if (q < mm && k < ncols) A[sh.mv_dst[q] * sr + (k < nl ? ca + k : xb + k - nl) * sc] = v[e];
    }
  }
}

// NB rows of one column (pitch up) by forward substitution, one fma per
// element in k order, in registers
template <typename T, int NB>
__device__ __forceinline__ void solve_column(T* uc, int up, const T* lt, int lp) {
  T u[NB];
#pragma unroll
  for (int i = 0; i < NB; i++) u[i] = uc[i * up];
#pragma unroll
  for (int p = 0; p < NB - 1; p++)
#pragma unroll
    for (int i = p + 1; i < NB; i++) u[i] = fma(-lt[i * lp + p], u[p], u[i]);
#pragma unroll
  for (int i = 1; i < NB; i++) uc[i * up] = u[i];
}

// U <- L^{-1} U by blocks of nb rows (4, 8, 16 or 32; Kp rows, a multiple of
// nb; w <= CW columns; L unit lower at lt, pitch lp a multiple of 4; U at ut,
// pitch up; all in shared memory): inside a block one thread per column; then
// the rows below take the block's products summed from zero, four rows of a
// column per thread.  Ends with a barrier.
template <typename T, int CW>
__device__ __forceinline__ void solve_rows(T* ut, int up, const T* lt, int lp, int Kp, int w, int nb) {
  constexpr int V = 16 / (int)sizeof(T), RG = BT / CW;
  const int tid = threadIdx.x, c = tid % CW, rg = tid / CW;
  for (int q0 = 0; q0 < Kp; q0 += nb) {
    if (rg == 0 && c < w) {
      T* uc = ut + q0 * up + c;
      const T* ld = lt + q0 * lp + q0;
      if (nb == 32) solve_column<T, 32>(uc, up, ld, lp);
      else if (nb == 16) solve_column<T, 16>(uc, up, ld, lp);
      else if (nb == 8) solve_column<T, 8>(uc, up, ld, lp);
      else solve_column<T, 4>(uc, up, ld, lp);
    }
    __syncthreads();
    if (c < w) {
      for (int i = q0 + nb + 4 * rg; i < Kp; i += 4 * RG) {  // Kp - q0 - nb is a multiple of 4
        T acc[4] = {};
        for (int p = 0; p < nb; p += V) {
          T u[V], l[4][V];
#pragma unroll
          for (int e = 0; e < V; e++) u[e] = ut[(q0 + p + e) * up + c];
#pragma unroll
          for (int r = 0; r < 4; r++) {
            const int4 q = *reinterpret_cast<const int4*>(&lt[(i + r) * lp + q0 + p]);
            memcpy(l[r], &q, 16);
#pragma unroll
            for (int e = 0; e < V; e++) acc[r] = fma(l[r][e], u[e], acc[r]);
          }
        }
#pragma unroll
        for (int r = 0; r < 4; r++) ut[(i + r) * up + c] -= acc[r];
      }
    }
    __syncthreads();
  }
}

// m x kw block at (k0, k0) of A into lb (column c of row r at lb[c * mp + r])
template <typename T>
__device__ __forceinline__ void copy_panel(const T* A, int n, int k0, int kw, int m, T* lb, int mp) {
  const int lg = kw > 1 ? 32 - __clz(kw - 1) : 0;
  for (int idx = threadIdx.x; idx < (m << lg); idx += BT) {
    const int r = idx >> lg, c = idx & ((1 << lg) - 1);
    if (c < kw) cp_async_elem<sizeof(T)>(lb + c * mp + r, A + (int64_t)(k0 + r) * n + k0 + c, true);
  }
  cp_async_commit_group();
  cp_async_wait_group<0>();
}

// Panel columns [k0, k0+kw), rows k0 .. k0+m, into lb, after the outer block's
// earlier panels (columns K0 .. k0 of L, U rows at ut, pitch up): per nb of
// them the products are summed from zero, then subtracted.
__device__ __forceinline__ void load_panel(const double* A, int n, int k0, int kw, int m, int K0, int nb, double* lb,
                                           int mp, const double* ut, int up, double*, int) {
  const int tid = threadIdx.x, Kp = k0 - K0;
  if (Kp == 0) {
    copy_panel(A, n, k0, kw, m, lb, mp);
    return;
  }
  // one warp per 16 rows x 16 columns; columns 4 (j + 2 e) + t of a register,
  // so a row's four lanes read 32 contiguous bytes
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nct = (kw + 15) / 16, nch = (m + 15) / 16;
  for (int w = warp; w < nch * nct; w += NWARP) {
    const int r = (w / nct) * 16 + g, cb = (w % nct) * 16;
    const bool ok0 = r < m, ok1 = r + 8 < m;
    const double* Ar = A + (int64_t)(k0 + r) * n;
    const double* Ar8 = Ar + (int64_t)8 * n;
    double cv[2][2][2];
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = cb + 4 * (j + 2 * e) + t;
        cv[0][j][e] = (ok0 && c < kw) ? Ar[k0 + c] : 0.0;
        cv[1][j][e] = (ok1 && c < kw) ? Ar8[k0 + c] : 0.0;
      }
    const int bc = cb + (g >> 1) + 8 * (g & 1);  // column of this lane's B values (tile j: + 4 j)
    for (int q = 0; q < Kp; q += nb) {
      double acc[2][4] = {};
      for (int kk = 0; kk < nb; kk += 16) {
        double a0[4], a1[4];
#pragma unroll
        for (int s = 0; s < 4; s++) {
          const int k = q + kk + 4 * s + t;
          const bool in = kk + 4 * s < nb;
          a0[s] = (in && ok0) ? Ar[K0 + k] : 0.0;
          a1[s] = (in && ok1) ? Ar8[K0 + k] : 0.0;
        }
#pragma unroll
        for (int s = 0; s < 4; s++) {
          if (kk + 4 * s < nb) {
            const double* ur = ut + (q + kk + 4 * s + t) * up;
#pragma unroll
            for (int j = 0; j < 2; j++) dmma_k4(acc[j], a0[s], a1[s], bc + 4 * j < kw ? ur[bc + 4 * j] : 0.0);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int e = 0; e < 2; e++) cv[h][j][e] -= acc[j][2 * h + e];
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int c = cb + 4 * (j + 2 * e) + t;
        if (c < kw) {
          if (ok0) lb[c * mp + r] = cv[0][j][e];
          if (ok1) lb[c * mp + r + 8] = cv[1][j][e];
        }
      }
  }
}
__device__ __forceinline__ void load_panel(const float* A, int n, int k0, int kw, int m, int K0, int nb, float* lb,
                                           int mp, const float* ut, int up, float* ls, int stage_rows) {
  const int tid = threadIdx.x, Kp = k0 - K0;
  copy_panel(A, n, k0, kw, m, lb, mp);
  if (Kp == 0) return;
  __syncthreads();
  // up to 256 rows of L (nb columns) at a time through shared memory, one row
  // and 16 of the panel's columns per thread, U broadcast
  const int lg = 31 - __clz(nb), row = tid & 255, cb = (tid >> 8) * 16;
  for (int q = 0; q < Kp; q += nb) {
    for (int r0 = 0; r0 < m; r0 += stage_rows) {
      const int nr = min(stage_rows, m - r0);
      for (int idx = tid; idx < (nr << lg); idx += BT) {
        const int i = idx >> lg, k = idx & (nb - 1);
        cp_async_elem<4>(ls + i * kStagePitch + k, A + (int64_t)(k0 + r0 + i) * n + K0 + q + k, true);
      }
      cp_async_commit_group();
      cp_async_wait_group<0>();
      __syncthreads();
      if (row < nr && cb < kw) {
        float acc[16] = {};
        for (int k = 0; k < nb; k++) {
          const float l = ls[row * kStagePitch + k];
          const float* ur = ut + (q + k) * up + cb;
          if (kw % 16 == 0) {
#pragma unroll
            for (int c = 0; c < 16; c += 4) {
              const float4 b = *reinterpret_cast<const float4*>(ur + c);
              acc[c] = fmaf(l, b.x, acc[c]);
              acc[c + 1] = fmaf(l, b.y, acc[c + 1]);
              acc[c + 2] = fmaf(l, b.z, acc[c + 2]);
              acc[c + 3] = fmaf(l, b.w, acc[c + 3]);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 16; c++)
              if (cb + c < kw) acc[c] = fmaf(l, ur[c], acc[c]);
          }
        }
#pragma unroll
        for (int c = 0; c < 16; c++)
          if (cb + c < kw) lb[(cb + c) * mp + r0 + row] -= acc[c];
      }
      __syncthreads();
    }
  }
}

// Trailing update of one column tile: C[r0:r1, ct:ct+TN] -= L U over TM-row
// tiles, L = A[.., kk0:kk0+K] streamed through two shared buffers of KS
// columns, U at ut in shared memory (K = outer_block<T>()).  One barrier per
// buffer; the copies of the next buffer and of the tile's own C values (each
// thread's into its own slots of shared memory) land while the products are
// summed (from zero, in k order), and C is prefetched into L2 two tiles ahead
// (thousands of systems are far larger than L2).
//
// FP64: 64 x 128 tiles, a warp owns 32 x 16 outputs on dmma_k4, which computes
// the transposed tile (A = U^T, B = L^T): the eight lanes of a fragment row
// then lie along a row of C, so an access of C touches 4 lines of 64 bytes
// instead of 8 of 32.  Both pitches are 4 mod 16 doubles: conflict-free
// fragments.  The copies are issued between the products: in one go behind the
// barrier they kept every warp from its products for a third of a tile (148
// systems of order 1024, this update: 5.4 -> 4.6 ms, 2.7 of them the products
// at the pipe's rate; 7.1 ms with 4 x 4 register blocks of plain fmas).
//
// FP32: 128 x 128 tiles, 8 rows x 4 columns per thread.  A warp's lanes share
// the rows, so an L value is a broadcast and four of a row come in one 16-byte
// load: 6 wavefronts per 32 fmas of a warp (2.7 ms at the same sizes; 3.1 with
// the copies between the products).
template <typename T>
struct Trail;
template <>
struct Trail<double> {
  static constexpr int TM = 64, TN = 128, K = 64, KS = 64, UP = TN + 4, LP = KS + 4;
};
template <>
struct Trail<float> {
  static constexpr int TM = 128, TN = 128, K = 128, KS = 64, UP = TN, LP = KS + 4;
};

// Step t of the stream: columns (t % (K / KS)) KS .. of row tile t / (K / KS);
// part p: BT elements of it
template <typename T>
__device__ __forceinline__ void stage_l_part(const T* A, int n, int r0, int r1, int kk0, int step, int p, T* lt) {
  using C = Trail<T>;
  constexpr int H = C::K / C::KS;
  const int r = r0 + step / H * C::TM, k0 = kk0 + step % H * C::KS;
  const int idx = threadIdx.x + p * BT, i = idx / C::KS, k = idx % C::KS;
  const bool ok = r + i < r1;
  cp_async_elem<sizeof(T)>(lt + (step & 1) * C::TM * C::LP + i * C::LP + k,
                           ok ? A + (int64_t)(r + i) * n + k0 + k : A, ok);
}
template <typename T>
__device__ __forceinline__ void stage_l(const T* A, int n, int r0, int r1, int kk0, int step, T* lt) {
  using C = Trail<T>;
#pragma unroll
  for (int p = 0; p < C::TM * C::KS / BT; p++) stage_l_part(A, n, r0, r1, kk0, step, p, lt);
  cp_async_commit_group();
}

// Rows [r, r + TM) of the column tile into L2
template <typename T>
__device__ __forceinline__ void prefetch_c(const T* A, int n, int r, int r1, int ct, int c1) {
  using C = Trail<T>;
  constexpr int LE = 128 / (int)sizeof(T), LPR = C::TN / LE;  // elements of a line, lines of a tile row
  static_assert(C::TM * LPR == BT, "one line per thread");
  const int i = r + threadIdx.x / LPR, j = ct + (threadIdx.x % LPR) * LE;
  if (i < r1 && j < c1) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + (int64_t)i * n + j));
}
constexpr int kAhead = 2;  // tiles between a prefetch and its use

// lt: two L buffers, the first one's copies already committed; cs: BT slots of
// TM TN / BT values
__device__ __forceinline__ void trail_tile(double* A, int n, int r0, int r1, int ct, int c1, int kk0,
                                           const double* ut, double* lt, double* cs) {
  using C = Trail<double>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wr = (warp >> 3) * 32, wc = (warp & 7) * 16;
  const int nrt = (r1 - r0 + C::TM - 1) / C::TM;
  const int cb = ct + wc + g;  // columns cb, cb + 8
  const bool okc[2] = {cb < c1, cb + 8 < c1};
  cs += tid;
  for (int tt = 0; tt < nrt; tt++) {
    cp_async_wait_group<0>();
    __syncthreads();  // L tile tt in shared memory; everyone is done with tile tt - 1
    // rows rb + 8 i + e
    const int rb = r0 + tt * C::TM + wr + 2 * t;
    double* Cp = A + (int64_t)rb * n + cb;
    prefetch_c(A, n, r0 + (tt + kAhead) * C::TM, r1, ct, c1);
    const double* ls = lt + (tt & 1) * C::TM * C::LP + (wr + g) * C::LP + t;
    const double* us = ut + t * C::UP + wc + g;
    double acc[4][4] = {};
#pragma unroll
    for (int s = 0; s < C::K / 4; s++) {
      const double u0 = us[4 * s * C::UP], u1 = us[4 * s * C::UP + 8];
#pragma unroll
      for (int i = 0; i < 4; i++) dmma_k4(acc[i], u0, u1, ls[8 * i * C::LP + 4 * s]);
      if (s < 8) {
        const int i = s >> 1, e = s & 1;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const bool ok = rb + 8 * i + e < r1 && okc[h];
          cp_async_elem<8>(cs + (2 * s + h) * BT, ok ? Cp + (int64_t)(8 * i + e) * n + 8 * h : A, ok);
        }
        if (s == 7) cp_async_commit_group();
      } else if (tt + 1 < nrt) {
        stage_l_part(A, n, r0, r1, kk0, tt + 1, s - 8, lt);
      }
    }
    cp_async_commit_group();
    cp_async_wait_group<1>();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int e = 0; e < 2; e++)
#pragma unroll
        for (int h = 0; h < 2; h++)
          if (rb + 8 * i + e < r1 && okc[h])
            Cp[(int64_t)(8 * i + e) * n + 8 * h] = cs[(4 * i + 2 * e + h) * BT] - acc[i][2 * h + e];
  }
}

__device__ __forceinline__ void trail_tile(float* A, int n, int r0, int r1, int ct, int c1, int kk0, const float* ut,
                                           float* lt, float* cs) {
  using C = Trail<float>;
  constexpr int H = C::K / C::KS;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wr = warp * 8;
  const int nrt = (r1 - r0 + C::TM - 1) / C::TM;
  cs += tid;
  for (int tt = 0; tt < nrt; tt++) {
    const int rb = r0 + tt * C::TM + wr, cb = ct + lane;  // columns cb + 32 j
    float* Cp = A + (int64_t)rb * n + cb;
    float acc[8][4] = {};
#pragma unroll 1
    for (int h = 0; h < H; h++) {
      const int step = tt * H + h;
      cp_async_wait_group<0>();
      __syncthreads();  // L buffer of this step in shared memory; everyone is done with the step before
      if (h == 0) {
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const bool ok = rb + i < r1 && cb + 32 * j < c1;
            cp_async_elem<4>(cs + (4 * i + j) * BT, ok ? Cp + (int64_t)i * n + 32 * j : A, ok);
          }
        prefetch_c(A, n, r0 + (tt + kAhead) * C::TM, r1, ct, c1);
      }
      if (step + 1 < nrt * H) stage_l(A, n, r0, r1, kk0, step + 1, lt);
      const float* ls = lt + (step & 1) * C::TM * C::LP + wr * C::LP;
      const float* us = ut + h * C::KS * C::UP + lane;
#pragma unroll 2
      for (int k = 0; k < C::KS; k += 4) {
        float b[4][4];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int j = 0; j < 4; j++) b[q][j] = us[(k + q) * C::UP + 32 * j];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float4 l = *reinterpret_cast<const float4*>(ls + i * C::LP + k);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            float v = acc[i][j];
            v = fmaf(l.x, b[0][j], v);
            v = fmaf(l.y, b[1][j], v);
            v = fmaf(l.z, b[2][j], v);
            v = fmaf(l.w, b[3][j], v);
            acc[i][j] = v;
          }
        }
      }
    }
    // C's copies were waited for with the last step's L buffer
    static_assert(H >= 2, "");
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 4; j++)
        if (rb + i < r1 && cb + 32 * j < c1) Cp[(int64_t)i * n + 32 * j] = cs[(4 * i + j) * BT] - acc[i][j];
  }
}

// The outer block [K0, Kend) (Kend < n, Kend - K0 = outer_block<T>()) on the
// columns right of it, one column tile at a time: its interchanges (sh.ob), its
// U rows by solve_rows, the trailing update.
template <typename T>
__device__ __forceinline__ void outer_update(T* A, int n, int K0, int nb, unsigned char* smem, const BShared<T>& sh) {
  using C = Trail<T>;
  constexpr int K = C::K;
  static_assert(K == outer_block<T>(), "");
  const int tid = threadIdx.x, Kend = K0 + K;
  T* ut = reinterpret_cast<T*>(smem);       // [K][UP]
  T* lt = ut + K * C::UP;                   // [2][TM][LP]
  T* cs = lt + 2 * C::TM * C::LP;           // [TM TN / BT][BT]
  T* l11 = cs;                              // [K][K], until the U rows are solved
  static_assert(C::TM * C::TN >= K * K, "");
  static_assert((size_t)(K * C::UP + 2 * C::TM * C::LP + C::TM * C::TN) * sizeof(T) <= kBatchSmem, "");
  for (int ct = Kend; ct < n; ct += C::TN) {
    const int w = min(C::TN, n - ct), c = tid % C::TN, i0 = tid / C::TN;
    constexpr int DI = BT / C::TN, E = K / DI;
    // the pivot rows into ut, the old top rows into registers
    T d[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int i = i0 + e * DI;
      cp_async_elem<sizeof(T)>(ut + i * C::UP + c, A + (int64_t)(K0 + sh.ob[i]) * n + ct + (c < w ? c : 0), c < w);
    }
    for (int idx = tid; idx < K * K; idx += BT)
      cp_async_elem<sizeof(T)>(l11 + idx, A + (int64_t)(K0 + idx / K) * n + K0 + idx % K, true);
    cp_async_commit_group();
#pragma unroll
    for (int e = 0; e < E; e++) d[e] = c < w ? A[(int64_t)(K0 + i0 + e * DI) * n + ct + c] : T(0);
    cp_async_wait_group<0>();
    __syncthreads();
    stage_l(A, n, Kend, n, K0, 0, lt);  // lands while the U rows are solved, as do the first tiles of C
    for (int tt = 0; tt < kAhead; tt++) prefetch_c(A, n, Kend + tt * C::TM, n, ct, n);
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int to = sh.to[i0 + e * DI];
      if (to >= Kend && c < w) A[(int64_t)to * n + ct + c] = d[e];
    }
    solve_rows<T, C::TN>(ut, C::UP, l11, K, K, w, nb);
#pragma unroll
    for (int e = 0; e < E; e++)
      if (c < w) A[(int64_t)(K0 + i0 + e * DI) * n + ct + c] = ut[(i0 + e * DI) * C::UP + c];
    trail_tile(A, n, Kend, n, ct, n, K0, ut, lt, cs);
    __syncthreads();  // ut, lt and cs free for the next column tile
  }
}

// LU of an n x n system in shared memory (n <= the bucket's threshold):
// a[c * mp + r], 16-column panels, everything right of a panel updated by one
// fma per element and column in column order, as the unblocked elimination
// does.
template <typename T>
__device__ int factor_small(T* A, int n, unsigned char* smem, BShared<T>& sh) {
  constexpr int W = 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mp = n | 1;
  T* a = reinterpret_cast<T*>(smem);
  T* rowbuf = &sh.diag[0][0];
  T* urow = rowbuf + 2 * NWARP * W;
  T* zero = urow + W * W;
  static_assert(2 * NWARP * W + W * W + W <= 32 * 33, "");
  for (int idx = tid; idx < n * n; idx += BT) a[(idx % n) * mp + idx / n] = A[idx];
  int info = 0;
  __syncthreads();
  for (int k0 = 0; k0 < n; k0 += W) {
    const int m = n - k0, kw = min(W, m), k1 = k0 + kw;
    T* lb = a + k0 * mp + k0;
    const int pi = panel_regs<T, W, 1>(lb, mp, m, kw, rowbuf, urow, zero, sh);
    if (pi && !info) info = k0 + pi;
    if (tid == 0) sh.mv_n = 0;
    __syncthreads();
    list_moves(sh, sh.src, m, k0);
    __syncthreads();
    apply_moves<T, 16>(a, 1, mp, sh, 0, k0, k1, n);
    // the panel's own columns: rows of the top block, and the moved rows below
    {
      T v[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int idx = tid + e * BT, d = idx / W, c = idx % W;  // top rows, then the list
        v[e] = T(0);
        if (d < W) {
          if (d < kw && c < kw) v[e] = panel_value(lb, mp, urow, W, sh.src, d, c);
        } else if (d - W < sh.mv_n && c < kw) {
          v[e] = lb[c * mp + sh.mv_src[d - W] - k0];
        }
      }
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int idx = tid + e * BT, d = idx / W, c = idx % W;
        if (d < W) {
          if (d < kw && c < kw) lb[c * mp + d] = v[e];
        } else if (d - W < sh.mv_n && c < kw && sh.mv_dst[d - W] >= k1) {
          lb[c * mp + sh.mv_dst[d - W] - k0] = v[e];
        }
      }
    }
    compose_map(sh, sh.perm, 0);
    __syncthreads();
    if (k1 >= n) break;
    // U rows: one thread per column
    if (k1 + tid < n) {
      T* uc = a + (k1 + tid) * mp + k0;
      T u[W];
#pragma unroll
      for (int i = 0; i < W; i++) u[i] = uc[i];
#pragma unroll
      for (int p = 0; p < W - 1; p++)
#pragma unroll
        for (int i = p + 1; i < W; i++) u[i] = fma(-lb[p * mp + i], u[p], u[i]);
#pragma unroll
      for (int i = 1; i < W; i++) uc[i] = u[i];
    }
    __syncthreads();
    // the rest: two rows per lane, their multipliers in registers
    const int rest = n - k1, nch = (rest + 63) / 64;
    for (int w = warp; w < NWARP; w += NWARP) {
      const int ch = w % nch, per = NWARP / nch;
      if (w / nch >= per) break;
      const int r0 = k1 + ch * 64 + lane, r1 = r0 + 32;
      T l0[W], l1[W];
#pragma unroll
      for (int k = 0; k < W; k++) {
        l0[k] = r0 < n ? a[(k0 + k) * mp + r0] : T(0);
        l1[k] = r1 < n ? a[(k0 + k) * mp + r1] : T(0);
      }
      for (int c = k1 + w / nch; c < n; c += per) {
        T* col = a + c * mp;
        T v0 = r0 < n ? col[r0] : T(0), v1 = r1 < n ? col[r1] : T(0);
#pragma unroll
        for (int k = 0; k < W; k++) {
          const T u = col[k0 + k];
          v0 = fma(-l0[k], u, v0);
          v1 = fma(-l1[k], u, v1);
        }
        if (r0 < n) col[r0] = v0;
        if (r1 < n) col[r1] = v1;
      }
    }
    __syncthreads();
  }
  for (int idx = tid; idx < n * n; idx += BT) A[idx] = a[(idx % n) * mp + idx / n];
  return info;
}

// Factor A (n x n row-major in global, ld = n) in place; sh.perm[i] = the
// original row that ends at row i.  Returns the 1-based first column without
// a usable pivot (0: none).
//
// Two-level blocking.  A panel of an outer block first gets the U rows of the
// block's earlier panels for its own columns, then its rows are loaded through
// the products with those panels, so inside the block no column is written
// before its panel comes up; after the panel its interchanges are applied to
// the block's other columns.  The columns left of the block take its composed
// interchanges when it is done, those right of it in outer_update.
template <typename T>
__device__ int factor_system(T* A, int n, unsigned char* smem, BShared<T>& sh) {
  const int tid = threadIdx.x;
  int nb, small;
  tuning_for<T>(n, nb, small);
  for (int i = tid; i < n; i += BT) sh.perm[i] = (unsigned short)i;
  if (n <= small) return factor_small<T>(A, n, smem, sh);
  constexpr int NB = outer_block<T>();
  T* ut = reinterpret_cast<T*>(smem);
  int info = 0;
  for (int k0 = 0; k0 < n; k0 += nb) {
    const PanelLayout<T> lay(n, nb, k0);
    const int kw = lay.kw, m = lay.m, mp = lay.mp, c1 = k0 + kw;
    const int Kp = lay.Kp, K0 = k0 - Kp, Kend = min(n, K0 + NB);
    const int up = lay.up, W = lay.W;
    T* lb = ut + lay.lb;  // [kw][mp]
    T* rowbuf = ut + lay.rowbuf;
    T* urow = ut + lay.urow;
    T* zero = ut + lay.zero;
    if (Kp == 0)
      for (int i = tid; i < n - K0; i += BT) sh.ob[i] = (unsigned short)i;
    if (Kp > 0) {
      T* lt = lb;  // [Kp][Kp + 4], before the panel takes the space
      const int lg = kw > 1 ? 32 - __clz(kw - 1) : 0;
      for (int idx = tid; idx < (Kp << lg); idx += BT) {
        const int i = idx >> lg, c = idx & ((1 << lg) - 1);
        if (c < kw) ut[i * up + c] = A[(int64_t)(K0 + i) * n + k0 + c];
      }
      for (int idx = tid; idx < Kp * Kp; idx += BT) {
        const int i = idx / Kp, k = idx - i * Kp;
        lt[i * (Kp + 4) + k] = A[(int64_t)(K0 + i) * n + K0 + k];
      }
      __syncthreads();
      solve_rows<T, 32>(ut, up, lt, Kp + 4, Kp, kw, nb);
      for (int idx = tid; idx < (Kp << lg); idx += BT) {
        const int i = idx >> lg, c = idx & ((1 << lg) - 1);
        if (c < kw) A[(int64_t)(K0 + i) * n + k0 + c] = ut[i * up + c];
      }
    }
    load_panel(A, n, k0, kw, m, K0, nb, lb, mp, ut, up, ut + lay.stage, lay.stage_rows);
    __syncthreads();
    int pi;
    if (W == 8) {
      if constexpr (sizeof(T) == 8) pi = panel_any<T, 8>(lb, mp, m, kw, rowbuf, urow, zero, sh);
      else pi = 0;
    } else if (W == 16) {
      pi = panel_any<T, 16>(lb, mp, m, kw, rowbuf, urow, zero, sh);
    } else {
      pi = panel_any<T, 32>(lb, mp, m, kw, rowbuf, urow, zero, sh);
    }
    if (pi && !info) info = k0 + pi;
    {
      const int lg = kw > 1 ? 32 - __clz(kw - 1) : 0;
      for (int idx = tid; idx < (m << lg); idx += BT) {
        const int d = idx >> lg, c = idx & ((1 << lg) - 1);
        if (c < kw) A[(int64_t)(k0 + d) * n + k0 + c] = panel_value(lb, mp, urow, W, sh.src, d, c);
      }
    }
    if (tid == 0) sh.mv_n = 0;
    __syncthreads();
    list_moves(sh, sh.src, m, k0);
    __syncthreads();
    apply_moves<T, 16>(A, n, 1, sh, K0, k0, c1, Kend);
    compose_map(sh, sh.ob, K0);
    __syncthreads();
    if (c1 < Kend) continue;
    // ---- the outer block is done
    if (tid == 0) sh.mv_n = 0;
    __syncthreads();
    list_moves(sh, sh.ob, n - K0, K0);
    for (int d = tid; d < n - K0; d += BT)
      if (sh.ob[d] < NB) sh.to[sh.ob[d]] = (unsigned short)(K0 + d);
    __syncthreads();
    apply_moves<T, 16>(A, n, 1, sh, 0, K0, K0, K0);
    compose_map(sh, sh.perm, 0);
    __syncthreads();
    if (Kend < n) outer_update<T>(A, n, K0, nb, smem, sh);
  }
  return info;
}

// Blocked forward (unit L) and backward (U) substitution, x in shared memory,
// 32-row blocks: a warp-parallel product over the solved part (two rows of a
// warp together), then one warp substitutes inside the 32 x 32 diagonal
// block, staged in shared memory meanwhile.
template <typename T>
__device__ __forceinline__ void solve_block_dots(const T* LU, int n, const T* xs, int I0, int rows, int j0, int j1,
                                                 BShared<T>& sh) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  T dg[2];
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int idx = tid + e * BT, i = idx >> 5, j = idx & 31;
    dg[e] = (i < rows && j < rows) ? LU[(int64_t)(I0 + i) * n + I0 + j] : T(0);
  }
  const bool two = warp + NWARP < rows;
  if (warp < rows) {
    const T* ra = LU + (int64_t)(I0 + warp) * n;
    const T* rb = LU + (int64_t)(I0 + (two ? warp + NWARP : warp)) * n;
    T sa = 0, sb = 0;
#pragma unroll 8
    for (int j = j0 + lane; j < j1; j += 32) {
      const T x = xs[j];
      sa = fma(ra[j], x, sa);
      sb = fma(rb[j], x, sb);
    }
    for (int o = 16; o > 0; o >>= 1) {
      sa += __shfl_xor_sync(0xffffffffu, sa, o);
      sb += __shfl_xor_sync(0xffffffffu, sb, o);
    }
    if (lane == 0) {
      sh.acc[warp] = sa;
      if (two) sh.acc[warp + NWARP] = sb;
    }
  }
#pragma unroll
  for (int e = 0; e < 2; e++) {
    const int idx = tid + e * BT;
    sh.diag[idx >> 5][idx & 31] = dg[e];
  }
  __syncthreads();
}

template <typename T>
__device__ void solve_system(const T* LU, int n, T* xs, BShared<T>& sh) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int I0 = 0; I0 < n; I0 += 32) {
    const int rows = min(32, n - I0);
    solve_block_dots(LU, n, xs, I0, rows, 0, I0, sh);
    if (warp == 0) {
      T v = lane < rows ? xs[I0 + lane] - sh.acc[lane] : T(0);
      for (int j = 0; j < rows; j++) {
        const T xj = __shfl_sync(0xffffffffu, v, j);
        if (lane > j && lane < rows) v = fma(-sh.diag[lane][j], xj, v);
      }
      if (lane < rows) xs[I0 + lane] = v;
    }
    __syncthreads();
  }
  const int nblk = (n + 31) / 32;
  for (int bi = nblk - 1; bi >= 0; bi--) {
    const int I0 = bi * 32, rows = min(32, n - I0);
    solve_block_dots(LU, n, xs, I0, rows, I0 + rows, n, sh);
    if (warp == 0) {
      T v = lane < rows ? xs[I0 + lane] - sh.acc[lane] : T(0);
      for (int j = rows - 1; j >= 0; j--) {
        if (lane == j) v = v / sh.diag[j][j];
        const T xj = __shfl_sync(0xffffffffu, v, j);
        if (lane < j) v = fma(-sh.diag[lane][j], xj, v);
      }
      if (lane < rows) xs[I0 + lane] = v;
    }
    __syncthreads();
  }
}

// One CTA per SM; T: the type of the factors.  FP32: the copy of each matrix
// is factored, then refined in FP64 against the matrix itself.
template <typename T>
__global__ void __launch_bounds__(BT, 1) batched_kernel(BatchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ BShared<T> sh;
  __shared__ int s_idx;
  __shared__ double s_red[4][NWARP];
  WorkHeader* hdr = reinterpret_cast<WorkHeader*>(a.work);
  if (ld_acquire_s32(&hdr->bad) != 0) return;
  const int* order = reinterpret_cast<const int*>(a.work + hdr->order);
  const int64_t* offA32 = reinterpret_cast<const int64_t*>(a.work + hdr->offA32);
  const int64_t* offV = reinterpret_cast<const int64_t*>(a.work + hdr->offV);
  float* A32s = reinterpret_cast<float*>(a.work + hdr->A32);
  double* r64s = reinterpret_cast<double*>(a.work + hdr->r64);
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) s_idx = (int)atomicAdd(&hdr->queue, 1u);
    __syncthreads();
    const int q = s_idx;
    __syncthreads();
    if (q >= a.count) break;
    const int sys = order[q];
    const int n = a.n[sys];
    double* A = a.A + a.a_off[sys];
    double* b = a.b + a.b_off[sys];
    int info = 0;
    if constexpr (sizeof(T) == 8) {
      info = factor_system<double>(A, n, smem, sh);
      __syncthreads();
      double* xs = reinterpret_cast<double*>(smem);
      for (int i = tid; i < n; i += BT) xs[i] = b[sh.perm[i]];
      __syncthreads();
      solve_system<double>(A, n, xs, sh);
      for (int i = tid; i < n; i += BT) b[i] = xs[i];
    } else {
      float* A32 = A32s + offA32[sys];
      double* r = r64s + 2 * offV[sys];  // [r | b] per system
      for (int base = tid; base < n * n; base += 16 * BT) {  // 16 loads in flight per thread
        double w[16];
#pragma unroll
        for (int e = 0; e < 16; e++) w[e] = base + e * BT < n * n ? A[base + e * BT] : 0.0;
#pragma unroll
        for (int e = 0; e < 16; e++)
          if (base + e * BT < n * n) A32[base + e * BT] = (float)w[e];
      }
      for (int i = tid; i < n; i += BT) r[n + i] = b[i];  // keep b for the residual
      __syncthreads();
      info = factor_system<float>(A32, n, smem, sh);
      __syncthreads();
      double* x = reinterpret_cast<double*>(smem);        // [n] the solution
      float* v = reinterpret_cast<float*>(x + kBatchMaxN);  // [n] the correction
      for (int i = tid; i < n; i += BT) v[i] = (float)b[sh.perm[i]];
      __syncthreads();
      solve_system<float>(A32, n, v, sh);
      // x = v, then FP64 refinement: r = b - A x (against the FP64 A), stop
      // when the scaled residual r_hpl < 16, else v = P r, FP32 solve, x += v
      for (int i = tid; i < n; i += BT) x[i] = (double)v[i];
      __syncthreads();
      const int warp = tid >> 5, lane = tid & 31;
      double anorm = 0.0, bmax = 0.0;
      for (int step = 0;; step++) {
        double rmax = 0.0, xmax = 0.0, an = 0.0;
        for (int i = warp; i < n; i += 2 * NWARP) {  // two rows of a warp together
          const bool two = i + NWARP < n;
          const double* ra = A + (int64_t)i * n;
          const double* rb = A + (int64_t)(two ? i + NWARP : i) * n;
          double aa = 0.0, ab = 0.0, sa = 0.0, sb = 0.0;
          if (step == 0) {
#pragma unroll 4
            for (int j = lane; j < n; j += 32) {
              const double va = ra[j], vb = rb[j], xj = x[j];
              aa = fma(va, xj, aa);
              ab = fma(vb, xj, ab);
              sa += fabs(va);
              sb += fabs(vb);
            }
          } else {
#pragma unroll 8
            for (int j = lane; j < n; j += 32) {
              const double xj = x[j];
              aa = fma(ra[j], xj, aa);
              ab = fma(rb[j], xj, ab);
            }
          }
          for (int o = 16; o > 0; o >>= 1) {
            aa += __shfl_xor_sync(0xffffffffu, aa, o);
            ab += __shfl_xor_sync(0xffffffffu, ab, o);
            sa += __shfl_xor_sync(0xffffffffu, sa, o);
            sb += __shfl_xor_sync(0xffffffffu, sb, o);
          }
          if (lane == 0) {
            const double ri = r[i + n] - aa;  // r[n + i] keeps b
            r[i] = ri;
            rmax = fmax(rmax, fabs(ri));
            an = fmax(an, sa);
            if (two) {
              const double rj = r[i + NWARP + n] - ab;
              r[i + NWARP] = rj;
              rmax = fmax(rmax, fabs(rj));
              an = fmax(an, sb);
            }
          }
        }
        for (int i = tid; i < n; i += BT) xmax = fmax(xmax, fabs(x[i]));
        if (step == 0)
          for (int i = tid; i < n; i += BT) bmax = fmax(bmax, fabs(r[i + n]));
        // block maxima
        for (int o = 16; o > 0; o >>= 1) {
          rmax = fmax(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
          xmax = fmax(xmax, __shfl_xor_sync(0xffffffffu, xmax, o));
          an = fmax(an, __shfl_xor_sync(0xffffffffu, an, o));
          bmax = fmax(bmax, __shfl_xor_sync(0xffffffffu, bmax, o));
        }
        if (lane == 0) { s_red[0][warp] = rmax; s_red[1][warp] = xmax; s_red[2][warp] = an; s_red[3][warp] = bmax; }
        __syncthreads();
        if (tid == 0) {
          double m0 = 0, m1 = 0, m2 = 0, m3 = 0;
          for (int w = 0; w < NWARP; w++) {
            m0 = fmax(m0, s_red[0][w]); m1 = fmax(m1, s_red[1][w]);
            m2 = fmax(m2, s_red[2][w]); m3 = fmax(m3, s_red[3][w]);
          }
          s_red[0][0] = m0; s_red[1][0] = m1; s_red[2][0] = m2; s_red[3][0] = m3;
        }
        __syncthreads();
        rmax = s_red[0][0];
        xmax = s_red[1][0];
        if (step == 0) { anorm = s_red[2][0]; bmax = s_red[3][0]; }
        __syncthreads();
        const double r_hpl = rmax / ((anorm * xmax + bmax) * (double)n * 2.220446049250313e-16);
        if (isnan(r_hpl)) {
          if (info == 0) info = LU_ERR_NONFINITE;
          if (tid == 0) atomicAdd(&hdr->refine_hist[kRefineHistBins - 1], 1);
          break;
        }
        if (r_hpl < 16.0) {
          if (tid == 0) atomicAdd(&hdr->refine_hist[step], 1);
          break;
        }
        if (step == kBatchRefineMax) {
          if (info == 0) info = LU_ERR_NOCONV;
          if (tid == 0) atomicAdd(&hdr->refine_hist[kRefineHistBins - 1], 1);
          break;
        }
        for (int i = tid; i < n; i += BT) v[i] = (float)r[sh.perm[i]];
        __syncthreads();
        solve_system<float>(A32, n, v, sh);
        for (int i = tid; i < n; i += BT) x[i] += (double)v[i];
        __syncthreads();
      }
      for (int i = tid; i < n; i += BT) b[i] = x[i];
    }
    if (tid == 0) a.info[sys] = info;
    __syncthreads();
  }
}

__host__ __device__ inline long long align256(long long x) { return (x + 255) & ~255LL; }

// Order systems by decreasing n (counting sort on n), prefix offsets of the
// per-system workspace regions, and the workspace layout.  One CTA.
__global__ void __launch_bounds__(1024) batched_prep_kernel(int count, const int* n, int precision,
                                                            unsigned char* work, long long work_bytes,
                                                            int* info) {
  __shared__ int hist[kBatchMaxN + 1];
  __shared__ int s_bad;
  WorkHeader* hdr = reinterpret_cast<WorkHeader*>(work);
  const int tid = threadIdx.x;
  long long o = 256;
  const long long o_order = o;
  o = align256(o + 4LL * count);
  const long long o_offA32 = o;
  o = align256(o + 8LL * count);
  const long long o_offV = o;
  o = align256(o + 8LL * count);
  int* order = reinterpret_cast<int*>(work + o_order);
  int64_t* offA32 = reinterpret_cast<int64_t*>(work + o_offA32);
  int64_t* offV = reinterpret_cast<int64_t*>(work + o_offV);
  for (int i = tid; i <= kBatchMaxN; i += blockDim.x) hist[i] = 0;
  if (tid == 0) s_bad = 0;
  __syncthreads();
  for (int i = tid; i < count; i += blockDim.x) {
    const int v = n[i];
    if (v < 1 || v > kBatchMaxN) { atomicAdd(&s_bad, 1); continue; }
    atomicAdd(&hist[v], 1);
  }
  __syncthreads();
  // start position of every order, descending: an exclusive scan of the
  // histogram from its end, two bins a thread; the offsets are a block scan
  // too.  One thread's loops over both took 125 us of a call at 4096 systems
  // (4096 systems of order 1: 0.306 -> 0.180 ms) and 35 us at 1000
  static_assert(kBatchMaxN == 2048, "two bins per thread");
  __shared__ long long w1[32], w2[32];
  __shared__ int wb[32];
  const int lane = tid & 31, warp = tid >> 5;
  const int v0 = kBatchMaxN - 2 * tid;  // bins v0, v0 - 1
  const int h0 = hist[v0], h1 = hist[v0 - 1];
  int hs = h0 + h1;
  // offsets of the systems: each thread a run of them
  const int per = (count + 1023) / 1024, i0 = min(count, tid * per), i1 = min(count, i0 + per);
  long long s1 = 0, s2 = 0;
  for (int i = i0; i < i1; i++) {
    const int v = n[i];
    if (v >= 1 && v <= kBatchMaxN) { s2 += (long long)v * v; s1 += v; }
  }
  const int hown = hs;
  const long long own1 = s1, own2 = s2;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int a = __shfl_up_sync(0xffffffffu, hs, o);
    const long long b1 = __shfl_up_sync(0xffffffffu, s1, o), b2 = __shfl_up_sync(0xffffffffu, s2, o);
    if (lane >= o) { hs += a; s1 += b1; s2 += b2; }
  }
  if (lane == 31) { wb[warp] = hs; w1[warp] = s1; w2[warp] = s2; }
  __syncthreads();
  int hb = 0;
  long long t1 = 0, t2 = 0;
  for (int w = 0; w < warp; w++) { hb += wb[w]; t1 += w1[w]; t2 += w2[w]; }
  hist[v0] = hb + hs - hown;
  hist[v0 - 1] = hb + hs - hown + h0;
  long long p1 = t1 + s1 - own1, p2 = t2 + s2 - own2;
  for (int i = i0; i < i1; i++) {
    const int v = n[i];
    offA32[i] = p2;
    offV[i] = p1;
    if (v >= 1 && v <= kBatchMaxN) { p2 += (long long)v * v; p1 += v; }
  }
  if (tid == 0) {
    s1 = 0;
    s2 = 0;
    for (int w = 0; w < 32; w++) { s1 += w1[w]; s2 += w2[w]; }
    hdr->queue = 0;
    for (int q = 0; q < kRefineHistBins; q++) hdr->refine_hist[q] = 0;
    hdr->s1 = s1;
    hdr->s2 = s2;
    hdr->order = o_order;
    hdr->offA32 = o_offA32;
    hdr->offV = o_offV;
    long long q = o;
    hdr->A32 = q;
    if (precision == LU_PREC_FP32) q = align256(q + 4 * s2);
    hdr->r64 = q;
    if (precision == LU_PREC_FP32) q = align256(q + 16 * s1);
    hdr->total = q;
    if (q > work_bytes) s_bad = 1;
  }
  __syncthreads();
  for (int i = tid; i < count; i += blockDim.x) {
    const int v = n[i];
    if (v < 1 || v > kBatchMaxN) { info[i] = LU_ERR_ARG; continue; }
    if (s_bad) { info[i] = LU_ERR_ARG; continue; }
    const int pos = atomicAdd(&hist[v], 1);
    order[pos] = i;
  }
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    hdr->bad = s_bad;
  }
}

std::mutex g_tune_mu;

}  // namespace
}  // namespace lub

using namespace lub;

extern "C" LU_API size_t lu_batched_work_bytes(int32_t count, const int32_t* n_host, int32_t precision) {
  if (count <= 0 || !n_host) return 0;
  long long s2 = 0, s1 = 0;
  for (int i = 0; i < count; i++) {
    s2 += (long long)n_host[i] * n_host[i];
    s1 += n_host[i];
  }
  long long o = 256;
  o = align256(o + 4LL * count);
  o = align256(o + 8LL * count);
  o = align256(o + 8LL * count);
  if (precision == LU_PREC_FP32) {
    o = align256(o + 4 * s2);
    o = align256(o + 16 * s1);
  }
  return (size_t)o;
}

extern "C" LU_API int lu_batched_refine_histogram(const void* dWork, int32_t* hist, void* stream) {
  if (!dWork || !hist) return LU_ERR_ARG;
  const WorkHeader* hdr = static_cast<const WorkHeader*>(dWork);
  cudaStream_t s = (cudaStream_t)stream;
  LUB_CUDA(cudaMemcpyAsync(hist, hdr->refine_hist, sizeof(int) * kRefineHistBins, cudaMemcpyDeviceToHost, s));
  LUB_CUDA(cudaStreamSynchronize(s));
  return LU_OK;
}

extern "C" LU_API int lu_batched_set_tuning(int32_t entries, const int32_t* table) {
  if (entries < 0 || entries > 16 || (entries > 0 && !table)) return LU_ERR_ARG;
  Tuning t[16] = {};
  for (int i = 0; i < entries; i++) {
    t[i].n_max = table[3 * i];
    t[i].nb = table[3 * i + 1];
    t[i].small = table[3 * i + 2];
    if (t[i].nb < 4 || t[i].nb > 32 || (t[i].nb & (t[i].nb - 1)) || t[i].small < 0) return LU_ERR_ARG;
    if (i > 0 && t[i].n_max <= t[i - 1].n_max) return LU_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(g_tune_mu);
  LUB_CUDA(cudaMemcpyToSymbol(c_tuning, t, sizeof(t)));
  LUB_CUDA(cudaMemcpyToSymbol(c_tuning_n, &entries, sizeof(int)));
  return LU_OK;
}

namespace {
template <typename T>
int layout_probe(int n, int nb, int* out) {
  nb = panel_width<T>(n, nb);
  out[0] = nb;
  out[1] = 0;
  out[2] = 256;
  for (int k0 = 0; k0 < n; k0 += nb) {
    const PanelLayout<T> lay(n, nb, k0);
    out[1] = std::max(out[1], lay.end * (int)sizeof(T));
    if (lay.stage_rows > 0) out[2] = std::min(out[2], lay.stage_rows);
  }
  return LU_OK;
}
}  // namespace

// Test hook (no GPU): out = panel width taken for order n where the table says
// nb, bytes of dynamic shared memory that its panels reach, fewest staged rows
// of L, bytes that the kernel asks for.
extern "C" __attribute__((visibility("default"))) int lub_test_batched_layout(int n, int nb, int esize, int* out) {
  out[3] = (int)kBatchSmem;
  return esize == 8 ? layout_probe<double>(n, nb, out) : layout_probe<float>(n, nb, out);
}

extern "C" LU_API int lu_batched_factor_solve(int32_t count, const int32_t* n, const int64_t* a_off,
                                              const int64_t* b_off, double* dA, double* db, int32_t* info,
                                              int32_t precision, void* dWork, size_t work_bytes, void* stream) {
  if (count <= 0 || !n || !a_off || !b_off || !dA || !db || !info || !dWork) return LU_ERR_ARG;
  if (precision != LU_PREC_FP64 && precision != LU_PREC_FP32) return LU_ERR_ARG;
  if (work_bytes < 256 + 20 * (size_t)count) return LU_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  static PerDeviceOnce once;
  LUB_TRY(once_per_device(once, [] {
    LUB_TRY(cuda_status(cudaFuncSetAttribute(batched_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)kBatchSmem)));
    return cuda_status(
        cudaFuncSetAttribute(batched_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchSmem));
  }));
  unsigned char* w = static_cast<unsigned char*>(dWork);
  batched_prep_kernel<<<1, 1024, 0, s>>>(count, n, precision, w, (long long)work_bytes, info);
  LUB_LAUNCH_CHECK();
  int dev = 0, sms = kNumSMsB200;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  BatchArgs a{count, n, a_off, b_off, dA, db, info, precision, w};
  if (precision == LU_PREC_FP64)
    batched_kernel<double><<<std::min(count, sms), BT, kBatchSmem, s>>>(a);
  else
    batched_kernel<float><<<std::min(count, sms), BT, kBatchSmem, s>>>(a);
  LUB_LAUNCH_CHECK();
  return LU_OK;
}
