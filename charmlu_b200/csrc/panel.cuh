// Unblocked panel factorisation (getf2) of a tall, narrow column block.
//
// Restates the per-column loop of factorDiagBlock / factorBelowDiagBlock
// (lu.ci:186-370) and its kernels:
//   findMaxElm          lu.C:197-205   (strict '>', first row wins)
//   MaxElm_max reducer  lu.C:207-218   (ties: lowest global row here; the
//                                       reference's order is message-arrival
//                                       dependent)
//   swapLocal / pivotRowSwap            lu.C:172-177, lu.ci:302-323
//   computeMultipliersAndFindColMax     lu.C:259-288 (true division)
//   updateLsubBlock (dger, offset 2)    lu.C:230-254
//   singularity check                   lu.ci:339-341 (reported, not aborted)
//   the row swap on the rest of the panel's columns (the reference swaps
//   whole rows of the panel block, lu.ci:302-323)
//
// What bounds it: a chain of W pivot searches over all rows, so latency per
// column, not bytes or flops.  The layout keeps that chain short:
//   * every thread holds RPT whole rows of the leaf in registers, and a row
//     is rotated by one after each column, so the current column is always
//     register 0 and one small copy of the code serves every column (copies
//     per column overflow the instruction cache: with eight, warps waited
//     for instructions half of the time).  Multipliers leave for shared
//     memory as they are made; the registers behind the unfinished columns
//     hold values that nothing reads;
//   * rows never move.  An interchange renames two rows: a row carries the
//     position it stands at, the chosen row leaves the set, the row standing
//     at the diagonal takes the chosen row's position;
//   * a CTA's candidate takes one barrier: each warp reduces its rows with
//     redux on the bit patterns of |a|, then a warp reduces the eight winners.
//     The best row reaches shared memory from the one lane that holds it, after
//     the winner is known: one lane stores 4 bytes a cycle, and eight warps
//     writing their candidates' rows ahead of the barrier took 290 - 520 cycles
//     of a column (FP64 256 x 32 36.3 -> 30.8 us, cluster 2048 x 32 48.6 ->
//     42.8).  In a grid, where L2 latency dominates and the row has to leave at
//     once, they are written ahead (FP32 36864 x 32: 84.5 us, 90 the other way);
//   * between CTAs there is no barrier.  In a cluster every CTA sends its
//     candidate (header and row) to every peer with st.async and waits on its
//     own mbarrier for G of them.  In a larger grid warp 0 publishes header
//     and row in global memory as 16-byte packets that carry the column's tag
//     (the data is its own flag), reads every CTA's header until the tags
//     match, and then the winner's row.  Both are double-buffered by column
//     parity, which is safe because a CTA sends column j + 2 only after it
//     has all of column j + 1, which every CTA sent after it was done with
//     column j.
// The rest of the enclosing panel's columns get the leaf's interchanges in
// one pass at the end, composed into one assignment of at most 2 W rows.
// Per element the arithmetic is one true division and one fma per column in
// column order, whatever the shape of the grid.
//
// Measured on B200, per column: FP64 order 2048 (cluster) 4.7 -> 1.5 us, FP32
// order 10000 (cluster) 5.0 -> 1.5 us, FP32 order 65536 beside the trailing
// update (48-CTA grid) 7.6 -> 4.3 us, against a leaf that kept its rows in
// shared memory and took a grid barrier per column; one CTA of 256 rows alone
// 1.1 us (FP64), 0.8 us (FP32).  About 180 instructions
// per warp and column remain, most of them waiting on the one before.
#pragma once
#include <climits>

#include "argmax.cuh"
#include "common.cuh"
#include "kernels.h"

namespace lub {
namespace {

constexpr int NT = 256;       // threads per CTA: 255 registers each, 8 warps to reduce over
constexpr int NW = NT / 32;
constexpr int kMaxCluster = 16;
enum { kSingle = 0, kGrid = 1, kCluster = 2 };

// Candidate (value, position) as a header's three words, and back
__device__ __forceinline__ void key_words(float v, unsigned& a, unsigned& b) { a = __float_as_uint(v); b = 0; }
__device__ __forceinline__ void key_words(double v, unsigned& a, unsigned& b) {
  a = (unsigned)__double2loint(v);
  b = (unsigned)__double2hiint(v);
}
__device__ __forceinline__ void key_value(unsigned a, unsigned, float& v) { v = __uint_as_float(a); }
__device__ __forceinline__ void key_value(unsigned a, unsigned b, double& v) { v = __hiloint2double((int)b, (int)a); }

// 16-byte packets in global memory: one 128-bit access each, so a packet is
// read whole or not at all
__device__ __forceinline__ void st_packet(ulonglong2* p, unsigned w0, unsigned w1, unsigned w2, unsigned tag) {
  const unsigned long long lo = ((unsigned long long)w1 << 32) | w0, hi = ((unsigned long long)tag << 32) | w2;
  asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
               "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ uint4 ld_packet(const ulonglong2* p) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}

// 16 bytes to a peer's shared memory, counted by the peer's mbarrier
__device__ __forceinline__ void st_async16(uint32_t local_dst, uint32_t local_bar, int peer, uint4 v) {
  asm volatile(
      "{\n .reg .b32 ra, rb;\n mapa.shared::cluster.u32 ra, %0, %2;\n mapa.shared::cluster.u32 rb, %1, %2;\n"
      " st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [ra], {%3, %4, %5, %6}, [rb];\n}" ::"r"(local_dst),
      "r"(local_bar), "r"(peer), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
      : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct LeafArgs {
  int64_t lda;
  int M, ncols, R;
  int32_t* ipiv;
  int row_base;
  ulonglong2* pkt;  // headers [2][kMaxLeafCTAs], then rows [2][kMaxLeafCTAs][kLeafRowPackets]
  unsigned tag0;
  DevStatus* st;
  int info_base;
  double thr;
  long long spin;
  int pw, lc0;
};

template <typename T, int W, int RPT, int XP>
struct LeafShared {
  // row j: the row chosen in column j, element i of it being column j + i
  // (cluster: this CTA's candidate, which is that row where it matters)
  alignas(16) T urow[W][W];
  // grid: each warp's candidate row, by column parity
  alignas(16) T row[XP == kGrid ? 2 : 1][XP == kGrid ? NW : 1][W];
  alignas(16) T zero[W];
  // cluster: every CTA's candidate, by column parity
  alignas(16) T crow[XP == kCluster ? 2 : 1][XP == kCluster ? kMaxCluster : 1][W];
  uint4 chdr[XP == kCluster ? 2 : 1][XP == kCluster ? kMaxCluster : 1];
  alignas(8) uint64_t bar[2];
  T key[2][NW];
  int pos[2][NW];
  T piv[W];  // the chosen pivots
  int p[W];  // position chosen in column j; -1: none usable, -2: a wait ran out
  int src[W];
  int mv_dst[2 * W], mv_src[2 * W];
  int mv_n;
  unsigned sink[NT];
};

template <typename T, int W, int RPT, int XP>
constexpr size_t leaf_smem() {
  return ((sizeof(LeafShared<T, W, RPT, XP>) + 15) & ~size_t(15)) + (size_t)W * NT * RPT * sizeof(T);
}

// One column's update of RPT rows over A registers, and their rotation
template <int A, typename T, int W, int RPT>
__device__ __forceinline__ void leaf_update(T (&v)[RPT][W], const T (&m)[RPT], const T* pr) {
  constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
  for (int c = 0; c < A; c += V) {
    T pv[V];
    const int4 q = *reinterpret_cast<const int4*>(pr + c);
    memcpy(pv, &q, 16);
#pragma unroll
    for (int e = 0; e < V; e++) {
      if (c + e == 0) continue;
#pragma unroll
      for (int u = 0; u < RPT; u++) v[u][c + e - 1] = fma(-m[u], pv[e], v[u][c + e]);
    }
  }
#pragma unroll
  for (int u = 0; u < RPT; u++) v[u][A - 1] = T(0);
}

template <typename T, int W, int RPT, int XP>
__global__ void __launch_bounds__(NT, 1) getf2_leaf_kernel(T* P, T* prow0, LeafArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using Sh = LeafShared<T, W, RPT, XP>;
  Sh& sh = *reinterpret_cast<Sh*>(smem_raw);
  T* lbuf = reinterpret_cast<T*>(smem_raw + ((sizeof(Sh) + 15) & ~size_t(15)));  // [W][NT * RPT] multipliers
  constexpr int LP = NT * RPT;
  constexpr int WPT = sizeof(T) / 4, NWORDS = W * WPT;
  constexpr int V = 16 / (int)sizeof(T);
  const int G = XP == kSingle ? 1 : gridDim.x, cta = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r_lo = cta * a.R, nr = min(a.M, r_lo + a.R) - r_lo, ncols = a.ncols;
  const bool vec = ncols == W && a.lda % V == 0 && (reinterpret_cast<uintptr_t>(P) & 15) == 0;
  if constexpr (XP != kGrid) after_previous_kernel();

  // ---- rows into registers
  T v[RPT][W];
  int pos[RPT];  // the row's position; ~j: chosen in column j; INT_MIN: no such row
  unsigned chk = 0;
#pragma unroll
  for (int u = 0; u < RPT; u++) {
    const int r = tid + u * NT;
    pos[u] = r < nr ? r_lo + r : INT_MIN;
    const T* src = P + (int64_t)(r_lo + r) * a.lda;
    if (vec && r < nr) {
#pragma unroll
      for (int i = 0; i < W; i += V) {
        const int4 q = *reinterpret_cast<const int4*>(src + i);
        memcpy(&v[u][i], &q, 16);
      }
    } else {
#pragma unroll
      for (int i = 0; i < W; i++) v[u][i] = (r < nr && i < ncols) ? src[i] : T(0);
    }
#pragma unroll
    for (int i = 0; i < W; i++) {
      unsigned w[WPT];
      memcpy(w, &v[u][i], sizeof(T));
#pragma unroll
      for (int k = 0; k < WPT; k++) chk ^= w[k];
    }
  }
  // Rows are written to their new positions at the end, where another CTA's
  // row may have been read from: this store depends on every value read, so
  // the first barrier, and with it column 0, follows all the reads.
  *(volatile unsigned*)&sh.sink[tid] = chk;
  if (tid < W) sh.zero[tid] = T(0);
  if constexpr (XP == kCluster) {
    if (tid == 0) {
      mbar_init(&sh.bar[0], 1);
      mbar_init(&sh.bar[1], 1);
      fence_mbar_init();
    }
    __syncthreads();
    cluster_sync();
  }
  bool dead = false;  // cluster: a wait ran out; go on without waiting, write nothing

#pragma unroll 1
  for (int j = 0; j < ncols; j++) {
    const int buf = j & 1;
    // ---- the CTA's candidate
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
    const int act = W - j;  // unfinished columns
    auto put_row = [&](T* dst) {
#pragma unroll
      for (int u = 0; u < RPT; u++)
        if (RPT == 1 || bu == u) {
#pragma unroll
          for (int i = 0; i < W; i += V) {
            if (i < act) {
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
      if constexpr (XP == kGrid) put_row(sh.row[buf][warp]);
    }
    if (XP == kCluster && tid == 0)
      mbar_arrive_expect_tx(&sh.bar[buf], (unsigned)(G * (((act + V - 1) / V) * 16 + 16)));
    __syncthreads();
    int cw = -1;  // the warp with the best row (grid: known to warp 0 only)
    if (XP != kGrid || warp == 0) {
      const T ck = lane < NW ? sh.key[buf][lane] : T(0);
      const int cp = lane < NW ? sh.pos[buf][lane] : -1;
      cw = warp_best(ck, cp >= 0, cp);
    }
    if (XP != kGrid && warp == cw && lane == wl) put_row(sh.urow[j]);
    const T* pr;
    bool none;
    [[maybe_unused]] int chosen = -1, chosen_lane = 0;  // cluster: the chosen position, in a lane
    if constexpr (XP == kSingle) {
      __syncthreads();
      none = cw < 0;
      pr = sh.urow[j];
      if (tid == 0) sh.p[j] = none ? -1 : sh.pos[buf][cw];
    } else if constexpr (XP == kCluster) {
      __syncthreads();  // the row is in shared memory: each warp sends it to its share of the peers
      // lanes 0 .. np-1 carry the row, the next one the header
      const int np = (act + V - 1) / V;
      unsigned k0, k1;
      key_words(sh.key[buf][max(cw, 0)], k0, k1);
      uint4 d = make_uint4(k0, k1, (unsigned)(cw >= 0 ? sh.pos[buf][cw] : -1), 0u);
      if (lane < np) d = *reinterpret_cast<const uint4*>(&sh.urow[j][lane * V]);
      const uint32_t dst = lane < np ? smem_u32(&sh.crow[buf][cta][lane * V]) : smem_u32(&sh.chdr[buf][cta]);
      const uint32_t bar = smem_u32(&sh.bar[buf]);
      if (lane <= np)
        for (int q = warp; q < G; q += NW) st_async16(dst, bar, q, d);
      if (!dead) {
        long long n = 0;
        while (!mbar_try_wait(&sh.bar[buf], (j >> 1) & 1)) {
          if (++n > a.spin) {
            dev_fail(a.st, LU_ERR_TIMEOUT, 201);
            dead = true;
            break;
          }
        }
      }
      __syncwarp();
      const uint4 hd = sh.chdr[buf][lane & (kMaxCluster - 1)];
      T hv;
      key_value(hd.x, hd.y, hv);
      const int hp = lane < G ? (int)hd.z : -1;
      const int q = warp_best(hv, hp >= 0, hp);
      none = q < 0;
      chosen = hp;
      chosen_lane = max(q, 0);
      pr = sh.crow[buf][max(q, 0)];
      if (warp == 0 && lane == max(q, 0)) sh.p[j] = none ? -1 : hp;
    } else {
      const unsigned tag = a.tag0 + (unsigned)j + 1u;
      ulonglong2* hdr = a.pkt + (size_t)buf * kMaxLeafCTAs;
      ulonglong2* rows = a.pkt + 2 * kMaxLeafCTAs + (size_t)buf * kMaxLeafCTAs * kLeafRowPackets;
      if (warp == 0) {
        // ---- publish header and row
        const int np = (act * WPT + 2) / 3;  // packets of the row's unfinished part
        unsigned w0, w1, w2 = (unsigned)(cw >= 0 ? sh.pos[buf][cw] : -1);
        key_words(sh.key[buf][max(cw, 0)], w0, w1);
        if (lane < np) {
          const unsigned* w = reinterpret_cast<const unsigned*>(sh.row[buf][max(cw, 0)]);
          w0 = w[3 * lane];
          w1 = 3 * lane + 1 < NWORDS ? w[3 * lane + 1] : 0u;
          w2 = 3 * lane + 2 < NWORDS ? w[3 * lane + 2] : 0u;
        }
        if (lane <= np) st_packet(lane < np ? rows + cta * kLeafRowPackets + lane : hdr + cta, w0, w1, w2, tag);
        // ---- every CTA's header, then the best one's row
        constexpr int E = (kMaxLeafCTAs + 31) / 32;
        uint4 h[E];
        long long polls = 0;
        int bad = 0;
        for (;;) {
          bool ok = true;
#pragma unroll
          for (int e = 0; e < E; e++)
            if (lane + 32 * e < G) h[e] = ld_packet(hdr + lane + 32 * e);
#pragma unroll
          for (int e = 0; e < E; e++)
            if (lane + 32 * e < G) ok = ok && h[e].w == tag;
          if (__all_sync(0xffffffffu, ok)) break;
          bool stop = ++polls > a.spin;
          if ((polls & 255) == 0 && ld_acquire_s32(&a.st->code) != 0) stop = true;
          if (__any_sync(0xffffffffu, stop)) { bad = 1; break; }
        }
        T gv = 0;
        int gp = -1, gq = 0;
#pragma unroll
        for (int e = 0; e < E; e++) {
          if (lane + 32 * e < G) {
            T x;
            key_value(h[e].x, h[e].y, x);
            const int ps = (int)h[e].z;
            if (ps >= 0 && (x > gv || (x == gv && gp >= 0 && ps < gp))) {
              gv = x;
              gp = ps;
              gq = lane + 32 * e;
            }
          }
        }
        const int gl = warp_best(gv, gp >= 0, gp);
        int p = -1;
        if (gl >= 0 && !bad) {
          const int q = __shfl_sync(0xffffffffu, gq, gl);
          p = __shfl_sync(0xffffffffu, gp, gl);
          uint4 d;
          for (polls = 0;;) {
            bool ok = true;
            if (lane < np) {
              d = ld_packet(rows + q * kLeafRowPackets + lane);
              ok = d.w == tag;
            }
            if (__all_sync(0xffffffffu, ok)) break;
            if (__any_sync(0xffffffffu, ++polls > a.spin)) { bad = 1; break; }
          }
          unsigned* dst = reinterpret_cast<unsigned*>(sh.urow[j]);
          if (lane < np) {
            dst[3 * lane] = d.x;
            if (3 * lane + 1 < NWORDS) dst[3 * lane + 1] = d.y;
            if (3 * lane + 2 < NWORDS) dst[3 * lane + 2] = d.z;
          }
        }
        if (bad && lane == 0) dev_fail(a.st, LU_ERR_TIMEOUT, 201);
        if (lane == 0) sh.p[j] = bad ? -2 : p;
      }
      __syncthreads();
      const int p = sh.p[j];
      if (p == -2) return;
      none = p < 0;
      pr = sh.urow[j];
    }

    // ---- rename, multipliers (true division), rank-1 update, rotation.  No
    //      usable pivot: the row at j stays, nothing is scaled or updated
    int pj = j;
    if (none) {
      pr = sh.zero;
#pragma unroll
      for (int u = 0; u < RPT; u++)
        if (pos[u] == j) {
          if (!(fabs((double)v[u][0]) > a.thr)) dev_singular(a.st, a.info_base + j + 1);
#pragma unroll
          for (int i = 0; i < W; i++) sh.urow[j][i] = v[u][i];
        }
    }
    const T piv = pr[0];
    if (!none) {
      if constexpr (XP == kSingle) pj = sh.pos[buf][cw];
      else if constexpr (XP == kGrid) pj = sh.p[j];
      else pj = __shfl_sync(0xffffffffu, chosen, chosen_lane);
    }
    if (tid == 0) sh.piv[j] = piv;
    T m[RPT];
#pragma unroll
    for (int u = 0; u < RPT; u++) {
      if (pos[u] == pj) pos[u] = ~j;
      else if (pos[u] == j) pos[u] = pj;
      // rows that are done or absent divide the pivot by itself: a zero
      // numerator leaves the division's fast path, and its warp with it
      const T l = none ? v[u][0] : (pos[u] >= 0 ? v[u][0] : piv) / piv;
      lbuf[j * LP + u * NT + tid] = l;
      m[u] = none ? T(0) : l;
    }
    if (j < W / 2) leaf_update<W>(v, m, pr);
    else leaf_update<W / 2>(v, m, pr);
  }

  if constexpr (XP == kCluster) {
    if (dead)  // bounded: let what the peers still send arrive
      for (int n = 0; n < 4096 && !mbar_try_wait(&sh.bar[0], 0); n++) {}
    dead = __syncthreads_or(dead) != 0;
    cluster_sync();  // no peer sends into this CTA's shared memory any more
    if (dead) return;
  } else {
    __syncthreads();
  }

  // ---- every row to its position: multipliers, and the U part of a chosen row
#pragma unroll
  for (int u = 0; u < RPT; u++) {
    if (pos[u] == INT_MIN) continue;
    const int row = pos[u] >= 0 ? pos[u] : ~pos[u];
    const int nl = pos[u] >= 0 ? ncols : row;
    T* dst = P + (int64_t)row * a.lda;
    const T* lb = lbuf + u * NT + tid;
    if (vec) {
#pragma unroll 2
      for (int c = 0; c < W; c += V) {
        T x[V];
#pragma unroll
        for (int e = 0; e < V; e++) x[e] = c + e < nl ? lb[(c + e) * LP] : sh.urow[nl][c + e - nl];
        int4 q;
        memcpy(&q, x, 16);
        *reinterpret_cast<int4*>(dst + c) = q;
      }
    } else {
      for (int c = 0; c < ncols; c++) dst[c] = c < nl ? lb[c * LP] : sh.urow[nl][c - nl];
    }
  }
  if (cta == 0 && tid < ncols) {
    const int p = sh.p[tid];
    a.ipiv[tid] = a.row_base + (p < 0 ? tid : p);
    if (p >= 0 && !(fabs((double)sh.piv[tid]) > a.thr)) dev_singular(a.st, a.info_base + tid + 1);
  }

  // ---- the interchanges on the enclosing panel's other columns
  const int others = a.pw - ncols;
  if (others <= 0) return;
  if (warp == 0) {
    // lane r follows the row that stood at r: it is chosen in column fin, or
    // ends at position cur below the top block
    const int pl = lane < ncols ? sh.p[lane] : -1;
    if (lane < ncols) sh.src[lane] = pl < 0 ? lane : pl;
    __syncwarp();
    int cur = lane, fin = lane < ncols ? -1 : 0;
    for (int j = 0; j < ncols; j++) {
      const int q = sh.p[j], p = q < 0 ? j : q;
      if (fin < 0) {
        if (cur == p) fin = j;
        else if (cur == j) cur = p;
      }
    }
    if (lane < ncols && fin >= 0) sh.src[fin] = lane;
    __syncwarp();
    const bool top = lane < ncols && sh.src[lane] != lane;
    const bool low = lane < ncols && fin < 0;
    const unsigned mt = __ballot_sync(0xffffffffu, top), ml = __ballot_sync(0xffffffffu, low);
    const unsigned below = (1u << lane) - 1u;
    if (top) {
      const int o = __popc(mt & below);
      sh.mv_dst[o] = lane;
      sh.mv_src[o] = sh.src[lane];
    }
    if (low) {
      const int o = __popc(mt) + __popc(ml & below);
      sh.mv_dst[o] = cur;
      sh.mv_src[o] = lane;
    }
    if (lane == 0) sh.mv_n = __popc(mt) + __popc(ml);
  }
  __syncthreads();
  const int mv = sh.mv_n;
  const int per = ((others + G - 1) / G + 7) & ~7;
  const int q1 = min(others, (cta + 1) * per);
  constexpr int E = 2 * W * 32 / NT;  // 32 columns of every moved row per pass
  for (int c0 = cta * per; c0 < q1; c0 += 32) {
    const int q = c0 + lane;
    const int col = q < a.lc0 ? q : q + ncols;
    T t[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int r = warp + e * NW;
      if (r < mv && q < q1) t[e] = prow0[(int64_t)sh.mv_src[r] * a.lda + col];
    }
    __syncthreads();  // every source read before any destination is written
#pragma unroll
    for (int e = 0; e < E; e++) {
      const int r = warp + e * NW;
      if (r < mv && q < q1) prow0[(int64_t)sh.mv_dst[r] * a.lda + col] = t[e];
    }
  }
}

template <typename T, int W, int RPT, int XP>
int launch_leaf(T* P, T* prow0, const LeafArgs& a, int G, cudaStream_t s) {
  const void* fn = (const void*)getf2_leaf_kernel<T, W, RPT, XP>;
  constexpr size_t smem = leaf_smem<T, W, RPT, XP>();
  static_assert(smem <= 227 * 1024, "leaf rows exceed shared memory");
  static PerDeviceOnce once;
  LUB_TRY(once_per_device(once, [&] {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && XP == kCluster)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return cuda_status(e);
  }));
  LeafArgs args = a;
  void* ptrs[] = {&P, &prow0, &args};
  if (XP == kCluster) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = may_overlap_launch(s) ? 2 : 1;
    LUB_CUDA(cudaLaunchKernelExC(&cfg, fn, ptrs));
  } else if (XP == kGrid) {
    LUB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(G), dim3(NT), ptrs, smem, s));
  } else {
    return launch_dependent(getf2_leaf_kernel<T, W, RPT, XP>, dim3(1), dim3(NT), smem, s, P, prow0, a);
  }
  __atomic_add_fetch(&g_kernel_launches, 1, __ATOMIC_RELAXED);
  return LU_OK;
}

// Rows per thread at most: W * RPT values fill 192 of a thread's 255
// registers, and as many words of shared memory hold the multipliers.
template <typename T, int W>
constexpr int max_rpt() { return 768 / (W * (int)sizeof(T)); }

template <typename T, int W, int XP>
int launch_leaf_w(T* P, T* prow0, const LeafArgs& a, int G, int rpt, cudaStream_t s) {
  constexpr int RM = max_rpt<T, W>();
  if (rpt <= 1) return launch_leaf<T, W, 1, XP>(P, prow0, a, G, s);
  if (rpt <= 2) return launch_leaf<T, W, 2, XP>(P, prow0, a, G, s);
  if constexpr (XP != kSingle) {
    if (rpt <= 3) return launch_leaf<T, W, 3, XP>(P, prow0, a, G, s);
    if constexpr (RM >= 6) {
      if (rpt <= 4) return launch_leaf<T, W, 4, XP>(P, prow0, a, G, s);
      if (rpt <= 6) return launch_leaf<T, W, 6, XP>(P, prow0, a, G, s);
    }
  }
  return LU_ERR_UNSUPPORTED;
}

// Largest cluster of leaf CTAs the device schedules: 16 needs 16 free SMs in
// one GPC and is not portable.
template <typename T>
int max_cluster() {
  auto probe = getf2_leaf_kernel<T, 16, 1, kCluster>;
  constexpr size_t smem = leaf_smem<T, 16, 6, kCluster>();
  cudaFuncSetAttribute(probe, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  cudaFuncSetAttribute(probe, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kMaxCluster);
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kMaxCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, (const void*)probe, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  return n >= 1 ? kMaxCluster : 8;
}

// Rows per thread of the grid and cluster instances (launch_leaf_w); 8 columns
// wide there is one grid instance of twice as many rows
template <typename T, int W>
constexpr int leaf_rows() { return max_rpt<T, W>() < 6 ? max_rpt<T, W>() : 6; }
constexpr int kTallRows = 12;

inline int leaf_cta_limit(int num_sms) { return std::min(num_sms, kMaxLeafCTAs); }

struct LeafPlan {
  int W, xp, G, R, rpt;  // instance, transport, CTAs, rows per CTA and per thread
};
// One CTA up to 512 rows (two per thread: no exchange at all); alone on the GPU
// (cluster > 0 CTAs in the largest cluster) one cluster, one row per thread
// first, then more CTAs, then more rows; else a cooperative grid, one CTA per
// SM, of at most max_ctas CTAs (more only when the rows need their registers).
template <typename T>
int leaf_plan(int M, int ncols, int num_sms, int max_ctas, int cluster, LeafPlan* p) {
  const int limit = leaf_cta_limit(num_sms);
  p->W = ncols <= 16 ? 16 : 32;
  const int rmax = p->W == 16 ? leaf_rows<T, 16>() : leaf_rows<T, 32>();
  p->G = 1;
  p->xp = kSingle;
  if (M > 2 * NT) {
    if (M <= (int64_t)cluster * NT * rmax) {
      p->xp = kCluster;
      p->G = 2;
      while (p->G < cluster && p->G * NT < M) p->G *= 2;
    } else {
      p->xp = kGrid;
      p->G = std::min(ceil_div(M, NT), std::min(max_ctas, limit));
      p->G = std::max(p->G, ceil_div(M, NT * rmax));
      if (p->G > limit) {  // twice the rows of half the width
        if (ncols > 8) return LU_ERR_UNSUPPORTED;
        p->W = 8;
        p->G = ceil_div(M, NT * kTallRows);
        if (p->G > limit) return LU_ERR_UNSUPPORTED;
      }
    }
  }
  p->R = ceil_div(M, p->G);
  if (p->xp == kGrid) p->G = ceil_div(M, p->R);
  p->rpt = p->W == 8 ? kTallRows : ceil_div(p->R, NT);
  return LU_OK;
}

}  // namespace

// Narrower than 16 only for panels too tall for the registers of every SM.
template <typename T>
int leaf_max_width(int M, int num_sms) {
  const int64_t rows = (int64_t)leaf_cta_limit(num_sms) * NT;
  if (M <= rows * leaf_rows<T, 32>()) return 32;
  if (M <= rows * leaf_rows<T, 16>()) return 16;
  return 8;
}

template <typename T>
int leaf_min_ctas(int M) { return ceil_div(M, NT * leaf_rows<T, 32>()); }

template <typename T>
int launch_getf2_leaf(T* P, int64_t lda, int M, int ncols, int32_t* ipiv, int row_base, ulonglong2* pkt,
                      unsigned tag0, DevStatus* st, int info_base, double thr, long long spin, int max_ctas,
                      bool alone, cudaStream_t s, T* prow0, int pw, int lc0) {
  if (M <= 0 || ncols <= 0) return LU_OK;
  if (ncols > 32) return LU_ERR_ARG;
  if (!prow0) {  // no enclosing panel: the leaf is the whole panel
    prow0 = P;
    pw = ncols;
    lc0 = 0;
  }
  if (lc0 < 0 || lc0 + ncols > pw) return LU_ERR_ARG;
  static int s_cluster[64], s_sms[64];
  static PerDeviceOnce once;
  int dev = 0;
  LUB_CUDA(cudaGetDevice(&dev));
  LUB_TRY(once_per_device(once, [&] {
    s_cluster[dev] = max_cluster<T>();
    return cuda_status(cudaDeviceGetAttribute(&s_sms[dev], cudaDevAttrMultiProcessorCount, dev));
  }));
  LeafPlan p;
  LUB_TRY(leaf_plan<T>(M, ncols, s_sms[dev], max_ctas, alone ? s_cluster[dev] : 0, &p));
  const LeafArgs a{lda, M, ncols, p.R, ipiv, row_base, pkt, tag0, st, info_base, thr, spin, pw, lc0};
  if (p.W == 8) return launch_leaf<T, 8, kTallRows, kGrid>(P, prow0, a, p.G, s);
  if (p.W == 16) {
    if (p.xp == kSingle) return launch_leaf_w<T, 16, kSingle>(P, prow0, a, p.G, p.rpt, s);
    if (p.xp == kGrid) return launch_leaf_w<T, 16, kGrid>(P, prow0, a, p.G, p.rpt, s);
    return launch_leaf_w<T, 16, kCluster>(P, prow0, a, p.G, p.rpt, s);
  }
  if (p.xp == kSingle) return launch_leaf_w<T, 32, kSingle>(P, prow0, a, p.G, p.rpt, s);
  if (p.xp == kGrid) return launch_leaf_w<T, 32, kGrid>(P, prow0, a, p.G, p.rpt, s);
  return launch_leaf_w<T, 32, kCluster>(P, prow0, a, p.G, p.rpt, s);
}

#define LUB_INSTANTIATE_LEAF(T)                                                                                    \
  template int leaf_min_ctas<T>(int);                                                                             \
  template int leaf_max_width<T>(int, int);                                                                       \
  template int launch_getf2_leaf<T>(T*, int64_t, int, int, int32_t*, int, ulonglong2*, unsigned, DevStatus*, int, \
                                    double, long long, int, bool, cudaStream_t, T*, int, int);

}  // namespace lub
