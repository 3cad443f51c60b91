// The small FP64 products and triangular solves of a panel step: C -= A B with
// few columns or few tiles, and B <- L^{-1} B for a whole panel's L in one
// launch (LUBlk::updateMatrix and computeU, lu.C:26-43, 180-189, at the
// sizes of the recursion's halves).
//
// What bounds them: latency.  At order 2048 the 128 x 128 tiles of
// gemm_f64.cu spend 4.3 us of tensor time per 32 of K on tiles of which a
// 32-wide product fills a quarter, on 16 of 148 SMs; and the recursive solve of
// 128 or 256 rows is a chain of 7 or 15 launches.
//
// Both kernels sum in the order of gemm_f64.cu, k 16 at a time as
// 0 2 4 6, 1 3 5 7, 8 10 12 14, 9 11 13 15 (one m16n8k4 each, which is the
// chain of its four fmas), starting from C with A negated, and the solve takes
// the blocks of at most 32 rows that the recursion takes, one fma per
// element and row inside them: the results have the recursion's bits.
//
// B200, whole solves, both kernels: n = 256 0.588 -> 0.508 ms, n = 2048 5.63 ->
// 4.54 ms, n = 4999 20.1 -> 15.7 ms, n = 16384 139.7 -> 131.1 ms.
#include "common.cuh"
#include "kernels.h"

namespace lub {
namespace {

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

// 16 bytes global -> shared of which `bytes` (0, 8 or 16) are read, the rest zero
__device__ __forceinline__ void cp16(void* sdst, const void* gsrc, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(sdst)), "l"(gsrc), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[MI][NJ] -= A[16 MI rows x 16] B[16 x 8 NJ] from shared memory: a at the
// lane's row g of A (pitch LP = 8 mod 16: the quarter-warps' 16-byte loads hit
// distinct banks), b at B's row 0, column g (pitch BP = 2 mod 8: rows 2 t
// apart fall 4 doubles apart)
template <int MI, int NJ, int LP, int BP>
__device__ __forceinline__ void mma16(double (&acc)[MI][NJ][4], const double* a, const double* b, int t) {
#pragma unroll
  for (int half = 0; half < 2; half++) {
    double2 af[MI][2];
#pragma unroll
    for (int mi = 0; mi < MI; mi++)
#pragma unroll
      for (int h = 0; h < 2; h++)
        af[mi][h] = *reinterpret_cast<const double2*>(a + (16 * mi + 8 * h) * LP + 2 * t + 8 * half);
    double bf[NJ][2];
#pragma unroll
    for (int nj = 0; nj < NJ; nj++)
#pragma unroll
      for (int q = 0; q < 2; q++) bf[nj][q] = b[(2 * t + q + 8 * half) * BP + 8 * nj];
#pragma unroll
    for (int q = 0; q < 2; q++)
#pragma unroll
      for (int mi = 0; mi < MI; mi++) {
        const double a0 = -(q == 0 ? af[mi][0].x : af[mi][0].y);
        const double a1 = -(q == 0 ? af[mi][1].x : af[mi][1].y);
#pragma unroll
        for (int nj = 0; nj < NJ; nj++) dmma(acc[mi][nj], a0, a1, bf[nj][q]);
      }
  }
}

// ---- C (M x N) -= A (M x K) B (K x N): 64 x 32 tiles, 4 warps of 32 x 16, K
// in double-buffered slices of 32
constexpr int GM = 64, GN = 32, GK = 32, GT = 128;
constexpr int GLP = GK + 8, GBP = GN + 2;
constexpr int kSmallStage = GM * GLP + GK * GBP;  // doubles
constexpr size_t kSmallSmem = 2 * kSmallStage * sizeof(double);

__global__ void __launch_bounds__(GT) gemm_f64_small_kernel(const double* A, int64_t lda, const double* B,
                                                            int64_t ldb, double* C, int64_t ldc, int M, int N, int K) {
  extern __shared__ __align__(16) double smem_d[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int r0 = blockIdx.x * GM, c0 = blockIdx.y * GN;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 16;
  const int KT = (K + GK - 1) / GK;
  auto stage = [&](int kt) {
    double* sa = smem_d + (kt & 1) * kSmallStage;
    double* sb = sa + GM * GLP;
    const int k0 = kt * GK;
#pragma unroll
    for (int u = 0; u < GM * GK / 2 / GT; u++) {
      const int idx = tid + u * GT, r = idx / (GK / 2), k = (idx % (GK / 2)) * 2;
      const int live = r0 + r < M ? max(0, min(2, K - k0 - k)) : 0;
      cp16(sa + r * GLP + k, live ? A + (int64_t)(r0 + r) * lda + k0 + k : A, 8 * live);
    }
#pragma unroll
    for (int u = 0; u < GK * GN / 2 / GT; u++) {
      const int idx = tid + u * GT, k = idx / (GN / 2), c = (idx % (GN / 2)) * 2;
      const int live = k0 + k < K ? max(0, min(2, N - c0 - c)) : 0;
      cp16(sb + k * GBP + c, live ? B + (int64_t)(k0 + k) * ldb + c0 + c : B, 8 * live);
    }
    cp_commit();
  };
  after_previous_kernel();
  stage(0);
  double acc[2][2][4];
  double* Cp[2][2];
  const int cc = c0 + wc + 2 * t;
#pragma unroll
  for (int mi = 0; mi < 2; mi++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = r0 + wr + 16 * mi + 8 * h + g;
      Cp[mi][h] = C + (int64_t)r * ldc + cc;
#pragma unroll
      for (int nj = 0; nj < 2; nj++) {
        double2 v = make_double2(0.0, 0.0);
        if (r < M) {
          if (cc + 8 * nj + 1 < N) v = *reinterpret_cast<const double2*>(Cp[mi][h] + 8 * nj);
          else if (cc + 8 * nj < N) v.x = Cp[mi][h][8 * nj];
        }
        acc[mi][nj][2 * h] = v.x;
        acc[mi][nj][2 * h + 1] = v.y;
      }
    }
  for (int kt = 0; kt < KT; kt++) {
    cp_wait<0>();
    __syncthreads();  // slice kt in shared memory; everyone is done with slice kt - 1
    if (kt + 1 < KT) stage(kt + 1);
    const double* sa = smem_d + (kt & 1) * kSmallStage;
    const double* sb = sa + GM * GLP;
#pragma unroll
    for (int k = 0; k < GK; k += 16) mma16<2, 2, GLP, GBP>(acc, sa + (wr + g) * GLP + k, sb + k * GBP + wc + g, t);
  }
#pragma unroll
  for (int mi = 0; mi < 2; mi++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      if (r0 + wr + 16 * mi + 8 * h + g >= M) continue;
#pragma unroll
      for (int nj = 0; nj < 2; nj++) {
        if (cc + 8 * nj + 1 < N)
          *reinterpret_cast<double2*>(Cp[mi][h] + 8 * nj) = make_double2(acc[mi][nj][2 * h], acc[mi][nj][2 * h + 1]);
        else if (cc + 8 * nj < N) Cp[mi][h][8 * nj] = acc[mi][nj][2 * h];
      }
    }
}

// ---- B (w x ncols) <- L^{-1} B, w <= 256: one CTA per CB columns, the columns
// in shared memory for the whole solve; L's block columns (rows from the
// diagonal block down) stream through two buffers, block j + 1 in flight
// while block j is applied
constexpr int kStripW = 256, ST = 256, SLP = 32 + 8;
struct StripBlocks {
  int n;
  int at[kStripW / 16 + 2];  // block boundaries; each block at most 32 rows
};
template <int CB>
constexpr size_t strip_smem(int w) {
  const int rows = (w + 31) & ~31;
  return ((size_t)rows * (CB + 2) + (size_t)(rows + std::max(rows - 16, 32)) * SLP) * sizeof(double);
}

template <int CB>
__global__ void __launch_bounds__(ST) trsm_strip_kernel(const double* L, int64_t ldl, double* B,
                                                        int64_t ldb, int w, int ncols,
                                                        const __grid_constant__ StripBlocks blk) {
  constexpr int XP = CB + 2;
  extern __shared__ __align__(16) double smem_d[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rows = (w + 31) & ~31;
  double* X = smem_d;                     // [rows][XP]
  double* Lb[2] = {X + (size_t)rows * XP, X + (size_t)rows * XP + (size_t)rows * SLP};
  const int c0 = blockIdx.x * CB, nc = min(CB, ncols - c0);
  after_previous_kernel();
  for (int idx = tid; idx < rows * (CB / 2); idx += ST) {
    const int r = idx / (CB / 2), c = (idx % (CB / 2)) * 2;
    const int live = r < w ? max(0, min(2, nc - c)) : 0;
    cp16(X + r * XP + c, live ? B + (int64_t)r * ldb + c0 + c : B, 8 * live);
  }
  auto stage = [&](int j) {
    const int l0 = blk.at[j], kb = blk.at[j + 1] - l0;
    double* dst = Lb[j & 1];
    for (int idx = tid; idx < (w - l0) * 16; idx += ST) {
      const int r = idx >> 4, k = (idx & 15) * 2;
      const int live = max(0, min(2, kb - k));
      cp16(dst + r * SLP + k, live ? L + (int64_t)(l0 + r) * ldl + l0 + k : L, 8 * live);
    }
    cp_commit();
  };
  stage(0);
  for (int j = 0; j < blk.n; j++) {
    const int l0 = blk.at[j], l1 = blk.at[j + 1], kb = l1 - l0;
    cp_wait<0>();
    __syncthreads();  // block j of L (and, at j = 0, the columns) in shared memory; block j - 1 applied
    if (j + 1 < blk.n) stage(j + 1);
    const double* ls = Lb[j & 1];
    if (tid < CB) {  // the diagonal block: one column per thread
      double x[32];
      double* xc = X + l0 * XP + tid;
#pragma unroll
      for (int i = 0; i < 32; i++) x[i] = i < kb ? xc[i * XP] : 0.0;
      solve_unit_lower32(x, ls, SLP, kb);
#pragma unroll
      for (int i = 1; i < 32; i++)
        if (i < kb) xc[i * XP] = x[i];
    }
    __syncthreads();
    // rows below, 16 x 16 per warp and turn
    const int nrt = (w - l1 + 15) / 16, units = nrt * (CB / 16);
    for (int u = warp; u < units; u += ST / 32) {
      const int r = l1 + (u / (CB / 16)) * 16, wc = (u % (CB / 16)) * 16;
      double acc[1][2][4];
      double* xp = X + (r + g) * XP + wc + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const bool ok = r + 8 * h + g < w;
#pragma unroll
        for (int nj = 0; nj < 2; nj++) {
          const double2 v = ok ? *reinterpret_cast<const double2*>(xp + 8 * h * XP + 8 * nj) : make_double2(0.0, 0.0);
          acc[0][nj][2 * h] = v.x;
          acc[0][nj][2 * h + 1] = v.y;
        }
      }
      // rows past w of the last tile read staged rows of an earlier block or
      // the padding; they are not stored
      const int lr = min(r - l0 + g, w - l0 - 1), lr8 = min(r - l0 + g + 8, w - l0 - 1);
      for (int k = 0; k < kb; k += 16) {
        const double* b = X + (l0 + k) * XP + wc + g;
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const double2 a0 = *reinterpret_cast<const double2*>(ls + lr * SLP + k + 2 * t + 8 * half);
          const double2 a1 = *reinterpret_cast<const double2*>(ls + lr8 * SLP + k + 2 * t + 8 * half);
          double bf[2][2];
#pragma unroll
          for (int nj = 0; nj < 2; nj++)
#pragma unroll
            for (int q = 0; q < 2; q++) bf[nj][q] = b[(2 * t + q + 8 * half) * XP + 8 * nj];
#pragma unroll
          for (int nj = 0; nj < 2; nj++) dmma(acc[0][nj], -a0.x, -a1.x, bf[nj][0]);
#pragma unroll
          for (int nj = 0; nj < 2; nj++) dmma(acc[0][nj], -a0.y, -a1.y, bf[nj][1]);
        }
      }
#pragma unroll
      for (int h = 0; h < 2; h++)
        if (r + 8 * h + g < w)
#pragma unroll
          for (int nj = 0; nj < 2; nj++)
            *reinterpret_cast<double2*>(xp + 8 * h * XP + 8 * nj) =
                make_double2(acc[0][nj][2 * h], acc[0][nj][2 * h + 1]);
    }
  }
  __syncthreads();
  for (int idx = tid; idx < w * (CB / 2); idx += ST) {
    const int r = idx / (CB / 2), c = (idx % (CB / 2)) * 2;
    double* dst = B + (int64_t)r * ldb + c0 + c;
    if (c + 1 < nc) *reinterpret_cast<double2*>(dst) = *reinterpret_cast<const double2*>(X + r * XP + c);
    else if (c < nc) *dst = X[r * XP + c];
  }
}

// the recursion's blocks: halves (a multiple of 16 first) down to 32 rows
void strip_blocks(int l0, int w, StripBlocks& b) {
  if (w <= 32) {
    b.at[b.n++] = l0;
    return;
  }
  const int h = w / 2, w1 = h >= 16 ? (h & ~15) : std::max(h & ~1, 2);
  strip_blocks(l0, w1, b);
  strip_blocks(l0 + w1, w - w1, b);
}

template <int CB>
int launch_strip(const double* L, int64_t ldl, double* B, int64_t ldb, int w, int ncols, const StripBlocks& blk,
                 cudaStream_t s) {
  static PerDeviceOnce once;
  LUB_TRY(once_per_device(once, [] {
    return cuda_status(cudaFuncSetAttribute(trsm_strip_kernel<CB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            (int)strip_smem<CB>(kStripW)));
  }));
  return launch_dependent(trsm_strip_kernel<CB>, dim3(ceil_div(ncols, CB)), dim3(ST), strip_smem<CB>(w), s, L, ldl, B,
                          ldb, w, ncols, blk);
}

}  // namespace

int launch_gemm_f64_small(const double* A, int64_t lda, const double* B, int64_t ldb, double* C, int64_t ldc, int M,
                          int N, int K, cudaStream_t s) {
  if (M <= 0 || N <= 0 || K <= 0) return LU_OK;
  static PerDeviceOnce once;
  LUB_TRY(once_per_device(once, [] {
    return cuda_status(
        cudaFuncSetAttribute(gemm_f64_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem));
  }));
  dim3 grid(ceil_div(M, GM), ceil_div(N, GN));
  if (grid.y > 65535) return LU_ERR_UNSUPPORTED;
  return launch_dependent(gemm_f64_small_kernel, grid, dim3(GT), kSmallSmem, s, A, lda, B, ldb, C, ldc, M, N, K);
}

int launch_trsm_f64_strip(const double* L, int64_t ldl, double* B, int64_t ldb, int w, int ncols, cudaStream_t s) {
  if (w <= 0 || ncols <= 0) return LU_OK;
  if (w > kStripW) return LU_ERR_ARG;
  StripBlocks blk;
  blk.n = 0;
  strip_blocks(0, w, blk);
  blk.at[blk.n] = w;
  // narrower strips while the wider ones would leave half of the SMs idle
  if (ncols <= 16 * kNumSMsB200) return launch_strip<16>(L, ldl, B, ldb, w, ncols, blk, s);
  return launch_strip<32>(L, ldl, B, ldb, w, ncols, blk, s);
}

}  // namespace lub
