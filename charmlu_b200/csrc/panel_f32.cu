// The FP32 instances of the panel leaf.
#include "panel.cuh"

namespace lub {
LUB_INSTANTIATE_LEAF(float)
}  // namespace lub

// Test hook: one FP32 leaf (ncols <= 32 at column lc0 of a panel of pw
// columns) with its own packet buffer; max_ctas and alone choose the grid.
// Returns the status word's code, or the 1-based first singular column.
extern "C" __attribute__((visibility("default"))) int lub_test_getf2_leaf(float* prow0, int64_t lda, int M, int ncols,
                                                                          int pw, int lc0, int32_t* ipiv,
                                                                          int max_ctas, int alone, void* stream) {
  using namespace lub;
  cudaStream_t s = (cudaStream_t)stream;
  ulonglong2* pkt = nullptr;
  const size_t bytes = sizeof(ulonglong2) * kLeafPackets;
  LUB_CUDA(cudaMallocAsync((void**)&pkt, bytes + sizeof(DevStatus), s));
  DevStatus* st = reinterpret_cast<DevStatus*>(pkt + kLeafPackets);
  LUB_CUDA(cudaMemsetAsync(pkt, 0, bytes + sizeof(DevStatus), s));
  int rc = launch_getf2_leaf<float>(prow0 + lc0, lda, M, ncols, ipiv, 0, pkt, 64, st, 0, 0.0, 1LL << 22, max_ctas,
                                    alone != 0, s, prow0, pw, lc0);
  DevStatus h;
  LUB_CUDA(cudaMemcpyAsync(&h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
  LUB_CUDA(cudaFreeAsync(pkt, s));
  LUB_CUDA(cudaStreamSynchronize(s));
  return rc != LU_OK ? rc : (h.code != 0 ? h.code : h.info);
}

// Test hook (no GPU): the launch taken for a leaf, out = {widest leaf for M
// rows, status, instance width, transport, CTAs, rows per CTA, rows per thread}.
// cluster: CTAs of the largest cluster (0: another kernel runs beside it).
extern "C" __attribute__((visibility("default"))) int lub_test_leaf_plan(int esize, int M, int ncols, int num_sms,
                                                                         int max_ctas, int cluster, int* out) {
  using namespace lub;
  LeafPlan p{};
  out[0] = esize == 8 ? leaf_max_width<double>(M, num_sms) : leaf_max_width<float>(M, num_sms);
  out[1] = esize == 8 ? leaf_plan<double>(M, ncols, num_sms, max_ctas, cluster, &p)
                      : leaf_plan<float>(M, ncols, num_sms, max_ctas, cluster, &p);
  out[2] = p.W;
  out[3] = p.xp;
  out[4] = p.G;
  out[5] = p.R;
  out[6] = p.rpt;
  return LU_OK;
}
