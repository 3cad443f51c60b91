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
