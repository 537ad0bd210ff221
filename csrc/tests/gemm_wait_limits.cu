// gemm_wait_limits.cu -- the GEMM that splits K over a cluster with a wait limit of 20 ms and a K
// step whose operands are not fetched, so that the waits for them run out.  They arrive after the
// CTA has given up.  tests/test_gpu_op_wait_limits.py checks what the kernel makes of that.
#define FLAGCX_GEMM_WAIT_NS 20000000ull
#define FLAGCX_GEMM_HELD_BACK(tile, kb) ((tile) == heldBack[0] && (kb) == heldBack[1])
#define FLAGCX_GEMM_GIVEN_UP(load)                                                                          \
  if (heldBack[1] >= kb0 && heldBack[1] < kb0 + issued) {                                                   \
    const int j = heldBack[1] - kb0;                                                                        \
    load(heldBack[1], j % STAGES);                                                                          \
    mbarWait(&s.full[j % STAGES], (uint32_t)(j / STAGES) & 1u, &never, kWaitLimitNs);                       \
  }
static __device__ int heldBack[2] = {-1, -1};
#define fcx fcx_gemmwait // in a process that has the library, whose functions would be taken for these
#include "../kernels/split_gemm.cu"

namespace {

int tensorMap(CUtensorMap *map, const void *base, int rows, int cols, int boxRows) {
  void *fn = nullptr;
  cudaDriverEntryPointQueryResult found;
  const cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
  if (e != cudaSuccess || !fn) return 1;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)boxRows}, steps[2] = {1, 1};
  return (int)((decltype(&cuTensorMapEncodeTiled))fn)(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims,
                                                      strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

} // namespace

extern "C" {

// Of the tile-th tile K step kb is held back (-1: none).
int hold_back_step(int tile, int kb) {
  const int held[2] = {tile, kb};
  return (int)cudaMemcpyToSymbol(heldBack, held, sizeof held);
}

int split_gemm(const void *a, const void *b, void *d, int M, int N, int K, int parts, int tileN) {
  CUtensorMap ta, tb;
  if (tensorMap(&ta, a, M, K, 128) || tensorMap(&tb, b, N, K, tileN)) return 1;
  fcx::SplitGemmPlan plan;
  plan.parts = parts;
  plan.tileN = tileN;
  const cudaError_t e = fcx::launchSplitGemm(nullptr, ta, tb, d, M, N, K, plan);
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}

} // extern "C"
