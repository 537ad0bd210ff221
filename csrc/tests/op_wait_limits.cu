// op_wait_limits.cu -- the model kernels with a wait limit of 20 ms and a row whose copy is never
// started, so that the waits for it run out; tests/test_gpu_op_wait_limits.py checks what the
// kernels make of that.
#define FLAGCX_OPS_WAIT_NS 20000000ull
#define FLAGCX_OPS_HELD_BACK(row) ((long)(row) == heldBackRow)
static __device__ long heldBackRow = -1;
#include "../../flagcx_b200/ops/csrc/fused_elementwise.cu"

extern "C" {

int hold_back(long row) { return cudaMemcpyToSymbol(heldBackRow, &row, sizeof row); }

int norm_partials(long rows, int H, int sms) { return fcxops::rmsnormPartials(rows, H, sms); }

int norm_backward(const void *g, const void *x, const void *w, const float *rstd, const void *add, void *dx, void *dw,
                  float *partial, long rows, int H, int sms) {
  const cudaError_t e = fcxops::rmsnormBackward(g, x, w, rstd, add, dx, dw, partial, rows, H, sms, nullptr);
  return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

int cross_entropy(void *logits, const long *targets, float *loss, long rows, int V, float gradScale, int sms) {
  const cudaError_t e = fcxops::crossEntropy(logits, targets, loss, rows, V, gradScale, sms, nullptr);
  return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

} // extern "C"
