// op_wait_limits.cu -- the model kernels with a wait limit of 20 ms and a row whose copy is never
// started, so that the waits for it run out, or with answers to requests for a row that count as
// not seen in time; tests/test_gpu_op_wait_limits.py checks what the kernels make of that.
#define FLAGCX_OPS_WAIT_NS 20000000ull
#define FLAGCX_OPS_HELD_BACK(row) ((long)(row) == heldBackRow)
#define FLAGCX_OPS_UNSEEN(request) (blockIdx.x == unseen[0] && (request) == unseen[1] ? unseen[2] : 0)
static __device__ long heldBackRow = -1;
static __device__ unsigned unseen[3] = {0, 0, 0};
#include "../../flagcx_b200/ops/csrc/fused_elementwise.cu"

extern "C" {

int hold_back(long row) { return cudaMemcpyToSymbol(heldBackRow, &row, sizeof row); }

// Of the requests of the cluster that starts with CTA `block`, `waits` waits for the nth do not see its answer.
int leave_unseen(unsigned block, unsigned nth, unsigned waits) {
  const unsigned u[3] = {block, nth, waits};
  return cudaMemcpyToSymbol(unseen, u, sizeof u);
}

int norm_forward(const void *x, const void *w, void *y, float *rstd, long rows, int H) {
  const cudaError_t e = fcxops::rmsnormForward(x, w, y, rstd, rows, H, 1e-5f, nullptr);
  return e != cudaSuccess ? e : cudaDeviceSynchronize();
}

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
