// fused_elementwise.h -- launchers of the model kernels in fused_elementwise.cu.  Pointers are
// device memory, 16-byte aligned where they name bf16 data; shapes have been checked by the
// caller (torch_ops.cpp); sms is the device's number of multiprocessors.  rows and tokens are
// at least 1.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace fcxops {

cudaError_t rmsnormForward(const void *x, const void *w, void *y, float *rstd, long rows, int H, float eps,
                           cudaStream_t stream);
// partial: scratch of rmsnormPartials(rows, H, sms) x H floats; add may be null
int rmsnormPartials(long rows, int H, int sms);
cudaError_t rmsnormBackward(const void *g, const void *x, const void *w, const float *rstd, const void *add, void *dx, void *dw,
                            float *partial, long rows, int H, int sms, cudaStream_t stream);
cudaError_t rope(void *x, const int *positions, int tokens, int heads, int D, float logTheta, float sign, cudaStream_t stream);
cudaError_t ropeQkv(const void *qkv, void *out, int tokens, int ropeHeads, int totalHeads, int D, float logTheta, float sign,
                    cudaStream_t stream);
cudaError_t swigluForward(const void *ab, void *out, size_t T, int F, cudaStream_t stream);
cudaError_t swigluBackward(const void *g, const void *ab, void *dab, size_t T, int F, cudaStream_t stream);
cudaError_t crossEntropy(void *logits, const long *targets, float *loss, long rows, int V, float gradScale, int sms,
                         cudaStream_t stream);
cudaError_t adamw(void *p, const void *g, void *m, void *v, size_t n, float lr, float beta1, float beta2, float eps, float wd,
                  float bc1, float bc2, cudaStream_t stream);

} // namespace fcxops
