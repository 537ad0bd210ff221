// split_gemm.h -- launcher of the GEMM that splits K over a cluster of CTAs.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace fcx {

constexpr int kSplitGemmMaxParts = 8; // the portable cluster size

struct SplitGemmPlan {
  int tileN = 0; // 256, 128 or 64; 0: use the persistent kernel
  int parts = 1; // CTAs that share a tile's K
};

// The last `count` tiles, from `first` on, of the persistent kernel's order: tileRows x 256
// outputs, walked in groups of groupRows row blocks, column by column.  count = 0: the whole
// output.
struct SplitGemmTail {
  int first = 0, count = 0, tileRows = 128, groupRows = 1;
};

// tmB's box is tileN rows; parts <= K / 64.
cudaError_t launchSplitGemm(cudaStream_t stream, const CUtensorMap &tmA, const CUtensorMap &tmB, void *D, int M, int N, int K,
                            const SplitGemmPlan &plan, const SplitGemmTail &tail = {});

} // namespace fcx
