// fused_elementwise.cu -- the memory-bound model kernels that sit between the GEMMs
// of a Llama-shaped decoder: RMSNorm (forward, backward), rotary embedding
// (in place, forward/backward by sign), SwiGLU (forward, backward), softmax
// cross-entropy with the gradient written in place of the logits, and a flat
// AdamW step.  All are sm_100a kernels with 16-byte accesses and fp32 math; each
// reads its operands once and writes its results once.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>

#include "fused_elementwise.h"
#include "launch_state.h"
#include "norm_route.h"

namespace cg = cooperative_groups;

namespace {

using bf16 = __nv_bfloat16;
using fcxops::kNormBwdThreads;
using fcxops::kNormFewRows;

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warpMax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide reductions through shared memory; `red` holds 32 floats.
__device__ __forceinline__ float blockSum(float v, float *red) {
  v = warpSum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
  if (threadIdx.x < 32) t = warpSum(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}
__device__ __forceinline__ float blockMax(float v, float *red) {
  v = warpMax(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : -INFINITY;
  if (threadIdx.x < 32) t = warpMax(t);
  if (threadIdx.x == 0) red[0] = t;
  __syncthreads();
  return red[0];
}

__device__ __forceinline__ uint32_t sharedAddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// How long a copy may take before a kernel gives up on it, the row that is never fetched, and how
// many of the two waits for the answer to a request are taken as having run out (a test of the waits
// that run out sets all three; there are none otherwise).
#ifndef FLAGCX_OPS_WAIT_NS
#define FLAGCX_OPS_WAIT_NS 1000000000ull
#define FLAGCX_OPS_HELD_BACK(row) false
#define FLAGCX_OPS_UNSEEN(request) 0
#endif

// Waits for a phase of an mbarrier for at most about one second.
__device__ __forceinline__ bool mbarWaitBounded(uint64_t *bar, uint32_t parity) {
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(sharedAddr(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 63) == 63) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > FLAGCX_OPS_WAIT_NS) return false;
    }
  }
}

// One bulk asynchronous copy global -> this CTA's shared memory, counted on an mbarrier.
// Both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulkLoad(void *dstShared, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   sharedAddr(dstShared)),
               "l"(src), "r"(bytes), "r"(sharedAddr(bar))
               : "memory");
}
__device__ __forceinline__ void mbarInit(uint64_t *bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sharedAddr(bar)) : "memory");
}
__device__ __forceinline__ void mbarExpect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sharedAddr(bar)), "r"(bytes) : "memory");
}

// The weight gradient's sum over CTAs is launched with programmatic serialization: it may be set up
// while the backward runs (letNextGridStart), and reads nothing before that is done and visible.
__device__ __forceinline__ void letNextGridStart() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void waitForEarlierGrid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

struct Pack8 {
  uint4 raw;
  __device__ float get(int i) const { return __bfloat162float(((const bf16 *)&raw)[i]); }
  __device__ void set(int i, float v) { ((bf16 *)&raw)[i] = __float2bfloat16_rn(v); }
};

// ---------------------------------------------------------------------------
// RMSNorm: y = x * rstd * w,  rstd = rsqrt(mean(x^2) + eps), H a multiple of 8.  A group of GT
// threads takes a row and holds it in registers (PPT packs of 8 per thread); a CTA has four warps
// or one group.  The row and the weights are on their way before the sum of squares is taken; the
// hardware deals the CTAs out.  Bound: HBM for many rows, the chain load -> sum -> store for few.
// Four packs per thread where they hold the row (eight of 256 threads beyond 8192 elements), us
// against one warp per row up to 4096 elements and 512 threads beyond: 128 x 4096 8.3 -> 3.4, 1021 x
// 4096 10.1 -> 6.1, 4096 x 4096 16.9 -> 14.4, 3000 x 2560 12.2 -> 9.1, 512 x 8192 6.2 -> 6.1, 1000 x
// 16384 16.4 -> 14.5; at 512 threads with one pack each 1021 x 4096 takes 8.0, at 256 with two 6.3.
// ---------------------------------------------------------------------------
template <int GT>
constexpr int kNormFwdThreads = GT < 128 ? 128 : GT;

template <int GT, int PPT>
__global__ void __launch_bounds__(kNormFwdThreads<GT>)
rmsnormFwd(const bf16 *__restrict__ x, const bf16 *__restrict__ w, bf16 *__restrict__ y, float *__restrict__ rstdOut, long rows,
           int H, float eps) {
  constexpr int T = kNormFwdThreads<GT>, G = T / GT;
  __shared__ float red[T / 32];
  const int group = threadIdx.x / GT, t = threadIdx.x % GT, nPacks = H / 8;
  const long row = (long)blockIdx.x * G + group;
  const bool live = row < rows;
  const uint4 *xr = (const uint4 *)(x + row * H);
  Pack8 px[PPT], pw[PPT];
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int p = t + k * GT;
    px[k].raw = live && p < nPacks ? xr[p] : make_uint4(0, 0, 0, 0);
  }
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int p = t + k * GT;
    if (p < nPacks) pw[k].raw = ((const uint4 *)w)[p];
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < PPT; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) { const float v = px[k].get(i); ss += v * v; }
  ss = warpSum(ss);
  if constexpr (GT > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < GT / 32; ++i) ss += red[group * (GT / 32) + i];
  }
  if (!live) return;
  const float rstd = rsqrtf(ss / H + eps);
  if (t == 0) rstdOut[row] = rstd;
  uint4 *yr = (uint4 *)(y + row * H);
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int p = t + k * GT;
    if (p < nPacks) {
      Pack8 po;
#pragma unroll
      for (int i = 0; i < 8; ++i) po.set(i, px[k].get(i) * rstd * pw[k].get(i));
      yr[p] = po.raw;
    }
  }
}

// Backward: dx = rstd * (g*w - x * rstd^2 * mean(g*w*x)); the weight gradient is summed
// per CTA in fp32 (thread t owns the same columns for all of its CTA's rows) and the
// partials are added up by columnSumToBf16.
//
// Few rows: one CTA of 512 threads per row, or two rows for each of the CTAs that run at once.
// Both come in by bulk asynchronous copies of (g, x, the gradient to be added) that complete on one
// mbarrier per row and are under way before the first is needed.  Bound: the latency of copy, dot
// product, block-wide sum and store (64 x 4096 takes 5.7 us with the sum over CTAs that follows).
template <int MAXP>
__global__ void __launch_bounds__(kNormBwdThreads)
rmsnormBwdFewRows(const bf16 *__restrict__ g, const bf16 *__restrict__ x, const bf16 *__restrict__ w,
                  const float *__restrict__ rstdIn, const bf16 *__restrict__ addIn, bf16 *__restrict__ dx,
                  float *__restrict__ dwPartial, int rows, int H) {
  extern __shared__ __align__(128) unsigned char slots[];
  __shared__ float red[32];
  __shared__ __align__(8) uint64_t full[kNormFewRows];
  letNextGridStart();
  const int nPacks = H / 8;
  const uint32_t rowBytes = (uint32_t)H * 2u;
  // a slot holds the g row, the x row and, when a gradient of the same shape is to be added
  // to dx (the residual branch around the norm), that gradient's row
  const uint32_t slotBytes = (addIn ? 3u : 2u) * rowBytes;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kNormFewRows; ++s) mbarInit(&full[s]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < kNormFewRows; ++s) {
      const size_t row = blockIdx.x + (size_t)s * gridDim.x;
      if (row >= (size_t)rows || FLAGCX_OPS_HELD_BACK(row)) continue;
      unsigned char *dst = slots + (size_t)s * slotBytes;
      mbarExpect(&full[s], slotBytes);
      bulkLoad(dst, g + row * H, rowBytes, &full[s]);
      bulkLoad(dst + rowBytes, x + row * H, rowBytes, &full[s]);
      if (addIn) bulkLoad(dst + 2 * rowBytes, addIn + row * H, rowBytes, &full[s]);
    }
  }
  __syncthreads();

  float dwAcc[MAXP][8];
  Pack8 pw[MAXP];
#pragma unroll
  for (int k = 0; k < MAXP; ++k) {
    int p = threadIdx.x + k * blockDim.x;
    if (p < nPacks) pw[k].raw = ((const uint4 *)w)[p];
#pragma unroll
    for (int i = 0; i < 8; ++i) dwAcc[k][i] = 0.f;
  }
  bool ok = true;
  for (int s = 0; s < kNormFewRows; ++s) {
    const size_t row = blockIdx.x + (size_t)s * gridDim.x;
    if (row >= (size_t)rows) break;
    const float rstd = rstdIn[row];
    // Every thread goes on through the same barriers whatever its wait returned.  After one that
    // ran out this CTA's row (or rows) from there on and its part of the weight gradient are NaN;
    // the copies that are out land (or are given as long again) first.
    if (ok && !(ok = mbarWaitBounded(&full[s], 0)) && threadIdx.x == 0)
      for (int k = s; k < kNormFewRows && blockIdx.x + (size_t)k * gridDim.x < (size_t)rows; ++k) mbarWaitBounded(&full[k], 0);
    const uint4 *gs = (const uint4 *)(slots + (size_t)s * slotBytes), *xs = gs + nPacks, *as = xs + nPacks;
    Pack8 pg[MAXP], px[MAXP], pa[MAXP];
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < MAXP; ++k) {
      int p = threadIdx.x + k * blockDim.x;
      if (p < nPacks) {
        pg[k].raw = gs[p];
        px[k].raw = xs[p];
        if (addIn) pa[k].raw = as[p];
#pragma unroll
        for (int i = 0; i < 8; ++i) dot += pg[k].get(i) * pw[k].get(i) * px[k].get(i);
      }
    }
    dot = blockSum(ok ? dot : NAN, red);
    const float c = dot * rstd * rstd / H;
    uint4 *dxr = (uint4 *)(dx + row * H);
#pragma unroll
    for (int k = 0; k < MAXP; ++k) {
      int p = threadIdx.x + k * blockDim.x;
      if (p < nPacks) {
        Pack8 po;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float gv = pg[k].get(i), xv = px[k].get(i);
          float d = rstd * (gv * pw[k].get(i) - xv * c);
          if (addIn) d += pa[k].get(i);
          po.set(i, d);
          dwAcc[k][i] += gv * xv * rstd;
        }
        dxr[p] = po.raw;
      }
    }
  }
  float *out = dwPartial + (size_t)blockIdx.x * H;
  const float bad = ok ? 0.f : NAN;
#pragma unroll
  for (int k = 0; k < MAXP; ++k) {
    int p = threadIdx.x + k * blockDim.x;
    if (p < nPacks) {
      *(float4 *)(out + p * 8) = make_float4(dwAcc[k][0] + bad, dwAcc[k][1] + bad, dwAcc[k][2] + bad, dwAcc[k][3] + bad);
      *(float4 *)(out + p * 8 + 4) = make_float4(dwAcc[k][4] + bad, dwAcc[k][5] + bad, dwAcc[k][6] + bad, dwAcc[k][7] + bad);
    }
  }
}

// The same for more rows (norm_route.h says where the line lies).  A CTA is cut into groups of GT
// threads, the fewest (a power of two from 32) that hold a row with four packs per thread; every
// group owns a ring of row slots in shared memory, which its first thread keeps full with bulk
// copies that complete on one mbarrier per slot, and reduces its rows by itself: shuffles, and for
// GT > 32 one named barrier of the group.  So a CTA has 512 / GT rows in work and as many or more
// on their way, and nothing waits for the whole block.  Bound: the chain wait -> dot product ->
// sum -> store of each row, and 128 registers (with four packs per thread and the weights widened
// ahead of the loop 16 bytes too few: 8192 x 8192 96.0 us instead of 86.0, which is 6.2 TB/s, 4096 x 4096
// 30.9 instead of 28.8).  Device time
// with the sum over CTAs and a skip gradient, against one row per CTA at every size: 8192 x 1024
// 37.1 -> 18.8 us, 8192 x 256 34.2 -> 8.7, 4096 x 2560 27.9 -> 20.4, 2048 x 5120 28.7 -> 19.0,
// 2048 x 16384 58.1 -> 51.0.
constexpr int kNormThreads = 512, kNormMaxStages = 6, kNormPacks = 4, kNormRingBytes = 200 << 10;

// Sum over a group of GT threads; every thread gets it.  red holds one float per warp of the
// CTA, alternately the first and the second 16 (parity), so that one barrier per sum is enough:
// a half is written again only after the next sum's barrier, which follows its last read.
template <int GT>
__device__ __forceinline__ float groupSum(float v, float (*red)[kNormThreads / 32], int parity, int group) {
  v = warpSum(v);
  if constexpr (GT > 32) {
    constexpr int W = GT / 32;
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red[parity][warp] = v;
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GT) : "memory");
    v = 0.f;
#pragma unroll
    for (int i = 0; i < W; ++i) v += red[parity][group * W + i];
  } else {
    __syncwarp();
  }
  return v;
}

// The weight gradient is summed in fp32 per group (a thread owns the same columns for all of
// its rows), then over the CTA's groups in their order, then over CTAs by columnSumToBf16.
template <int GT, int PPT>
__global__ void __launch_bounds__(kNormThreads)
rmsnormBwdRing(const bf16 *__restrict__ g, const bf16 *__restrict__ x, const bf16 *__restrict__ w,
               const float *__restrict__ rstdIn, const bf16 *__restrict__ addIn, bf16 *__restrict__ dx,
               float *__restrict__ dwPartial, long rows, int H, int stages) {
  extern __shared__ __align__(128) unsigned char ring[];
  constexpr int G = kNormThreads / GT;
  __shared__ float red[2][kNormThreads / 32];
  __shared__ __align__(8) uint64_t full[G * kNormMaxStages];
  letNextGridStart();
  const int group = threadIdx.x / GT, t = threadIdx.x % GT;
  const int nPacks = H / 8;
  const uint32_t rowBytes = (uint32_t)H * 2u;
  // a slot holds the g row, the x row and, when a gradient of the same shape is to be added
  // to dx (the residual branch around the norm), that gradient's row
  const uint32_t slotBytes = (addIn ? 3u : 2u) * rowBytes;
  unsigned char *slots = ring + (size_t)group * stages * slotBytes;
  uint64_t *bars = full + group * kNormMaxStages;
  const long first = (long)blockIdx.x * G + group, step = (long)gridDim.x * G;
  auto issue = [&](long row, int s) { // the group's first thread: a row into slot s
    if (row >= rows || FLAGCX_OPS_HELD_BACK(row)) return;
    unsigned char *dst = slots + (size_t)s * slotBytes;
    mbarExpect(&bars[s], slotBytes);
    bulkLoad(dst, g + (size_t)row * H, rowBytes, &bars[s]);
    bulkLoad(dst + rowBytes, x + (size_t)row * H, rowBytes, &bars[s]);
    if (addIn) bulkLoad(dst + 2 * rowBytes, addIn + (size_t)row * H, rowBytes, &bars[s]);
  };
  if (t == 0) {
    for (int s = 0; s < stages; ++s) mbarInit(&bars[s]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int s = 0; s < stages; ++s) issue(first + s * step, s);
  }
  __syncthreads();
  float dwAcc[PPT][8];
  Pack8 pw[PPT];
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int p = t + k * GT;
    if (p < nPacks) pw[k].raw = ((const uint4 *)w)[p];
#pragma unroll
    for (int i = 0; i < 8; ++i) dwAcc[k][i] = 0.f;
  }
  bool ok = true; // of the whole warp
  int s = 0, half = 0;
  uint32_t phase = 0;
  long row = first;
  for (; row < rows; row += step) {
    const float rstd = rstdIn[row];
    ok = __all_sync(0xffffffffu, mbarWaitBounded(&bars[s], phase));
    if (!ok) break;
    const uint4 *gs = (const uint4 *)(slots + (size_t)s * slotBytes), *xs = gs + nPacks, *as = xs + nPacks;
    if constexpr (PPT == 4) // the weights stay packed: widened ahead of the loop they take 16 registers more than there are
#pragma unroll
      for (int k = 0; k < PPT; ++k)
        asm volatile("" : "+r"(pw[k].raw.x), "+r"(pw[k].raw.y), "+r"(pw[k].raw.z), "+r"(pw[k].raw.w));
    Pack8 pg[PPT], px[PPT], pa[PPT];
    float dot = 0.f;
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int p = t + k * GT;
      if (p < nPacks) {
        pg[k].raw = gs[p];
        px[k].raw = xs[p];
        if (addIn) pa[k].raw = as[p];
#pragma unroll
        for (int i = 0; i < 8; ++i) dot += pg[k].get(i) * pw[k].get(i) * px[k].get(i);
      }
    }
    dot = groupSum<GT>(dot, red, half, group); // the whole group has read the slot
    half ^= 1;
    if (t == 0) issue(row + stages * step, s);
    if (++s == stages) { s = 0; phase ^= 1u; }
    const float c = dot * rstd * rstd / H;
    uint4 *dxr = (uint4 *)(dx + (size_t)row * H);
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int p = t + k * GT;
      if (p < nPacks) {
        Pack8 po;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float gv = pg[k].get(i), xv = px[k].get(i);
          float d = rstd * (gv * pw[k].get(i) - xv * c);
          if (addIn) d += pa[k].get(i);
          po.set(i, d);
          dwAcc[k][i] += gv * xv * rstd;
        }
        dxr[p] = po.raw;
      }
    }
  }
  // A wait ran out: nothing more is fetched, copies still under way land (or are given as long
  // again), and the rows from there on and the warp's part of the weight gradient are NaN.
  if (!ok) {
    if (t == 0)
      for (long r = row; r < rows && r < row + stages * step; r += step) {
        mbarWaitBounded(&bars[s], phase);
        if (++s == stages) { s = 0; phase ^= 1u; }
      }
    __syncwarp();
    for (; row < rows; row += step, half ^= 1) {
      groupSum<GT>(NAN, red, half, group);
      for (int p = t; p < nPacks; p += GT)
        ((uint4 *)(dx + (size_t)row * H))[p] = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
    }
  }
  // The groups' sums meet at the start of the ring: G x H floats fit since a slot holds at least
  // two rows of 16 bits.  They lie across slots of other groups, so every group is through with
  // its rows first, and no copy is under way then.
  const float bad = ok ? 0.f : NAN;
  float *mine = (float *)ring + (size_t)group * H;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int p = t + k * GT;
    if (p < nPacks) {
      *(float4 *)(mine + p * 8) = make_float4(dwAcc[k][0] + bad, dwAcc[k][1] + bad, dwAcc[k][2] + bad, dwAcc[k][3] + bad);
      *(float4 *)(mine + p * 8 + 4) = make_float4(dwAcc[k][4] + bad, dwAcc[k][5] + bad, dwAcc[k][6] + bad, dwAcc[k][7] + bad);
    }
  }
  __syncthreads();
  float *out = dwPartial + (size_t)blockIdx.x * H;
  for (int c = threadIdx.x; c < H / 4; c += kNormThreads) {
    float4 sum = ((const float4 *)ring)[c];
    for (int q = 1; q < G; ++q) {
      const float4 v = ((const float4 *)((const float *)ring + (size_t)q * H))[c];
      sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
    }
    ((float4 *)out)[c] = sum;
  }
}

// dw[c] = sum over the CTAs' partials, in a fixed order, rounded to bf16 once.
// Block (32, 32): 32 neighbouring columns, 32 lanes over the rows.  The partials may still be in
// writing when this kernel starts, so they are read through L2, never as read-only data.
__global__ void columnSumToBf16(const float *partial, bf16 *__restrict__ dw, int R, int H) {
  __shared__ float tile[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  waitForEarlierGrid();
  float acc = 0.f;
  if (c < H)
    for (int r = threadIdx.y; r < R; r += 32) acc += __ldcg(partial + (size_t)r * H + c);
  tile[threadIdx.y][threadIdx.x] = acc;
  __syncthreads();
  if (threadIdx.y == 0 && c < H) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) t += tile[i][threadIdx.x];
    dw[c] = __float2bfloat16_rn(t);
  }
}

// ---------------------------------------------------------------------------
// Rotary embedding, in place, half-split layout: for a head of dimension D,
// (x[i], x[i+D/2]) is rotated by angle pos * theta^(-2i/D).  sign=-1 is the backward.
// x: [tokens, heads, D]; one thread per pair of 8-element packs.
// ---------------------------------------------------------------------------
__global__ void ropeKernel(bf16 *__restrict__ x, const int *__restrict__ positions, int tokens, int heads, int D,
                           float logTheta, float sign) {
  const int half = D / 2, packsPerHalf = half / 8;
  const size_t total = (size_t)tokens * heads * packsPerHalf;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  int pk = idx % packsPerHalf;
  size_t th = idx / packsPerHalf;
  int tok = th / heads;
  float pos = positions ? (float)positions[tok] : (float)tok;
  bf16 *base = x + th * D;
  Pack8 a, b, oa, ob;
  a.raw = *(uint4 *)(base + pk * 8);
  b.raw = *(uint4 *)(base + half + pk * 8);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int d = pk * 8 + i;
    float inv = __expf(-logTheta * (2.0f * d / D));
    float s, c;
    sincosf(pos * inv, &s, &c);
    s *= sign;
    float x1 = a.get(i), x2 = b.get(i);
    oa.set(i, x1 * c - x2 * s);
    ob.set(i, x2 * c + x1 * s);
  }
  *(uint4 *)(base + pk * 8) = oa.raw;
  *(uint4 *)(base + half + pk * 8) = ob.raw;
}

// The same rotation applied to a fused projection [tokens, totalHeads, D] whose first
// ropeHeads heads (queries, then keys) are rotated and whose other heads (values) are
// copied through: one pass that reads src once and writes dst once, so the model needs no
// separate q / k copies before or after the rotation.
__global__ void ropeFusedQkv(const bf16 *__restrict__ src, bf16 *__restrict__ dst, int tokens, int ropeHeads,
                             int totalHeads, int D, float logTheta, float sign) {
  const int half = D / 2, packsPerHalf = half / 8;
  const size_t total = (size_t)tokens * totalHeads * packsPerHalf;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int pk = idx % packsPerHalf;
  const size_t th = idx / packsPerHalf;
  const int head = th % totalHeads;
  const int tok = th / totalHeads;
  const bf16 *in = src + th * D;
  bf16 *out = dst + th * D;
  Pack8 a, b, oa, ob;
  a.raw = *(const uint4 *)(in + pk * 8);
  b.raw = *(const uint4 *)(in + half + pk * 8);
  if (head < ropeHeads) {
    const float pos = (float)tok;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int d = pk * 8 + i;
      const float inv = __expf(-logTheta * (2.0f * d / D));
      float s, c;
      sincosf(pos * inv, &s, &c);
      s *= sign;
      const float x1 = a.get(i), x2 = b.get(i);
      oa.set(i, x1 * c - x2 * s);
      ob.set(i, x2 * c + x1 * s);
    }
  } else {
    oa = a;
    ob = b;
  }
  *(uint4 *)(out + pk * 8) = oa.raw;
  *(uint4 *)(out + half + pk * 8) = ob.raw;
}

// ---------------------------------------------------------------------------
// SwiGLU on a fused projection ab = [a | b] of shape [T, 2F]: out = silu(a) * b.
// ---------------------------------------------------------------------------
__global__ void swigluFwd(const bf16 *__restrict__ ab, bf16 *__restrict__ out, size_t T, int F) {
  const int packs = F / 8;
  const size_t total = T * packs;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  size_t t = idx / packs;
  int p = idx % packs;
  Pack8 a, b, o;
  a.raw = *(const uint4 *)(ab + t * 2 * F + p * 8);
  b.raw = *(const uint4 *)(ab + t * 2 * F + F + p * 8);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float av = a.get(i);
    o.set(i, av / (1.f + __expf(-av)) * b.get(i));
  }
  *(uint4 *)(out + t * F + p * 8) = o.raw;
}

__global__ void swigluBwd(const bf16 *__restrict__ g, const bf16 *__restrict__ ab, bf16 *__restrict__ dab, size_t T,
                          int F) {
  const int packs = F / 8;
  const size_t total = T * packs;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx >= total) return;
  size_t t = idx / packs;
  int p = idx % packs;
  Pack8 a, b, gg, da, db;
  a.raw = *(const uint4 *)(ab + t * 2 * F + p * 8);
  b.raw = *(const uint4 *)(ab + t * 2 * F + F + p * 8);
  gg.raw = *(const uint4 *)(g + t * F + p * 8);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float av = a.get(i), bv = b.get(i), gv = gg.get(i);
    float sig = 1.f / (1.f + __expf(-av));
    float silu = av * sig;
    da.set(i, gv * bv * (sig + silu * (1.f - sig)));
    db.set(i, gv * silu);
  }
  *(uint4 *)(dab + t * 2 * F + p * 8) = da.raw;
  *(uint4 *)(dab + t * 2 * F + F + p * 8) = db.raw;
}

// ---------------------------------------------------------------------------
// Softmax cross-entropy, one CTA per row.  Writes the per-row loss and overwrites
// the logits with gradScale * (softmax - onehot): the [T, V] tensor is read three
// times out of L2 and written once; no fp32 copy of the logits is ever made.
// ---------------------------------------------------------------------------
__global__ void crossEntropyFwdBwd(bf16 *__restrict__ logits, const long *__restrict__ targets,
                                   float *__restrict__ loss, int V, float gradScale) {
  __shared__ float red[32];
  const size_t row = blockIdx.x;
  bf16 *lr = logits + row * V;
  const int packs = V / 8; // V a multiple of 8
  float mx = -INFINITY;
  for (int p = threadIdx.x; p < packs; p += blockDim.x) {
    Pack8 v;
    v.raw = ((const uint4 *)lr)[p];
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = fmaxf(mx, v.get(i));
  }
  mx = blockMax(mx, red);
  float sum = 0.f;
  for (int p = threadIdx.x; p < packs; p += blockDim.x) {
    Pack8 v;
    v.raw = ((const uint4 *)lr)[p];
#pragma unroll
    for (int i = 0; i < 8; ++i) sum += __expf(v.get(i) - mx);
  }
  sum = blockSum(sum, red);
  const long tgt = targets[row];
  const float lse = mx + __logf(sum);
  if (threadIdx.x == 0) loss[row] = lse - __bfloat162float(lr[tgt]);
  __syncthreads(); // the target logit was read before anybody overwrites it
  const float inv = 1.f / sum;
  for (int p = threadIdx.x; p < packs; p += blockDim.x) {
    Pack8 v, o;
    v.raw = ((const uint4 *)lr)[p];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float pr = __expf(v.get(i) - mx) * inv;
      if ((long)p * 8 + i == tgt) pr -= 1.f;
      o.set(i, pr * gradScale);
    }
    ((uint4 *)lr)[p] = o.raw;
  }
}

// ---------------------------------------------------------------------------
// The same operation, persistent, for vocabularies up to 262144.  A cluster
// of C CTAs walks over rows; each CTA's 1/C of a row comes into a shared-memory slot by bulk
// copy, moves on into registers (PPT packs of 8 per thread), and the copy of the next row
// into the slot starts at once: while a row is being reduced, scaled and stored, the next one
// is already on its way.  The exponentials are taken relative to the WARP's maximum and stay
// in registers (as bf16), so that a row needs one exchange only: every warp publishes its
// (maximum, sum), one cluster barrier, and every warp combines all pairs of the cluster.  A
// warp whose logits are all -inf (a masked stretch) contributes nothing.
//
// DEAL: rows are not cut into equal shares; the grid has a cluster for every row, and a cluster that
// runs takes over rows whose clusters have not started (cluster launch control) until none is left.
// The answer for the row after next is asked for while a row is worked on and reaches the other
// CTAs with the pairs.
//
// Bound: HBM (one read and one write of the logits).  The kernel below it in this file, which
// loads, reduces and stores one row per CTA with nothing overlapped, took 458 us for
// 4096 x 128256; this one takes 331 (6.3 TB/s, 0.97 of a copy).  The CTAs of a cluster wait for one
// another at every row, so a row goes to as few as can hold it: with up to 21 packs per thread (two
// CTAs per SM, and all of their 128 registers: 12 bytes spilled made it 449) 3 instead of 4 here,
// 349 -> 331; 2048 x 151936 in 4 instead of 8 261 -> 214; with 5, 6 and 7 CTAs 376, 400 and 445.  Dealt
// against equal shares: 4096 x 32000 93.4 -> 85.2,
// 8192 x 8192 46.6 -> 45.5, 16384 x 1024 45.2 -> 47.0: from four packs per thread on.
// ---------------------------------------------------------------------------
constexpr int kCeRowThreads = 256, kCeRowWarps = kCeRowThreads / 32;
constexpr int kCeRowPacks = 21 * kCeRowThreads;         // packs of a row that one CTA can hold
constexpr int kCeRowMaxPacks = 8 * 16 * kCeRowThreads;  // longer rows go to crossEntropyCluster
constexpr uint32_t kCeBulkPiece = 32768;

// Cluster launch control: asks for a cluster of this grid that has not started yet; the answer (16
// bytes) arrives at `answer` and is counted on the mbarrier.
__device__ __forceinline__ void askForCluster(uint4 *answer, uint64_t *bar) {
  mbarExpect(bar, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(
                   sharedAddr(answer)),
               "r"(sharedAddr(bar))
               : "memory");
}
// blockIdx.x of the first CTA of the cluster that the answer hands over, -1: none is left.
__device__ __forceinline__ int clusterHandedOver(const uint4 *answer) {
  uint32_t ok, x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "ld.shared.b128 h, [%2];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "mov.u32 %1, 0;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %1, h;\n\t}"
      : "=r"(ok), "=r"(x)
      : "r"(sharedAddr(answer))
      : "memory");
  return ok ? (int)x : -1;
}

__device__ __forceinline__ void clusterSyncAll() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ float lowBf16(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float highBf16(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
__device__ __forceinline__ uint32_t packBf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t maxBf16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}

template <int PPT, bool DEAL>
__global__ void __launch_bounds__(kCeRowThreads, PPT > 10 ? 2 : PPT > 8 ? 3 : PPT == 8 ? 4 : PPT == 4 ? 5 : 8)
crossEntropyRows(bf16 *__restrict__ logits, const long *__restrict__ targets, float *__restrict__ loss, long rows, int V,
                 float gradScale, int packsPerCta) {
  extern __shared__ __align__(128) unsigned char ceSlot[];
  __shared__ float2 stat[2][kCeRowWarps]; // (maximum, sum) of every warp, two rows deep
  __shared__ __align__(8) uint64_t bar, dealBar;
  __shared__ __align__(16) uint4 answer[2];
  // of the cluster's first CTA: the row after next (-1: none); 0, or no more requests (bit 1: an answer was not seen)
  __shared__ int dealt[2], dealOver;
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), cr = (int)cluster.block_rank();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long step = gridDim.x / C;
  const bool dealer = DEAL && cr == 0 && tid == 0;
  // Dealer: what came of the nth request.  The row that it hands over is nobody else's, so the answer
  // is given as long again to be seen; if it is not, a row may be done by nobody, and which one is not
  // known: the rows that this cluster has become NaN.
  auto takeAnswer = [&](uint32_t nth) {
    for (int wait = 0; wait < 2; ++wait)
      if (mbarWaitBounded(&dealBar, nth & 1u) && wait >= FLAGCX_OPS_UNSEEN(nth)) {
        const int first = clusterHandedOver(&answer[nth & 1u]);
        return first < 0 ? -1 : first / C;
      }
    dealOver = 2;
    return -1;
  };
  const int p0 = cr * packsPerCta, n = max(0, min(packsPerCta, V / 8 - p0));
  const uint32_t bytes = (uint32_t)n * 16u;
  const uint4 *slot = (const uint4 *)ceSlot;
  auto part = [&](long row) { return (unsigned char *)(logits + (size_t)row * V + (size_t)p0 * 8); };
  auto issue = [&](long row) { // thread 0
    if (FLAGCX_OPS_HELD_BACK(row)) return;
    mbarExpect(&bar, bytes);
    for (uint32_t off = 0; off < bytes; off += kCeBulkPiece)
      bulkLoad(ceSlot + off, part(row) + off, min(kCeBulkPiece, bytes - off), &bar);
  };
  long row = blockIdx.x / C, next = row + step;
  if (tid == 0) {
    mbarInit(&bar);
    if (DEAL) mbarInit(&dealBar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (row < rows && n > 0) issue(row);
  }
  if constexpr (DEAL) {
    if (dealer) {
      dealOver = 0;
      askForCluster(&answer[0], &dealBar);
      dealt[1] = takeAnswer(0);
    }
    if (C > 1) {
      __syncwarp(); // the cluster barrier wants whole warps, and the dealer's lane has been away
      clusterSyncAll();
    } else {
      __syncthreads();
    }
    next = *cluster.map_shared_rank(&dealt[1], 0);
  } else {
    __syncthreads();
  }
  constexpr float kLog2e = 1.4426950408889634f;
  // A copy that never arrived makes the loss and the gradient of its row NaN, and those of the rows
  // after it, which are not fetched; it is given as long again to land before the CTA may leave.
  bool ok = true;
  for (int it = 0; DEAL || row < rows; ++it) {
    if (dealer && next >= 0 && !dealOver) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the last answer has been read
      askForCluster(&answer[(it + 1) & 1], &dealBar);
    }
    if (n > 0 && ok && !(ok = mbarWaitBounded(&bar, (uint32_t)it & 1u)) && tid == 0) mbarWaitBounded(&bar, (uint32_t)it & 1u);
    const long tLocal = targets[row] - (long)p0 * 8; // index of the target inside this CTA's part, if it is here
    const bool own = tLocal >= 0 && tLocal < (long)n * 8;
    const float tgtLogit = own ? __bfloat162float(((const bf16 *)ceSlot)[tLocal]) : 0.f;
    uint32_t v[PPT][4];
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int p = tid + k * kCeRowThreads;
      const uint4 q = p < n ? slot[p] : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u); // -inf
      v[k][0] = q.x; v[k][1] = q.y; v[k][2] = q.z; v[k][3] = q.w;
    }
    __syncthreads(); // the slot has been read
    if (tid == 0 && (DEAL ? next >= 0 : next < rows) && n > 0 && ok) issue(next);
    uint32_t m2 = 0xff80ff80u;
#pragma unroll
    for (int k = 0; k < PPT; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) m2 = maxBf16x2(m2, v[k][i]);
    const float wmax = warpMax(fmaxf(lowBf16(m2), highBf16(m2)));
    // exponentials: 2^(v*log2e - max*log2e), one FMA and one MUFU each
    const float ref = wmax == -INFINITY ? 0.f : wmax * kLog2e;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < PPT; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float e0 = exp2f(fmaf(lowBf16(v[k][i]), kLog2e, -ref)), e1 = exp2f(fmaf(highBf16(v[k][i]), kLog2e, -ref));
        sum += e0 + e1;
        v[k][i] = packBf16x2(e0, e1);
      }
    sum = warpSum(ok ? sum : NAN);
    if (lane == 0) stat[it & 1][warp] = make_float2(wmax, sum);
    if (dealer) {
      dealt[it & 1] = next >= 0 && !dealOver ? takeAnswer(it + 1) : -1;
      if (dealOver & 2) stat[it & 1][0].y = NAN;
    }
    __syncwarp();
    // One barrier per row: the pairs of the row before last are overwritten only now, when
    // every CTA has passed the last row's barrier and so has read them.
    if (C > 1) clusterSyncAll(); else __syncthreads();
    const long after = DEAL ? *cluster.map_shared_rank(&dealt[it & 1], 0) : next + step;
    float M = -INFINITY, S = 0.f;
    float2 st[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int i = lane + 32 * j;
      st[j] = i < C * kCeRowWarps ? cluster.map_shared_rank(&stat[it & 1][0], i / kCeRowWarps)[i % kCeRowWarps]
                                  : make_float2(-INFINITY, 0.f);
      M = fmaxf(M, st[j].x);
    }
    M = warpMax(M);
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (st[j].y != 0.f) S += st[j].y * __expf(st[j].x - M);
    S = warpSum(S);
    // A cluster that has lost a copy takes no further row (nor one that has met a NaN, which its
    // sums do not tell apart): rows that nobody takes over start clusters of their own.
    if (dealer && S != S) dealOver |= 1;
    if (own && tid == 0) loss[row] = M + __logf(S) - tgtLogit;
    const float f = __expf(wmax - M) / S * gradScale;
    uint4 *out = (uint4 *)part(row);
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int p = tid + k * kCeRowThreads;
      if (p < n) {
        uint4 o;
        o.x = packBf16x2(lowBf16(v[k][0]) * f, highBf16(v[k][0]) * f);
        o.y = packBf16x2(lowBf16(v[k][1]) * f, highBf16(v[k][1]) * f);
        o.z = packBf16x2(lowBf16(v[k][2]) * f, highBf16(v[k][2]) * f);
        o.w = packBf16x2(lowBf16(v[k][3]) * f, highBf16(v[k][3]) * f);
        out[p] = o;
      }
    }
    // the one element that is softmax - 1, redone in fp32 by the thread that stored its pack
    if (own && tid == (int)((tLocal >> 3) % kCeRowThreads))
      ((bf16 *)out)[tLocal] = __float2bfloat16_rn(exp2f(fmaf(tgtLogit, kLog2e, -ref)) * f - gradScale);
    if (DEAL && next < 0) break;
    row = next;
    next = after;
  }
  __syncwarp();
  if (C > 1) clusterSyncAll(); // no CTA leaves while another may still read its pairs
}

// ---------------------------------------------------------------------------
// The same operation for vocabularies beyond that (part of a row stays in shared memory, up to
// 200 KiB per CTA).  A thread-block cluster of C CTAs
// owns one row; each CTA brings its 1/C of the row into shared memory with one
// bulk asynchronous copy, finds its own maximum and sum of exponentials (the
// exponentials replace the logits in shared memory, as bf16), trades (max, sum)
// with the other CTAs of the cluster through distributed shared memory, scales
// its exponentials into gradients and sends them back with one bulk store.  The
// [T, V] tensor crosses L2/HBM once in each direction and every element costs one
// exponential instead of two.
// ---------------------------------------------------------------------------
constexpr int kCeMaxThreads = 1024, kCePartBytes = 200 << 10;

__global__ void __launch_bounds__(kCeMaxThreads)
crossEntropyCluster(bf16 *__restrict__ logits, const long *__restrict__ targets, float *__restrict__ loss, int V,
                    float gradScale, int packsPerCta) {
  extern __shared__ __align__(128) unsigned char ceRow[];
  __shared__ float red[32];
  __shared__ float stat[2];
  __shared__ __align__(8) uint64_t bar;
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned C = cluster.num_blocks(), cr = cluster.block_rank();
  const size_t row = blockIdx.x / C;
  const int packs = V / 8, p0 = (int)cr * packsPerCta;
  const int n = max(0, min(packsPerCta, packs - p0));
  unsigned char *gRow = (unsigned char *)(logits + row * V + (size_t)p0 * 8);
  uint4 *buf = (uint4 *)ceRow;
  const uint32_t bytes = (uint32_t)n * 16u;

  if (threadIdx.x == 0) {
    mbarInit(&bar);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  bool ok = true;
  if (n > 0) {
    if (threadIdx.x == 0 && !FLAGCX_OPS_HELD_BACK(row)) {
      mbarExpect(&bar, bytes);
      for (uint32_t off = 0; off < bytes; off += kCeBulkPiece) bulkLoad(ceRow + off, gRow + off, min(kCeBulkPiece, bytes - off), &bar);
    }
    ok = mbarWaitBounded(&bar, 0);
    if (!ok && threadIdx.x == 0) mbarWaitBounded(&bar, 0); // nothing is written over a copy that is under way
  }

  const long tLocal = targets[row] - (long)p0 * 8; // index of the target inside this CTA's part, if it is here
  const bool own = tLocal >= 0 && tLocal < (long)n * 8;
  const float tgtLogit = own ? __bfloat162float(((const bf16 *)ceRow)[tLocal]) : 0.f;
  // maximum: on packed bf16 pairs, no conversion
  __nv_bfloat162 m2 = __float2bfloat162_rn(-INFINITY);
  for (int p = threadIdx.x; p < n; p += (int)blockDim.x) {
    const uint4 v = buf[p];
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&v;
    m2 = __hmax2(m2, __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3])));
  }
  float mx = fmaxf(__low2float(m2), __high2float(m2));
  mx = blockMax(mx, red); // its barriers also order the read of the target logit before the overwrite below
  // exponentials: 2^(v*log2e - mx*log2e), one FMA and one MUFU each
  constexpr float kLog2e = 1.4426950408889634f;
  const float mxs = mx == -INFINITY ? 0.f : mx * kLog2e; // a part that is all -inf contributes nothing
  float sum = 0.f;
  for (int p = threadIdx.x; p < n; p += (int)blockDim.x) {
    const uint4 v = buf[p];
    uint4 e;
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&v;
    __nv_bfloat162 *eo = (__nv_bfloat162 *)&e;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      const float e0 = exp2f(fmaf(f.x, kLog2e, -mxs)), e1 = exp2f(fmaf(f.y, kLog2e, -mxs));
      sum += e0 + e1;
      eo[i] = __floats2bfloat162_rn(e0, e1);
    }
    buf[p] = e;
  }
  sum = blockSum(ok ? sum : NAN, red); // a copy that never arrived makes the whole row's loss and gradient NaN
  if (threadIdx.x == 0) {
    stat[0] = mx;
    stat[1] = sum;
  }
  cluster.sync();
  float M = -INFINITY, S = 0.f;
  for (unsigned r = 0; r < C; ++r) M = fmaxf(M, cluster.map_shared_rank(stat, r)[0]);
  for (unsigned r = 0; r < C; ++r) {
    const float *rs = cluster.map_shared_rank(stat, r);
    const float si = rs[1];
    if (si != 0.f) S += si * __expf(rs[0] - M);
  }
  if (own && threadIdx.x == 0) loss[row] = M + __logf(S) - tgtLogit;
  const float f = n > 0 ? __expf(mx - M) / S * gradScale : 0.f;
  for (int p = threadIdx.x; p < n; p += (int)blockDim.x) {
    const uint4 e = buf[p];
    uint4 o;
    const __nv_bfloat162 *h = (const __nv_bfloat162 *)&e;
    __nv_bfloat162 *oo = (__nv_bfloat162 *)&o;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 v = __bfloat1622float2(h[i]);
      oo[i] = __floats2bfloat162_rn(v.x * f, v.y * f);
    }
    buf[p] = o;
  }
  // the one element that is softmax - 1, redone in fp32 by the thread that wrote its pack
  if (own && threadIdx.x == (int)((tLocal >> 3) % blockDim.x))
    ((bf16 *)ceRow)[tLocal] = __float2bfloat16_rn(exp2f(fmaf(tgtLogit, kLog2e, -mxs)) * f - gradScale);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the stores above, before the engine reads them
  __syncthreads();
  if (threadIdx.x == 0 && n > 0) {
    for (uint32_t off = 0; off < bytes; off += kCeBulkPiece) {
      const uint32_t sz = min(kCeBulkPiece, bytes - off);
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gRow + off),
                   "r"(sharedAddr(ceRow + off)), "r"(sz)
                   : "memory");
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  }
  cluster.sync(); // no CTA leaves while another may still read its (max, sum)
}

// ---------------------------------------------------------------------------
// AdamW on flat bf16 tensors (parameters, gradients, both moments), fp32 math.
// ---------------------------------------------------------------------------
__global__ void adamwFlat(bf16 *__restrict__ p, const bf16 *__restrict__ g, bf16 *__restrict__ m, bf16 *__restrict__ v,
                          size_t n, float lr, float beta1, float beta2, float eps, float wd, float bc1, float bc2) {
  const size_t packs = n / 8;
  const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (idx < packs) {
    Pack8 pp, pg, pm, pv;
    pp.raw = ((const uint4 *)p)[idx];
    pg.raw = ((const uint4 *)g)[idx];
    pm.raw = ((const uint4 *)m)[idx];
    pv.raw = ((const uint4 *)v)[idx];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float gv = pg.get(i), mv = pm.get(i), vv = pv.get(i), pw = pp.get(i);
      mv = beta1 * mv + (1.f - beta1) * gv;
      vv = beta2 * vv + (1.f - beta2) * gv * gv;
      float upd = (mv / bc1) / (sqrtf(vv / bc2) + eps);
      pw = pw * (1.f - lr * wd) - lr * upd;
      pp.set(i, pw); pm.set(i, mv); pv.set(i, vv);
    }
    ((uint4 *)p)[idx] = pp.raw;
    ((uint4 *)m)[idx] = pm.raw;
    ((uint4 *)v)[idx] = pv.raw;
  }
  // tail (n not a multiple of 8)
  const size_t tail = packs * 8 + idx;
  if (tail < n) {
    float gv = __bfloat162float(g[tail]), mv = __bfloat162float(m[tail]), vv = __bfloat162float(v[tail]);
    float pw = __bfloat162float(p[tail]);
    mv = beta1 * mv + (1.f - beta1) * gv;
    vv = beta2 * vv + (1.f - beta2) * gv * gv;
    pw = pw * (1.f - lr * wd) - lr * (mv / bc1) / (sqrtf(vv / bc2) + eps);
    p[tail] = __float2bfloat16_rn(pw);
    m[tail] = __float2bfloat16_rn(mv);
    v[tail] = __float2bfloat16_rn(vv);
  }
}

// The element-wise kernels (rope, SwiGLU, AdamW) take one item per thread and as many CTAs as that
// needs, whatever their number.  Bound: HBM.  Cut into equal shares for 8 CTAs of 256 threads per
// SM, as they once were, a pass lasts as long as the SM farthest from the memory takes for its
// share; dealt out by the hardware, SMs that are done sooner take more.  Device us, equal shares
// against this: AdamW of 218 M elements 498 -> 438 (6.97 TB/s), SwiGLU 4099 x 14336 forward 57.3
// -> 53.4, backward 102.1 -> 88.0 (6.67), rope 8192 x 48 x 128 36.9 -> 33.0 (6.1), 1021 tokens the
// same as before.  Between 64 and 512 threads, one or two items each, all but 64 (forward 63.6) are
// within 1 %.
constexpr int kItemThreads = 128;
unsigned gridFor(size_t items) { return (unsigned)std::max<size_t>(1, (items + kItemThreads - 1) / kItemThreads); }

#define RETURN_IF(e)                        \
  do {                                      \
    const cudaError_t err_ = (e);           \
    if (err_ != cudaSuccess) return err_;   \
  } while (0)

// Lets every launch of Kern on this device have `bytes` of dynamic shared memory, the most that any
// of its sizes asks for.  The limit belongs to the kernel, not to a launch: set to each call's own
// size, two threads could lower it between the other's call and launch.
template <auto Kern>
cudaError_t allowShared(int bytes) {
  static fcxops::OncePerDevice once;
  int dev = 0;
  RETURN_IF(cudaGetDevice(&dev));
  return once(dev, [&] { return cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
}

// Calls f(GT, PPT) for rows of `packs` packs of 8: the smallest group whose threads hold a row
// with at most four packs each, so three or four in every group but the smallest.  MOST is the largest
// group there is to be (512 threads and four packs: 16384 elements); a row that it cannot hold is refused.
template <int MOST, typename F>
cudaError_t withNormShape(int packs, F &&f) {
  auto ppt = [&](auto gt) -> cudaError_t {
    constexpr int GT = decltype(gt)::value;
    const int n = (packs + GT - 1) / GT;
    if constexpr (GT == 32) {
      if (n <= 1) return f(gt, std::integral_constant<int, 1>());
      if (n <= 2) return f(gt, std::integral_constant<int, 2>());
    }
    if (n <= 3) return f(gt, std::integral_constant<int, 3>());
    return f(gt, std::integral_constant<int, 4>());
  };
  if (packs <= 32 * kNormPacks) return ppt(std::integral_constant<int, 32>());
  if (packs <= 64 * kNormPacks) return ppt(std::integral_constant<int, 64>());
  if (packs <= 128 * kNormPacks) return ppt(std::integral_constant<int, 128>());
  if (packs <= 256 * kNormPacks) return ppt(std::integral_constant<int, 256>());
  if constexpr (MOST == 512)
    if (packs <= 512 * kNormPacks) return ppt(std::integral_constant<int, 512>());
  return cudaErrorInvalidValue;
}

template <int PPT, bool DEAL>
cudaError_t launchCeRows(bf16 *logits, const long *targets, float *loss, long rows, int V, float gradScale, int C, int per,
                         int sms, cudaStream_t stream) {
  auto kern = crossEntropyRows<PPT, DEAL>;
  const int smem = per * 16;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.blockDim = dim3(kCeRowThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  constexpr int kMost = PPT * kCeRowThreads * 16;
  if constexpr (kMost > (47 << 10)) RETURN_IF((allowShared<crossEntropyRows<PPT, DEAL>>(kMost))); // beyond what a kernel gets without asking
  // Equal shares: as many clusters as run at once, a second wave would be waste.
  long clusters = rows;
  if (!DEAL && rows * C > sms) {
    static fcxops::ClusterCount count;
    int dev = 0, active = 0;
    RETURN_IF(cudaGetDevice(&dev));
    cfg.gridDim = dim3((unsigned)C);
    RETURN_IF(count(dev, smem, C, [&](int *n) { return cudaOccupancyMaxActiveClusters(n, kern, &cfg); }, &active));
    clusters = std::min<long>(rows, active);
  }
  cfg.gridDim = dim3((unsigned)(clusters * C));
  return cudaLaunchKernelEx(&cfg, kern, logits, targets, loss, rows, V, gradScale, per);
}

} // namespace

// ---------------------------------------------------------------------------
// launchers (see fused_elementwise.h)
// ---------------------------------------------------------------------------
namespace fcxops {

cudaError_t rmsnormForward(const void *x, const void *w, void *y, float *rstd, long rows, int H, float eps,
                           cudaStream_t stream) {
  auto launch = [&](auto gt, auto ppt) {
    constexpr int GT = decltype(gt)::value, PPT = decltype(ppt)::value, G = kNormFwdThreads<GT> / GT;
    rmsnormFwd<GT, PPT><<<(unsigned)((rows + G - 1) / G), kNormFwdThreads<GT>, 0, stream>>>(
        (const bf16 *)x, (const bf16 *)w, (bf16 *)y, rstd, rows, H, eps);
    return cudaGetLastError();
  };
  const int packs = H / 8;
  if (packs > 256 * kNormPacks && packs <= 256 * 8) return launch(std::integral_constant<int, 256>(), std::integral_constant<int, 8>());
  return withNormShape<256>(packs, launch);
}

int rmsnormPartials(long rows, int H, int sms) {
  if (rmsnormRowPerCta(rows, H, sms)) return (int)std::max<long>(1, std::min<long>(rows, sms * 2));
  int ctas = 0;
  withNormShape<512>(H / 8, [&](auto gt, auto) {
    constexpr int G = kNormThreads / decltype(gt)::value;
    ctas = (int)std::max<long>(1, std::min<long>((rows + G - 1) / G, sms));
    return cudaSuccess;
  });
  return ctas;
}

cudaError_t rmsnormBackward(const void *g, const void *x, const void *w, const float *rstd, const void *add, void *dx, void *dw,
                            float *partial, long rows, int H, int sms, cudaStream_t stream) {
  const int ctas = rmsnormPartials(rows, H, sms);
  if (rmsnormRowPerCta(rows, H, sms)) {
    const int shared = H * (add ? 6 : 4) * (rows > ctas ? kNormFewRows : 1);
    auto launch = [&](auto tag) {
      constexpr int MAXP = decltype(tag)::value;
      constexpr auto kern = rmsnormBwdFewRows<MAXP>;
      RETURN_IF(allowShared<kern>(kNormFewRows * MAXP * kNormBwdThreads * 8 * 6));
      kern<<<ctas, kNormBwdThreads, shared, stream>>>((const bf16 *)g, (const bf16 *)x, (const bf16 *)w, rstd, (const bf16 *)add,
                                                      (bf16 *)dx, partial, (int)rows, H);
      return cudaGetLastError();
    };
    if (H / 8 <= kNormBwdThreads) RETURN_IF(launch(std::integral_constant<int, 1>()));
    else RETURN_IF(launch(std::integral_constant<int, 2>()));
  } else {
    RETURN_IF(withNormShape<512>(H / 8, [&](auto gt, auto ppt) {
      constexpr int GT = decltype(gt)::value, PPT = decltype(ppt)::value, G = kNormThreads / GT;
      // slots of all groups, two for each at least: one CTA per SM
      const size_t slots = (size_t)H * (add ? 6 : 4) * G;
      const int stages = (int)std::min<size_t>(kNormMaxStages, kNormRingBytes / slots);
      const size_t smem = slots * stages;
      constexpr auto kern = rmsnormBwdRing<GT, PPT>;
      RETURN_IF(allowShared<kern>(kNormRingBytes));
      kern<<<ctas, kNormThreads, smem, stream>>>((const bf16 *)g, (const bf16 *)x, (const bf16 *)w, rstd, (const bf16 *)add,
                                                 (bf16 *)dx, partial, rows, H, stages);
      return cudaGetLastError();
    }));
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)((H + 31) / 32));
  cfg.blockDim = dim3(32, 32);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, columnSumToBf16, (const float *)partial, (bf16 *)dw, ctas, H);
}

cudaError_t rope(void *x, const int *positions, int tokens, int heads, int D, float logTheta, float sign, cudaStream_t stream) {
  const size_t items = (size_t)tokens * heads * (D / 16);
  ropeKernel<<<gridFor(items), kItemThreads, 0, stream>>>((bf16 *)x, positions, tokens, heads, D, logTheta, sign);
  return cudaGetLastError();
}

cudaError_t ropeQkv(const void *qkv, void *out, int tokens, int ropeHeads, int totalHeads, int D, float logTheta, float sign,
                    cudaStream_t stream) {
  const size_t items = (size_t)tokens * totalHeads * (D / 16);
  ropeFusedQkv<<<gridFor(items), kItemThreads, 0, stream>>>((const bf16 *)qkv, (bf16 *)out, tokens, ropeHeads, totalHeads,
                                                             D, logTheta, sign);
  return cudaGetLastError();
}

cudaError_t swigluForward(const void *ab, void *out, size_t T, int F, cudaStream_t stream) {
  swigluFwd<<<gridFor(T * (F / 8)), kItemThreads, 0, stream>>>((const bf16 *)ab, (bf16 *)out, T, F);
  return cudaGetLastError();
}

cudaError_t swigluBackward(const void *g, const void *ab, void *dab, size_t T, int F, cudaStream_t stream) {
  swigluBwd<<<gridFor(T * (F / 8)), kItemThreads, 0, stream>>>((const bf16 *)g, (const bf16 *)ab, (bf16 *)dab, T, F);
  return cudaGetLastError();
}

cudaError_t crossEntropy(void *logits, const long *targets, float *loss, long rows, int V, float gradScale, int sms,
                         cudaStream_t stream) {
  // Many rows: the fewest CTAs whose part of a row fits the registers of crossEntropyRows, rows dealt
  // out.  From eight rounds of the CTAs that run at once on: with 8 it gains 2 % (1230 x 48440), with 14
  // 5 to 9 (1410 x 86736, 4096 x 32000), with 3 to 5 the first requests cost more (700 x 65536 42.0 ->
  // 43.2, 2228 x 5520 14.4 -> 16.4).  Fewer rows: equal shares, at most 64 KiB of a row per CTA, and more
  // CTAs per row while that leaves SMs idle and a CTA still has two packs per thread.  Longer
  // rows: up to 200 KiB of shared memory per CTA; failing that, the kernel that streams the
  // row three times.
  const int packs = V / 8;
  int cluster = 0, per = 0;
  static const size_t partKb = std::getenv("FLAGCX_OPS_CE_PART_KB") ? (size_t)atoi(std::getenv("FLAGCX_OPS_CE_PART_KB")) : kCeRowPacks * 16 >> 10;
  static const bool forceStreaming = std::getenv("FLAGCX_OPS_CE_STREAMING") && atoi(std::getenv("FLAGCX_OPS_CE_STREAMING")) != 0;
  if (!forceStreaming) {
    if (packs <= kCeRowMaxPacks) {
      auto fits = [&](int c, int most, size_t kb) {
        per = (packs + c - 1) / c;
        return per <= most && ((size_t)per * 16 <= kb << 10 || c == 8);
      };
      cluster = 1;
      while (!fits(cluster, kCeRowPacks, partKb)) ++cluster; // 8 do
      const int perSm = per <= 4 * kCeRowThreads ? 5 : per <= 8 * kCeRowThreads ? 4 : per <= 10 * kCeRowThreads ? 3 : 2;
      const bool deal = per > 2 * kCeRowThreads && rows * cluster >= 8L * perSm * sms && rows * cluster <= 0x7fffffffL;
      if (!deal) {
        cluster = 1;
        while (!fits(cluster, 16 * kCeRowThreads, std::min<size_t>(partKb, 64))) cluster *= 2;
        while (cluster < 8 && rows * cluster < 2 * sms && packs >= 4 * kCeRowThreads * cluster) cluster *= 2;
        per = (packs + cluster - 1) / cluster;
      }
      // Packs per thread decide the registers (4 each), and they how many CTAs share an SM: 10 let
      // three, 21 two, 13, 16 and 18 leave fewer threads without a pack.  Without 10 and 13 1024 x 65544
      // took 79.9 us instead of 61.2, 4096 x 100352 327.5 instead of 295.5.
      auto go = [&](auto tag) {
        constexpr int PPT = decltype(tag)::value;
        auto launch = deal ? launchCeRows<PPT, (PPT > 2)> : launchCeRows<PPT, (PPT > 16)>;
        return launch((bf16 *)logits, targets, loss, rows, V, gradScale, cluster, per, sms, stream);
      };
      if (per <= kCeRowThreads) return go(std::integral_constant<int, 1>());
      if (per <= 2 * kCeRowThreads) return go(std::integral_constant<int, 2>());
      if (per <= 4 * kCeRowThreads) return go(std::integral_constant<int, 4>());
      if (per <= 8 * kCeRowThreads) return go(std::integral_constant<int, 8>());
      if (per <= 10 * kCeRowThreads) return go(std::integral_constant<int, 10>());
      if (per <= 13 * kCeRowThreads) return go(std::integral_constant<int, 13>());
      if (per <= 16 * kCeRowThreads) return go(std::integral_constant<int, 16>());
      if (per <= 18 * kCeRowThreads) return go(std::integral_constant<int, 18>());
      return go(std::integral_constant<int, 21>());
    }
    per = (packs + 7) / 8;
    if (per * 16 <= kCePartBytes) cluster = 8;
  }
  if (!cluster || rows * cluster > 0x7fffffffLL) {
    crossEntropyFwdBwd<<<(unsigned)rows, 1024, 0, stream>>>((bf16 *)logits, targets, loss, V, gradScale);
    return cudaGetLastError();
  }
  const size_t smem = (size_t)per * 16;
  RETURN_IF(allowShared<crossEntropyCluster>(kCePartBytes));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * cluster));
  static const int ceThreads = std::getenv("FLAGCX_OPS_CE_THREADS") ? std::min(kCeMaxThreads, std::max(32, atoi(std::getenv("FLAGCX_OPS_CE_THREADS")) / 32 * 32)) : 256;
  cfg.blockDim = dim3(ceThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, crossEntropyCluster, (bf16 *)logits, targets, loss, V, gradScale, per);
}

cudaError_t adamw(void *p, const void *g, void *m, void *v, size_t n, float lr, float beta1, float beta2, float eps, float wd,
                  float bc1, float bc2, cudaStream_t stream) {
  // a small step is the host's: this launch reports its own error
  void *args[] = {&p, &g, &m, &v, &n, &lr, &beta1, &beta2, &eps, &wd, &bc1, &bc2};
  return cudaLaunchKernel((const void *)adamwFlat, dim3(gridFor(n / 8 + 8)), dim3(kItemThreads), args, 0, stream);
}

} // namespace fcxops
