// split_gemm.cu -- the plain tcgen05 GEMM D[M,N] = A[M,K] * B[N,K]^T for outputs that have
// too few 256-wide tiles to occupy the chip (few rows: decoding, short prompts).
//
// The persistent kernel of tp_gemm.cu gives a whole K to one CTA (pair) per tile: 128 x 3584
// x 8192 is 14 tiles, so 14 of 148 SMs stream the 59 MB of weights.  Here a cluster of S
// CTAs owns a tile and each takes 1/S of K, so tiles x S SMs stream at once; tiles are 128 x
// BN with BN = 256, 128 or 64.  Each CTA accumulates its part in TMEM, leaves it as fp32 in
// its own shared memory (the operand ring is free by then), and after one cluster barrier
// every CTA adds up 1/S of the tile's rows out of the S shared memories (distributed shared
// memory, fixed order 0..S-1: the result does not depend on timing) and stores it as bf16.
// The same kernel takes the last, nearly empty wave of a large product (SplitGemmTail): the
// persistent kernel stops after its full waves.
// The partial sums never leave the chip, no workspace is needed, and no CTA waits for
// another except at that barrier, which the hardware's cluster scheduling makes safe.
//
// Bound, 128 x 3584 x 8192 (112 CTAs, 4 parts): 10 us in which the weights come out of HBM at 5.9
// TB/s, and 3.6 us behind them: accumulators to shared memory 0.6, cluster barrier 0.7, the sum 2.3,
// which is 48 KB into every SM at the 14 bytes a clock that distributed shared memory gives (loads,
// stores and bulk copies alike).  The sum's loads are all under way at once, the marks of
// parts that failed come with them (0.1 us with 8 parts: 128 x 256 x 8192 9.09 -> 9.24), the last
// barrier publishes nothing, and the kernel is launched while the one in front of it ends: 20.5 -> 17.5
// us back to back.
#include <cuda_bf16.h>

#include <atomic>

#include "split_gemm.h"
#include "tcgen05.cuh"

namespace fcx {
namespace {

using bf16 = __nv_bfloat16;
using namespace tc;

constexpr int BM = 128, BK = 64, kThreads = 256;

// How long a wait may take, the K step whose operands are not fetched, and what is done about them
// once the CTA has given up (a test of the waits that run out sets all three).
#ifndef FLAGCX_GEMM_WAIT_NS
#define FLAGCX_GEMM_WAIT_NS 4000000000ull
#define FLAGCX_GEMM_HELD_BACK(tile, kb) false
#define FLAGCX_GEMM_GIVEN_UP(load)
#endif
constexpr unsigned long long kWaitLimitNs = FLAGCX_GEMM_WAIT_NS;

template <int BN>
struct __align__(1024) Smem {
  static constexpr int STAGES = 192 * 1024 / ((BM + BN) * BK * 2); // 4, 6, 8
  bf16 a[STAGES][BM * BK];
  bf16 b[STAGES][BN * BK];
  uint64_t full[STAGES], empty[STAGES], done;
  uint32_t tmemBase;
  int abortFlag;
  int lost; // this part has no sum.  Outside the ring, where copies may land late
};

__device__ __forceinline__ float4 ldCluster16(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

__device__ __forceinline__ int ldClusterInt(uint32_t addr) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// Rows [r0, r1) of the tile: the parts' fp32 values out of the cluster's shared memories (tile
// buffers at `base` in each), added in the order of the parts, to bf16 rows at `out`.  The loads of
// kBatch chunks and all parts are under way before any is used.
template <int BN, int S>
__device__ __forceinline__ void addParts(uint32_t base, int parts, int r0, int r1, bf16 *out, int N) {
  constexpr int kChunks = BN / 4, kMost = S ? S : kSplitGemmMaxParts, kBatch = S ? (S < 16 ? 16 / S : 1) : 2;
  const int n = S ? S : parts, items = (r1 - r0) * kChunks;
  uint32_t from[kMost];
#pragma unroll
  for (int p = 0; p < kMost; ++p) from[p] = mapToCta(base, p < n ? p : 0);
  for (int i0 = threadIdx.x; i0 < items; i0 += kBatch * kThreads) {
    float4 v[kBatch][kMost];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = i0 + u * kThreads, row = r0 + i / kChunks, ch = i % kChunks;
      if (i < items) {
#pragma unroll
        for (int p = 0; p < kMost; ++p)
          if (p < n) v[u][p] = ldCluster16(from[p] + (uint32_t)(row * kChunks + (ch ^ (row & 7))) * 16u);
      }
    }
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int i = i0 + u * kThreads, row = r0 + i / kChunks, ch = i % kChunks;
      if (i < items) {
        float4 t = v[u][0];
#pragma unroll
        for (int p = 1; p < kMost; ++p)
          if (p < n) { t.x += v[u][p].x; t.y += v[u][p].y; t.z += v[u][p].z; t.w += v[u][p].w; }
        __align__(8) __nv_bfloat162 o[2] = {__floats2bfloat162_rn(t.x, t.y), __floats2bfloat162_rn(t.z, t.w)};
        *reinterpret_cast<uint2 *>(out + (size_t)row * N + ch * 4) = *reinterpret_cast<uint2 *>(o);
      }
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
    splitGemmKernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    bf16 *__restrict__ D, int N, int kBlocks, int tilesM, int S, const SplitGemmTail tail) {
  extern __shared__ uint8_t rawSmem[];
  using SmemT = Smem<BN>;
  constexpr int STAGES = SmemT::STAGES;
  constexpr uint32_t kStageBytes = (BM + BN) * BK * 2;
  constexpr int kChunks = BN / 4; // 16-byte chunks of an fp32 tile row
  static_assert(BM * BN * 4 <= (int)(STAGES * kStageBytes), "the fp32 tile reuses the operand ring");
  SmemT &s = *reinterpret_cast<SmemT *>((reinterpret_cast<uintptr_t>(rawSmem) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int part = (int)clusterCtaRank(), tile = blockIdx.x / S;
  int tm = tile % tilesM, tn = tile / tilesM; // neighbours share the rows of B
  if (tail.count) {
    // part q of one of the persistent kernel's tiles (its order: tileCoords in tp_gemm.cu)
    const int down = tail.tileRows / BM, per = down * (256 / BN), t = tail.first + tile / per, q = tile % per;
    const int wide = N / 256, g = t / (tail.groupRows * wide), wg = t - g * tail.groupRows * wide;
    const int gsize = min(tail.groupRows, (tilesM + down - 1) / down - g * tail.groupRows);
    tm = (g * tail.groupRows + wg % gsize) * down + q % down;
    tn = wg / gsize * (256 / BN) + q / down;
    if (tm >= tilesM) return; // the whole cluster: half a tile that lies beyond the output
  }
  const int kb0 = (int)((long)kBlocks * part / S), kb1 = (int)((long)kBlocks * (part + 1) / S);

  if (threadIdx.x == 0) {
    prefetchTensorMap(&tmA);
    prefetchTensorMap(&tmB);
    for (int i = 0; i < STAGES; ++i) { mbarInit(&s.full[i], 1); mbarInit(&s.empty[i], 1); }
    mbarInit(&s.done, 1);
    s.abortFlag = 0;
    s.lost = 0;
    mbarInitFence();
  }
  if (warp == 1) { tmemAlloc(&s.tmemBase, BN); tmemRelinquish(); }
  fenceBeforeSync();
  __syncthreads();
  fenceAfterSync();
  waitForEarlierGrid();
  letNextGridStart();
  const uint32_t tmemBase = s.tmemBase;
  volatile int *abortFlag = &s.abortFlag;

  int issued = 0; // K steps whose operands thread 0 has asked for
  auto load = [&](int kb, int stage) {
    mbarExpectTx(&s.full[stage], kStageBytes);
    tmaLoad2d(s.a[stage], &tmA, kb * BK, tm * BM, &s.full[stage]);
    tmaLoad2d(s.b[stage], &tmB, kb * BK, tn * BN, &s.full[stage]);
  };
  if (warp == 0) {
    if (lane == 0) { // TMA producer
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbarWait(&s.empty[stage], phase ^ 1, abortFlag, kWaitLimitNs)) break;
        if (!FLAGCX_GEMM_HELD_BACK(tile, kb)) load(kb, stage);
        ++issued;
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) { // MMA issuer
      constexpr uint32_t idesc = instrDescBf16(BM, BN);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbarWait(&s.full[stage], phase, abortFlag, kWaitLimitNs)) { ok = false; break; }
        fenceAfterSync();
        const uint64_t da = smemDescSw128(s.a[stage]), db = smemDescSw128(s.b[stage]);
#pragma unroll
        for (int k4 = 0; k4 < BK / 16; ++k4) mmaBf16(tmemBase, da + 2 * k4, db + 2 * k4, idesc, (kb > kb0) || k4 != 0);
        mmaCommit(&s.empty[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) mmaCommit(&s.done);
    }
    __syncwarp();
  }
  // every MMA has finished (and with them every load and every read of the ring)
  const bool ok = mbarWait(&s.done, 0, abortFlag, kWaitLimitNs);
  fenceAfterSync();
  float4 *tileBuf = reinterpret_cast<float4 *>(s.a);
  if (__syncthreads_and(ok ? 1 : 0)) {
    // warp w reads TMEM lanes 32 (w % 4) .. and half of the columns; a row's chunks are
    // swizzled by its number, so that the eight lanes of a phase hit different banks
    const int row = (warp & 3) * 32 + lane;
#pragma unroll 1
    for (int c = (warp >> 2) * (BN / 2); c < ((warp >> 2) + 1) * (BN / 2); c += 32) {
      uint32_t r[32];
      tmemLoad32(tmemBase + ((uint32_t)((warp & 3) * 32) << 16) + c, r);
      tmemLoadWait();
#pragma unroll
      for (int i = 0; i < 8; ++i)
        tileBuf[row * kChunks + ((c / 4 + i) ^ (row & 7))] =
            make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]),
                        __uint_as_float(r[4 * i + 3]));
    }
  } else if (threadIdx.x == 0) {
    s.lost = 1;
    // given up: copies that are still under way land before the CTA goes on
    int never = 0;
    for (int j = issued > STAGES ? issued - STAGES : 0; j < issued; ++j)
      mbarWait(&s.full[j % STAGES], (uint32_t)(j / STAGES) & 1u, &never, kWaitLimitNs);
    FLAGCX_GEMM_GIVEN_UP(load);
  }
  fenceBeforeSync();
  __syncwarp();
  clusterSync();
  const uint32_t base = smemAddr(tileBuf);
  const int lost = lane < S ? ldClusterInt(mapToCta(smemAddr(&s.lost), lane)) : 0; // on its way during the sum
  const int r0 = BM * part / S, r1 = BM * (part + 1) / S;
  bf16 *out = D + (size_t)tm * BM * N + tn * BN;
  switch (S) {
    case 1: addParts<BN, 1>(base, S, r0, r1, out, N); break;
    case 2: addParts<BN, 2>(base, S, r0, r1, out, N); break;
    case 4: addParts<BN, 4>(base, S, r0, r1, out, N); break;
    case 8: addParts<BN, 8>(base, S, r0, r1, out, N); break;
    default: addParts<BN, 0>(base, S, r0, r1, out, N);
  }
  if (__any_sync(0xffffffffu, lost)) { // the tile becomes NaN, in every CTA of the cluster: each thread's sums again
    __align__(8) const __nv_bfloat162 o[2] = {__floats2bfloat162_rn(NAN, NAN), __floats2bfloat162_rn(NAN, NAN)};
    for (int i = threadIdx.x; i < (r1 - r0) * kChunks; i += kThreads)
      *reinterpret_cast<uint2 *>(out + (size_t)(r0 + i / kChunks) * N + i % kChunks * 4) = *reinterpret_cast<const uint2 *>(o);
  }
  // no CTA leaves while another may still read its part: the stores above have taken what they read
  __syncwarp();
  clusterSyncRelaxed();
  if (warp == 1) tmemDealloc(tmemBase, BN);
}

template <int BN>
cudaError_t launch(cudaStream_t stream, const CUtensorMap &tmA, const CUtensorMap &tmB, void *D, int M, int N, int K, int S,
                   const SplitGemmTail &tail) {
  static std::atomic<unsigned long long> ready{0}; // bit per device: the attribute belongs to the device's context
  const size_t smem = sizeof(Smem<BN>) + 1024;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (dev > 63 || !(ready.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(splitGemmKernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (dev <= 63) ready.fetch_or(bit, std::memory_order_release);
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)S;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  const int tiles = tail.count ? tail.count * (tail.tileRows / BM) * (256 / BN) : (M / BM) * (N / BN);
  cfg.gridDim = dim3((unsigned)(tiles * S));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, splitGemmKernel<BN>, tmA, tmB, (bf16 *)D, N, K / BK, M / BM, S, tail);
}

} // namespace

cudaError_t launchSplitGemm(cudaStream_t stream, const CUtensorMap &tmA, const CUtensorMap &tmB, void *D, int M, int N, int K,
                            const SplitGemmPlan &p, const SplitGemmTail &tail) {
  if (p.parts < 1 || p.parts > kSplitGemmMaxParts || p.parts > K / BK) return cudaErrorInvalidValue;
  switch (p.tileN) {
    case 256: return launch<256>(stream, tmA, tmB, D, M, N, K, p.parts, tail);
    case 128: return launch<128>(stream, tmA, tmB, D, M, N, K, p.parts, tail);
    case 64: return launch<64>(stream, tmA, tmB, D, M, N, K, p.parts, tail);
    default: return cudaErrorInvalidValue;
  }
}

} // namespace fcx
