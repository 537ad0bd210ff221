// tp_gemm.cc -- host side of the tcgen05 GEMM and of the fused tensor-parallel kernels
// (all-gather -> GEMM, GEMM -> reduce-scatter): symmetric buffers and flags, TMA tensor
// maps, launches.
#include <algorithm>
#include <map>

#include "../kernels/launch.h"
#include "../kernels/split_gemm.h"
#include "../kernels/tp_gemm_args.h"
#include "comm.h"
#include "flagcx_ext.h"

namespace fcx {
size_t tpGemmSmemBytes(bool pair);
cudaError_t launchTpGemm(cudaStream_t stream, const CUtensorMap &tmA, const CUtensorMap &tmB, const TpStoreMaps *maps,
                         const flagcxDevComm &c, const TpGemmArgs &a, int nCtas, bool pair);
} // namespace fcx

using namespace fcx;

struct flagcxTpGemm {
  flagcxComm *comm;
  int mode, M, N, K, rowsPerRank;
  void *buf = nullptr, *flags = nullptr;
  Window *wBuf = nullptr, *wFlags = nullptr;
  bool vmmBuf = false, vmmFlags = false;
  unsigned long long epoch = 0;
  CUtensorMap tmGather;
  TpStoreMaps storeMaps;
  std::map<const void *, CUtensorMap> mapsA, mapsB;
};

namespace {

// CTA pairs (256-row tiles, cta_group::2) whenever the row blocks allow it.
bool usePair(int rowsPerOwner) { return readParam("GEMM_PAIR", 1) != 0 && rowsPerOwner % 256 == 0; }

// Row blocks walked together by the tile order: the grid (74 pairs or 148 CTAs) then
// covers a near-square patch of the output at any moment.
int groupRows(bool pair) { return std::max(1, (int)readParam("GEMM_GROUP", pair ? 8 : 16)); }

int smCount() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms > 0 ? sms : 1;
}

// Estimates for split_gemm.cu: fixed cost and cost of a K step (us) by tile width, and how many
// CTAs run at once by cluster size.
struct { int tileN; double fixedUs, stepUs; } const kSplitKinds[] = {{256, 11.5, 0.384}, {128, 10.3, 0.27}, {64, 8.7, 0.2875}};
struct { int parts, ctas; } const kSplits[] = {{8, 112}, {4, 132}, {2, 148}, {1, 148}};

// Which kernel takes a plain product: the persistent one (tileN = 0), or K split over clusters
// of S CTAs that own 128 x tileN tiles.  The split pays while the persistent kernel's 128 x 256
// tiles leave most SMs idle (back-to-back calls, operands not in L2, us: 128 x 3584 x 8192
// 54.6 -> 20.2, 256 x 3584 x 8192 45.2 -> 25.1, 128 x 256 x 8192 47.7 -> 12.4, 512 x 3584 x
// 8192 45.5 -> 36.8); from about 64 tiles on the persistent kernel's CTA pairs and overlapped
// epilogues win (1024 x 3584 x 8192: 53 against 68 us).  Below that the smallest of the
// estimates decides: a fixed cost plus the largest of one CTA's K steps, the operands out of
// HBM (6.4 TB/s) and what all CTAs together pull out of L2 (13 TB/s); the figures are fitted to
// 26 shapes from 128 x 256 x 4096 to 1024 x 1280 x 8192 and within 2 us of all of them.
// Clusters stay within what is co-resident (33 of 4 CTAs, 14 of 8): a second wave costs more
// than the split gains (28 clusters of 5: 37 us against 27).
SplitGemmPlan splitPlan(int M, int N, int K, bool pair) {
  SplitGemmPlan best;
  const int kb = K / 64;
  const int forced = (int)readParam("GEMM_SPLIT", 0);
  if (forced == 1) return best;
  if (forced > 1 && forced <= kSplitGemmMaxParts && forced <= kb) {
    best.parts = forced;
    best.tileN = (int)readParam("GEMM_SPLIT_N", 256);
    return best;
  }
  const long tiles256 = (long)(M / 128) * (N / 256);
  if (tiles256 > 64 || kb < 4) return best;
  const double hbmUs = ((double)M + N) * K * 2 / 6.4e6;
  double bestUs = pair ? 7.2 + kb * 0.33 : 8.5 + kb * 0.38;
  for (auto &k : kSplitKinds) {
    const long tiles = tiles256 * (256 / k.tileN);
    for (auto &sp : kSplits) {
      if (tiles * sp.parts > sp.ctas || sp.parts * 4 > kb) continue;
      const double steps = (kb + sp.parts - 1) / sp.parts * k.stepUs;
      const double bytes = (double)tiles * kb * (128 + k.tileN) * 128;
      const double us = k.fixedUs + std::max({steps, hbmUs, bytes / 13e6});
      if (us < bestUs) {
        bestUs = us;
        best.tileN = k.tileN;
        best.parts = sp.parts;
      }
    }
  }
  return best;
}

// The tiles of the persistent kernel's last wave, where handing them to the split kernel (parts
// CTAs per tile) is quicker than a wave of whole tiles in which most SMs are idle.  8192 x 3584
// x 8192 is 6 waves of 74 CTA pairs and 4 tiles: 336 -> 325 us; 2048 x 5120 x 4096 119 -> 86,
// 1408 x 3584 x 8192 99 -> 76.  3 us are asked for as margin (the second launch; 2304 x 2560 x
// 3072 lost 2 %), and beyond 9 waves the last one no longer counts.
SplitGemmTail tailPlan(int M, int N, int K, bool pair, int units, SplitGemmPlan *plan) {
  SplitGemmTail t;
  const int kb = K / 64, tiles = (M / (pair ? 256 : 128)) * (N / 256), rest = tiles % units;
  if (tiles <= units || tiles > 9 * units || rest == 0 || readParam("GEMM_SPLIT", 0) == 1) return t;
  const int parts128 = rest * (pair ? 2 : 1);
  for (auto &sp : kSplits) {
    if (sp.parts < 2 || parts128 * sp.parts > sp.ctas || sp.parts * 4 > kb) continue;
    const double steps = (kb + sp.parts - 1) / sp.parts * kSplitKinds[0].stepUs;
    const double bytes = (double)parts128 * kb * (128 + 256) * 128;
    if (kSplitKinds[0].fixedUs + std::max(steps, bytes / 13e6) + 3.0 > kb * 0.38) break;
    plan->tileN = 256;
    plan->parts = sp.parts;
    t.first = tiles - rest;
    t.count = rest;
    t.tileRows = pair ? 256 : 128;
    t.groupRows = groupRows(pair);
    break;
  }
  return t;
}

flagcxResult_t checkShape(int M, int N, int K) {
  FCX_ARGCHECK(M > 0 && N > 0 && K > 0 && M % 128 == 0 && N % 256 == 0 && K % 64 == 0,
               "tcgen05 GEMM needs M %% 128 == 0, N %% 256 == 0, K %% 64 == 0 (got %d x %d x %d)", M, N, K);
  return flagcxSuccess;
}

flagcxResult_t symAlloc(flagcxComm *c, size_t bytes, void **ptr, Window **win, bool *isVmm) {
  cu::VmmBlock b;
  if (cu::vmmSupported(c->cudaDev) && readParam("VMM_ENABLE", 1) != 0) {
    FCXCHECK(cu::vmmAlloc(bytes, c->cudaDev, &b));
    *ptr = b.ptr;
    *isVmm = true;
  } else {
    FCX_CUDACHECK(cudaMalloc(ptr, bytes));
    *isVmm = false;
  }
  return windowRegister(c, *ptr, bytes, FLAGCX_WIN_COLL_SYMMETRIC, win);
}

void symFree(flagcxComm *c, void *ptr, Window *win, bool isVmm) {
  if (!ptr) return;
  if (win) windowDeregister(c, win);
  if (isVmm) {
    if (const cu::VmmBlock *b = cu::vmmLookup(ptr)) { cu::VmmBlock copy = *b; cu::vmmFree(&copy); }
  } else {
    cudaFree(ptr);
  }
}

flagcxResult_t cachedMap(std::map<const void *, CUtensorMap> &cache, const void *base, uint64_t rows, uint64_t cols,
                         uint32_t boxRows, const CUtensorMap **out) {
  auto it = cache.find(base);
  if (it == cache.end()) {
    CUtensorMap m;
    FCXCHECK(cu::tensorMap2dBf16(&m, base, rows, cols, boxRows, 64));
    if (cache.size() > 256) cache.clear();
    it = cache.emplace(base, m).first;
  }
  *out = &it->second;
  return flagcxSuccess;
}

} // namespace

extern "C" {

flagcxResult_t flagcxGemmBf16(const void *A, const void *B, void *D, int M, int N, int K, flagcxStream_t stream) {
  if (!A || !B || !D) return flagcxInvalidArgument;
  if (!cu::available()) return flagcxNotSupported;
  FCXCHECK(checkShape(M, N, K));
  CUtensorMap ta, tb;
  FCXCHECK(cu::tensorMap2dBf16(&ta, A, M, K, 128, 64));
  const bool pair = usePair(M);
  SplitGemmPlan plan = splitPlan(M, N, K, pair);
  if (plan.tileN) {
    FCXCHECK(cu::tensorMap2dBf16(&tb, B, N, K, plan.tileN, 64));
    cudaError_t e = launchSplitGemm(stream ? stream->base : nullptr, ta, tb, D, M, N, K, plan);
    if (e != cudaSuccess) { FCX_WARN("GEMM launch failed: %s", cudaGetErrorString(e)); return flagcxUnhandledDeviceError; }
    return flagcxSuccess;
  }
  FCXCHECK(cu::tensorMap2dBf16(&tb, B, N, K, pair ? 128 : 256, 64));
  flagcxDevComm c;
  memset(&c, 0, sizeof c);
  c.nRanks = 1;
  c.timeoutNs = 4000000000ull;
  TpGemmArgs a;
  memset(&a, 0, sizeof a);
  a.D = (__nv_bfloat16 *)D;
  a.M = M; a.N = N; a.K = K;
  a.mode = kPlain;
  a.rowsPerRank = M;
  a.groupRows = groupRows(pair);
  int tiles = (M / 128) * (N / 256);
  if (pair) tiles = 2 * ((M / 256) * (N / 256));
  const int sms = smCount();
  const SplitGemmTail tail = tailPlan(M, N, K, pair, pair ? sms / 2 : sms, &plan);
  a.tiles = tail.first;
  cudaError_t e = launchTpGemm(stream ? stream->base : nullptr, ta, tb, nullptr, c, a, std::min(tiles, sms), pair);
  if (e == cudaSuccess && tail.count) {
    CUtensorMap tb256;
    FCXCHECK(cu::tensorMap2dBf16(&tb256, B, N, K, 256, 64));
    e = launchSplitGemm(stream ? stream->base : nullptr, ta, tb256, D, M, N, K, plan, tail);
  }
  if (e != cudaSuccess) { FCX_WARN("GEMM launch failed: %s", cudaGetErrorString(e)); return flagcxUnhandledDeviceError; }
  return flagcxSuccess;
}

flagcxResult_t flagcxTpGemmCreate(flagcxComm_t comm, int mode, int M, int N, int K, flagcxTpGemm_t *out) {
  if (!commValid(comm) || !out) return flagcxInvalidArgument;
  if (!comm->devicePath || comm->emu) return flagcxNotSupported;
  FCXCHECK(checkShape(M, N, K));
  const int n = comm->nranks;
  FCX_ARGCHECK((mode == kAllGatherGemm || mode == kGemmReduceScatter) && M % (128 * n) == 0,
               "flagcxTpGemmCreate: mode must be 1 (all-gather->GEMM) or 2 (GEMM->reduce-scatter) and M a multiple of 128 x ranks");
  auto *h = new flagcxTpGemm();
  h->comm = comm;
  h->mode = mode;
  h->M = M; h->N = N; h->K = K;
  h->rowsPerRank = M / n;
  const int chunks = h->rowsPerRank / 128;
  size_t bufBytes = mode == kAllGatherGemm ? (size_t)M * K * 2 : (size_t)M * N * 2;
  size_t flagBytes = alignUp(128 * (size_t)n * chunks, 4096); // one counter per 128-byte line
  flagcxResult_t r = symAlloc(comm, bufBytes, &h->buf, &h->wBuf, &h->vmmBuf);
  if (r == flagcxSuccess) r = symAlloc(comm, flagBytes, &h->flags, &h->wFlags, &h->vmmFlags);
  if (r != flagcxSuccess) { delete h; return r; }
  FCX_CUDACHECK(cudaMemset(h->flags, 0, flagBytes));
  FCX_CUDACHECK(cudaDeviceSynchronize());
  if (mode == kAllGatherGemm) FCXCHECK(cu::tensorMap2dBf16(&h->tmGather, h->buf, M, K, 128, 64));
  memset(&h->storeMaps, 0, sizeof h->storeMaps);
  if (mode == kGemmReduceScatter)
    for (int p = 0; p < n; ++p) FCXCHECK(cu::tensorMap2dBf16(&h->storeMaps.m[p], h->wBuf->peer[p], M, N, 32, 64));
  FCXCHECK(comm->bootstrap->barrier()); // flags are zero everywhere before anyone raises one
  *out = h;
  return flagcxSuccess;
}

flagcxResult_t flagcxTpGemmDestroy(flagcxTpGemm_t h) {
  if (!h) return flagcxSuccess;
  flagcxComm *c = h->comm;
  cudaDeviceSynchronize();
  if (c->bootstrap) c->bootstrap->barrier();
  symFree(c, h->buf, h->wBuf, h->vmmBuf);
  symFree(c, h->flags, h->wFlags, h->vmmFlags);
  delete h;
  return flagcxSuccess;
}

flagcxResult_t flagcxTpGemmGetShard(flagcxTpGemm_t h, void **localShard) {
  if (!h || !localShard || h->mode != kAllGatherGemm) return flagcxInvalidArgument;
  *localShard = (char *)h->buf + (size_t)h->comm->rank * h->rowsPerRank * h->K * 2;
  return flagcxSuccess;
}

flagcxResult_t flagcxTpAllGatherGemm(flagcxTpGemm_t h, const void *B, void *D, flagcxStream_t stream) {
  if (!h || !B || !D || h->mode != kAllGatherGemm) return flagcxInvalidArgument;
  flagcxComm *c = h->comm;
  if (c->asyncError.load() != flagcxSuccess) return (flagcxResult_t)c->asyncError.load();
  const CUtensorMap *tb;
  const bool pair = usePair(h->rowsPerRank);
  FCXCHECK(cachedMap(h->mapsB, B, h->N, h->K, pair ? 128 : 256, &tb));
  TpGemmArgs a;
  memset(&a, 0, sizeof a);
  a.D = (__nv_bfloat16 *)D;
  a.M = h->M; a.N = h->N; a.K = h->K;
  a.mode = kAllGatherGemm;
  a.rowsPerRank = h->rowsPerRank;
  a.groupRows = groupRows(pair);
  a.epoch = ++h->epoch;
  for (int p = 0; p < c->nranks; ++p) {
    a.gathered[p] = (__nv_bfloat16 *)h->wBuf->peer[p];
    a.chunkFlags[p] = (unsigned long long *)h->wFlags->peer[p];
  }
  const int sms = smCount();
  a.piecesPerChunk = h->K / 16; // a chunk is 128 rows of K bf16 = K/16 pieces of 4 KiB
  cudaError_t e = launchTpGemm(stream ? stream->base : nullptr, h->tmGather, *tb, nullptr, c->dev, a, sms, pair);
  if (e != cudaSuccess) { FCX_WARN("all-gather GEMM launch failed: %s", cudaGetErrorString(e)); return flagcxUnhandledDeviceError; }
  return flagcxSuccess;
}

flagcxResult_t flagcxTpGemmReduceScatter(flagcxTpGemm_t h, const void *A, const void *B, void *out,
                                         flagcxStream_t stream) {
  if (!h || !A || !B || !out || h->mode != kGemmReduceScatter) return flagcxInvalidArgument;
  flagcxComm *c = h->comm;
  if (c->asyncError.load() != flagcxSuccess) return (flagcxResult_t)c->asyncError.load();
  const CUtensorMap *ta, *tb;
  const bool pair = usePair(h->rowsPerRank);
  FCXCHECK(cachedMap(h->mapsA, A, h->M, h->K, 128, &ta));
  FCXCHECK(cachedMap(h->mapsB, B, h->N, h->K, pair ? 128 : 256, &tb));
  TpGemmArgs a;
  memset(&a, 0, sizeof a);
  a.M = h->M; a.N = h->N; a.K = h->K;
  a.mode = kGemmReduceScatter;
  a.rowsPerRank = h->rowsPerRank;
  a.groupRows = groupRows(pair);
  a.epoch = ++h->epoch;
  a.out = (__nv_bfloat16 *)out;
  for (int p = 0; p < c->nranks; ++p) {
    a.partial[p] = (__nv_bfloat16 *)h->wBuf->peer[p];
    a.rowFlags[p] = (unsigned long long *)h->wFlags->peer[p];
  }
  cudaError_t e = launchTpGemm(stream ? stream->base : nullptr, *ta, *tb, &h->storeMaps, c->dev, a, smCount(), pair);
  if (e != cudaSuccess) { FCX_WARN("GEMM reduce-scatter launch failed: %s", cudaGetErrorString(e)); return flagcxUnhandledDeviceError; }
  return flagcxSuccess;
}

} // extern "C"
