// launch.h -- host-callable launchers of the collective kernels.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "coll_args.h"

namespace fcx {

struct MoeArgs;

struct LaunchCtx {
  const flagcxDevComm *comm = nullptr; // host copy, passed to the kernel by value
  cudaStream_t stream = nullptr;
  int nCtas = 1;
  int nThreads = FLAGCX_DEVICE_THREADS_PER_CTA;
  // Emulated world (several ranks of one process on one GPU): one cooperative
  // launch with gridDim.y = emuRanks; the per-rank blocks (host arrays) become its arguments.
  int emuRanks = 0;
  const flagcxDevComm *emuComms = nullptr;
  const CollArgs *emuArgs = nullptr;
  const P2pArgs *emuP2p = nullptr;
  const MoeArgs *emuMoe = nullptr;
  bool emuBulk = false;          // some emulated rank takes a bulk-copy path: the launch needs the shared-memory ring
};

// Arguments of an emulated world's kernel: blockIdx.y picks its rank's.  They travel with the
// launch, up to 9.2 KB of the 32 KB that arguments may take.  Copied to the device before each
// launch, as they once were, they cost two copies of 1.2 us in front of the kernel, the host time
// for them, and a load from memory for every field that a barrier looks at.  Eight ranks' all-reduce
// of 32 KiB: kernel 20.8 -> 10.0 us; of 16 KiB, back to back: 19.3 -> 16.5 us.
template <typename Args>
struct EmuLaunch {
  flagcxDevComm comm[FLAGCX_MAX_RANKS];
  Args args[FLAGCX_MAX_RANKS];
};
template <typename Args>
cudaError_t launchEmu(void (*kernel)(EmuLaunch<Args>), const LaunchCtx &lc, const Args *args, dim3 grid, dim3 block,
                      size_t sharedBytes) {
  EmuLaunch<Args> e;
  for (int r = 0; r < lc.emuRanks; ++r) {
    e.comm[r] = lc.emuComms[r];
    e.args[r] = args[r];
  }
  void *params[] = {&e};
  return cudaLaunchCooperativeKernel((const void *)kernel, grid, block, params, sharedBytes, lc.stream);
}

// How many CTAs per rank of a kernel may be part of such a launch (all must run at once): at least 1
// where one fits at all.  The answer is the device's and is kept per kernel.
template <auto Kernel>
cudaError_t emuCtasPerRank(int threads, int ranks, int *ctas) {
  static std::atomic<int> perDevice[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int all = dev < 64 ? perDevice[dev].load(std::memory_order_relaxed) : 0;
  if (!all) {
    int sms = 0, perSm = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, (const void *)Kernel, threads, 0);
    if (e != cudaSuccess) return e;
    all = sms * perSm;
    if (dev < 64) perDevice[dev].store(all, std::memory_order_relaxed);
  }
  *ctas = all / ranks > 1 ? all / ranks : 1;
  return cudaSuccess;
}

cudaError_t launchMoeDispatch(const LaunchCtx &lc, const MoeArgs &a);
cudaError_t launchMoeCombine(const LaunchCtx &lc, const MoeArgs &a);

cudaError_t launchReduceKernel(const LaunchCtx &lc, const CollArgs &a, int nRanks);
cudaError_t launchCopyKernel(const LaunchCtx &lc, const CollArgs &a);
cudaError_t launchP2pKernel(const LaunchCtx &lc, const P2pArgs &a);
cudaError_t launchNvlsKernel(const LaunchCtx &lc, const CollArgs &a);
cudaError_t launchLlKernel(const LaunchCtx &lc, const CollArgs &a);
// One-sided host API (onesided.cu).  `arrival` is a zero-initialised device word the
// CTAs of one put count themselves in; puts on one stream may share it.
cudaError_t launchPutSignal(cudaStream_t s, void *dst, const void *src, size_t bytes, unsigned long long *peerSignal,
                            unsigned long long addValue, unsigned int *arrival, int nCtas);
cudaError_t launchWaitSignal(cudaStream_t s, const flagcxDevComm &c, const unsigned long long *sig,
                             unsigned long long want, unsigned int peer);
// Upper bound on grid size (x * y) for the cooperative emulated-world launch.
int maxCoresidentCtas(int nThreads);

} // namespace fcx
