// moe.cu -- expert-parallel dispatch and combine as NVLink kernels.
//
// dispatch: every (token, chosen expert) pair ends up in the destination rank's receive
// buffer, already grouped by expert (rows of expert e from rank 0, then rank 1, ...),
// i.e. the all-to-all and the token permutation are one pass over the data.  A token that
// several experts of ONE rank want crosses NVLink once; the receiver makes the other
// copies locally.  Counting the routing table and exchanging the counts that place the
// rows happen inside the same kernel.
// combine: the mirror image.  The token's owner pushes the gate weights to the expert
// ranks; each expert rank adds up, in fp32, the weighted outputs a token has on it (one
// bf16 row per token and rank); the owner pulls those rows and sums them: one row per
// (token, rank) crosses NVLink instead of one per (token, expert), the all-to-all back and
// the weighted sum are one kernel, and the un-permutation is implicit.  With
// preReduce = 0 the owner pulls every (token, expert) row and weights it itself.
//
// FlagCX offers only flagcxAlltoAllv for this (plugin/torch/flagcx/src/
// backend_flagcx.cpp:926-993 in the FlagCX project); permutation and the weighted
// sum are separate framework kernels there.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "launch.h"
#include "moe_args.h"
#include "prims.cuh"

namespace fcx {
namespace {

// CTAs of 8 warps: the combine keeps eight 16-byte loads per lane in flight and wants the
// registers for them; the host launches twice as many CTAs as it would of the 512-thread kind.
constexpr int kMoeThreads = 256;
// In the emulated world, where all ranks' CTAs share the SMs, the dispatch runs as one CTA of twice
// the threads per SM: CTAs of one SM wait for each other's system-wide releases in a barrier (8
// tokens of 7168 a rank 22.5 -> 18.8 us against two CTAs per SM, 400 of 2048 22.7 -> 18.2, 512 of 7168
// the same).
constexpr int kMoeEmuThreads = 512;

// A row of vecs 16-byte vectors is copied in pieces of at most 32 x kMoePiece vectors, one warp
// each, so that the warps of a CTA share its rows evenly however few they are.
constexpr int kMoePiece = 8;
struct RowPieces {
  int count, vecs; // pieces per row, vectors per piece
  __device__ __forceinline__ explicit RowPieces(int rowVecs) {
    count = (rowVecs + 32 * kMoePiece - 1) / (32 * kMoePiece);
    vecs = ((rowVecs + count - 1) / count + 31) & ~31;
  }
};

// One warp copies the vectors [first, end) of a row to the first n of the rows dst.  The piece is
// read once, all of a lane's loads in flight, and then goes to every destination.
__device__ __forceinline__ void warpCopyPiece(char *const *dst, int n, const char *src, int first, int end, int lane,
                                              bool srcIsPeerWritten) {
  uint4 r[kMoePiece];
#pragma unroll
  for (int u = 0; u < kMoePiece; ++u) {
    const int v = first + lane + 32 * u;
    if (v < end) r[u] = srcIsPeerWritten ? ldSys16((const uint4 *)src + v) : ((const uint4 *)src)[v];
  }
  for (int k = 0; k < n; ++k) {
    uint4 *d = (uint4 *)dst[k];
#pragma unroll
    for (int u = 0; u < kMoePiece; ++u) {
      const int v = first + lane + 32 * u;
      if (v < end) st16(d + v, r[u]);
    }
  }
}

// A group record (FLAGCX_MOE_MAX_TOPK ints written by a peer) as two 16-byte loads.
__device__ __forceinline__ void loadGroup(const int *rec, int rows[FLAGCX_MOE_MAX_TOPK]) {
  static_assert(FLAGCX_MOE_MAX_TOPK == 8, "a group record is two 16-byte vectors");
  const uint4 lo = ldSys16(rec), hi = ldSys16(rec + 4);
  rows[0] = (int)lo.x; rows[1] = (int)lo.y; rows[2] = (int)lo.z; rows[3] = (int)lo.w;
  rows[4] = (int)hi.x; rows[5] = (int)hi.y; rows[6] = (int)hi.z; rows[7] = (int)hi.w;
}

// dst row = sum over M rows of w[j] * rows[j], fp32 accumulation, one warp.  U vectors of
// every row are loaded before any is used, so a lane has M*U 16-byte loads in flight.
template <int M, int U>
__device__ __forceinline__ void rowSumFixed(const char *const *rows, const float *w, uint4 *dst, int vecs, int lane,
                                            bool peerWritten) {
  for (int v0 = lane; v0 < vecs; v0 += 32 * U) {
    uint4 r[U][M];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + 32 * u;
      if (v < vecs) {
#pragma unroll
        for (int j = 0; j < M; ++j)
          r[u][j] = peerWritten ? ldSys16(rows[j] + (size_t)v * 16) : *(const uint4 *)(rows[j] + (size_t)v * 16);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int v = v0 + 32 * u;
      if (v < vecs) {
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < M; ++j) {
          const __nv_bfloat16 *e = (const __nv_bfloat16 *)&r[u][j];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] += w[j] * __bfloat162float(e[i]);
        }
        uint4 o;
        __nv_bfloat16 *oe = (__nv_bfloat16 *)&o;
#pragma unroll
        for (int i = 0; i < 8; ++i) oe[i] = __float2bfloat16_rn(acc[i]);
        st16(dst + v, o);
      }
    }
  }
}

// dst row = sum of the first m rows, weighted (m = 0: zeros).  Few rows mean more vectors
// per row in flight: 8 loads per lane either way.  m is the same for all lanes of the warp.
__device__ __forceinline__ void weightedRowSum(const char *rows[FLAGCX_MOE_MAX_TOPK], float w[FLAGCX_MOE_MAX_TOPK], int m,
                                               uint4 *dst, int vecs, int lane, bool rowsArePeerWritten) {
  if (m == 0) {
    for (int v = lane; v < vecs; v += 32) st16(dst + v, make_uint4(0, 0, 0, 0));
  } else if (m == 1) {
    rowSumFixed<1, 8>(rows, w, dst, vecs, lane, rowsArePeerWritten);
  } else if (m == 2) {
    rowSumFixed<2, 4>(rows, w, dst, vecs, lane, rowsArePeerWritten);
  } else if (m <= 4) {
#pragma unroll
    for (int j = 2; j < 4; ++j)
      if (j >= m) { rows[j] = rows[0]; w[j] = 0.f; } // pad with a weightless repeat of a valid row
    rowSumFixed<4, 2>(rows, w, dst, vecs, lane, rowsArePeerWritten);
  } else {
#pragma unroll
    for (int j = 4; j < FLAGCX_MOE_MAX_TOPK; ++j)
      if (j >= m) { rows[j] = rows[0]; w[j] = 0.f; }
    rowSumFixed<8, 1>(rows, w, dst, vecs, lane, rowsArePeerWritten);
  }
}

// Start of CTA b's range of T tokens: at most ceil(T / g) of them, every CTA within one of that.
__device__ __forceinline__ int firstToken(int T, int b, int g) { return (int)((long)T * b / g); }

// The whole dispatch is this one kernel: histogram of the routing, exchange of the
// counts, the copies, and the local fan-out of rows that several experts of one rank want.
// Bound: memory (eight emulated ranks, 512 tokens x 7168, top 8 of 256: 640 MB, 97 us of the 126
// at the rate of a copy), then two barriers and about 6 us of counting and routing.  One warp per
// row, one load of the routing table at a time, and one CTA of 8 warps per SM took 173 us; the
// routes of four tokens at once, pieces of rows and 16 warps per SM brought it here.
constexpr int kMoeTable = 256; // tokens, or group records, that a CTA looks at before it moves their rows
static_assert(kMoeThreads >= kMoeTable, "a thread looks at one record");
struct DispatchShared {
  int base[FLAGCX_MOE_MAX_EXPERTS];
  union {
    struct { int tot[FLAGCX_MOE_MAX_EXPERTS], before[FLAGCX_MOE_MAX_EXPERTS], mine[FLAGCX_MOE_MAX_EXPERTS]; };
    struct { // rows that a token goes to, or the row that a group has and then those it is copied to
      char *row[kMoeTable][FLAGCX_MOE_MAX_TOPK];
      int nRows[kMoeTable];
    };
  };
  int grpN[FLAGCX_MAX_RANKS], nRec;
};

__device__ void dispatchBody(const flagcxDevComm &c, const MoeArgs &a) {
  __shared__ DispatchShared s;
  const int b = blockIdx.x, g = gridDim.x, rank = c.rank, n = c.nRanks;
  const int t = threadIdx.x, nt = blockDim.x;
  // this CTA's tokens: a contiguous range, so that "how many earlier pairs chose expert e"
  // splits into the pairs of earlier CTAs' ranges and the pairs of this range
  const int tlo = firstToken(a.T, b, g), thi = firstToken(a.T, b + 1, g);
  const int lo = tlo * a.K, hi = thi * a.K, items = a.T * a.K;
  // 0. every CTA counts the whole routing table (a few dozen shared-memory atomics per
  // thread): no separate counting kernel, no global atomics, no memset
  for (int e = t; e < a.E; e += nt) s.tot[e] = s.before[e] = s.mine[e] = 0;
  if (t < FLAGCX_MAX_RANKS) s.grpN[t] = 0;
  __syncthreads();
  constexpr int kAhead = 8; // entries of the table that a thread has on their way
  for (int i0 = t; i0 < items; i0 += kAhead * nt) {
    int es[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) es[u] = i0 + u * nt < items ? a.topkIdx[i0 + u * nt] : 0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + u * nt, e = es[u];
      if (i >= items) break;
      const bool valid = e >= 0 && e < a.E;
      if (i < lo) { if (valid) atomicAdd(&s.before[e], 1); }
      else if (i < hi) {
        if (valid) a.pos[i] = atomicAdd(&s.mine[e], 1); // index within this CTA's range, completed below
        else {
          a.pos[i] = -1;
          fcxdev::reportError(c.status, FLAGCX_DEV_BOUNDS, FLAGCX_DEV_AT_KERNEL, 0xffffffffu, (unsigned long long)i);
        }
      } else if (valid) atomicAdd(&s.tot[e], 1);
    }
  }
  __syncthreads();
  // 1. publish my per-expert counts in every rank's table (row `rank`), mine included;
  // every CTA writes the same values and reads them back from its own peers' CTA
  for (int e = t; e < a.E; e += nt) {
    const int cnt = s.tot[e] + s.before[e] + s.mine[e];
#pragma unroll
    for (int p = 0; p < FLAGCX_MAX_RANKS; ++p)
      if (p < n) a.countsAll[p][(size_t)rank * a.E + e] = cnt;
  }
  if (!ctaBarrier(c, b)) return;
  // 2. where my rows start inside each destination's expert-grouped buffer
  const int *tab = a.countsAll[rank];
  for (int e = t; e < a.E; e += nt) {
    int cnt[FLAGCX_MAX_RANKS], all = 0, lower = 0;
    // rows written by peers: system-scope loads, never a stale cached line
#pragma unroll
    for (int q = 0; q < FLAGCX_MAX_RANKS; ++q) cnt[q] = q < n ? ldSysElem(tab + (size_t)q * a.E + e) : 0;
#pragma unroll
    for (int q = 0; q < FLAGCX_MAX_RANKS; ++q) {
      all += cnt[q];
      if (q < rank) lower += cnt[q];
    }
    s.tot[e] = all;
    s.base[e] = lower + s.before[e]; // pairs of lower ranks and of earlier CTAs' ranges come first
  }
  __syncthreads();
  for (int e = t; e < a.E; e += nt) {
    int sum = 0;
    for (int e2 = e / a.EPR * a.EPR; e2 < e; ++e2) sum += s.tot[e2];
    s.base[e] += sum;
  }
  if (b == 0) {
    // this rank's own expert boundaries, for whoever runs the experts
    for (int le = t; le <= a.EPR; le += nt) {
      int sum = 0;
      for (int e2 = 0; e2 < le; ++e2) sum += s.tot[rank * a.EPR + e2];
      a.expertOffsets[le] = sum;
    }
    if (t == 0) {
      long total = 0;
      for (int le = 0; le < a.EPR; ++le) total += s.tot[rank * a.EPR + le];
      if ((size_t)total > a.capacity)
        fcxdev::reportError(c.status, FLAGCX_DEV_BOUNDS, FLAGCX_DEV_AT_KERNEL, (unsigned)rank, (unsigned long long)total);
    }
  }
  // 3. eight lanes per token work out where its rows go.  The first expert of each destination
  // rank gets the row over NVLink, straight into its final place; the destination is left a group
  // record (all rows of that token there, leader first) from which it makes the other copies
  // locally.  Then one warp per piece of a row moves the data.
  const int warps = nt >> 5, warp = t >> 5, lane = t & 31;
  const int vecs = a.H / 8; // 16-byte vectors per row
  const size_t rowBytes = (size_t)a.H * 2;
  const int capPer = ((a.maxT + g - 1) / g) * a.K;
  const RowPieces pieces(vecs);
  static_assert(FLAGCX_MOE_MAX_TOPK == 8, "a quarter of a warp per token");
  for (int tok0 = tlo; tok0 < thi; tok0 += kMoeTable) {
    const int nTok = thi - tok0 < kMoeTable ? thi - tok0 : kMoeTable;
    __syncthreads(); // the tables of counts, or the last batch's rows, have been read
    for (int j0 = warp * 4; j0 < nTok; j0 += warps * 4) { // the whole warp stays together
      const int j = j0 + (lane >> 3), k = lane & 7, tok = tok0 + j;
      int d = 0, row = 0;
      bool valid = false;
      if (j < nTok && k < a.K) {
        const int i = tok * a.K + k, e = a.topkIdx[i], rel = a.pos[i];
        valid = rel >= 0;
        if (valid) {
          d = e / a.EPR;
          row = s.base[e] + rel;
          a.pos[i] = row; // any value >= 0 tells combine that the pair is real
          a.route[2 * i] = d;
          a.route[2 * i + 1] = row;
          valid = (size_t)row < a.capacity; // rows past the capacity are reported by the receiver and dropped
        }
      }
      // pairs of one token that go to one rank form a group; others (no pair, bad pair) are alone
      const int alone = FLAGCX_MAX_RANKS * 4 + lane;
      const unsigned members = __match_any_sync(0xffffffffu, valid && a.dedup ? (lane >> 3) * FLAGCX_MAX_RANKS + d : alone);
      const int leader = __ffs(members) - 1, member = __popc(members & ((1u << lane) - 1u));
      const bool isLeader = valid && lane == leader;
      int idx = 0;
      if (isLeader) idx = atomicAdd(&s.grpN[d], 1);
      idx = __shfl_sync(0xffffffffu, idx, leader);
      // the token's groups, packed: entry j = pair index of the j-th leader, -1 after the last
      const unsigned leaders = (__ballot_sync(0xffffffffu, isLeader) >> (lane & 24)) & 0xffu;
      const int at = __popc(leaders & ((1u << k) - 1u)), nLead = __popc(leaders);
      if (j < nTok) {
        if (isLeader) {
          a.lead[tok * a.K + at] = k;
          s.row[j][at] = a.recv[d] + (size_t)row * rowBytes;
        }
        if (k >= nLead && k < a.K) a.lead[tok * a.K + k] = -1;
        if (k == 0) s.nRows[j] = nLead;
      }
      if (valid && idx < capPer) {
        int *rec = a.grpList[d] + ((size_t)rank * a.grpRecordsPerSender + (size_t)b * capPer + idx) * FLAGCX_MOE_MAX_TOPK;
        rec[member] = row;
        if (isLeader)
          for (int m = __popc(members); m < FLAGCX_MOE_MAX_TOPK; ++m) rec[m] = -1;
      }
    }
    __syncthreads();
    for (int i = warp; i < nTok * pieces.count; i += warps) {
      const int j = i / pieces.count, first = (i - j * pieces.count) * pieces.vecs;
      const int end = first + pieces.vecs < vecs ? first + pieces.vecs : vecs;
      warpCopyPiece(s.row[j], s.nRows[j], (const char *)(a.x + (size_t)(tok0 + j) * a.H), first, end, lane, false);
    }
  }
  __syncthreads();
  if (t < n) a.grpCount[t][(size_t)rank * FLAGCX_COLL_BARRIER_SLOTS + b] = s.grpN[t] < capPer ? s.grpN[t] : capPer;
  if (!ctaBarrier(c, b)) return;
  // 4. the copies the senders' CTA b left to this rank: row to row inside my own buffer.  A thread
  // looks at one record; those with more than one row are collected, and their pieces shared out.
  int start[FLAGCX_MAX_RANKS + 1]; // records of senders 0 .. q-1
  start[0] = 0;
#pragma unroll
  for (int q = 0; q < FLAGCX_MAX_RANKS; ++q)
    start[q + 1] = q < n ? ldSysElem(a.grpCount[rank] + (size_t)q * FLAGCX_COLL_BARRIER_SLOTS + b) : 0;
#pragma unroll
  for (int q = 0; q < FLAGCX_MAX_RANKS; ++q) start[q + 1] += start[q];
  for (int r0 = 0; r0 < start[FLAGCX_MAX_RANKS]; r0 += kMoeTable) {
    if (t == 0) s.nRec = 0;
    __syncthreads();
    const int r = r0 + t;
    if (t < kMoeTable && r < start[FLAGCX_MAX_RANKS]) {
      int q = 0, before = 0;
#pragma unroll
      for (int p = 1; p < FLAGCX_MAX_RANKS; ++p)
        if (r >= start[p]) { q = p; before = start[p]; }
      const int *rec = a.grpList[rank] +
                       ((size_t)q * a.grpRecordsPerSender + (size_t)b * capPer + (r - before)) * FLAGCX_MOE_MAX_TOPK;
      int rows[FLAGCX_MOE_MAX_TOPK];
      loadGroup(rec, rows);
      if (rows[1] >= 0 && (size_t)rows[0] < a.capacity) { // packed: no row after -1
        const int at = atomicAdd(&s.nRec, 1);
        int m = 0;
#pragma unroll
        for (int k = 0; k < FLAGCX_MOE_MAX_TOPK; ++k)
          if (rows[k] >= 0 && (size_t)rows[k] < a.capacity) s.row[at][m++] = a.recv[rank] + (size_t)rows[k] * rowBytes;
        s.nRows[at] = m;
      }
    }
    __syncthreads();
    const int nRec = s.nRec;
    for (int i = warp; i < nRec * pieces.count; i += warps) {
      const int j = i / pieces.count, first = (i - j * pieces.count) * pieces.vecs;
      const int end = first + pieces.vecs < vecs ? first + pieces.vecs : vecs;
      warpCopyPiece(s.row[j] + 1, s.nRows[j] - 1, s.row[j][0], first, end, lane, true);
    }
    __syncthreads();
  }
}

// Pull-everything combine: the token's owner reads each (token, expert) row and weights it.
// Independent of the dispatch's CTA layout (it needs only the route), so it runs as CTAs of
// 512 threads: measured faster that way (402 against 527 us on two B200s for the same
// number of warps in 256-thread CTAs).  A warp draws a part of a token at a time, so that few tokens
// occupy all warps and many end together.  Eight emulated ranks, 512 tokens x 7168: 135 -> 99 us with
// twice the CTAs (107), the parts drawn by ticket, and a cheaper barrier; 530 MB, 81 us for a copy.
__device__ void combinePullBody(const flagcxDevComm &c, const MoeArgs &a) {
  const int b = blockIdx.x, g = gridDim.x;
  const int t = threadIdx.x, nt = blockDim.x;
  const int warpsPerCta = nt >> 5, lane = t & 31;
  const int vecs = a.H / 8;
  const size_t rowBytes = (size_t)a.H * 2;
  constexpr int U = 2; // vectors of every row in flight per lane
  // four parts or more per warp, of whole rounds of the loop below
  const int rounds = (vecs + 32 * U - 1) / (32 * U), wanted = a.T > 0 ? (4 * g * warpsPerCta + a.T - 1) / a.T : 1;
  const int perPart = (rounds + wanted - 1) / wanted, parts = (rounds + perPart - 1) / perPart;
  const Tickets tickets{a.tickets};
  const bool met = ctaBarrier(c, b); // every rank's expert outputs are complete
  int item = met ? (int)tickets.take() : a.T * parts;
  while (item < a.T * parts) {
    const int next = (int)tickets.take(); // on its way while this one is worked on
    const int tok = item / parts, first = (item - tok * parts) * perPart * 32 * U;
    const int end = first + perPart * 32 * U < vecs ? first + perPart * 32 * U : vecs;
    const char *rows[FLAGCX_MOE_MAX_TOPK];
    float w[FLAGCX_MOE_MAX_TOPK];
#pragma unroll
    for (int k = 0; k < FLAGCX_MOE_MAX_TOPK; ++k) {
      if (k < a.K) {
        int i = tok * a.K + k;
        int d = a.route[2 * i], row = a.route[2 * i + 1];
        bool ok = a.pos[i] >= 0 && (size_t)row < a.capacity;
        rows[k] = ok ? a.expertOut[d] + (size_t)row * rowBytes : nullptr;
        w[k] = ok ? a.topkW[i] : 0.f;
      } else {
        rows[k] = nullptr;
        w[k] = 0.f;
      }
    }
    uint4 *dst = (uint4 *)(a.out + (size_t)tok * a.H);
    for (int v0 = first + lane; v0 < end; v0 += 32 * U) {
      uint4 r[U][FLAGCX_MOE_MAX_TOPK];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int v = v0 + 32 * u;
        if (v < end) {
#pragma unroll
          for (int k = 0; k < FLAGCX_MOE_MAX_TOPK; ++k)
            if (rows[k]) r[u][k] = ldSys16(rows[k] + (size_t)v * 16);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int v = v0 + 32 * u;
        if (v < end) {
          float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
          for (int k = 0; k < FLAGCX_MOE_MAX_TOPK; ++k)
            if (rows[k]) {
              const __nv_bfloat16 *e = (const __nv_bfloat16 *)&r[u][k];
#pragma unroll
              for (int j = 0; j < 8; ++j) acc[j] += w[k] * __bfloat162float(e[j]);
            }
          uint4 o;
          __nv_bfloat16 *oe = (__nv_bfloat16 *)&o;
#pragma unroll
          for (int j = 0; j < 8; ++j) oe[j] = __float2bfloat16_rn(acc[j]);
          dst[v] = o;
        }
      }
    }
    item = next;
  }
  tickets.leave();
  if (met) ctaBarrier(c, b); // peers may overwrite their expert outputs only after everyone has read them
}

// Pre-reducing combine.  Everything is organised per CTA index, like the dispatch: the
// groups that sender q's CTA b recorded here are reduced by this rank's CTA b and pulled
// by q's CTA b, so the per-CTA barriers across ranks are all the ordering it needs.
__device__ void combineReduceBody(const flagcxDevComm &c, const MoeArgs &a) {
  const int b = blockIdx.x, g = gridDim.x, rank = c.rank, n = c.nRanks;
  const int t = threadIdx.x, nt = blockDim.x;
  const int warpsPerCta = nt >> 5, warp = t >> 5, lane = t & 31;
  const int vecs = a.H / 8;
  const size_t rowBytes = (size_t)a.H * 2;
  const int tlo = firstToken(a.T, b, g), thi = firstToken(a.T, b + 1, g); // the dispatch's token ranges
  const int capPer = ((a.maxT + g - 1) / g) * a.K;
  // 0. the gate weight of each of my pairs goes next to the row it weights
  for (int i = tlo * a.K + t; i < thi * a.K; i += nt) {
    const int d = a.route[2 * i], row = a.route[2 * i + 1];
    if (a.pos[i] >= 0 && (size_t)row < a.capacity) a.wRow[d][row] = a.topkW[i];
  }
  if (!ctaBarrier(c, b)) return; // weights have landed; every rank's expert outputs are complete
  // A. one row per group: the weighted sum of the group's expert outputs, all local reads
  for (int q = 0; q < n; ++q) {
    const int cnt = ldSysElem(a.grpCount[rank] + (size_t)q * FLAGCX_COLL_BARRIER_SLOTS + b);
    const int *recs = a.grpList[rank] + ((size_t)q * a.grpRecordsPerSender + (size_t)b * capPer) * FLAGCX_MOE_MAX_TOPK;
    for (int r = warp; r < cnt; r += warpsPerCta) {
      int rowIdx[FLAGCX_MOE_MAX_TOPK];
      loadGroup(recs + (size_t)r * FLAGCX_MOE_MAX_TOPK, rowIdx);
      if ((size_t)rowIdx[0] >= a.capacity) continue;
      const char *rows[FLAGCX_MOE_MAX_TOPK];
      float w[FLAGCX_MOE_MAX_TOPK];
      int m = 0; // the record is packed: valid rows first
#pragma unroll
      for (int j = 0; j < FLAGCX_MOE_MAX_TOPK; ++j) {
        const bool ok = j == m && rowIdx[j] >= 0 && (size_t)rowIdx[j] < a.capacity;
        rows[j] = ok ? a.expertOut[rank] + (size_t)rowIdx[j] * rowBytes : nullptr;
        w[j] = ok ? ldSysElem(a.wRow[rank] + rowIdx[j]) : 0.f;
        m += ok ? 1 : 0;
      }
      weightedRowSum(rows, w, m, (uint4 *)(a.partial[rank] + (size_t)rowIdx[0] * rowBytes), vecs, lane, false);
    }
  }
  if (!ctaBarrier(c, b)) return; // the partial rows of my tokens are complete on every rank
  // B. each token adds up one row per rank it has experts on
  for (int tok = tlo + warp; tok < thi; tok += warpsPerCta) {
    const char *rows[FLAGCX_MOE_MAX_TOPK];
    float w[FLAGCX_MOE_MAX_TOPK];
    int m = 0;
#pragma unroll
    for (int j = 0; j < FLAGCX_MOE_MAX_TOPK; ++j) {
      rows[j] = nullptr;
      w[j] = 1.f;
      if (j < a.K) {
        const int k = a.lead[tok * a.K + j]; // pair index of this token's j-th group, -1 after the last
        if (j == m && k >= 0) {
          const int i = tok * a.K + k;
          rows[j] = a.partial[a.route[2 * i]] + (size_t)a.route[2 * i + 1] * rowBytes;
          ++m;
        }
      }
    }
    weightedRowSum(rows, w, m, (uint4 *)(a.out + (size_t)tok * a.H), vecs, lane, true);
  }
  ctaBarrier(c, b); // weights and partial rows may be overwritten only after everyone has read them
}


__global__ void __launch_bounds__(kMoeThreads)
    moeDispatchKernel(const __grid_constant__ flagcxDevComm c, const __grid_constant__ MoeArgs a) {
  dispatchBody(c, a);
}
__global__ void __launch_bounds__(kMoeEmuThreads)
    moeDispatchKernelEmu(const __grid_constant__ EmuLaunch<MoeArgs> e) {
  dispatchBody(e.comm[blockIdx.y], e.args[blockIdx.y]);
}
__global__ void __launch_bounds__(kMoeThreads)
    moeCombineKernel(const __grid_constant__ flagcxDevComm c, const __grid_constant__ MoeArgs a) {
  combineReduceBody(c, a);
}
__global__ void __launch_bounds__(kMoeThreads)
    moeCombineKernelEmu(const __grid_constant__ EmuLaunch<MoeArgs> e) {
  combineReduceBody(e.comm[blockIdx.y], e.args[blockIdx.y]);
}
__global__ void __launch_bounds__(FLAGCX_DEVICE_THREADS_PER_CTA)
    moeCombinePullKernel(const __grid_constant__ flagcxDevComm c, const __grid_constant__ MoeArgs a) {
  combinePullBody(c, a);
}
__global__ void __launch_bounds__(FLAGCX_DEVICE_THREADS_PER_CTA)
    moeCombinePullKernelEmu(const __grid_constant__ EmuLaunch<MoeArgs> e) {
  combinePullBody(e.comm[blockIdx.y], e.args[blockIdx.y]);
}

} // namespace

// The emulated world has fewer CTAs per rank to offer than a GPU of its own.  The pre-reducing
// combine must run as many as the dispatch that left it its records: what both kernels have room for.
static cudaError_t emuMoeCtas(const LaunchCtx &lc, bool preReduce, int *ctas) {
  int forDispatch = 0, forCombine = lc.nCtas;
  cudaError_t e = emuCtasPerRank<moeDispatchKernelEmu>(kMoeEmuThreads, lc.emuRanks, &forDispatch);
  if (e == cudaSuccess && preReduce) e = emuCtasPerRank<moeCombineKernelEmu>(kMoeThreads, lc.emuRanks, &forCombine);
  *ctas = std::min(lc.nCtas, std::min(forDispatch, forCombine));
  return e;
}

cudaError_t launchMoeDispatch(const LaunchCtx &lc, const MoeArgs &a) {
  if (lc.emuRanks > 0) {
    int ctas = 0;
    const cudaError_t e = emuMoeCtas(lc, a.preReduce != 0, &ctas);
    return e != cudaSuccess ? e : launchEmu(moeDispatchKernelEmu, lc, lc.emuMoe, dim3(ctas, lc.emuRanks), dim3(kMoeEmuThreads), 0);
  }
  moeDispatchKernel<<<lc.nCtas, kMoeThreads, 0, lc.stream>>>(*lc.comm, a);
  return cudaGetLastError();
}

// a.preReduce picks the kernel; the pull kind takes half as many CTAs of twice the threads.
cudaError_t launchMoeCombine(const LaunchCtx &lc, const MoeArgs &a) {
  const bool pull = a.preReduce == 0;
  const int pullCtas = (lc.nCtas + 1) / 2, pullThreads = FLAGCX_DEVICE_THREADS_PER_CTA;
  if (lc.emuRanks > 0) {
    int ctas = 0;
    cudaError_t e = pull ? emuCtasPerRank<moeCombinePullKernelEmu>(pullThreads, lc.emuRanks, &ctas) : emuMoeCtas(lc, true, &ctas);
    if (e != cudaSuccess) return e;
    if (pull)
      return launchEmu(moeCombinePullKernelEmu, lc, lc.emuMoe, dim3(std::min(ctas, pullCtas), lc.emuRanks), dim3(pullThreads), 0);
    return launchEmu(moeCombineKernelEmu, lc, lc.emuMoe, dim3(ctas, lc.emuRanks), dim3(kMoeThreads), 0);
  }
  if (pull) moeCombinePullKernel<<<pullCtas, pullThreads, 0, lc.stream>>>(*lc.comm, a);
  else moeCombineKernel<<<lc.nCtas, kMoeThreads, 0, lc.stream>>>(*lc.comm, a);
  return cudaGetLastError();
}

} // namespace fcx
