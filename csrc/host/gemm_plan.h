// gemm_plan.h -- which kernel takes which part of a plain bf16 product (flagcxGemmBf16).
#pragma once
#include <algorithm>

#include "../kernels/split_gemm.h"

namespace fcx {

// Estimates for split_gemm.cu by tile width: fixed cost, cost of exchanging a whole tile of fp32
// parts between CTAs and cost of a K step (us), and what all CTAs together pull out of L2 (TB/s);
// and how many CTAs run at once by cluster size on the 148 SMs of this chip (33 clusters of 4, 14 of 8).
struct SplitGemmKind { int tileN; double fixedUs, exchangeUs, stepUs, l2TBs; };
struct SplitGemmSize { int parts, ctas; };
constexpr SplitGemmKind kSplitKinds[] = {{256, 5.0, 4.0, 0.35, 14}, {128, 4.1, 2.0, 0.30, 15}, {64, 3.6, 1.25, 0.2875, 10}};
constexpr SplitGemmSize kSplitSizes[] = {{8, 112}, {4, 132}, {2, 148}, {1, 148}};

// K split over `parts` CTAs for `tiles` tiles of that kind: a fixed cost, the exchange, and the
// largest of one CTA's K steps, the operands out of HBM (hbmUs) and all CTAs' operands out of L2.
inline double splitUs(const SplitGemmKind &k, int parts, long tiles, int kb, double hbmUs) {
  const double steps = (kb + parts - 1) / parts * k.stepUs, bytes = (double)tiles * kb * (128 + k.tileN) * 128;
  return k.fixedUs + k.exchangeUs * (parts - 1) / parts + std::max({steps, hbmUs, bytes / (k.l2TBs * 1e6)});
}

// The persistent kernel (tileN = 0), or K split over clusters of `parts` CTAs that own 128 x
// tileN tiles.  The split pays while the persistent kernel's 128 x 256 tiles leave half of the SMs
// idle (operands not in L2, us: 128 x 3584 x 8192 52 -> 16.4, 128 x 256 x 8192 51 -> 9.1, 1664 x
// 1280 x 4544 29.2 -> 20.2, which is 65 tiles); with more tiles there is no room for two CTAs each.
// Up to there the smallest of the estimates decides, the persistent kernel's less 0.6 us (the fit's
// spread).  The figures are fitted to device times (calls captured in a graph) of 179 shapes from
// 128 x 256 x 256 to 2048 x 6144 x 8192, every kind and size that the shape allows: the smallest
// estimate takes 1.002 of the quickest on average, 1.08 at worst (256 x 2816 x 3072).  Beyond 32
// tiles the persistent kernel keeps what it had when a split cost 2 us more: two parts or more, and
// 1.7 us to be gained (given away: 3456 x 512 x 1472 12.0 against 12.6, 2432 x 512 x 1152 10.5 against
// 10.9, 1664 x 768 x 1024 10.1 against 10.3; with the pairs that this takes now the persistent kernel has
// caught up at 128 x 9728 x 1280, 12.8 against 12.7).
// pair: that the number of 128-row blocks is even.  The persistent kernel may yet take pairs for an odd
// one (pairsQuicker); its estimate here stays that of single CTAs, with which the split was right on
// all of 30 shapes where the estimate for pairs would have left it (3 to 22 % quicker: 1152 x 2048 x 2816
// 16.1 against 19.7, 128 x 13312 x 11328 58.4 against 65.6).
// Clusters stay within what is co-resident: a second wave costs more than the split gains (28
// clusters of 5: 37 us against 27).
// forced: 1 = never split, 2 to 8 = split over so many CTAs with tiles of forcedTileN.
inline SplitGemmPlan splitPlan(int M, int N, int K, bool pair, int forced = 0, int forcedTileN = 256) {
  SplitGemmPlan best;
  const int kb = K / 64;
  if (forced == 1) return best;
  if (forced > 1 && forced <= kSplitGemmMaxParts && forced <= kb) {
    best.parts = forced;
    best.tileN = forcedTileN;
    return best;
  }
  const long tiles256 = (long)(M / 128) * (N / 256);
  if (tiles256 > 74 || kb < 4) return best;
  const double hbmUs = ((double)M + N) * K * 2 / 5.5e6;
  const bool few = tiles256 <= 32;
  double bestUs = (pair ? 5.6 + kb * 0.2915 : 4.7 + kb * 0.359) - (few ? 0.6 : 1.7);
  for (auto &k : kSplitKinds) {
    const long tiles = tiles256 * (256 / k.tileN);
    for (auto &sp : kSplitSizes) {
      if (tiles * sp.parts > sp.ctas || sp.parts * 4 > kb || (sp.parts == 1 && !few)) continue;
      const double us = splitUs(k, sp.parts, tiles, kb, hbmUs);
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
// CTAs per tile) is quicker than a wave of whole tiles in which most SMs are idle: 8192 x 3584
// x 8192 is 6 waves of 74 CTA pairs and 4 tiles, 327 -> 314 us in short runs (under the power limit of a
// long one 370 to 380, and the difference within what the clock moves).  A wave costs 0.363 us per K step, of
// pairs 0.33 (several waves: the clock is lower than in splitPlan's single one); the split kernel
// the larger of its K steps and its operands out of L2, and 14.5 us for the exchange and the second
// launch.  Measured on 90 shapes, none lost (6400 x 768 x 8896 90 -> 68, 1792 x 3072 x 7424 75 -> 63).
// Since the second launch starts while the first kernel ends it costs less: with 10.5 us 1024 x 4864 x
// 3072 would take 32.7 instead of 35.2 us, 768 x 8448 x 6336 65.3 instead of 67.5, 6400 x 4096 x 7040 246
// instead of 249, 5504 x 3584 x 2880 the same.  The gain falls with the number of full waves (on average
// 17 % after one, 11 after two, 3 after six, 1 after eight); beyond nine it is within the noise.
inline SplitGemmTail tailPlan(int M, int N, int K, bool pair, int units, int groupRows, SplitGemmPlan *plan) {
  SplitGemmTail t;
  const int kb = K / 64, tiles = (M / (pair ? 256 : 128)) * (N / 256), rest = tiles % units;
  if (tiles <= units || tiles > 9 * units || rest == 0) return t;
  const int parts128 = rest * (pair ? 2 : 1);
  for (auto &sp : kSplitSizes) {
    if (sp.parts < 2 || parts128 * sp.parts > sp.ctas || sp.parts * 4 > kb) continue;
    const double steps = (kb + sp.parts - 1) / sp.parts * 0.3625, bytes = (double)parts128 * kb * (128 + 256) * 128;
    if (std::max(steps, bytes / 13e6) + 14.5 > kb * (pair ? 0.33 : 0.363)) break;
    plan->tileN = 256;
    plan->parts = sp.parts;
    t.first = tiles - rest;
    t.count = rest;
    t.tileRows = pair ? 256 : 128;
    t.groupRows = groupRows;
    break;
  }
  return t;
}

// Whether the persistent kernel takes CTA pairs.  A K step of pairs is quicker (single CTAs load every
// tile of B once for 128 rows, not 256); the end of a wave of pairs costs more, where two CTAs wait for
// each other; and with an odd number of 128-row blocks the pairs' last row of tiles is half empty.  So
// single CTAs are the quicker side up to seven K steps, and about where pairs need a wave more.  In a
// single wave they are up to eleven, where 75 tiles or more occupy half of the SMs with either kind
// (2560 x 1792 x 576 9.3 against 9.7 us, 512 x 9472 x 896 12.6 against 12.1), and up to eight with
// fewer tiles (384 x 4096 x 512 8.3 against 8.4, 256 x 3584 x 832 10.0 against 9.5; a lone block of 128
// rows gains from the second CTA that fetches half of B: 128 x 14848 x 7296 56.0 against 47.3).
// Several waves were set by 550 shapes of 256 to 6272 rows and tried on 240 others against pairs for
// even numbers of blocks and single CTAs for odd ones: 1.8 % less time over the even ones (5888 x 4608
// x 256 24.6 -> 21.0 us, 5888 x 5888 x 384 33.9 -> 30.2), 4.3 % over the odd (1152 x 4608 x 2304
// 32.8 -> 28.6, 640 x 4608 x 7104 45.9 -> 40.6), none slower by more than the 0.3 us that two
// runs of one route differ by; 2.0 and 4.6 % if the better side were always known.  5504 x 4352 x 896
// stays with single CTAs, 37.4 against 35.8.  A single wave by 244 shapes: at worst 0.2 us are given
// away, for odd and even numbers of blocks alike.
inline bool pairsQuicker(int M, int N, int K, int sms, int groupPair, int groupSingle, bool noTail) {
  const int kb = K / 64;
  auto us = [&](bool pair) {
    const int rows = pair ? (M + 255) / 256 * 256 : M, units = pair ? sms / 2 : sms;
    const int tiles = rows / (pair ? 256 : 128) * (N / 256), waves = (tiles + units - 1) / units;
    const double wave = pair ? kb * 0.30 + 0.45 : kb * 0.363, only = M / 128 * (N / 256) > sms / 2 ? 0.27 : 0.085;
    SplitGemmPlan plan;
    if (noTail || !tailPlan(rows, N, K, pair, units, pair ? groupPair : groupSingle, &plan).count)
      return waves * wave + (pair && waves == 1 ? only : 0);
    return (waves - 1) * wave + 10.5 + (kb + plan.parts - 1) / plan.parts * 0.3625;
  };
  return us(true) < us(false);
}

} // namespace fcx
