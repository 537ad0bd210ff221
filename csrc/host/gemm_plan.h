// gemm_plan.h -- which kernel takes which part of a plain bf16 product (flagcxGemmBf16).
#pragma once
#include <algorithm>

#include "../kernels/split_gemm.h"

namespace fcx {

// Estimates for split_gemm.cu: fixed cost and cost of a K step (us) by tile width, and how many
// CTAs run at once by cluster size on the 148 SMs of this chip (33 clusters of 4, 14 of 8).
struct SplitGemmKind { int tileN; double fixedUs, stepUs; };
struct SplitGemmSize { int parts, ctas; };
constexpr SplitGemmKind kSplitKinds[] = {{256, 9.25, 0.3625}, {128, 7.25, 0.3125}, {64, 6.0, 0.30}};
constexpr SplitGemmSize kSplitSizes[] = {{8, 112}, {4, 132}, {2, 148}, {1, 148}};

// The persistent kernel (tileN = 0), or K split over clusters of `parts` CTAs that own 128 x
// tileN tiles.  The split pays while the persistent kernel's 128 x 256 tiles leave most SMs idle
// (operands not in L2, us: 128 x 3584 x 8192 54.6 -> 20.2, 256 x 3584 x 8192 45.2 -> 25.1, 128 x
// 256 x 8192 47.7 -> 12.4, 512 x 3584 x 8192 45.5 -> 36.8); from about 64 tiles on the
// persistent kernel's CTA pairs and overlapped epilogues win (1024 x 3584 x 8192: 53 against 68
// us).  Below that the smallest of the estimates decides, the persistent kernel's less 0.6 us
// (the fit's spread): a fixed cost plus the largest of one CTA's K steps, the operands out of
// HBM (6.4 TB/s) and what all CTAs together pull out of L2 (13 TB/s).  The figures are fitted to
// device times (calls captured in a graph) of 170 shapes from 128 x 256 x 256 to 8192 x 256 x
// 10240.  An earlier fit to back-to-back calls, which hid 13 us of host time, sent small K to
// the split where it lost: 1664 x 768 x 1024 11.1 -> 12.6, 2432 x 512 x 1152 12.0 -> 13.4, 128 x
// 9728 x 1280 14.1 -> 15.6.
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
  if (tiles256 > 64 || kb < 4) return best;
  const double hbmUs = ((double)M + N) * K * 2 / 6.4e6;
  double bestUs = (pair ? 6.83 + kb * 0.283 : 5.0 + kb * 0.363) - 0.6;
  for (auto &k : kSplitKinds) {
    const long tiles = tiles256 * (256 / k.tileN);
    for (auto &sp : kSplitSizes) {
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
// x 8192 is 6 waves of 74 CTA pairs and 4 tiles: 339 -> 328 us; 1408 x 5120 x 12352 213 -> 177,
// 6400 x 768 x 8896 142 -> 92.  A wave costs 0.363 us per K step, of pairs 0.33 (several waves:
// the clock is lower than in splitPlan's single one); the split kernel its estimate and 5.25 us
// for the second launch.  Measured on 283 shapes with both routes: at 0.38 us for pairs,
// too, 21 of the 162 that took a second launch lost 1 to 5 % (6400 x 4096 x 7040 269 -> 282, 768 x 8448 x 6336 80 -> 83), and
// with less for the launch 5504 x 3584 x 2880 did (123 -> 130).  The gain falls
// with the number of full waves (on average 17 % after one, 11 after two, 3 after six, 1 after
// eight); beyond nine it is within the noise (twelve shapes to 13 waves: 0.95 to 1.05).
inline SplitGemmTail tailPlan(int M, int N, int K, bool pair, int units, int groupRows, SplitGemmPlan *plan) {
  SplitGemmTail t;
  const int kb = K / 64, tiles = (M / (pair ? 256 : 128)) * (N / 256), rest = tiles % units;
  if (tiles <= units || tiles > 9 * units || rest == 0) return t;
  const int parts128 = rest * (pair ? 2 : 1);
  for (auto &sp : kSplitSizes) {
    if (sp.parts < 2 || parts128 * sp.parts > sp.ctas || sp.parts * 4 > kb) continue;
    const double steps = (kb + sp.parts - 1) / sp.parts * kSplitKinds[0].stepUs;
    const double bytes = (double)parts128 * kb * (128 + 256) * 128;
    if (kSplitKinds[0].fixedUs + std::max(steps, bytes / 13e6) + 5.25 > kb * (pair ? 0.33 : 0.363)) break;
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

} // namespace fcx
