// norm_route.h -- which kernel of fused_elementwise.cu takes an RMSNorm backward.
#pragma once

namespace fcxops {

constexpr int kNormBwdThreads = 512;
constexpr int kNormFewRows = 2; // rows of a CTA of rmsnormBwdFewRows, of which an SM holds two

// True: one CTA of 512 threads per row (rmsnormBwdFewRows, two CTAs per SM and at most two rows
// each).  False: groups of threads that hold a row each (rmsnormBwdRing, one CTA per SM).  Groups
// win by having more rows in work; with few rows there are none to have, and the shorter chain of
// 512 threads decides (device us, groups against one row per CTA): 257 x 2048 7.6 -> 6.1, 64 x 4096
// 7.3 -> 5.7, 592 x 1024 7.6 -> 7.1, 148 x 8192 8.3 -> 7.6.  The lines, in rows per SM, with the
// ratios measured below and above them (above 1: one row per CTA is quicker):
//   1 up to 32 packs of 8 (0.93 to 1.12; 0.84 to 1.0) and for two packs per thread, 4104 to 8192
//     columns (0.94 to 1.23; 0.69 to 0.87)
//   2 else (0.93 to 1.36; 0.67 to 1.0)
//   3 from 448 packs on, where the 512 threads are 7/8 full (0.94 to 1.44; 0.79 to 1.04, most at 800 x 3584)
//   4 where a group of 32 or 64 threads walks four packs per thread (1.02 to 1.62; 0.38 to 0.97)
// Rows of more than two packs per thread are quicker in groups of 512 threads (0.67 to 0.98).
inline bool rmsnormRowPerCta(long rows, int H, int sms) {
  const int packs = H / 8;
  if (packs > 2 * kNormBwdThreads) return false;
  const bool four = (packs > 96 && packs <= 128) || (packs > 192 && packs <= 256);
  return rows <= (packs <= 32 || packs > kNormBwdThreads ? 1L : four ? 4L : packs >= 448 ? 3L : 2L) * sms; // 2 x kNormFewRows at most
}

} // namespace fcxops
