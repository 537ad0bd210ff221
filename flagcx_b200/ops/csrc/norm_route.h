// norm_route.h -- which kernel of fused_elementwise.cu takes an RMSNorm backward.
#pragma once

namespace fcxops {

constexpr int kNormBwdThreads = 512;

// One CTA of 512 threads per row (rmsnormBwdPipelined, two CTAs per SM), or groups of threads
// that hold a row each (rmsnormBwdRing, one CTA per SM).  Groups win by having more rows in work;
// with few rows there are none to have, and the shorter chain of 512 threads decides (device us,
// groups against one row per CTA): 257 x 2048 7.9 -> 6.2, 64 x 4096 7.6 -> 5.7, 592 x 1024 7.8 ->
// 7.1, 800 x 3584 12.6 -> 11.9, 148 x 8192 8.3 -> 7.2.  The lines, in rows per SM, by packs of 8:
//   up to two packs per thread: 1 (every size: 1.01 to 1.62 times as fast; more than two: groups)
//   one pack per thread: 2 up to 64 packs, the CTAs that run at once (0.92 to 1.3), 4 up to 256,
//   whose groups of 32 or 64 threads walk three or four packs each (0.95 to 1.4), 3 beyond (1.0
//   to 1.4), but 6 where 512 threads are at least 7/8 full (0.93 to 1.5)
// With many rows and a third tensor added, rows that fill the threads need fewer registers and
// barriers pay: from 0.9 full always (4096 x 4096 33.6 against 35.4, 16384 x 4096 100.1 against
// 104.4), two packs at least 7/8 full from 16 rows per SM (8192 x 7168 88.1 against 95.6; 1021 x
// 7168 0.93).  Without the third tensor groups win (16384 x 4096 90.4 against 96.3) but for two
// packs and 40 rows per SM (8192 x 8192 87.4 against 90.3).
inline bool rmsnormRowPerCta(long rows, int H, bool add, int sms) {
  const int packs = H / 8, perThread = (packs + kNormBwdThreads - 1) / kNormBwdThreads;
  if (perThread > 2) return false;
  const bool full = packs * 8 >= 7 * perThread * kNormBwdThreads;
  if (rows <= sms) return true;
  if (perThread == 1 && rows <= (packs <= 64 ? 2L : packs <= 256 ? 4L : full ? 6L : 3L) * sms) return true;
  if (add && packs * 10 > 9 * perThread * kNormBwdThreads) return true;
  return perThread == 2 && full && rows >= (add ? 16L : 40L) * sms;
}

} // namespace fcxops
