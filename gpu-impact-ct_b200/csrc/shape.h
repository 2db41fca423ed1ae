// shape.h -- launch shapes of the streaming passes (march.cu) as functions of the grid
// and of the device's SM count (host code, no CUDA: tests/test_launch_shapes.py runs it).
#pragma once
#include <algorithm>

namespace impact {

// Steps of a thread that marches along an axis of na steps, `threads` threads side by side: the
// largest power of two up to `most` that leaves `per_sm` threads per SM.  A longer segment re-reads
// fewer of the CNT - 1 values before it and pays its set-up once; a thread too few costs a small grid
// more than that (56 x 56 x 56 FP64 upwind term along x 7.4 us at 4 to 8 steps and 49 blocks, 6.2 at one; JOR
// sweep on 48 x 48 x 48 5.2 and 4.2).  320 threads and 8 steps (along y and z, JOR sweep), 256 and
// 16 (along x, whose set-up loads coefficient rows) lie within 1 to 4 % of each pass's best of 1 to 32
// steps and 64 to 256 threads a block, on average over 24^3 to 256^3.
inline int march_seg(long long threads, int na, int sms, int per_sm, int most) {
  int seg = 1;
  while (2 * seg <= most && 2 * seg <= na && threads * na >= (long long)sms * per_sm * 2 * seg) seg *= 2;
  return seg;
}

}  // namespace impact
