// shape.h -- launch shapes of the streaming passes (march.cu, stencil3.cu) as functions of the grid
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

// Planes per block of a three-axis pass: gxy blocks side by side, n3 planes, `sms` SMs (a batch's
// grids each take their share of them).  The depth minimises rounds of blocks x (planes + a block's
// set-up).  Vectors of points: a round is the 2 blocks of 256 threads and 128 registers that an SM
// holds, the set-up about 3 planes' time.  Single points: 6 and 6, both fitted (2 or 3 blocks are
// resident, but the next ones' set-up hides behind them).  A last round that is not full takes half to
// all of a full one's time; beyond 3 rounds the blocks have drifted apart, only their number counts, and
// 32 planes are enough (256 x 256 x 512 FP64: Helmholtz 253 us at 32, 266 at 64).
// 192 x 192 x 192 FP64: Helmholtz 57 us at the 48 planes of one round (a count of 3 vector blocks per SM
// chose 8: 71), divergence2 54 (72); 128 x 128 x 128: 18.5 (22.8), 17.3 (21.4).
inline int tri_depth(double gxy, int n3, double sms, bool vec) {
  const int slots = vec ? 2 : 6, setup = vec ? 3 : 6;
  double best = -1.0;
  int depth = 64;
  for (int kz : {64, 48, 32, 24, 16, 12, 8, 4, 2, 1}) {
    const double per_sm = gxy * ((n3 + kz - 1) / kz) / sms;
    double rounds = per_sm / slots;
    if (rounds > 3.0 && kz > 32) continue;
    if (rounds <= 3.0) {
      const int m = (int)(per_sm + 0.999999), part = m % slots;
      rounds = m / slots + (part ? 0.5 + 0.5 * part / slots : 0.0);
    }
    const double cost = rounds * (std::min(kz, n3) + setup);
    if (best < 0.0 || cost < best) {
      best = cost;
      depth = kz;
    }
  }
  return depth;
}

}  // namespace impact
