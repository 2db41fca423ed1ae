// shape.h -- launch shapes of the streaming passes (march.cu, stencil3.cu) and of the Krylov kernels
// (engine.cu) as functions of the grids and of the device's SM count (host code, no CUDA: tests/test_launch_shapes.py runs it).
#pragma once
#include <algorithm>
#include <vector>

namespace impact {

constexpr int MAX_GRID_YZ = 65535;  // blocks of a launch along y or z

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
  while ((na - 1) / seg + 1 > MAX_GRID_YZ) seg *= 2;
  return seg;
}

// Planes per block of a three-axis pass: gxy blocks side by side, n3 planes, `sms` SMs (a batch's
// grids each take their share of them).  The depth minimises waves of blocks x (planes + a block's
// set-up).  Vectors of points: a wave is the 2 blocks of 256 threads and 128 registers that an SM
// holds, the set-up about 3 planes' time.  Single points: 6 and 6, both fitted (2 or 3 blocks are
// resident, but the next ones' set-up hides behind them).  A last wave that is not full takes half to
// all of a full one's time; beyond 3 waves the blocks have drifted apart, only their number counts, and
// 32 planes are enough (256 x 256 x 512 FP64: Helmholtz 253 us at 32, 266 at 64).
// 192 x 192 x 192 FP64: Helmholtz 57 us at the 48 planes of one wave (a count of 3 vector blocks per SM
// chose 8: 71), divergence2 54 (72); 128 x 128 x 128: 18.5 (22.8), 17.3 (21.4).
inline int tri_depth(double gxy, int n3, double sms, bool vec) {
  const int slots = vec ? 2 : 6, setup = vec ? 3 : 6;
  double best = -1.0;
  int depth = 64;
  for (int kz : {64, 48, 32, 24, 16, 12, 8, 4, 2, 1}) {
    const double per_sm = gxy * ((n3 + kz - 1) / kz) / sms;
    double waves = per_sm / slots;
    if (waves > 3.0 && kz > 32) continue;
    if (waves <= 3.0) {
      const int m = (int)(per_sm + 0.999999), part = m % slots;
      waves = m / slots + (part ? 0.5 + 0.5 * part / slots : 0.0);
    }
    const double cost = waves * (std::min(kz, n3) + setup);
    if (best < 0.0 || cost < best) {
      best = cost;
      depth = kz;
    }
  }
  while ((n3 - 1) / depth + 1 > MAX_GRID_YZ) depth *= 2;
  return depth;
}

// A grid cut into tiles of tx x rows columns and kc planes for a Krylov kernel.  ks: the planes of one unit of
// summation (one partial sum each); stack: a tile may hold several units.
struct TileGrid {
  int tx, rows, n1, n2, n3;
  bool stack;
  int ks, kc;
};
inline long long tiles_at(const TileGrid& g, int kc) {
  return (long long)((g.n1 + g.tx - 1) / g.tx) * ((g.n2 + g.rows - 1) / g.rows) * ((g.n3 + kc - 1) / kc);
}

// Tile depth, at most kc (the solver parameter tile_kc or its default), for `tiles(depth)` tiles over
// grids of up to n3 planes.  A tile is a serial chain of planes after a prologue of about 8 planes' time
// (the job's scalars; in the operator the z window and the first staged group), so the depth minimises
// waves of tiles over the kernel's `slots` resident blocks x (depth + 8), among kc, the multiples of 8
// below it (the vector updates walk blocks of 8 planes) and 4, or as far down as `least`.
template <typename Tiles>
inline int depth_for(Tiles&& tiles, int n3, int kc, int slots, int least = 4) {
  int best = kc;
  long long cost = -1;
  auto consider = [&](int d) {
    const long long c = (tiles(d) + slots - 1) / slots * (std::min(d, n3) + 8);
    if (cost < 0 || c < cost) {
      cost = c;
      best = d;
    }
  };
  consider(kc);
  for (int d = (kc - 1) / 8 * 8; d >= 8; d -= 8) consider(d);
  for (int d = 4; d >= least; d /= 2)
    if (kc > d) consider(d);
  return best;
}

// The depth of one grid, from the grid alone: the unit of its partial sums, so that a case's sums do not
// depend on its batch.  Grids of many waves keep kc; on 32 x 32 x 64 the 4 tiles of 64 planes become 64 of 4
// (FP32 operator 26.6 -> 6.2 us, x update 14.4 -> 4.3 us); kernels of two rows per thread (tiles of more than
// 8 rows) step by 2 planes and may take as few.
inline int grid_depth(const TileGrid& g, int kc, int slots) {
  return depth_for([&](int d) { return tiles_at(g, d); }, g.n3, kc, slots, g.rows > 8 ? 2 : 4);
}

// the depth of a list without partial sums: the same rule over all its grids together (the small
// grids of a batch need no shallow tiles of their own to fill the GPU)
inline int list_depth(const std::vector<TileGrid>& gs, int kc, int slots) {
  int n3 = 0;
  for (const TileGrid& g : gs) n3 = std::max(n3, g.n3);
  auto tiles = [&](int d) {
    long long t = 0;
    for (const TileGrid& g : gs) t += tiles_at(g, d);
    return t;
  };
  return depth_for(tiles, n3, kc, slots);
}

// Tile depths of an operator list of several grids whose units ks are chosen.  A grid whose tiles of ks planes
// would fill the GPU alone shares it here, where each tile's prologue is paid for nothing: a tile holds
// as many whole units as the list's common depth allows, and its kernel sums each unit by itself.  The
// depth minimises the planes and prologues of the most loaded of `slots` blocks, which take the list's tiles
// in turn, + those of the average one (a block that is done leaves its SM to another).  step: the
// planes per step of the kernel, of which a unit must be a multiple.  48 cases of 32 to 152 cells a
// side: FP64 operator 32.0 ms a step with tiles of one unit, 29.4 with several (29.2 with 64 planes in every
// tile and unit), FP32 operator 14.4 and 13.4.  Lists of fewer than 3 waves of one-unit tiles keep those: the
// prologues hide behind the other blocks' planes, and fewer tiles leave SMs idle (FP64 cases of 72 and 64
// cells a side, step 9.22 ms; with tiles of 32 planes 9.54).
inline void stack_units(std::vector<TileGrid>& gs, int kc, int slots, int step) {
  auto depth = [&](const TileGrid& g, int d) { return g.stack && g.ks % step == 0 ? g.ks * std::max(1, d / g.ks) : g.ks; };
  int best = 1;
  double least = -1.0;
  std::vector<long long> change(slots + 1);
  auto consider = [&](int d) {
    std::fill(change.begin(), change.end(), 0);  // of the load from one block to the next
    long long first = 0, work = 0;
    for (const TileGrid& g : gs) {
      const int e = depth(g, d), len = std::min(e, g.n3) + 8;
      const long long tiles = tiles_at(g, e), part = tiles % slots, at = first % slots;
      change[0] += tiles / slots * len;
      change[at] += len;
      change[(at + part) % slots] -= len;  // (at slots: past the last block, undone by the next line)
      if (at + part >= slots) change[0] += len;
      first += tiles;
      work += tiles * len;
    }
    long long load = 0, longest = 0;
    for (int b = 0; b < slots; ++b) longest = std::max(longest, load += change[b]);
    const double cost = (double)longest + (double)work / slots;
    if (least < 0.0 || cost < least) {
      least = cost;
      best = d;
    }
  };
  long long alone = 0;
  for (const TileGrid& g : gs) alone += tiles_at(g, g.ks);
  if (gs.size() > 1 && alone >= 3LL * slots) {
    consider(kc);
    for (int d = (kc - 1) / 8 * 8; d >= 8; d -= 8) consider(d);
    for (int d : {4, 1})
      if (kc > d) consider(d);
  }
  for (TileGrid& g : gs) g.kc = depth(g, best);
}

// Blocks per coarse tail of a list of `ntails`: the largest power of two up to `most` whose cut into slabs fits
// (fits(blocks)) and of which the device can hold a cluster for every tail at once (held(blocks): clusters;
// 15 of 8, 33 of 4 and 74 of 2 on a whole B200, whose SMs stand in groups; a part of one may hold none);
// else one.
template <typename Fits, typename Held>
inline int tail_cluster(int ntails, int most, Fits&& fits, Held&& held) {
  for (int cb = most; cb > 1; cb /= 2)
    if (fits(cb) && held(cb) >= ntails) return cb;
  return 1;
}

}  // namespace impact
