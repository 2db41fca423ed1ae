// Test harness: the launch-shape rules of gpu-impact-ct_b200/csrc/shape.h, compiled for the host.
// Built by tests/test_launch_shapes.py into a temporary directory; nothing in the product loads it.
#include "shape.h"

extern "C" int host_march_seg(long long threads, int na, int sms, int per_sm, int most) {
  return impact::march_seg(threads, na, sms, per_sm, most);
}
extern "C" int host_tri_depth(double gxy, int n3, double sms, int vec) { return impact::tri_depth(gxy, n3, sms, vec != 0); }
// depths of a list of n cubes-like grids (n x n x 2n): units and stacked tiles
extern "C" void host_stack(const int* n, int count, int rows, int kc, int slots, int step, int* ks, int* depth) {
  std::vector<impact::TileGrid> g;
  for (int q = 0; q < count; ++q) {
    g.push_back({32, rows, n[q], n[q], 2 * n[q], true, 0, 0});
    g[q].ks = g[q].kc = impact::grid_depth(g[q], kc, slots);
  }
  impact::stack_units(g, kc, slots, step);
  for (int q = 0; q < count; ++q) {
    ks[q] = g[q].ks;
    depth[q] = g[q].kc;
  }
}
// held: clusters of 2, 4 and 8 blocks that the device holds; fitted: most blocks that the slabs of every case fit
extern "C" int host_tail_cluster(int ntails, const int* held, int fitted) {
  return impact::tail_cluster(ntails, 8, [&](int cb) { return cb <= fitted; },
                              [&](int cb) { return held[cb == 2 ? 0 : (cb == 4 ? 1 : 2)]; });
}
