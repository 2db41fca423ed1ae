// Test harness: the launch-shape rules of gpu-impact-ct_b200/csrc/shape.h, compiled for the host.
// Built by tests/test_launch_shapes.py into a temporary directory; nothing in the product loads it.
#include "shape.h"

extern "C" int host_march_seg(long long threads, int na, int sms, int per_sm, int most) {
  return impact::march_seg(threads, na, sms, per_sm, most);
}
extern "C" int host_tri_depth(double gxy, int n3, double sms, int vec) { return impact::tri_depth(gxy, n3, sms, vec != 0); }
