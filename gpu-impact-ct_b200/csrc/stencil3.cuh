// stencil3.cuh -- the passes whose stencils run along all three axes, as z-marching passes
// (stencil3.cu; internal):
//
//   divergence2        D1 u + D2 v + D3 w                                  (mod_diff.f90:130-215)
//   interpolate_vel    the three velocities to the pressure points         (mod_diff.f90:1436-1472),
//                      optionally with get_dtime's bound of every block    (mod_lib.f90:46-250)
//   projection         vel_m = rhs_m - G_m pre, three components           (mod_solvers.f90:180-330)
//   Helmholtz_explicit nl -= multL (cx u_xx + cy u_yy + cz u_zz)           (mod_diff.f90:549-762)
//
// Every point sums its terms in table order with fused multiply-adds, x first, then y, then z.
#pragma once
#include "common.cuh"

namespace impact {

enum TriKind { TRI_DIV2 = 0, TRI_INTERP, TRI_PROJECT, TRI_HELM };

// per-axis row sums of get_dtime: sum_l |cpp(l,i)| and sum_l |cp1(l,i)|
struct DtRows {
  const double* spp[3];
  const double* sp1[3];
};

// One pass over one grid.  T: fields and arithmetic; TO: the results (float: the FP32
// interpolated velocities of a mixed-precision case).
template <typename T, typename TO>
struct TriArgs {
  const T* c[3];   // the tables of the three axes
  const T* f[3];   // DIV2, INTERP: the three velocities; PROJECT: f[0] = pre; HELM: f[0] = vel
  const T* s[3];   // PROJECT: rhs; HELM: s[0] = nl (may be o[0])
  TO* o[3];        // results
  T alpha;         // HELM: multL
  int ahead;       // prefetch planes into L2 (tri_ahead)
  // INTERP: when partial is given, the maximum of get_dtime's bound over every block
  DtRows dr;
  const double* Re;  // device (batches); null: ReV
  double ReV;
  double* partial;
};

// blocks of a pass: gx x gy x gz, kz planes each; vec: 16-byte vectors of points per thread
struct TriGrid {
  int vec, gx, gy, gz, kz;
  int blocks() const { return gx * gy * gz; }
};
// n1 divisible by the vector width and every field 16-byte aligned
bool tri_vectorable(const Geom& g, int elt, const void* const* fields, int n);
// the pass's fields exceed what the L2 keeps between its planes
bool tri_ahead(const Geom& g, int elt);
// depth by tri_depth (shape.h).  total_points: grids advanced by the same launch share the GPU (0: this
// grid alone)
TriGrid tri_grid(const Geom& g, int elt, bool vec, long long total_points = 0);

template <int KIND, typename T, typename TO>
void launch_tri(const Geom& g, const TriArgs<T, TO>& a, const TriGrid& tg, cudaStream_t s);

// one case of a batched pass (FP64 fields): block b of the launch is block b - b0 of its grid
struct TriJob {
  Geom g;
  TriGrid tg;
  TriArgs<double, double> a[3];   // by kind (DIV2, INTERP, PROJECT)
  TriArgs<double, float> a32;     // INTERP with FP32 results
  int b0;
};
// f32: TRI_INTERP writing the FP32 fields; dt: TRI_INTERP with get_dtime's bounds
void launch_tri_batch(int kind, int f32, int dt, const TriJob* jobs, int nj, int blocks, cudaStream_t s);

// the stability limits of get_dtime (41 rays), uploaded before the first pass that needs them
int tri_upload_limits(const double* lim41, cudaStream_t s);

}  // namespace impact
