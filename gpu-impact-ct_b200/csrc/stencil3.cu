// stencil3.cu -- the three-axis passes of the time step and of the launcher FFI (stencil3.cuh).
//
// A block owns LX x LY vectors of V points (V = 16 bytes, rows holding whole vectors; V = 1 on the
// other grids) and walks them along z over kz planes.  A thread keeps the x and y coefficients of
// its points and the z window of its column in registers for the whole march; x and y neighbours
// are vectors of the row and of the rows around it, which the block's other threads read too (L1).
// On grids whose fields exceed the L2 the planes PD ahead are prefetched into it, so that a step
// waits for L2 and not for DRAM (256 x 256 x 512 FP64: Helmholtz 325 -> 250 us, divergence2 340 ->
// 256 us; where the fields stay in L2 the prefetches only cost issue slots).  No barrier ties the
// warps of a block together.
//
// The passes these replace gave every thread one point: 18 scalar loads per point and, for the
// x stencil, one strided table load per tap, which cost more of the L1 data path than the fields
// themselves.  Now bound by that path still (65 % of its cycles; 12 vector loads per 2 points) and by
// the latency of 16 warps per SM.  256 x 256 x 512 FP64: Helmholtz 253 us (294), divergence2 263 us
// (390); 128 x 128 x 224 FP32: 16.5 us (19), 16 us (40); 187 x 131 x 157 FP32: 31 us (51), 27 us (43).
// 384 x 384 x 768 FP64, in the time step: interpolate_vel 1.09 ms (1.44; with get_dtime's bound
// in the same pass, which took another 1.94), divergence2 0.82 ms (1.33), projection 1.35 (1.44).
// The same with the tiles staged in shared memory by cp.async, four planes in a ring: 255 and
// 262 us, and slower on small grids.
#include <algorithm>

#include "kernels.cuh"
#include "shape.h"
#include "stencil3.cuh"

namespace impact {
namespace {

__constant__ double c_lim[41];

template <typename T, int V>
struct TriCfg {
  static constexpr int LX = V == 1 ? 32 : 16, LY = 256 / LX, NT = LX * LY;
  static constexpr int NX = LX * V;
};
// stencil ranges and operands of a kind
template <int KIND>
struct TriKindCfg {
  static constexpr int CNT = KIND == TRI_HELM ? NB : ND;
  static constexpr int LO = KIND == TRI_HELM ? B_LO : (KIND == TRI_PROJECT ? G_LO : D_LO);
  static constexpr int HI = LO + CNT - 1;
  static constexpr bool XY = KIND == TRI_PROJECT || KIND == TRI_HELM;  // one field with both halos
  static constexpr int NS = KIND == TRI_PROJECT ? 3 : (KIND == TRI_HELM ? 1 : 0);  // streamed operands
};
constexpr int PD = 4;  // planes prefetched ahead
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

template <typename T, int V>
__device__ __forceinline__ void ldv(const T* p, T (&o)[V]) {
  if constexpr (V == 1) {
    o[0] = __ldg(p);
  } else if constexpr (V == 2) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    o[0] = v.x;
    o[1] = v.y;
  } else {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
}
template <typename T, int V>
__device__ __forceinline__ void ldv_plain(const T* p, T (&o)[V]) {  // a field the pass writes
  if constexpr (V == 1) {
    o[0] = p[0];
  } else if constexpr (V == 2) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    o[0] = v.x;
    o[1] = v.y;
  } else {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
}
template <typename TO, typename T, int V>
__device__ __forceinline__ void stv(TO* p, const T (&o)[V]) {
  if constexpr (V == 1) {
    p[0] = (TO)o[0];
  } else if constexpr (V == 2 && sizeof(TO) == 8) {
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  } else if constexpr (V == 2) {
    *reinterpret_cast<float2*>(p) = make_float2((float)o[0], (float)o[1]);
  } else {
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  }
}
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }

// The first two terms of a sum.  The Helmholtz term rounds the first product and adds the second
// by fused multiply-add, as the one-axis passes do; the others round the second product, as the
// passes of the time step always have (a velocity's last bit decides which way the mixed solve's
// FP32 image of the residual rounds).
template <int KIND, typename T>
__device__ __forceinline__ T head(T c0, T f0, T c1, T f1) {
  return KIND == TRI_HELM ? fma_(c1, f1, mul_(c0, f0)) : fma_(c0, f0, mul_(c1, f1));
}

// get_dtime's bound radius / limit(angle) of one point, raised into `best`.  The limit of a ray is
// at least the smallest of the table, so a point whose radius cannot beat `best` even there is
// left out before the square root, the arc tangent and the divisions (the margin covers their
// rounding): the maximum is the same.
__device__ __forceinline__ void dt_bound(double spp, double s0, double s1, double s2, double Re, double w1, double w2,
                                         double w3, double lmin, double& best) {
  const double are = spp / Re;
  double aim = s0 * fabs(w1);
  aim = aim + s1 * fabs(w2);
  aim = aim + s2 * fabs(w3);
  const double r2 = are * are + aim * aim;
  const double top = best * lmin;
  if (r2 <= top * top * (1.0 - 1e-9)) return;
  const double pi = 3.14159265358979323846;
  const double angle = (fabs(aim) < 1e-16) ? pi / 2.0 : atan(are / aim);
  const double radius = sqrt(r2);
  long long idx = llround(2.0 * 40.0 * angle / pi);
  idx = idx < 0 ? 0 : (idx > 40 ? 40 : idx);
  best = fmax(best, radius / c_lim[idx]);
}

template <int KIND, typename T, typename TO, int V, bool DT>
__device__ __forceinline__ void tri_block(const Geom& g, const TriArgs<T, TO>& A, int kz, int bx, int by, int bz,
                                          int blk) {
  using C = TriCfg<T, V>;
  using K = TriKindCfg<KIND>;
  constexpr int CNT = K::CNT, LO = K::LO, HI = K::HI, NT = C::NT;
  const int tid = threadIdx.x, tx = tid % C::LX, ty = tid / C::LX;
  const int k0 = bz * kz + 1, k1 = min(g.n3, k0 + kz - 1), nk = k1 - k0 + 1;
  const int i = bx * C::NX + V * tx + 1, j = by * C::LY + ty + 1;
  const bool act = i <= g.n1 && j <= g.n2;  // V > 1: n1 % V == 0, the V points are valid together
  if (!DT && !act) return;
  const int ic = act ? i : 1, jc = act ? j : 1;
  const int own = (ic + 3) + g.nx * (jc + 3);
  const T* const fx = A.f[0];                   // the fields of the x, y and z stencils
  const T* const fy = K::XY ? A.f[0] : A.f[1];
  const T* const fz = K::XY ? A.f[0] : A.f[2];
  auto zoff = [&](int k) -> long long {         // plane k, at most one period outside 1..n3
    return (long long)((k < 1 ? k + g.n3 : (k > g.n3 ? k - g.n3 : k)) + 3) * g.nxy;
  };
  // coefficients of the thread's points and the z window's first CNT - 1 planes
  T cx[V][CNT], cy[CNT], win[CNT][V];
#pragma unroll
  for (int l = 0; l < CNT; ++l) {
#pragma unroll
    for (int v = 0; v < V; ++v) cx[v][l] = __ldg(A.c[0] + (size_t)(ic + v) * CNT + l);
    cy[l] = __ldg(A.c[1] + (size_t)jc * CNT + l);
  }
#pragma unroll
  for (int v = 0; v < V; ++v) win[0][v] = T(0);
#pragma unroll
  for (int l = 1; l < CNT; ++l) ldv<T, V>(fz + zoff(k0 - 1 + LO + l) + own, win[l]);
  double beta = 0.0, lmin = 0.0, dRe = 1.0, sx[V], s1x[V], sy = 0.0, s1y = 0.0;
  if constexpr (DT) {
    lmin = c_lim[0];
    for (int q = 1; q < 41; ++q) lmin = fmin(lmin, c_lim[q]);
    dRe = A.Re ? *A.Re : A.ReV;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      sx[v] = A.dr.spp[0][ic + v];
      s1x[v] = A.dr.sp1[0][ic + v];
    }
    sy = A.dr.spp[1][jc];
    s1y = A.dr.sp1[1][jc];
  }
  constexpr int FV = (LO - (V - 1)) / V, LV = (V - 1 + HI) / V, NV = LV - FV + 1;  // vectors of the x stencils
  int ox[NV], oy[CNT];  // in-plane offsets of the row's vectors and of the rows (periodic images)
  const int nvx = g.n1 / V, vx = (ic - 1) / V;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int u = vx + FV + n;
    ox[n] = 4 + V * (u < 0 ? u + nvx : (u >= nvx ? u - nvx : u)) + g.nx * (jc + 3);
  }
#pragma unroll
  for (int l = 0; l < CNT; ++l) {
    const int jj = jc + LO + l;
    oy[l] = (ic + 3) + g.nx * ((jj < 1 ? jj + g.n2 : (jj > g.n2 ? jj - g.n2 : jj)) + 3);
  }
  long long p = (long long)(k0 + 3) * g.nxy + own;
  const int nka = act ? nk : 0;
  for (int t = 0; t < nka; ++t, p += g.nxy) {
    const long long pz = (long long)(k0 + t + 3) * g.nxy;
    if (A.ahead && t + PD < nk) {
      const long long q = p + PD * g.nxy;
      if (!K::XY) prefetch_l2(fx + q);
      if (!K::XY) prefetch_l2(fy + q);
      prefetch_l2(fz + zoff(k0 + t + HI + PD) + own);
#pragma unroll
      for (int n = 0; n < K::NS; ++n) prefetch_l2(A.s[n] + q);
    }
#pragma unroll
    for (int l = 0; l + 1 < CNT; ++l)
#pragma unroll
      for (int v = 0; v < V; ++v) win[l][v] = win[l + 1][v];
    ldv<T, V>(fz + zoff(k0 + t + HI) + own, win[CNT - 1]);
    T cz[CNT];
#pragma unroll
    for (int l = 0; l < CNT; ++l) cz[l] = __ldg(A.c[2] + (size_t)(k0 + t) * CNT + l);
    // x neighbours: the aligned vectors of the thread's row
    T xv[NV * V], yv[CNT][V];
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      T tmp[V];
      if (K::XY && n == -FV) {
#pragma unroll
        for (int v = 0; v < V; ++v) tmp[v] = win[-LO][v];
      } else {
        ldv<T, V>(fx + pz + ox[n], tmp);
      }
#pragma unroll
      for (int v = 0; v < V; ++v) xv[n * V + v] = tmp[v];
    }
#pragma unroll
    for (int l = 0; l < CNT; ++l) {
      if (K::XY && l == -LO) {
#pragma unroll
        for (int v = 0; v < V; ++v) yv[l][v] = win[-LO][v];
      } else {
        ldv<T, V>(fy + pz + oy[l], yv[l]);
      }
    }
    T old[V];
    if constexpr (KIND == TRI_HELM) ldv_plain<T, V>(A.s[0] + p, old);
    T X[V], Y[V], Z[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      X[v] = head<KIND>(cx[v][0], xv[v + LO - FV * V], cx[v][1], xv[v + LO + 1 - FV * V]);
#pragma unroll
      for (int l = 2; l < CNT; ++l) X[v] = fma_(cx[v][l], xv[v + LO + l - FV * V], X[v]);
    }
    constexpr bool CHAIN = KIND == TRI_DIV2 || KIND == TRI_HELM;  // one sum over the axes
#pragma unroll
    for (int l = 0; l < CNT; ++l)
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (CHAIN)
          X[v] = fma_(cy[l], yv[l][v], X[v]);
        else if (l > 0)
          Y[v] = l == 1 ? head<KIND>(cy[0], yv[0][v], cy[1], yv[1][v]) : fma_(cy[l], yv[l][v], Y[v]);
      }
#pragma unroll
    for (int l = 0; l < CNT; ++l)
#pragma unroll
      for (int v = 0; v < V; ++v) {
        if (CHAIN)
          X[v] = fma_(cz[l], win[l][v], X[v]);
        else if (l > 0)
          Z[v] = l == 1 ? head<KIND>(cz[0], win[0][v], cz[1], win[1][v]) : fma_(cz[l], win[l][v], Z[v]);
      }
    if constexpr (KIND == TRI_DIV2) {
      stv<TO, T, V>(A.o[0] + p, X);
    } else if constexpr (KIND == TRI_HELM) {
#pragma unroll
      for (int v = 0; v < V; ++v) X[v] = fma_(-A.alpha, X[v], old[v]);
      stv<TO, T, V>(A.o[0] + p, X);
    } else if constexpr (KIND == TRI_INTERP) {
      stv<TO, T, V>(A.o[0] + p, X);
      stv<TO, T, V>(A.o[1] + p, Y);
      stv<TO, T, V>(A.o[2] + p, Z);
      if constexpr (DT) {
        const double sz = A.dr.spp[2][k0 + t], s1z = A.dr.sp1[2][k0 + t];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          double are = sx[v] + sy;
          are = are + sz;
          dt_bound(are, s1x[v], s1y, s1z, dRe, X[v], Y[v], Z[v], lmin, beta);
        }
      }
    } else {
      T r[V];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        ldv<T, V>(A.s[q] + p, r);
#pragma unroll
        for (int v = 0; v < V; ++v) r[v] = r[v] - (q == 0 ? X[v] : (q == 1 ? Y[v] : Z[v]));
        stv<TO, T, V>(A.o[q] + p, r);
      }
    }
  }
  if constexpr (DT) {
    __shared__ double sh[NT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) beta = fmax(beta, __shfl_xor_sync(0xffffffffu, beta, o));
    if ((tid & 31) == 0) sh[tid >> 5] = beta;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < NT / 32; ++w) beta = fmax(beta, sh[w]);
      A.partial[blk] = beta;
    }
  }
}

template <int KIND, typename T, typename TO, int V, bool DT>
__global__ void __launch_bounds__(256, V == 1 && sizeof(T) == 4 ? 3 : 2) k_tri(Geom g, TriArgs<T, TO> A, int kz) {
  const int blk = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  tri_block<KIND, T, TO, V, DT>(g, A, kz, blockIdx.x, blockIdx.y, blockIdx.z, blk);
}

// the pass over the cases of a batch (FP64 fields; a case with odd rows takes the scalar form)
template <int KIND, typename TO, bool DT>
__global__ void __launch_bounds__(256, 2) k_tri_batch(const TriJob* __restrict__ jobs, int nj) {
  int lo = 0, hi = nj - 1;
  const int b = blockIdx.x;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].b0 <= b) lo = mid; else hi = mid - 1;
  }
  const TriJob& J = jobs[lo];
  const int lb = b - J.b0;
  const int bx = lb % J.tg.gx, by = (lb / J.tg.gx) % J.tg.gy, bz = lb / (J.tg.gx * J.tg.gy);
  const Geom g = J.g;
  auto args = [&]() {
    if constexpr (sizeof(TO) == 4)
      return J.a32;
    else
      return J.a[KIND];
  };
  const TriArgs<double, TO> A = args();
  if (J.tg.vec)
    tri_block<KIND, double, TO, 2, DT>(g, A, J.tg.kz, bx, by, bz, lb);
  else
    tri_block<KIND, double, TO, 1, DT>(g, A, J.tg.kz, bx, by, bz, lb);
}

template <int KIND, typename T, typename TO, int V, bool DT>
void launch_tri_v(const Geom& g, const TriArgs<T, TO>& a, const TriGrid& tg, cudaStream_t s) {
  k_tri<KIND, T, TO, V, DT><<<dim3(tg.gx, tg.gy, tg.gz), 256, 0, s>>>(g, a, tg.kz);
}

template <int KIND, typename TO, bool DT>
void launch_tri_batch_k(const TriJob* jobs, int nj, int blocks, cudaStream_t s) {
  k_tri_batch<KIND, TO, DT><<<blocks, 256, 0, s>>>(jobs, nj);
}

}  // namespace

bool tri_ahead(const Geom& g, int elt) { return 3.0 * (double)g.nfield * elt > 96e6; }

bool tri_vectorable(const Geom& g, int elt, const void* const* fields, int n) {
  bool ok = g.n1 % (16 / elt) == 0;
  for (int q = 0; q < n; ++q) ok = ok && (reinterpret_cast<uintptr_t>(fields[q]) & 15) == 0;
  return ok;
}

TriGrid tri_grid(const Geom& g, int elt, bool vec, long long total_points) {
  TriGrid t;
  t.vec = vec ? 1 : 0;
  const int nx = vec ? 16 * (16 / elt) : 32, ny = vec ? 16 : 8;
  t.gx = (g.n1 + nx - 1) / nx;
  t.gy = (g.n2 + ny - 1) / ny;
  // a grid of a batch: its share of the SMs, by its points
  const double share = total_points > 0 ? (double)g.n1 * g.n2 * g.n3 / (double)total_points : 1.0;
  t.kz = tri_depth((double)t.gx * t.gy, g.n3, device_sms() * share, vec);
  t.gz = (g.n3 + t.kz - 1) / t.kz;
  return t;
}

template <int KIND, typename T, typename TO>
void launch_tri(const Geom& g, const TriArgs<T, TO>& a, const TriGrid& tg, cudaStream_t s) {
  constexpr int W = 16 / (int)sizeof(T);
  if constexpr (KIND == TRI_INTERP) {
    if (a.partial) {
      if (tg.vec)
        launch_tri_v<KIND, T, TO, W, true>(g, a, tg, s);
      else
        launch_tri_v<KIND, T, TO, 1, true>(g, a, tg, s);
      return;
    }
  }
  if (tg.vec)
    launch_tri_v<KIND, T, TO, W, false>(g, a, tg, s);
  else
    launch_tri_v<KIND, T, TO, 1, false>(g, a, tg, s);
}
template void launch_tri<TRI_DIV2, double, double>(const Geom&, const TriArgs<double, double>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_DIV2, float, float>(const Geom&, const TriArgs<float, float>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_HELM, double, double>(const Geom&, const TriArgs<double, double>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_HELM, float, float>(const Geom&, const TriArgs<float, float>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_INTERP, double, double>(const Geom&, const TriArgs<double, double>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_INTERP, double, float>(const Geom&, const TriArgs<double, float>&, const TriGrid&, cudaStream_t);
template void launch_tri<TRI_PROJECT, double, double>(const Geom&, const TriArgs<double, double>&, const TriGrid&, cudaStream_t);

void launch_tri_batch(int kind, int f32, int dt, const TriJob* jobs, int nj, int blocks, cudaStream_t s) {
  if (kind == TRI_DIV2) {
    launch_tri_batch_k<TRI_DIV2, double, false>(jobs, nj, blocks, s);
  } else if (kind == TRI_PROJECT) {
    launch_tri_batch_k<TRI_PROJECT, double, false>(jobs, nj, blocks, s);
  } else if (f32) {
    if (dt)
      launch_tri_batch_k<TRI_INTERP, float, true>(jobs, nj, blocks, s);
    else
      launch_tri_batch_k<TRI_INTERP, float, false>(jobs, nj, blocks, s);
  } else {
    if (dt)
      launch_tri_batch_k<TRI_INTERP, double, true>(jobs, nj, blocks, s);
    else
      launch_tri_batch_k<TRI_INTERP, double, false>(jobs, nj, blocks, s);
  }
}

int tri_upload_limits(const double* lim41, cudaStream_t s) {
  IMPACT_CUDA_CHECK(cudaMemcpyToSymbolAsync(c_lim, lim41, 41 * sizeof(double), 0, cudaMemcpyHostToDevice, s));
  return 0;
}

}  // namespace impact
