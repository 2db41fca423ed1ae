// march.cu -- the one-axis stencil operators of the launcher FFI, the JOR sweep and axpby as
// streaming passes.
//
// gradient (mod_diff.f90:309-414), divergence per axis (:52-118), both interpolations
// (:1567-1648, :1740-1825) and the upwind advection term (:784-1424) are 6- or 7-point stencils
// along one axis a: out(q) = sum_{l} c(l, q) f(q + LO + l), q the coordinate along a, with the
// row of coefficients c(., q) of that coordinate.  A thread owns one vector of V x points (V = 16
// bytes where the rows hold whole aligned vectors, else V = 1) and walks a segment in blocks of U
// steps, all loads of a block issued before its stores:
//   a = y or z: marches along a, the stencil's values in registers, one new vector per step; the
//               coefficient row of a step is the same for the whole block;
//   a = x:      marches z with the coefficient rows of its points loaded once; each plane takes the
//               aligned vectors of the row that its points' stencils span (V = 1: its taps).
// Threads are numbered along the vectors of a row and then along the rows, so that narrow grids
// fill their warps, and a segment is as short as one step where a small grid would otherwise leave
// SMs idle (march_seg, shape.h).  Periodic wrapping is applied to the coordinate along a only; each
// point sums its terms in table order with fused multiply-adds.
//
// Bound by DRAM on large grids and by latency on small ones.  256 x 256 x 512 FP64 (270 MB a
// field, 6.5 TB/s copy bandwidth): the y and z interpolations 90 and 87 us (6.0 and 6.2 TB/s; 95 and 94
// with blocks of 256 threads, 118 - 125 with one step's loads at a time and segments of 64), along x
// 113 us (125 with spilled planes), the upwind terms 234 / 198 us, axpby 123 us.  187 x 131 x 157
// FP32, rows of odd length: 12.4 us (one point per thread with its taps wrapped one by one: 25), the
// upwind terms 16.5 - 18.6 us (29 - 31).  64 x 64 x 128 FP64: JOR sweep 6.3 us (10.7), interpolations
// 4.7 us (8.3).
#include "kernels.cuh"
#include "shape.h"

namespace impact {
namespace {

template <typename T>
struct V16;
template <>
struct V16<double> {
  using t = double2;
  static constexpr int W = 2;
};
template <>
struct V16<float> {
  using t = float4;
  static constexpr int W = 4;
};
template <typename T>
__device__ __forceinline__ void vld(const T* p, T (&o)[V16<T>::W]) {
  const typename V16<T>::t v = __ldg(reinterpret_cast<const typename V16<T>::t*>(p));
  if constexpr (V16<T>::W == 2) {
    o[0] = v.x;
    o[1] = v.y;
  } else {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
}
template <typename T>
__device__ __forceinline__ void vld_plain(const T* p, T (&o)[V16<T>::W]) {  // may alias the output
  const typename V16<T>::t v = *reinterpret_cast<const typename V16<T>::t*>(p);
  if constexpr (V16<T>::W == 2) {
    o[0] = v.x;
    o[1] = v.y;
  } else {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
}
template <typename T>
__device__ __forceinline__ void vst(T* p, const T (&o)[V16<T>::W]) {
  if constexpr (V16<T>::W == 2)
    *reinterpret_cast<double2*>(p) = make_double2(o[0], o[1]);
  else
    *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ float fmaT(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fmaT(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mulT(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mulT(double a, double b) { return __dmul_rn(a, b); }

// OP 0: out = S f;  OP 1: out = out + S f (terms added to the old value in order);
// OP 2: upwind, out = S_sel f * pp (first axis) or out + S_sel f * pp, S_sel the cA row where
// pp >= 0 and the cB row elsewhere
template <typename T, int CNT, int OP>
__device__ __forceinline__ T point_value(const T* __restrict__ ca, const T* __restrict__ cb, const T (&win)[CNT],
                                         T old, T ppv, int first) {
  if (OP == 1) {
    T s = old;
#pragma unroll
    for (int l = 0; l < CNT; ++l) s = fmaT(ca[l], win[l], s);
    return s;
  }
  const T* c = (OP == 2 && !(ppv >= T(0))) ? cb : ca;
  T s = mulT(c[0], win[0]);
#pragma unroll
  for (int l = 1; l < CNT; ++l) s = fmaT(c[l], win[l], s);
  if (OP == 2) return first ? mulT(s, ppv) : fmaT(s, ppv, old);
  return s;
}

constexpr int MT = 128;  // threads per block

template <typename T, int V>
__device__ __forceinline__ void ldv(const T* p, T (&o)[V]) {
  if constexpr (V == 1)
    o[0] = __ldg(p);
  else
    vld(p, o);
}
template <typename T, int V>
__device__ __forceinline__ void ldv_plain(const T* p, T (&o)[V]) {  // may alias the output
  if constexpr (V == 1)
    o[0] = p[0];
  else
    vld_plain(p, o);
}
template <typename T, int V>
__device__ __forceinline__ void stv(T* p, const T (&o)[V]) {
  if constexpr (V == 1)
    p[0] = o[0];
  else
    vst(p, o);
}
// a = 1 (y) or 2 (z): thread (vector, other in-plane coordinate o) marches q = q0 .. q1
template <typename T, int V, int LO, int CNT, int OP>
__global__ void __launch_bounds__(MT) k_march_yz(int a, Geom g, const T* __restrict__ cA, const T* __restrict__ cB,
                                                 const T* __restrict__ f, const T* __restrict__ pp,
                                                 T* __restrict__ out, int first, int seg) {
  // steps at a time: 4, or 2 where the operands of 4 take the registers of too many warps
  constexpr bool wide = OP == 1 ? V == 2 : (OP == 2 && (V == 4 || (V == 1 && sizeof(T) == 8)));
  constexpr int U = wide ? 2 : 4, NW = CNT - 1 + U;
  const int nvx = g.n1 / V;
  const unsigned idx = blockIdx.x * MT + threadIdx.x;
  const int o = (int)(idx / (unsigned)nvx) + 1;
  const int i = 1 + V * (int)(idx % (unsigned)nvx);
  const int na = a == 2 ? g.n3 : g.n2, no = a == 2 ? g.n2 : g.n3;
  if (o > no) return;
  const long long sa = a == 2 ? g.nxy : (long long)g.nx;
  const long long so = a == 2 ? (long long)g.nx : g.nxy;
  const long long base = (i + 3) + so * (o + 3) + sa * 3;  // (i, o, q = 0)
  const int q0 = blockIdx.y * seg + 1, q1 = min(na, q0 + seg - 1);
  T win[NW][V];
#pragma unroll
  for (int l = 0; l < CNT - 1; ++l) ldv<T, V>(f + base + sa * wrapi(q0 + LO + l, na), win[l]);
  for (int q = q0; q <= q1; q += U) {
    T old[U][V], pv[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || q + u <= q1) {
        ldv<T, V>(f + base + sa * wrapi(q + u + LO + CNT - 1, na), win[CNT - 1 + u]);
        const long long p = base + sa * (q + u);
        if (OP != 0) ldv_plain<T, V>(out + p, old[u]);
        if (OP == 2) ldv<T, V>(pp + p, pv[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || q + u <= q1) {
        T ca[CNT], cb[CNT], r[V];
#pragma unroll
        for (int l = 0; l < CNT; ++l) {
          ca[l] = __ldg(cA + (long long)(q + u) * CNT + l);
          cb[l] = OP == 2 ? __ldg(cB + (long long)(q + u) * CNT + l) : ca[l];
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          T wv[CNT];
#pragma unroll
          for (int l = 0; l < CNT; ++l) wv[l] = win[u + l][v];
          r[v] = point_value<T, CNT, OP>(ca, cb, wv, OP != 0 ? old[u][v] : T(0), OP == 2 ? pv[u][v] : T(0), first);
        }
        stv<T, V>(out + base + sa * (q + u), r);
      }
#pragma unroll
    for (int l = 0; l < CNT - 1; ++l)
#pragma unroll
      for (int v = 0; v < V; ++v) win[l][v] = win[l + U][v];
  }
}

// Resident blocks of k_march_x, which set its registers: as many as hold the coefficient rows and the
// planes in flight without spills (vectors one plane at a time: 64 registers.  With 2 or 4 planes in those
// 64 a thread spilled 24 to 268 bytes: 128^3 FP64 20.5 us, now 8.3; 192^3 FP32 22.6, now 12.5)
template <typename T, int V, int OP>
constexpr int march_x_blocks() {
  if (V > 1) return OP == 2 ? 4 : 8;
  return OP != 2 ? 4 : (sizeof(T) == 8 ? 6 : 8);
}
// a = 0 (x): thread (vector, row j) marches z
template <typename T, int V, int LO, int CNT, int OP>
__global__ void __launch_bounds__(MT, march_x_blocks<T, V, OP>()) k_march_x(Geom g, const T* __restrict__ cA,
                                                                            const T* __restrict__ cB,
                                                                            const T* __restrict__ f,
                                                                            const T* __restrict__ pp,
                                                                            T* __restrict__ out, int first, int seg) {
  constexpr int U = OP == 2 || V > 1 ? 1 : 4;
  constexpr int FV = (LO - (V - 1)) / V;          // floor(LO / V) for LO < 0
  constexpr int LV = (V - 1 + LO + CNT - 1) / V;  // floor of the last position / V (>= 0)
  constexpr int NV = LV - FV + 1;
  const int nvx = g.n1 / V;
  const unsigned idx = blockIdx.x * MT + threadIdx.x;
  const int j = (int)(idx / (unsigned)nvx) + 1;
  const int vx = (int)(idx % (unsigned)nvx);
  if (j > g.n2) return;
  const int i = 1 + V * vx;
  const int k0 = blockIdx.y * seg + 1, k1 = min(g.n3, k0 + seg - 1);
  T ca[V][CNT], cb[V][CNT];
#pragma unroll
  for (int v = 0; v < V; ++v)
#pragma unroll
    for (int l = 0; l < CNT; ++l) {
      ca[v][l] = __ldg(cA + (long long)(i + v) * CNT + l);
      cb[v][l] = OP == 2 ? __ldg(cB + (long long)(i + v) * CNT + l) : ca[v][l];
    }
  int us[NV];
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int u = vx + FV + n;
    us[n] = V * (u < 0 ? u + nvx : (u >= nvx ? u - nvx : u));
  }
  const long long rowj = 4 + (long long)g.nx * (j + 3);  // offset of (1, j, k = -3)
  for (int k = k0; k <= k1; k += U) {
    T val[U][NV * V], old[U][V], pv[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        const long long row = rowj + g.nxy * (k + u + 3);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          T tmp[V];
          ldv<T, V>(f + row + us[n], tmp);
#pragma unroll
          for (int v = 0; v < V; ++v) val[u][n * V + v] = tmp[v];
        }
        const long long p = row + (i - 1);
        if (OP != 0) ldv_plain<T, V>(out + p, old[u]);
        if (OP == 2) ldv<T, V>(pp + p, pv[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        T r[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          T wv[CNT];
#pragma unroll
          for (int l = 0; l < CNT; ++l) wv[l] = val[u][v + LO + l - FV * V];
          r[v] = point_value<T, CNT, OP>(ca[v], cb[v], wv, OP != 0 ? old[u][v] : T(0), OP == 2 ? pv[u][v] : T(0), first);
        }
        stv<T, V>(out + rowj + g.nxy * (k + u + 3) + (i - 1), r);
      }
  }
}

// relaxation_div_grad / the JOR sweep (mod_laplace.f90:339-613, jacobi_kernel.cu):
// out = omega (bb - sum of the six off-diagonal terms of cdg) / diag + (1 - omega) rel.  Thread
// (vector, row j) marches z with the column's rel at k-1..k+1 in registers.
template <typename T, int V>
__global__ void __launch_bounds__(MT, 5) k_jacobi_march(Geom g, const T* __restrict__ c1, const T* __restrict__ c2,
                                                     const T* __restrict__ c3, T omega, const T* __restrict__ bb,
                                                     const T* __restrict__ rel, T* __restrict__ out, int seg) {
  constexpr int U = 2;
  const int nvx = g.n1 / V;
  const unsigned idx = blockIdx.x * MT + threadIdx.x;
  const int j = (int)(idx / (unsigned)nvx) + 1;
  const int i = 1 + V * (int)(idx % (unsigned)nvx);
  if (j > g.n2) return;
  const int k0 = blockIdx.y * seg + 1, k1 = min(g.n3, k0 + seg - 1);
  const long long row = (i + 3) + (long long)g.nx * (j + 3);  // (i, j, k = -3)
  const int dW = i == 1 ? g.n1 - 1 : -1, dE = i + V - 1 == g.n1 ? 1 - i : V;
  const int dS = (wrapi(j - 1, g.n2) - j) * g.nx, dN = (wrapi(j + 1, g.n2) - j) * g.nx;
  T a0[V], a1[V], a2[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const T* a = c1 + 3 * (i + v - 1);
    a0[v] = __ldg(a);
    a1[v] = __ldg(a + 1);
    a2[v] = __ldg(a + 2);
  }
  const T b0 = __ldg(c2 + 3 * (j - 1)), b1 = __ldg(c2 + 3 * (j - 1) + 1), b2 = __ldg(c2 + 3 * (j - 1) + 2);
  T zc[2 + U][V];
  ldv<T, V>(rel + row + (long long)g.nxy * (wrapi(k0 - 1, g.n3) + 3), zc[0]);
  ldv<T, V>(rel + row + (long long)g.nxy * (k0 + 3), zc[1]);
  for (int k = k0; k <= k1; k += U) {
    T w[U], e[U], ym[U][V], yp[U][V], bv[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        const long long p = row + (long long)g.nxy * (k + u + 3);
        ldv<T, V>(rel + row + (long long)g.nxy * (wrapi(k + u + 1, g.n3) + 3), zc[2 + u]);
        w[u] = __ldg(rel + p + dW);
        e[u] = __ldg(rel + p + dE);
        ldv<T, V>(rel + p + dS, ym[u]);
        ldv<T, V>(rel + p + dN, yp[u]);
        ldv<T, V>(bb + p, bv[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        const T e0 = __ldg(c3 + 3 * (k + u - 1)), e1 = __ldg(c3 + 3 * (k + u - 1) + 1), e2 = __ldg(c3 + 3 * (k + u - 1) + 2);
        T r[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const T xm = v == 0 ? w[u] : zc[1 + u][v == 0 ? 0 : v - 1];
          const T xp = v == V - 1 ? e[u] : zc[1 + u][v == V - 1 ? v : v + 1];
          r[v] = omega * (bv[u][v] - a0[v] * xm - a2[v] * xp - b0 * ym[u][v] - b2 * yp[u][v] - e0 * zc[u][v] -
                          e2 * zc[2 + u][v]) /
                     (a1[v] + b1 + e1) +
                 (T(1) - omega) * zc[1 + u][v];
        }
        stv<T, V>(out + row + (long long)g.nxy * (k + u + 3), r);
      }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      zc[0][v] = zc[U][v];
      zc[1][v] = zc[U + 1][v];
    }
  }
}

// z = a x + b y (axpby_kernel.cu:6-17)
template <typename T, int V>
__global__ void __launch_bounds__(MT) k_axpby(Geom g, T a, T b, const T* __restrict__ x, const T* __restrict__ y,
                                              T* __restrict__ z, int seg) {
  constexpr int U = 4;
  const int nvx = g.n1 / V;
  const unsigned idx = blockIdx.x * MT + threadIdx.x;
  const int j = (int)(idx / (unsigned)nvx) + 1;
  const int i = 1 + V * (int)(idx % (unsigned)nvx);
  if (j > g.n2) return;
  const int k0 = blockIdx.y * seg + 1, k1 = min(g.n3, k0 + seg - 1);
  long long p = off(g, i, j, k0);
  for (int k = k0; k <= k1; k += U, p += U * g.nxy) {
    T xv[U][V], yv[U][V];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        ldv<T, V>(x + p + u * g.nxy, xv[u]);
        ldv<T, V>(y + p + u * g.nxy, yv[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u == 0 || k + u <= k1) {
        T r[V];
#pragma unroll
        for (int v = 0; v < V; ++v) r[v] = fmaT(a, xv[u][v], mulT(b, yv[u][v]));
        stv<T, V>(z + p + u * g.nxy, r);
      }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_axpby_points(Geom g, T a, T b, const T* __restrict__ x,
                                                      const T* __restrict__ y, T* __restrict__ z) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1, j = blockIdx.y * 8 + threadIdx.y + 1;
  if (i > g.n1 || j > g.n2) return;
  const long long p = off(g, i, j, blockIdx.z + 1);
  z[p] = fmaT(a, x[p], mulT(b, y[p]));
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// grid of a pass: threads (vectors of one row x no rows), na steps, segments by march_seg
inline dim3 march_grid(const Geom& g, int V, int no, int na, int& seg, int per_sm = 320, int most = 8) {
  const long long threads = (long long)(g.n1 / V) * no;
  seg = march_seg(threads, na, device_sms(), per_sm, most);
  return dim3((unsigned)((threads + MT - 1) / MT), (na + seg - 1) / seg);
}

template <typename T, int V, int LO, int CNT, int OP>
void march1(int a, const Geom& g, const T* cA, const T* cB, const T* f, const T* pp, T* out, int first,
            cudaStream_t s) {
  int seg = 0;
  if (a == 0) {
    const dim3 grid = march_grid(g, V, g.n2, g.n3, seg, 256, 16);
    k_march_x<T, V, LO, CNT, OP><<<grid, MT, 0, s>>>(g, cA, cB, f, pp, out, first, seg);
  } else {
    const dim3 grid = march_grid(g, V, a == 2 ? g.n2 : g.n3, a == 2 ? g.n3 : g.n2, seg);
    k_march_yz<T, V, LO, CNT, OP><<<grid, MT, 0, s>>>(a, g, cA, cB, f, pp, out, first, seg);
  }
}

}  // namespace

template <typename T, int LO, int CNT, int OP>
void launch_march1(int a, const Geom& g, const T* cA, const T* cB, const T* f, const T* pp, T* out, int first,
                   cudaStream_t s) {
  constexpr int W = V16<T>::W;
  if (g.n1 % W == 0 && aligned16(f) && aligned16(out) && (OP != 2 || aligned16(pp)))
    march1<T, W, LO, CNT, OP>(a, g, cA, cB, f, pp, out, first, s);
  else
    march1<T, 1, LO, CNT, OP>(a, g, cA, cB, f, pp, out, first, s);
}

template <typename T>
void launch_jacobi(const Geom& g, const T* c1, const T* c2, const T* c3, T omega, const T* bb, const T* rel, T* out,
                   cudaStream_t s) {
  constexpr int W = V16<T>::W;
  int seg = 0;
  if (g.n1 % W == 0 && aligned16(bb) && aligned16(rel) && aligned16(out)) {
    const dim3 grid = march_grid(g, W, g.n2, g.n3, seg);
    k_jacobi_march<T, W><<<grid, MT, 0, s>>>(g, c1, c2, c3, omega, bb, rel, out, seg);
  } else {
    const dim3 grid = march_grid(g, 1, g.n2, g.n3, seg);
    k_jacobi_march<T, 1><<<grid, MT, 0, s>>>(g, c1, c2, c3, omega, bb, rel, out, seg);
  }
}
template <typename T>
void launch_axpby(const Geom& g, T a, T b, const T* x, const T* y, T* z, cudaStream_t s) {
  constexpr int W = V16<T>::W;
  int seg = 0;
  // fewer vectors than 320 threads per SM (46 points a side in FP64, 57 in FP32): all latency, one point
  // per thread without a march (32 x 32 x 64: 3.1 us against 3.6 to 4.1)
  if ((long long)g.n1 * g.n2 * g.n3 < 320LL * W * device_sms()) {
    const dim3 grid((g.n1 + 31) / 32, (g.n2 + 7) / 8, g.n3);
    k_axpby_points<T><<<grid, dim3(32, 8), 0, s>>>(g, a, b, x, y, z);
  } else if (g.n1 % W == 0 && aligned16(x) && aligned16(y) && aligned16(z)) {
    const dim3 grid = march_grid(g, W, g.n2, g.n3, seg, 640);
    k_axpby<T, W><<<grid, MT, 0, s>>>(g, a, b, x, y, z, seg);
  } else {
    const dim3 grid = march_grid(g, 1, g.n2, g.n3, seg, 640);
    k_axpby<T, 1><<<grid, MT, 0, s>>>(g, a, b, x, y, z, seg);
  }
}

#define MARCH_INST(T)                                                                                             \
  template void launch_march1<T, G_LO, NG, 0>(int, const Geom&, const T*, const T*, const T*, const T*, T*, int,  \
                                              cudaStream_t);                                                      \
  template void launch_march1<T, D_LO, ND, 0>(int, const Geom&, const T*, const T*, const T*, const T*, T*, int,  \
                                              cudaStream_t);                                                      \
  template void launch_march1<T, D_LO, ND, 1>(int, const Geom&, const T*, const T*, const T*, const T*, T*, int,  \
                                              cudaStream_t);                                                      \
  template void launch_march1<T, B_LO, NB, 2>(int, const Geom&, const T*, const T*, const T*, const T*, T*, int,  \
                                              cudaStream_t);                                                      \
  template void launch_jacobi<T>(const Geom&, const T*, const T*, const T*, T, const T*, const T*, T*,            \
                                 cudaStream_t);                                                                   \
  template void launch_axpby<T>(const Geom&, T, T, const T*, const T*, T*, cudaStream_t);
MARCH_INST(double)
MARCH_INST(float)
#undef MARCH_INST

}  // namespace impact
