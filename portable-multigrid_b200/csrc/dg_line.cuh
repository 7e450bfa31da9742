// DG-SIPG operator on axis-aligned boxes, cell and face terms in one kernel, one thread per line of a
// cell (the interior-penalty operator of include/operators/portable_laplace_operator_dg.h).
//
// On a uniform Cartesian box the operator is a sum over the directions of a 1D interior-penalty
// operator times mass matrices across: with T_d the 1D operator along d (cell stiffness, own traces
// and the two neighbours' traces),
//   A u = Mz (My T_x u + Mx T_y u) + My Mx T_z u.
// T_d acts on u itself, so a neighbour enters only through the line that continues a thread's own
// one: its end value and end derivative, read from L1 or L2 -- no face buffers, no tiles, no
// face mass of its own.  Per cell N^2 threads:
//   each thread's x, y and z line: g_d = T_d u, into three buffers
//   x lines:  q = Mx g_y, r = Mx g_z
//   y lines:  s = My g_x + q, r' = My r
//   z lines:  A u = Mz s + r', written once (or the Chebyshev step from it)
// with one barrier in between.  8 contractions per cell and three barriers against 240 face
// evaluations per 64 cells and five block barriers of the tile kernel.
#pragma once

#include "line_kernels.cuh"
#include "pdl.cuh"

namespace pmg {
namespace kern {

template <int N, typename T> struct DGLineTab {
  EvenOdd<N, T> eM, eK;
  T dphi0[N], dphi1[N];
};
struct DGLineGeo {
  double area_h[3], area[3], sigma[3], rh[3]; // area / h, face area, c_pen / h, 1 / h per direction
  int dirichlet;                              // face mask
};
// the Chebyshev step that may take the place of storing A x (STEP):
// out = x + f1 (x - x_prev) + f2 D^{-1} (b - A x), x = src; prev null: x_prev = 0
template <typename T> struct DGLineStep {
  const T *prev, *b, *invd;
  T f1, f2;
};

template <int N, typename T, typename SH> constexpr size_t dg_line_smem() {
  return size_t(3) * SH::CPB * LineLayout<N, T>::CS * sizeof(T);
}

// N values ST apart; VEC: consecutive ones as the widest loads that fit (p aligned to them)
template <int N, int ST, bool VEC, typename T> __device__ __forceinline__ void load_line(const T *p, T (&u)[N]) {
  constexpr int bytes = N * (int)sizeof(T);
  if constexpr (VEC && ST == 1 && bytes % 16 == 0) {
#pragma unroll
    for (int v = 0; v < bytes / 16; ++v) {
      const uint4 q = reinterpret_cast<const uint4 *>(p)[v];
      memcpy(reinterpret_cast<char *>(u) + 16 * v, &q, 16);
    }
  } else if constexpr (VEC && ST == 1 && bytes % 8 == 0) {
#pragma unroll
    for (int v = 0; v < bytes / 8; ++v) {
      const uint2 q = reinterpret_cast<const uint2 *>(p)[v];
      memcpy(reinterpret_cast<char *>(u) + 8 * v, &q, 8);
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) u[i] = p[i * ST];
  }
}

// g = T_D u on a line; at: the line's offset in a cell (entries ST apart); nb0, nb1: the neighbour
// cells below and above (-1: boundary)
template <int N, typename T, int D, int ST, bool VEC>
__device__ __forceinline__ void dg_line(const DGLineTab<N, T> &tab, const DGLineGeo &geo, const T *src, int at,
                                        int32_t nb0, int32_t nb1, const T (&u)[N], T (&g)[N]) {
  constexpr int N3 = N * N * N;
  const T rh = (T)geo.rh[D], sigma = (T)geo.sigma[D], area = (T)geo.area[D], ck = (T)geo.area_h[D];
  T d0 = T(0), d1 = T(0);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    d0 = fma(tab.dphi0[i], u[i], d0);
    d1 = fma(tab.dphi1[i], u[i], d1);
  }
  // value jump and sum of the derivatives along +d, per side (mirror u+ = -u-, d_n u+ = d_n u- on a
  // Dirichlet face; nothing on another boundary face)
  T j0, s0, j1, s1;
  if (nb0 >= 0) {
    T w[N], d = T(0);
    load_line<N, ST, VEC>(src + int64_t(nb0) * N3 + at, w);
#pragma unroll
    for (int i = 0; i < N; ++i) d = fma(tab.dphi1[i], w[i], d);
    j0 = u[0] - w[N - 1];
    s0 = d0 + d;
  } else {
    const bool dir = (geo.dirichlet >> (2 * D)) & 1;
    j0 = dir ? T(2) * u[0] : T(0);
    s0 = dir ? T(2) * d0 : T(0);
  }
  if (nb1 >= 0) {
    T w[N], d = T(0);
    load_line<N, ST, VEC>(src + int64_t(nb1) * N3 + at, w);
#pragma unroll
    for (int i = 0; i < N; ++i) d = fma(tab.dphi0[i], w[i], d);
    j1 = u[N - 1] - w[0];
    s1 = d1 + d;
  } else {
    const bool dir = (geo.dirichlet >> (2 * D + 1)) & 1;
    j1 = dir ? T(2) * u[N - 1] : T(0);
    s1 = dir ? T(2) * d1 : T(0);
  }
  const T hr = T(0.5) * rh;
  const T v0 = area * (sigma * j0 + hr * s0), v1 = area * (sigma * j1 - hr * s1); // value tests
  const T n0 = area * hr * j0, n1 = -(area * hr) * j1;                            // derivative tests
  eo_apply<N, T, 1>(tab.eK, u, [&](int q, T v) { g[q] = ck * v; });
#pragma unroll
  for (int i = 0; i < N; ++i) g[i] += n0 * tab.dphi0[i] + n1 * tab.dphi1[i];
  g[0] += v0;
  g[N - 1] += v1;
}

template <int N, typename T, typename SH, bool VEC, bool STEP>
__global__ void __launch_bounds__(line_threads<N, SH>(), SH::MINB)
    dg_line_kernel(const __grid_constant__ DGLineTab<N, T> tab, const __grid_constant__ DGLineGeo geo, const T *src, T *dst,
                   const int32_t *__restrict__ nbr, int64_t n_cells, const DGLineStep<T> step) {
  using L = LineLayout<N, T>;
  using E1 = typename L::E1;
  using E2 = typename L::E2;
  using E3 = typename L::E3;
  constexpr int N2 = N * N, N3 = N2 * N, CPB = SH::CPB;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const LinePlace<N, T, SH> at;
  const int e = at.e, r = at.r;
  const int64_t c = int64_t(blockIdx.x) * CPB + e;
  const bool in = at.active && c < n_cells;
  const int ra = r % N, rb = r / N, yi = L::YK ? rb : ra, yk = L::YK ? ra : rb;
  // three buffers; an array is laid out for the lines that read it next (LineLayout), so where the
  // layout changes every thread reads its lines before any writes
  T *X = reinterpret_cast<T *>(smem_raw), *Y = X + CPB * L::CS, *Z = Y + CPB * L::CS;
  const int z3 = e * L::CS + ra * E3::I + rb * E3::J, x3 = e * L::CS + ra * E3::J + rb * E3::K;
  int32_t nb[6]; // (fixed at setup: read before the wait)
#pragma unroll
  for (int f = 0; f < 6; ++f) nb[f] = in ? __ldg(nbr + c * 6 + f) : -1;
  pdl_wait();
  src = pdl_after(src);
  const T *own = src + c * N3;
  T uz[N];
  if (in) {
    T u[N], g[N];
    load_line<N, 1, VEC>(own + r * N, u);
    load_line<N, N2, false>(own + r, uz);
    dg_line<N, T, 0, 1, VEC>(tab, geo, src, r * N, nb[0], nb[1], u, g);
#pragma unroll
    for (int i = 0; i < N; ++i) X[at.x2 + i * E2::I] = g[i];
    const int y = yi + yk * N2;
    load_line<N, N, false>(own + y, u);
    dg_line<N, T, 1, N, false>(tab, geo, src, y, nb[2], nb[3], u, g);
#pragma unroll
    for (int j = 0; j < N; ++j) Y[at.y2 + j * E2::J] = g[j];
    dg_line<N, T, 2, N2, false>(tab, geo, src, r, nb[4], nb[5], uz, g);
#pragma unroll
    for (int k = 0; k < N; ++k) Z[z3 + k * E3::K] = g[k];
  }
  at.sync();
  {
    T a[N], b[N];
    if (in) {
#pragma unroll
      for (int i = 0; i < N; ++i) {
        a[i] = Y[at.x2 + i * E2::I];
        b[i] = Z[x3 + i * E3::I];
      }
      eo_apply<N, T, 1>(tab.eM, a, [&](int q, T v) { Y[at.x2 + q * E2::I] = v; });
    }
    at.sync();
    if (in) eo_apply<N, T, 1>(tab.eM, b, [&](int q, T v) { Z[at.x2 + q * E2::I] = v; });
  }
  at.sync();
  {
    T a[N], b[N], d[N];
    if (in) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        a[j] = X[at.y2 + j * E2::J];
        b[j] = Y[at.y2 + j * E2::J];
        d[j] = Z[at.y2 + j * E2::J];
      }
    }
    at.sync();
    if (in) {
      eo_apply<N, T, 1>(tab.eM, a, [&](int q, T v) { X[at.y1 + q * E1::J] = v + b[q]; });
      eo_apply<N, T, 1>(tab.eM, d, [&](int q, T v) { Z[at.y1 + q * E1::J] = v; });
    }
  }
  at.sync();
  if (in) {
    T a[N], b[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      a[k] = X[at.z1 + k * E1::K];
      b[k] = Z[at.z1 + k * E1::K];
    }
    const int64_t o = c * N3 + r;
    if constexpr (STEP) {
      // out (dst) may be prev, whose entry only this thread reads, never src, which the neighbours read
      eo_apply<N, T, 1>(tab.eM, a, [&](int q, T v) { b[q] += v; });
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const T x = uz[k], xo = step.prev ? step.prev[o + k * N2] : T(0);
        b[k] = x + step.f1 * (x - xo) + step.f2 * step.invd[o + k * N2] * (step.b[o + k * N2] - b[k]);
      }
#pragma unroll
      for (int k = 0; k < N; ++k) dst[o + k * N2] = b[k];
    } else {
      eo_apply<N, T, 1>(tab.eM, a, [&](int q, T v) { dst[o + q * N2] = b[q] + v; });
    }
  }
}

} // namespace kern
} // namespace pmg
