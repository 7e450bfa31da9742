// Kernels of the adjoint path: the FE mass matrix, its diagonal, and the density of the
// Laplace form at every quadrature point.  None of them exists in the reference; they use the
// layouts and the two thread schemes of the Laplace kernels: one lane per line of a cell at
// degrees >= 3 (line_kernels.cuh), one lane per plane below and for the diagonal
// (laplace_kernels.cuh).
//
//   mass:    v = Sz Sy Sx u at the Gauss points, times |det J| w_q, back by the transposes.
//   qp form: grad_ref u and grad_ref v at the Gauss points as in the Laplace kernel's first
//            half, and e_q = alpha * grad u^T G_q grad v, written lexicographically per cell.
#pragma once

#include "laplace_kernels.cuh"
#include "line_kernels.cuh"

namespace pmg {
namespace kern {

// MG 1: affine cell without a weight field, |det J| = geo[cell][6];
// MG 0: per-point weights |det J| w_q (times a coefficient) in wts, a value per point as CellData
// places it.
template <int N, typename T, typename SH> constexpr size_t mass_line_smem() {
  return size_t(2) * SH::CPB * LineLayout<N, T>::CS * sizeof(T);
}
template <int N, typename T, int MG, typename SH>
__global__ void __launch_bounds__(line_threads<N, SH>(), SH::MINB)
    mass_line_kernel(const __grid_constant__ LineTab<N, T> tab, const T *__restrict__ src, T *__restrict__ dst,
                     const uint32_t *__restrict__ idx, const T *__restrict__ geo, const T *__restrict__ wts,
                     int64_t n_cells) {
  using L = LineLayout<N, T>;
  using E1 = typename L::E1;
  using E2 = typename L::E2;
  constexpr int N2 = N * N, N3 = N2 * N, CPB = SH::CPB;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *A = reinterpret_cast<T *>(smem_raw), *B = A + CPB * L::CS; // E1 and E2
  const LinePlace<N, T, SH> at;
  const int r = at.r;
  const int64_t c = int64_t(blockIdx.x) * CPB + at.e;
  const bool in = at.active && c < n_cells;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  uint32_t id[N];
  line_index<N>(idx, c, r, in, pol_first, id);
  T w[N]; // the weights on the x line
  if constexpr (MG == 1) {
    const T vyz = (in ? __ldg(geo + c * 8 + 6) : T(0)) * line_weight<N, T>(tab.W, r % N) * line_weight<N, T>(tab.W, r / N);
#pragma unroll
    for (int p = 0; p < N; ++p) w[p] = vyz * tab.W[p];
  } else {
#pragma unroll
    for (int p = 0; p < N; ++p) w[p] = in ? ld_keep_early(wts + c * N3 + p * N2 + r, pol_first) : T(0);
  }
  T u[N];
  if (at.active) {
#pragma unroll
    for (int k = 0; k < N; ++k) u[k] = id[k] != kInvalidIdx ? ld_keep(src + id[k], pol_last) : T(0);
    eo_apply<N, T, 1>(tab.eS, u, [&](int q, T v) { A[at.z1 + q * E1::K] = v; });
  }
  at.sync();
  if (at.active) {
#pragma unroll
    for (int j = 0; j < N; ++j) u[j] = A[at.y1 + j * E1::J];
    eo_apply<N, T, 1>(tab.eS, u, [&](int q, T v) { B[at.y2 + q * E2::J] = v; });
  }
  at.sync();
  if (at.active) {
    T v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) u[i] = B[at.x2 + i * E2::I];
    eo_apply<N, T, 1>(tab.eS, u, [&](int q, T x) { v[q] = w[q] * x; });
    eo_apply<N, T, 1>(tab.eST, v, [&](int q, T x) { B[at.x2 + q * E2::I] = x; });
  }
  at.sync();
  if (at.active) {
#pragma unroll
    for (int j = 0; j < N; ++j) u[j] = B[at.y2 + j * E2::J];
    eo_apply<N, T, 1>(tab.eST, u, [&](int q, T v) { A[at.y1 + q * E1::J] = v; });
  }
  at.sync();
  if (at.active) {
#pragma unroll
    for (int k = 0; k < N; ++k) u[k] = A[at.z1 + k * E1::K];
    eo_apply<N, T, 1>(tab.eST, u, [&](int q, T v) {
      if (id[q] != kInvalidIdx) red_keep(dst + id[q], v, pol_last);
    });
  }
}

template <int N, typename T, int MG>
__global__ void __launch_bounds__(128, 1) mass_slab_kernel(const __grid_constant__ Tab<N, T> tab,
                                                        const T *__restrict__ src, T *__restrict__ dst,
                                                        const uint32_t *__restrict__ idx,
                                                        const T *__restrict__ geo,
                                                        const T *__restrict__ wts, int64_t n_groups) {
  using Lo = Layout<N>;
  constexpr int CPW = Lo::CPW, LANES = Lo::LANES, N2 = Lo::N2;
  constexpr int CS = Stride<N>::CELL;
  constexpr unsigned MASK = Lo::MASK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  if (lane >= LANES) return;
  const int e = lane / N;
  const int s = lane - e * N;
  T *buf = reinterpret_cast<T *>(smem_raw) + (threadIdx.x >> 5) * (CPW * CS) + e * CS;
  const int64_t warp0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  static_assert(!mass_line_layout(N), "mass_line_kernel");
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  constexpr int UNR = N;
  T wr = tab.W[0];
#pragma unroll
  for (int r = 1; r < N; ++r)
    if (s == r) wr = tab.W[r];

  for (int64_t g = warp0; g < n_groups; g += nwarps) {
    const uint32_t *ig = idx + g * (N2 * LANES) + lane;
    // Y-slab y = s: gather, x and z interpolation -> buf (z, y = s, x)
    {
      T u[N][N];
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const uint32_t id = ld_stream(ig + (k * N + i) * LANES, pol_first);
          u[k][i] = (id != kInvalidIdx) ? ld_keep(src + id, pol_last) : T(0);
        }
#pragma unroll UNR
      for (int p = 0; p < N; ++p) {
        T t[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
          T a = T(0);
#pragma unroll
          for (int i = 0; i < N; ++i) a = fma(tab.S[i * N + p], u[k][i], a);
          t[k] = a;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) {
          T w = T(0);
#pragma unroll
          for (int k = 0; k < N; ++k) w = fma(tab.S[k * N + r], t[k], w);
          buf[(r * N + s) * N + p] = w;
        }
      }
    }
    __syncwarp(MASK);
    // Z-slab z = s: y interpolation, weights, and the transposed x and y contractions
    {
      const T vol = MG == 1 ? __ldg(geo + (g * CPW + e) * 8 + 6) * wr : T(1);
      T a[N][N];
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) a[j][i] = T(0);
#pragma unroll UNR
      for (int p = 0; p < N; ++p) {
        T Wc[N];
#pragma unroll
        for (int j = 0; j < N; ++j) Wc[j] = buf[(s * N + j) * N + p];
        T f[N];
#pragma unroll
        for (int q = 0; q < N; ++q) {
          T v = T(0);
#pragma unroll
          for (int j = 0; j < N; ++j) v = fma(tab.S[j * N + q], Wc[j], v);
          const T wq = MG == 1 ? vol * tab.W[q] * tab.W[p]
                               : ld_stream(wts + g * (N2 * LANES) + (q * N + p) * LANES + lane, pol_first);
          f[q] = wq * v;
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
          T y = T(0);
#pragma unroll
          for (int q = 0; q < N; ++q) y = fma(tab.S[j * N + q], f[q], y);
#pragma unroll
          for (int i = 0; i < N; ++i) a[j][i] = fma(tab.S[i * N + p], y, a[j][i]);
        }
      }
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) buf[(s * N + j) * N + i] = a[j][i];
    }
    __syncwarp(MASK);
    // Y-slab y = s: transposed z contraction and scatter
#pragma unroll UNR
    for (int i = 0; i < N; ++i) {
      T A[N];
#pragma unroll
      for (int r = 0; r < N; ++r) A[r] = buf[(r * N + s) * N + i];
#pragma unroll
      for (int k = 0; k < N; ++k) {
        T v = T(0);
#pragma unroll
        for (int r = 0; r < N; ++r) v = fma(tab.S[k * N + r], A[r], v);
        const uint32_t id = ld_stream(ig + (k * N + i) * LANES, pol_first);
        if (id != kInvalidIdx) red_keep(dst + id, v, pol_last);
      }
    }
    __syncwarp(MASK);
  }
}

// diag(M)(i,j,k) = sum_{p,q,r} S2[i,p] S2[j,q] S2[k,r] w(p,q,r), S2 = S*S elementwise.
template <int N, typename T, int MG>
__global__ void __launch_bounds__(128) mass_diag_slab_kernel(const __grid_constant__ Tab2<N, T> tab,
                                                             T *__restrict__ diag,
                                                             const uint32_t *__restrict__ idx,
                                                             const T *__restrict__ geo,
                                                             const T *__restrict__ wts, int64_t n_groups) {
  using Lo = Layout<N>;
  using CD = CellData<N, mass_line_layout(N)>;
  constexpr int CPW = Lo::CPW, LANES = Lo::LANES;
  constexpr int CS = Stride<N>::CELL;
  constexpr unsigned MASK = Lo::MASK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  if (lane >= LANES) return;
  const int e = lane / N;
  const int s = lane - e * N;
  T *buf = reinterpret_cast<T *>(smem_raw) + (threadIdx.x >> 5) * (CPW * CS) + e * CS;
  const int64_t warp0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  T wr = tab.W[0];
#pragma unroll
  for (int r = 1; r < N; ++r)
    if (s == r) wr = tab.W[r];
  for (int64_t g = warp0; g < n_groups; g += nwarps) {
    const T vol = MG == 1 ? __ldg(geo + (g * CPW + e) * 8 + 6) * wr : T(1);
    T w[N][N]; // [q][p] on the Z-slab z = s
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int p = 0; p < N; ++p)
        w[q][p] = MG == 1 ? vol * tab.W[q] * tab.W[p] : __ldg(wts + CD::point(g * CPW + e, p, q, s));
#pragma unroll
    for (int i = 0; i < N; ++i) {
      T x[N];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        T a = T(0);
#pragma unroll
        for (int p = 0; p < N; ++p) a = fma(tab.S2[i * N + p], w[q][p], a);
        x[q] = a;
      }
#pragma unroll
      for (int j = 0; j < N; ++j) {
        T b = T(0);
#pragma unroll
        for (int q = 0; q < N; ++q) b = fma(tab.S2[j * N + q], x[q], b);
        buf[(s * N + j) * N + i] = b;
      }
    }
    __syncwarp(MASK);
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        T v = T(0);
#pragma unroll
        for (int r = 0; r < N; ++r) v = fma(tab.S2[k * N + r], buf[(r * N + s) * N + i], v);
        const uint32_t id = __ldg(idx + CD::idx(g * CPW + e, i, s, k));
        if (id != kInvalidIdx) atomic_add(diag + id, v);
      }
    __syncwarp(MASK);
  }
}

// e_q = alpha * grad_ref(u)^T G_q grad_ref(v) at every Gauss point, written as
// out[cell][(z*N + y)*N + x] (FP64).  G_q is the operator's stored geometry (GEOM 0 full, 1
// axis-aligned, 2 axis-aligned times the per-point coefficient), so the
// coefficient is included: e summed over the points of all cells is a(u, v).
// The gradient of u waits in registers while that of v passes through the same buffers; the
// results leave through shared memory as one contiguous run per block.
template <int N, typename T, int GEOM, typename SH>
__global__ void __launch_bounds__(line_threads<N, SH>(), SH::MINB)
    qp_form_line_kernel(const __grid_constant__ LineTab<N, T> tab, const T *__restrict__ u, const T *__restrict__ v,
                        double *__restrict__ out, const uint32_t *__restrict__ idx, const T *__restrict__ geo,
                        const T *__restrict__ coef, T cd0, T cd3, T cd5, int64_t n_cells, double alpha) {
  static_assert(SH::WC == 0, "the cells of a block leave as one run");
  using L = LineLayout<N, T>;
  using E1 = typename L::E1;
  using E2 = typename L::E2;
  constexpr int N2 = N * N, N3 = N2 * N, CPB = SH::CPB, GF = geo_cell_elems<N, T>(6);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *A0 = reinterpret_cast<T *>(smem_raw), *A1 = A0 + CPB * L::CS, *A2 = A1 + CPB * L::CS;
  const LinePlace<N, T, SH> at;
  const int r = at.r;
  const int64_t c0 = int64_t(blockIdx.x) * CPB, c = c0 + at.e;
  const bool in = at.active && c < n_cells;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  uint32_t id[N];
  line_index<N>(idx, c, r, in, pol_first, id);
  T g[2][3][N]; // gradients of u and v at the points of the x line
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const T *src = w == 0 ? u : v;
    if (at.active) {
      T x[N];
#pragma unroll
      for (int k = 0; k < N; ++k) x[k] = id[k] != kInvalidIdx ? ld_keep(src + id[k], pol_last) : T(0);
      eo_apply<N, T, 1>(tab.eS, x, [&](int q, T y) { A0[at.z1 + q * E1::K] = y; });
      eo_apply<N, T, -1>(tab.eSD, x, [&](int q, T y) { A1[at.z1 + q * E1::K] = y; });
    }
    at.sync();
    {
      T a[N], z[N];
      if (at.active) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
          a[j] = A0[at.y1 + j * E1::J];
          z[j] = A1[at.y1 + j * E1::J];
        }
      }
      at.sync();
      if (at.active) {
        eo_apply<N, T, 1>(tab.eS, a, [&](int q, T y) { A0[at.y2 + q * E2::J] = y; });
        eo_apply<N, T, -1>(tab.eSD, a, [&](int q, T y) { A1[at.y2 + q * E2::J] = y; });
        eo_apply<N, T, 1>(tab.eS, z, [&](int q, T y) { A2[at.y2 + q * E2::J] = y; });
      }
    }
    at.sync();
    if (at.active) {
      T l[N];
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A0[at.x2 + i * E2::I];
      eo_apply<N, T, -1>(tab.eSD, l, [&](int q, T y) { g[w][0][q] = y; });
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A1[at.x2 + i * E2::I];
      eo_apply<N, T, 1>(tab.eS, l, [&](int q, T y) { g[w][1][q] = y; });
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A2[at.x2 + i * E2::I];
      eo_apply<N, T, 1>(tab.eS, l, [&](int q, T y) { g[w][2][q] = y; });
    }
    at.sync(); // the buffers are free again
  }
  if (at.active) {
    const T wyz = GEOM == 0 ? T(0) : line_weight<N, T>(tab.W, r % N) * line_weight<N, T>(tab.W, r / N);
#pragma unroll
    for (int p = 0; p < N; ++p) {
      const T *a = &g[0][0][p], *b = &g[1][0][p]; // components N apart
      T e;
      if constexpr (GEOM == 0) {
        T m[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) m[k] = in ? ld_keep(geo + c * GF + (p * 6 + k) * N2 + r, pol_first) : T(0);
        e = a[0] * (m[0] * b[0] + m[1] * b[N] + m[2] * b[2 * N]) + a[N] * (m[1] * b[0] + m[3] * b[N] + m[4] * b[2 * N]) +
            a[2 * N] * (m[2] * b[0] + m[4] * b[N] + m[5] * b[2 * N]);
      } else {
        T f = wyz * tab.W[p];
        if constexpr (GEOM == 2) f *= in ? ld_keep(coef + c * N3 + p * N2 + r, pol_first) : T(0);
        e = a[0] * ((f * cd0) * b[0]) + a[N] * ((f * cd3) * b[N]) + a[2 * N] * ((f * cd5) * b[2 * N]);
      }
      A0[at.e * N3 + r * N + p] = e; // x lines are numbered z*N + y
    }
  }
  at.sync();
  const int64_t left = n_cells - c0;
  const int n = (left < CPB ? (int)left : CPB) * N3;
  for (int t = threadIdx.x; t < n; t += line_threads<N, SH>()) out[c0 * N3 + t] = alpha * double(A0[t]);
}

// The same at degrees 1 and 2, one lane per plane.
// Shared memory per warp: six exchange buffers (w, wz, wx of u and of v).
template <int N, typename T, int GEOM>
__global__ void __launch_bounds__(64, 1) qp_form_slab_kernel(const __grid_constant__ Tab<N, T> tab,
                                                          const T *__restrict__ u, const T *__restrict__ v,
                                                          double *__restrict__ out,
                                                          const uint32_t *__restrict__ idx,
                                                          const T *__restrict__ geo,
                                                          const T *__restrict__ coef, int64_t n_groups,
                                                          int64_t n_cells, double alpha) {
  using Lo = Layout<N>;
  constexpr int CPW = Lo::CPW, LANES = Lo::LANES, N3 = Lo::N3;
  constexpr int CS = Stride<N>::CELL;
  constexpr unsigned MASK = Lo::MASK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  if (lane >= LANES) return;
  const int e = lane / N;
  const int s = lane - e * N;
  static_assert(N <= 3, "qp_form_line_kernel");
  using CD = CellData<N, line_layout(N, GEOM)>;
  constexpr int UNR = N;
  T *wbase = reinterpret_cast<T *>(smem_raw) + (threadIdx.x >> 5) * (6 * CPW * CS);
  T *const B0 = wbase + e * CS; // buffer b of this cell: B0 + b * CPW * CS
  const int64_t warp0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  T wr = tab.W[0];
#pragma unroll
  for (int r = 1; r < N; ++r)
    if (s == r) wr = tab.W[r];

  for (int64_t g = warp0; g < n_groups; g += nwarps) {
    // Y-slab y = s, for u (buffers 0..2) and v (buffers 3..5)
#pragma unroll 1
    for (int vec = 0; vec < 2; ++vec) {
      const T *src = vec == 0 ? u : v;
      T *bW = B0 + (3 * vec) * (CPW * CS), *bZ = bW + CPW * CS, *bX = bZ + CPW * CS;
      T x[N][N];
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const uint32_t id = __ldg(idx + CD::idx(g * CPW + e, i, s, k));
          x[k][i] = (id != kInvalidIdx) ? ld_keep(src + id, pol_last) : T(0);
        }
#pragma unroll UNR
      for (int p = 0; p < N; ++p) {
        T t[N], tx[N];
#pragma unroll
        for (int k = 0; k < N; ++k) {
          T a = T(0), b = T(0);
#pragma unroll
          for (int i = 0; i < N; ++i) {
            a = fma(tab.S[i * N + p], x[k][i], a);
            b = fma(tab.SD[i * N + p], x[k][i], b);
          }
          t[k] = a;
          tx[k] = b;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) {
          T w = T(0), wz = T(0), wx = T(0);
#pragma unroll
          for (int k = 0; k < N; ++k) {
            w = fma(tab.S[k * N + r], t[k], w);
            wz = fma(tab.SD[k * N + r], t[k], wz);
            wx = fma(tab.S[k * N + r], tx[k], wx);
          }
          const int o = (r * N + s) * N + p;
          bW[o] = w;
          bZ[o] = wz;
          bX[o] = wx;
        }
      }
    }
    __syncwarp(MASK);
    // Z-slab z = s: gradients at the points (., ., s), the form, into buffer 0 in place
#pragma unroll 1
    for (int p = 0; p < N; ++p) {
      T c[6][N];
#pragma unroll
      for (int b = 0; b < 6; ++b)
#pragma unroll
        for (int j = 0; j < N; ++j) c[b][j] = B0[b * (CPW * CS) + (s * N + j) * N + p];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        T du[3] = {T(0), T(0), T(0)}, dv[3] = {T(0), T(0), T(0)};
#pragma unroll
        for (int j = 0; j < N; ++j) {
          du[0] = fma(tab.S[j * N + q], c[2][j], du[0]);
          du[1] = fma(tab.SD[j * N + q], c[0][j], du[1]);
          du[2] = fma(tab.S[j * N + q], c[1][j], du[2]);
          dv[0] = fma(tab.S[j * N + q], c[5][j], dv[0]);
          dv[1] = fma(tab.SD[j * N + q], c[3][j], dv[1]);
          dv[2] = fma(tab.S[j * N + q], c[4][j], dv[2]);
        }
        T gc[6];
        load_g6<N, T, GEOM>(geo, coef, tab, g * CPW + e, s, q, p, wr, gc);
        const T g0 = gc[0] * dv[0] + gc[1] * dv[1] + gc[2] * dv[2];
        const T g1 = gc[1] * dv[0] + gc[3] * dv[1] + gc[4] * dv[2];
        const T g2 = gc[2] * dv[0] + gc[4] * dv[1] + gc[5] * dv[2];
        B0[(s * N + q) * N + p] = du[0] * g0 + du[1] * g1 + du[2] * g2;
      }
    }
    __syncwarp(MASK);
    // the group's cells are consecutive: one contiguous, coalesced run of CPW*N^3 values
    const int64_t c0 = g * CPW;
    for (int t = lane; t < CPW * N3; t += LANES) {
      const int ec = t / N3, r = t - ec * N3;
      if (c0 + ec < n_cells) out[c0 * N3 + t] = alpha * double(wbase[ec * CS + r]);
    }
    __syncwarp(MASK);
  }
}

} // namespace kern
} // namespace pmg
