// Cell kernels of the continuous Q_p Laplace operator with one thread per line of a cell.
//
// What they compute is the BK3 cell operator of the reference
// (include/kernels/bk3_kokkos_kernel.h:25-746): per cell gather the nodal values (Dirichlet
// entries read as 0), differentiate at the Gauss points, apply the symmetric geometry tensor,
// integrate against the gradients and scatter-add.
//
// N^2 threads work on a cell, N = p+1.  A thread owns one line of N nodes along the direction
// being contracted, so a 1D contraction is a register product against tables in the constant
// bank; changing the direction is one exchange through shared memory.
// vmult_line_kernel (any geometry) takes the lines z, y, x to the Gauss points and x, y, z back:
//   z:  t = Sz u, tz = SDz u                                    (E1: 2 arrays)
//   y:  w = Sy t, wy = SDy t, wz = Sy tz                        (E2: 3 arrays)
//   x:  dx = SDx w, dy = Sx wy, dz = Sx wz;  f = G grad u;
//       ax = SDx^T fx, ay = Sx^T fy, az = Sx^T fz               (E2: 3 arrays)
//   y:  b = Sy^T ax + SDy^T ay, c = Sy^T az                     (E1: 2 arrays)
//   z:  out = Sz^T b + SDz^T c, scatter
// vmult_box_kernel (axis-aligned cells, no coefficient) uses that the cell matrix is the sum
// cx K x M x M + cy M x K x M + cz M x M x K of Kronecker products of the 1D mass matrix M and
// stiffness matrix K (the Gauss rule is exact for the products of two basis derivatives and
// the same rule defines M), which takes 7 instead of 16 contractions:
//   z:  a = Mz u, b = Kz u                                      (E1: 2 arrays)
//   y:  v = My a, w = cy Ky a + cz My b                         (E2: 2 arrays)
//   x:  out = cx Kx v + Mx w                                    (E3: 1 array)
//   z:  scatter
// Lines along z carry the gather and the scatter because the lanes of a warp then hold
// neighbouring nodes of an (x, y) plane, which are neighbours in the first-visit numbering too.
//
// Against one lane per plane of a cell (laplace_kernels.cuh) a line needs a third of the
// registers and its exchange buffers hold a third of the cell per thread, so 20 to 45 warps
// are resident per SM instead of 7 or 8, at twice the shared-memory traffic.
#pragma once

#include "laplace_kernels.cuh"
#include "pdl.cuh"

namespace pmg {
namespace kern {

// Two FP32 values moved and computed together, the same place of two neighbouring cells: one packed
// instruction for two scalar ones, each rounded as the scalar one is.
struct alignas(8) F2 {
  float x, y;
  F2() = default;
  __host__ __device__ __forceinline__ F2(float a, float b) : x(a), y(b) {}
  __host__ __device__ __forceinline__ explicit F2(double a) : x((float)a), y((float)a) {}
  __device__ __forceinline__ static F2 of(unsigned long long b) {
    F2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(b));
    return v;
  }
  __device__ __forceinline__ unsigned long long bits() const {
    unsigned long long b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(x), "f"(y));
    return b;
  }
  friend __device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a.bits()), "l"(b.bits()));
    return of(d);
  }
  friend __device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a.bits()), "l"(b.bits()));
    return of(d);
  }
  friend __device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a.bits()), "l"(b.bits()));
    return of(d);
  }
  friend __device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a.bits()), "l"(b.bits()), "l"(c.bits()));
    return of(d);
  }
};
// what a kernel's element V stands for: CELLS cells' values of type T
template <typename V> struct Elem {
  using T = V;
  static constexpr int CELLS = 1;
  template <typename F> __device__ __forceinline__ static V make(F &&f) { return f(0); }
  template <typename F> __device__ __forceinline__ static void each(V v, F &&f) { f(0, v); }
};
template <> struct Elem<F2> {
  using T = float;
  static constexpr int CELLS = 2;
  template <typename F> __device__ __forceinline__ static F2 make(F &&f) { return F2(f(0), f(1)); }
  template <typename F> __device__ __forceinline__ static void each(F2 v, F &&f) {
    f(0, v.x);
    f(1, v.y);
  }
};

// Layouts of the exchange buffers: node (i, j, k) of cell e is at e*CS + i*I + j*J + k*K.
// Lanes: z lines r = j*N + i, x lines r = k*N + j, y lines r = k*N + i (YK = 0) or i*N + k
// (YK = 1).  The strides are those with the fewest bank conflicts for the two access patterns
// of each exchange (z and y, y and x, x and z), found by exhaustive search over permuted,
// padded strides: for FP64 Q6, 467 shared-memory wavefronts per cell against 747 with one
// layout for every exchange (429 without any conflict).
template <int I_, int J_, int K_> struct XLayout {
  static constexpr int I = I_, J = J_, K = K_;
};
template <int N, typename T> struct LineLayout;
template <typename T> struct LineLayout<2, T> {
  using E1 = XLayout<1, 2, 6>;
  using E2 = XLayout<1, 3, 6>;
  using E3 = XLayout<1, 2, 5>;
  static constexpr int YK = 0, CS = 12;
};
template <typename T> struct LineLayout<3, T> {
  using E1 = XLayout<3, 1, 9>;
  using E2 = XLayout<1, 3, 9>;
  using E3 = XLayout<1, 3, 9>;
  static constexpr int YK = 0, CS = 27;
};
template <> struct LineLayout<4, float> {
  using E1 = XLayout<1, 4, 20>;
  using E2 = XLayout<1, 5, 20>;
  using E3 = XLayout<1, 4, 17>;
  static constexpr int YK = 0, CS = 80;
};
template <> struct LineLayout<4, double> {
  using E1 = XLayout<4, 1, 17>;
  using E2 = XLayout<1, 17, 4>;
  using E3 = XLayout<1, 4, 17>;
  static constexpr int YK = 0, CS = 67;
};
template <> struct LineLayout<5, float> {
  using E1 = XLayout<5, 1, 25>;
  using E2 = XLayout<1, 5, 25>;
  using E3 = XLayout<1, 5, 25>;
  static constexpr int YK = 0, CS = 125;
};
template <> struct LineLayout<5, double> {
  using E1 = XLayout<5, 25, 1>;
  using E2 = XLayout<25, 1, 5>;
  using E3 = XLayout<1, 5, 25>;
  static constexpr int YK = 1, CS = 125;
};
template <> struct LineLayout<6, float> {
  using E1 = XLayout<1, 6, 38>;
  using E2 = XLayout<1, 37, 6>;
  using E3 = XLayout<1, 6, 37>;
  static constexpr int YK = 0, CS = 228;
};
template <> struct LineLayout<6, double> {
  using E1 = XLayout<1, 6, 38>;
  using E2 = XLayout<1, 41, 6>;
  using E3 = XLayout<1, 6, 37>;
  static constexpr int YK = 0, CS = 244;
};
template <> struct LineLayout<7, float> {
  using E1 = XLayout<7, 49, 1>;
  using E2 = XLayout<49, 1, 7>;
  using E3 = XLayout<1, 7, 49>;
  static constexpr int YK = 1, CS = 343;
};
template <> struct LineLayout<7, double> {
  using E1 = XLayout<7, 1, 49>;
  using E2 = XLayout<1, 49, 7>;
  using E3 = XLayout<1, 7, 49>;
  static constexpr int YK = 0, CS = 353;
};

// elements of 8 bytes
template <> struct LineLayout<4, F2> : LineLayout<4, double> {};
template <> struct LineLayout<5, F2> : LineLayout<5, double> {};
template <> struct LineLayout<6, F2> : LineLayout<6, double> {};
template <> struct LineLayout<7, F2> : LineLayout<7, double> {};

// The tables a line kernel reads
template <int N, typename T> struct LineTab {
  EvenOdd<N, T> eS, eSD, eST, eSDT;
  T W[N];
};
// even/odd tables of the 1D mass matrix M and stiffness matrix K on the reference interval
template <int N, typename T> struct BoxTab {
  EvenOdd<N, T> eM, eK;
};

// CPB cells per block.  WC > 0: WC cells per warp, which only warp barriers order; WC = 0: the
// N^2 threads of the cells follow one another across warps and block barriers order them.
// MINB: blocks per SM that the registers are allocated for.
template <int CPB_, int WC_, int MINB_> struct LineShape {
  static constexpr int CPB = CPB_, WC = WC_, MINB = MINB_;
};
template <int N, typename SH> constexpr int line_threads() {
  return SH::WC ? SH::CPB / (SH::WC ? SH::WC : 1) * 32 : (SH::CPB * N * N + 31) / 32 * 32;
}

// Position of a thread: its cell in the block and its lines in each direction and layout
template <int N, typename T, typename SH> struct LinePlace {
  using L = LineLayout<N, T>;
  int e, r;      // cell of the block, line of the cell
  bool active;   // holds a line
  int z1, y1, y2, x2;
  __device__ __forceinline__ LinePlace() {
    constexpr int N2 = N * N;
    const int t = threadIdx.x, u = SH::WC ? (t & 31) : t, c = u / N2;
    r = u - c * N2;
    e = SH::WC ? (t >> 5) * SH::WC + c : c;
    active = SH::WC ? c < SH::WC : e < SH::CPB;
    const int ra = r % N, rb = r / N, yi = L::YK ? rb : ra, yk = L::YK ? ra : rb, o = e * L::CS;
    z1 = o + ra * L::E1::I + rb * L::E1::J;
    y1 = o + yi * L::E1::I + yk * L::E1::K;
    y2 = o + yi * L::E2::I + yk * L::E2::K;
    x2 = o + ra * L::E2::J + rb * L::E2::K;
  }
  __device__ __forceinline__ static void sync() {
    if constexpr (SH::WC != 0 || line_threads<N, SH>() == 32) __syncwarp();
    else __syncthreads();
  }
};

// the N entries of the index map on a z line (the sentinel for a cell past the end)
template <int N> __device__ __forceinline__ void line_index(const uint32_t *__restrict__ idx, int64_t c, int r,
                                                            bool in, uint64_t pol, uint32_t (&id)[N]) {
  const uint32_t *ip = idx + c * (N * N * N) + r;
#pragma unroll
  for (int k = 0; k < N; ++k) id[k] = in ? ld_keep_early(ip + k * (N * N), pol) : kInvalidIdx;
}

template <int N, typename T, typename SH> constexpr size_t line_smem() {
  return size_t(3) * SH::CPB * LineLayout<N, T>::CS * sizeof(T);
}
template <int N, typename T, typename SH> constexpr size_t box_smem() {
  return size_t(4) * SH::CPB * LineLayout<N, T>::CS * sizeof(T);
}

// GEOM 0: full geometry [cell][x point][6][z point, y point]; 2: axis-aligned cells (diagonal
// tensor cd0, cd3, cd5) times a coefficient per point, [cell][x point][z point, y point];
// 3: inverse-Jacobian layout, as 0 with 10 components.
// E1 and E2 share the three buffers (A0, A1 and B0, B1, B2), so a y line is read by every
// thread before any is written; buffers of their own, with two barriers less, cost a fifth of
// the resident warps and measured slower (FP64 Q4 455 against 419 us at 64^3).
// The loop over the batches of cells is the grid: a loop in the kernel made the compiler keep
// the tables in registers (FP64 Q6 207 instead of 88 registers, 652 against 330 us).
// Full geometry is prefetched into L2 as one bulk request per block, issued before the index
// map is read, and loaded where it is used: staging it in shared memory takes the room of a
// block more per SM (FP64 Q4 419 against 376 us, Q3 211 against 163 us at 64^3).
template <int N, typename V, int GEOM, typename SH>
__global__ void __launch_bounds__(line_threads<N, SH>(), SH::MINB)
    vmult_line_kernel(const __grid_constant__ LineTab<N, V> tab, const typename Elem<V>::T *__restrict__ src,
                      typename Elem<V>::T *__restrict__ dst, const uint32_t *__restrict__ idx,
                      const typename Elem<V>::T *__restrict__ geo, const typename Elem<V>::T *__restrict__ coef,
                      V cd0, V cd3, V cd5, int64_t n_cells) {
  using EL = Elem<V>;
  using T = typename EL::T;
  constexpr int CELLS = EL::CELLS;
  using L = LineLayout<N, V>;
  using E1 = typename L::E1;
  using E2 = typename L::E2;
  constexpr int N2 = N * N, N3 = N2 * N, CPB = SH::CPB, NCOMP = GEOM == 3 ? 10 : 6;
  constexpr int GF = geo_cell_elems<N, T>(NCOMP);
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *A0 = reinterpret_cast<V *>(smem_raw), *A1 = A0 + CPB * L::CS, *A2 = A1 + CPB * L::CS;
  const LinePlace<N, V, SH> at;
  const int r = at.r;
  const int64_t c0 = int64_t(blockIdx.x) * (CPB * CELLS), c = c0 + at.e * CELLS; // the first cell of the block, of the element
  auto in = [&](int m) { return at.active && c + m < n_cells; };
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  if constexpr (GEOM == 0 || GEOM == 3) {
    if (threadIdx.x == 0) {
      const int64_t left = n_cells - c0;
      prefetch_l2(geo + c0 * GF, (uint32_t)((left < CPB * CELLS ? (int)left : CPB * CELLS) * GF * (int)sizeof(T)), pol_first);
    }
  }
  uint32_t id[CELLS][N];
#pragma unroll
  for (int m = 0; m < CELLS; ++m) line_index<N>(idx, c + m, r, in(m), pol_first, id[m]); // (fixed at setup: read before the wait)
  pdl_wait();
  src = pdl_after(src);
  geo = pdl_after(geo);
  coef = pdl_after(coef);
  V cf[GEOM == 2 ? N : 1]; // the coefficient on the x line, requested before the gather
  if constexpr (GEOM == 2) {
    const T *cp = coef + c * N3 + r;
#pragma unroll
    for (int p = 0; p < N; ++p)
      cf[p] = EL::make([&](int m) { return in(m) ? ld_keep_early(cp + m * N3 + p * N2, pol_first) : T(0); });
  }
  if (at.active) {
    V u[N];
#pragma unroll
    for (int k = 0; k < N; ++k) 
      u[k] = EL::make([&](int m) { return id[m][k] != kInvalidIdx ? ld_keep(src + id[m][k], pol_last) : T(0); });
    eo_apply<N, V, 1>(tab.eS, u, [&](int q, V v) { A0[at.z1 + q * E1::K] = v; });
    eo_apply<N, V, -1>(tab.eSD, u, [&](int q, V v) { A1[at.z1 + q * E1::K] = v; });
  }
  at.sync();
  {
    V a[N], z[N];
    if (at.active) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        a[j] = A0[at.y1 + j * E1::J];
        z[j] = A1[at.y1 + j * E1::J];
      }
    }
    at.sync();
    if (at.active) {
      eo_apply<N, V, 1>(tab.eS, a, [&](int q, V v) { A0[at.y2 + q * E2::J] = v; });
      eo_apply<N, V, -1>(tab.eSD, a, [&](int q, V v) { A1[at.y2 + q * E2::J] = v; });
      eo_apply<N, V, 1>(tab.eS, z, [&](int q, V v) { A2[at.y2 + q * E2::J] = v; });
    }
  }
  at.sync();
  if (at.active) {
    if constexpr (GEOM == 2) {
      // the tensor is diagonal: one direction at a time
      const V wyz = line_weight<N, V>(tab.W, r % N) * line_weight<N, V>(tab.W, r / N);
#pragma unroll
      for (int p = 0; p < N; ++p) cf[p] = cf[p] * (tab.W[p] * wyz);
      V l[N], d[N];
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A0[at.x2 + i * E2::I];
      eo_apply<N, V, -1>(tab.eSD, l, [&](int q, V v) { d[q] = (cf[q] * cd0) * v; });
      eo_apply<N, V, -1>(tab.eSDT, d, [&](int q, V v) { A0[at.x2 + q * E2::I] = v; });
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A1[at.x2 + i * E2::I];
      eo_apply<N, V, 1>(tab.eS, l, [&](int q, V v) { d[q] = (cf[q] * cd3) * v; });
      eo_apply<N, V, 1>(tab.eST, d, [&](int q, V v) { A1[at.x2 + q * E2::I] = v; });
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = A2[at.x2 + i * E2::I];
      eo_apply<N, V, 1>(tab.eS, l, [&](int q, V v) { d[q] = (cf[q] * cd5) * v; });
      eo_apply<N, V, 1>(tab.eST, d, [&](int q, V v) { A2[at.x2 + q * E2::I] = v; });
    } else {
      V dx[N], dy[N], dz[N];
      {
        V l[N];
#pragma unroll
        for (int i = 0; i < N; ++i) l[i] = A0[at.x2 + i * E2::I];
        eo_apply<N, V, -1>(tab.eSD, l, [&](int q, V v) { dx[q] = v; });
#pragma unroll
        for (int i = 0; i < N; ++i) l[i] = A1[at.x2 + i * E2::I];
        eo_apply<N, V, 1>(tab.eS, l, [&](int q, V v) { dy[q] = v; });
#pragma unroll
        for (int i = 0; i < N; ++i) l[i] = A2[at.x2 + i * E2::I];
        eo_apply<N, V, 1>(tab.eS, l, [&](int q, V v) { dz[q] = v; });
      }
      const T *gp = geo + c * GF + r;
#pragma unroll
      for (int p = 0; p < N; ++p) {
        V g[NCOMP];
#pragma unroll
        for (int m = 0; m < NCOMP; ++m)
          g[m] = EL::make([&](int k) { return in(k) ? ld_keep(gp + k * GF + (p * NCOMP + m) * N2, pol_first) : T(0); });
        const V x = dx[p], y = dy[p], z = dz[p];
        if constexpr (GEOM == 0) {
          dx[p] = fma(g[2], z, fma(g[1], y, g[0] * x));
          dy[p] = fma(g[4], z, fma(g[3], y, g[1] * x));
          dz[p] = fma(g[5], z, fma(g[4], y, g[2] * x));
        } else { // J^{-1} row by row, then JxW: the physical gradient, times JxW, and back
          V gx[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) gx[k] = g[NCOMP - 1] * fma(g[(6 + k) % NCOMP], z, fma(g[3 + k], y, g[k] * x));
          dx[p] = fma(g[2], gx[2], fma(g[1], gx[1], g[0] * gx[0]));
          dy[p] = fma(g[5], gx[2], fma(g[4], gx[1], g[3] * gx[0]));
          dz[p] = fma(g[8 % NCOMP], gx[2], fma(g[7 % NCOMP], gx[1], g[6 % NCOMP] * gx[0]));
        }
      }
      eo_apply<N, V, -1>(tab.eSDT, dx, [&](int q, V v) { A0[at.x2 + q * E2::I] = v; });
      eo_apply<N, V, 1>(tab.eST, dy, [&](int q, V v) { A1[at.x2 + q * E2::I] = v; });
      eo_apply<N, V, 1>(tab.eST, dz, [&](int q, V v) { A2[at.x2 + q * E2::I] = v; });
    }
  }
  at.sync();
  {
    V a[N], z[N], o[N];
    if (at.active) {
#pragma unroll
      for (int j = 0; j < N; ++j) {
        a[j] = A0[at.y2 + j * E2::J];
        z[j] = A1[at.y2 + j * E2::J];
      }
      eo_apply<N, V, 1>(tab.eST, a, [&](int q, V v) { o[q] = v; });
      eo_apply<N, V, -1>(tab.eSDT, z, [&](int q, V v) { o[q] = o[q] + v; });
#pragma unroll
      for (int j = 0; j < N; ++j) a[j] = A2[at.y2 + j * E2::J];
    }
    at.sync();
    if (at.active) {
#pragma unroll
      for (int j = 0; j < N; ++j) A0[at.y1 + j * E1::J] = o[j];
      eo_apply<N, V, 1>(tab.eST, a, [&](int q, V v) { A1[at.y1 + q * E1::J] = v; });
    }
  }
  at.sync();
  if (at.active) {
    V a[N], z[N], o[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      a[k] = A0[at.z1 + k * E1::K];
      z[k] = A1[at.z1 + k * E1::K];
    }
    eo_apply<N, V, 1>(tab.eST, a, [&](int q, V v) { o[q] = v; });
    eo_apply<N, V, -1>(tab.eSDT, z, [&](int q, V v) { o[q] = o[q] + v; });
#pragma unroll
    for (int k = 0; k < N; ++k)
      EL::each(o[k], [&](int m, T v) {
        if (id[m][k] != kInvalidIdx) red_keep(dst + id[m][k], v, pol_last);
      });
  }
}

// axis-aligned cells without a coefficient: (cx, cy, cz) = vol / h^2 per direction.  E1, E2 and
// E3 have buffers of their own (E3 over E1's first), so three barriers order a cell.
template <int N, typename V, typename SH>
__global__ void __launch_bounds__(line_threads<N, SH>(), SH::MINB)
    vmult_box_kernel(const __grid_constant__ BoxTab<N, V> tab, const typename Elem<V>::T *__restrict__ src,
                     typename Elem<V>::T *__restrict__ dst, const uint32_t *__restrict__ idx, V cx, V cy, V cz,
                     int64_t n_cells) {
  using EL = Elem<V>;
  using T = typename EL::T;
  constexpr int CELLS = EL::CELLS;
  using L = LineLayout<N, V>;
  using E1 = typename L::E1;
  using E2 = typename L::E2;
  using E3 = typename L::E3;
  constexpr int CPB = SH::CPB;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V *A0 = reinterpret_cast<V *>(smem_raw), *A1 = A0 + CPB * L::CS, *B0 = A1 + CPB * L::CS, *B1 = B0 + CPB * L::CS;
  const LinePlace<N, V, SH> at;
  const int ra = at.r % N, rb = at.r / N;
  const int64_t c = (int64_t(blockIdx.x) * CPB + at.e) * CELLS;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  uint32_t id[CELLS][N];
#pragma unroll
  for (int m = 0; m < CELLS; ++m)
    line_index<N>(idx, c + m, at.r, at.active && c + m < n_cells, pol_first, id[m]); // (fixed at setup: read before the wait)
  pdl_wait();
  src = pdl_after(src);
  if (at.active) {
    V u[N];
#pragma unroll
    for (int k = 0; k < N; ++k) 
      u[k] = EL::make([&](int m) { return id[m][k] != kInvalidIdx ? ld_keep(src + id[m][k], pol_last) : T(0); });
    eo_apply<N, V, 1>(tab.eM, u, [&](int q, V v) { A0[at.z1 + q * E1::K] = v; });
    eo_apply<N, V, 1>(tab.eK, u, [&](int q, V v) { A1[at.z1 + q * E1::K] = cz * v; });
  }
  at.sync();
  if (at.active) {
    V a[N], b[N], o[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      a[j] = A0[at.y1 + j * E1::J];
      b[j] = A1[at.y1 + j * E1::J];
    }
    eo_apply<N, V, 1>(tab.eM, a, [&](int q, V v) { B0[at.y2 + q * E2::J] = v; });
    eo_apply<N, V, 1>(tab.eK, a, [&](int q, V v) { o[q] = v; });
    eo_apply<N, V, 1>(tab.eM, b, [&](int q, V v) { B1[at.y2 + q * E2::J] = fma(cy, o[q], v); });
  }
  at.sync();
  if (at.active) {
    V a[N], b[N], o[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      a[i] = B0[at.x2 + i * E2::I];
      b[i] = B1[at.x2 + i * E2::I];
    }
    V *x3 = A0 + at.e * L::CS + ra * E3::J + rb * E3::K;
    eo_apply<N, V, 1>(tab.eK, a, [&](int q, V v) { o[q] = v; });
    eo_apply<N, V, 1>(tab.eM, b, [&](int q, V v) { x3[q * E3::I] = fma(cx, o[q], v); });
  }
  at.sync();
  if (at.active) {
    const V *z3 = A0 + at.e * L::CS + ra * E3::I + rb * E3::J;
#pragma unroll
    for (int k = 0; k < N; ++k)
      EL::each(z3[k * E3::K], [&](int m, T v) {
        if (id[m][k] != kInvalidIdx) red_keep(dst + id[m][k], v, pol_last);
      });
  }
}

} // namespace kern
} // namespace pmg
