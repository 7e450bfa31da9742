// Slab kernels of the continuous Q_p Laplace operator for sm_100a: the vmult at degrees 1 and 2
// with stored geometry or a coefficient, and the diagonal at every degree.  (The vmult at
// degrees 3 to 6, and of axis-aligned cells without a coefficient at every degree, is in
// line_kernels.cuh: one lane per line of a cell.  At degrees 1 and 2 a line is too short: full
// geometry at 64^3, FP64 Q2 82 against 101 us, FP32 Q2 48 against 62 us with lines.)
//
// What they compute is the BK3 cell operator of the reference
// (include/kernels/bk3_kokkos_kernel.h:25-746): per cell gather the nodal values (Dirichlet
// entries read as 0), interpolate to the Gauss points, take collocation gradients, apply
// the symmetric geometry tensor G, integrate against the gradients and scatter-add.
//
//  * A warp owns a group of CPW = floor(32/N) consecutive cells (N = p+1 nodes per
//    direction), N lanes per cell.  Lane s of a cell works on a slab of the cell: the
//    plane y = s ("Y-slab") while gathering, contracting along x and z and scattering,
//    and the plane z = s ("Z-slab") while contracting along x and y and applying G.
//    Contractions along the slab stay in registers; switching slabs is one warp-local
//    exchange through shared memory.  The operator is factored (SD = S*D, the derivative of
//    the nodal basis at the Gauss points) so that only two switches are needed per cell:
//        Y-slab:  w = Sz Sx u,  wz = SDz Sx u,  wx = Sz SDx u
//        Z-slab:  dx = Sy wx, dy = SDy w, dz = Sy wz;  f = G grad u;
//                 a = Sy^T SDx^T fx + SDy^T Sx^T fy,  c = Sy^T Sx^T fz
//        Y-slab:  out = Sz^T a + SDz^T c
//    No block-wide barrier is used; warps are independent.
//  * The index map and the geometry are stored lane-contiguous per group ([group][point][lane]),
//    so every load of them is a fully coalesced warp access; G is column-major per group (one
//    contiguous chunk per x point). The ring variant streams the columns of the current
//    group through a two-slot shared-memory ring filled by TMA bulk copies one column ahead;
//    the direct-load variant bulk-prefetches the next group's G into L2
//    (cp.async.bulk.prefetch.L2) instead.
//  * Scatter with native FP64/FP32 atomic adds (red.global.add) into L2.
//  * The 1D tables are kernel parameters (constant bank), indexed at compile time.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "pdl.cuh"

namespace pmg {
namespace kern {

constexpr uint32_t kInvalidIdx = 0xFFFFFFFFu;

// Even/odd form of a 1D apply out_q = sum_i M(i, q) in_i for a matrix with the mirror
// symmetry M(N-1-i, N-1-q) = SIG M(i, q) (SIG = +1: S and its transpose; -1: SD and its
// transpose, from the symmetric GLL nodes and Gauss points): with e_i = in_i + in_{N-1-i},
// o_i = in_i - in_{N-1-i} (i < H = N/2) and E_q = sum_i A(i,q) e_i + C(q) in_H (odd N),
// O_q = sum_i B(i,q) o_i, out_q = E_q + O_q and out_{N-1-q} = SIG (E_q - O_q): about half
// the multiply-adds of the plain product.  A = (M(i,q) + M(N-1-i,q))/2, B = (M(i,q) -
// M(N-1-i,q))/2, C(q) = M(H,q), for q < Q = (N+1)/2.
template <int N, typename T> struct EvenOdd {
  static constexpr int H = N / 2, Q = (N + 1) / 2;
  T A[H * Q > 0 ? H * Q : 1], B[H * Q > 0 ? H * Q : 1], C[Q];
};

template <int N, typename T> struct Tab {
  T S[N * N];  // S[i*N+q]  = phi_i(g_q)
  T SD[N * N]; // SD[i*N+q] = phi_i'(g_q)
  T D[N * N];  // D[n*N+q]  = l_n'(g_q) on the Gauss points
  T W[N];      // Gauss weights
  EvenOdd<N, T> eS, eSD;   // S and SD (input node i, output point q)
  EvenOdd<N, T> eST, eSDT; // their transposes (input point q, output node i)
};

// even/odd table of the matrix M(i, q) (host)
template <int N, typename T, typename F> inline void fill_even_odd(EvenOdd<N, T> &e, F &&M) {
  constexpr int H = N / 2, Q = (N + 1) / 2;
  for (int i = 0; i < H; ++i)
    for (int q = 0; q < Q; ++q) {
      e.A[i * Q + q] = (T)(0.5 * (M(i, q) + M(N - 1 - i, q)));
      e.B[i * Q + q] = (T)(0.5 * (M(i, q) - M(N - 1 - i, q)));
    }
  for (int q = 0; q < Q; ++q) e.C[q] = (N & 1) ? (T)M(H, q) : T(0);
}
// those of S and SD (row-major N x N) and their transposes into tab.eS, eSD, eST, eSDT
template <int N, typename TAB> inline void fill_even_odd(TAB &tab, const double *S, const double *SD) {
  fill_even_odd(tab.eS, [&](int i, int q) { return S[i * N + q]; });
  fill_even_odd(tab.eSD, [&](int i, int q) { return SD[i * N + q]; });
  fill_even_odd(tab.eST, [&](int r, int k) { return S[k * N + r]; });
  fill_even_odd(tab.eSDT, [&](int r, int k) { return SD[k * N + r]; });
}

// out_q = sum_i M(i, q) in_i by the even/odd form; f(q, out_q) is called once for every q
template <int N, typename T, int SIG, typename F>
__device__ __forceinline__ void eo_apply(const EvenOdd<N, T> &m, const T (&in)[N], F &&f) {
  constexpr int H = N / 2, Q = (N + 1) / 2;
  T e[H > 0 ? H : 1], o[H > 0 ? H : 1];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    e[i] = in[i] + in[N - 1 - i];
    o[i] = in[i] - in[N - 1 - i];
  }
#pragma unroll
  for (int q = 0; q < H; ++q) {
    T E = (N & 1) ? m.C[q] * in[H] : T(0), O = T(0);
#pragma unroll
    for (int i = 0; i < H; ++i) {
      E = fma(m.A[i * Q + q], e[i], E);
      O = fma(m.B[i * Q + q], o[i], O);
    }
    f(q, E + O);
    f(N - 1 - q, SIG > 0 ? E - O : O - E);
  }
  if (N & 1) {
    T v = T(0);
    if (SIG > 0) {
      v = m.C[H] * in[H];
#pragma unroll
      for (int i = 0; i < H; ++i) v = fma(m.A[i * Q + H], e[i], v);
    } else {
#pragma unroll
      for (int i = 0; i < H; ++i) v = fma(m.B[i * Q + H], o[i], v);
    }
    f(H, v);
  }
}

// squared tables for the diagonal: S2 = S*S, SS = S*SD, D2 = SD*SD (elementwise)
template <int N, typename T> struct Tab2 {
  T S2[N * N];
  T SS[N * N];
  T D2[N * N];
  T W[N];
};

template <int N> struct Layout {
  static constexpr int CPW = 32 / N;
  static constexpr int LANES = CPW * N;
  static constexpr unsigned MASK = LANES == 32 ? 0xffffffffu : ((1u << LANES) - 1u);
  static constexpr int N2 = N * N;
  static constexpr int N3 = N * N * N;
};

// elements of a cell's geometry in the line layout, [N][ncomp][N^2], padded to 16 bytes (the
// unit of the bulk prefetch)
template <int N, typename T> __host__ __device__ constexpr int geo_cell_elems(int ncomp) {
  return (ncomp * N * N * N * (int)sizeof(T) + 15) / 16 * 16 / (int)sizeof(T);
}

// whether a Laplace operator of geometry code GEOM (0 full, 1 axis-aligned, 2 with a coefficient,
// 3 inverse Jacobian) is applied by the line kernels and keeps its cell data in the line layout:
// degrees >= 3, axis-aligned cells at every degree, and degree 1 with a coefficient (64^3 cells,
// FP64 / FP32: 18.8 / 12.5 us against 25.5 / 16.5 us with slabs; degree 2: 76 / 43 against 66 / 43)
__host__ __device__ constexpr bool line_layout(int N, int geom) {
  return N >= 4 || geom == 1 || (N == 2 && geom == 2);
}
// Operators applied by patches of 2 x 2 x 2 cells where the cell order allows it (patch_kernels.cuh):
// axis-aligned cells without a coefficient of degrees >= 2, from 1024 lines of patches per SM on.  Fewer
// leave warps missing: vmult of Q4 at 16^3 (280 lines per SM) 8.6 us against 6.8 by cells in FP64, 8.0
// against 6.7 in FP32; at 32^3 (2240) 21.2 against 26.0 and 14.0 against 16.6; Q2 at 32^3 (690) 8.0 against
// 8.7 and 7.4 against 6.7.
__host__ __device__ constexpr bool patch_layout(int N, int geom) { return N >= 3 && geom == 1; }
inline bool patches_fill(int N, int64_t n_cells, int sms) {
  return n_cells / 8 * ((2 * N - 1) * (2 * N - 1)) >= int64_t(1024) * sms;
}
// the same for mass matrices
__host__ __device__ constexpr bool mass_line_layout(int N) { return N >= 4; }

// Where an operator's cell data lie.  LINE: cell by cell, the index map lexicographic, a value per point as [x point][z point,
// y point].  Otherwise by warp group: the index map as [group][k*N + i][e*N + j], a full geometry
// as [group][x point][y point][component][e*N + z point], a value per point as
// [group][y point, x point][e*N + z point].
template <int N, bool LINE> struct CellData {
  using Lo = Layout<N>;
  static __device__ __forceinline__ int64_t idx(int64_t c, int i, int j, int k) {
    if (LINE) return c * Lo::N3 + (k * N + j) * N + i;
    const int64_t g = c / Lo::CPW;
    return (g * Lo::N2 + k * N + i) * Lo::LANES + int(c - g * Lo::CPW) * N + j;
  }
  // value m of the `ncomp` values of point (p, q, r)
  template <typename T> static __device__ __forceinline__ int64_t geo(int64_t c, int p, int q, int r, int m, int ncomp) {
    if (LINE) return c * geo_cell_elems<N, T>(ncomp) + (p * ncomp + m) * Lo::N2 + r * N + q;
    const int64_t g = c / Lo::CPW;
    return ((g * Lo::N2 + p * N + q) * ncomp + m) * Lo::LANES + int(c - g * Lo::CPW) * N + r;
  }
  static __device__ __forceinline__ int64_t point(int64_t c, int p, int q, int r) {
    if (LINE) return c * Lo::N3 + p * Lo::N2 + r * N + q;
    const int64_t g = c / Lo::CPW;
    return (g * Lo::N2 + q * N + p) * Lo::LANES + int(c - g * Lo::CPW) * N + r;
  }
};

// L2 eviction policies: the geometry and index streams are read once and should not push
// the reused src/dst lines out of L2; src gathers and dst atomics should stay.
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t policy_evict_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ void prefetch_l2(const void *p, uint32_t bytes, uint64_t pol) {
  asm volatile("cp.async.bulk.prefetch.L2.global.L2::cache_hint [%0], %1, %2;" ::"l"(p), "r"(bytes),
               "l"(pol)
               : "memory");
}

// loads with an L2 policy, not allocated in L1 (index maps through the read-only path)
__device__ __forceinline__ double ld_stream(const double *p, uint64_t pol) {
  double v;
  asm("ld.global.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_stream(const float *p, uint64_t pol) {
  float v;
  asm("ld.global.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ uint32_t ld_stream(const uint32_t *p, uint64_t pol) {
  uint32_t v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
// gathered or streamed loads as volatile asm: issued where they stand in the program, not sunk
// towards their first use
__device__ __forceinline__ double ld_keep_early(const double *p, uint64_t pol) {
  double v;
  asm volatile("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_keep_early(const float *p, uint64_t pol) {
  float v;
  asm volatile("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ uint32_t ld_keep_early(const uint32_t *p, uint64_t pol) {
  uint32_t v;
  asm volatile("ld.global.nc.L2::cache_hint.u32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
// W[s] for a runtime s without a divergent constant-bank access
template <int N, typename T> __device__ __forceinline__ T line_weight(const T (&W)[N], int s) {
  T w = W[0];
#pragma unroll
  for (int r = 1; r < N; ++r)
    if (s == r) w = W[r];
  return w;
}
// gathered loads that are reused by neighbouring cells
__device__ __forceinline__ double ld_keep(const double *p, uint64_t pol) {
  double v;
  asm("ld.global.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_keep(const float *p, uint64_t pol) {
  float v;
  asm("ld.global.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}

__device__ __forceinline__ void atomic_add(double *p, double v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add(float *p, float v) { atomicAdd(p, v); }
__device__ __forceinline__ void red_keep(double *p, double v, uint64_t pol) {
  asm volatile("red.global.add.L2::cache_hint.f64 [%0], %1, %2;" ::"l"(p), "d"(v), "l"(pol) : "memory");
}
__device__ __forceinline__ void red_keep(float *p, float v, uint64_t pol) {
  asm volatile("red.global.add.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}

// ---- bulk copies into shared memory completed on an mbarrier (sm_90+ async proxy) ----
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void bulk_load(void *dst_smem, const void *src, uint32_t bytes,
                                          uint64_t *bar, uint64_t pol) {
  // order earlier generic-proxy reads of the destination before the async-proxy write
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
               " [%0], [%1], %2, [%3], %4;" ::"r"(smem_u32(dst_smem)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(smem_u32(bar)), "r"(parity)
               : "memory");
  return ok != 0;
}
// bounded wait: gives up after `limit` polls, records the event in *err and returns false
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity,
                                                  unsigned int *err, uint32_t limit) {
  for (uint32_t it = 0; it < limit; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  if (err) atomicOr(err, 1u);
  return false;
}

// ---- per-thread asynchronous copies into shared memory (cp.async, completion per thread) ----
__device__ __forceinline__ void cp_async(void *dst_smem, const void *src, int bytes, int src_bytes,
                                         uint64_t pol) {
  if (bytes == 8)
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 8, %2, %3;" ::"r"(smem_u32(dst_smem)),
                 "l"(src), "r"(src_bytes), "l"(pol)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global.L2::cache_hint [%0], [%1], 4, %2, %3;" ::"r"(smem_u32(dst_smem)),
                 "l"(src), "r"(src_bytes), "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// GEOM 0: full G per quadrature point, geo = [group][N (x point p)][N (y point q)][6][LANES]
// GEOM 1: affine, geo = [cell][8] (6 used) multiplied by the tensor Gauss weight; affine cells
//         are axis-aligned boxes, so only rr, ss, tt are nonzero (the vmult uses those three)
// GEOM 2: affine as 1, times coef = [group][N^2][LANES] per quadrature point
//
// Register budget: every phase streams over one index so that at most ~2 N^2 values are
// live per lane (the accumulators of the back-contraction plus one column):
//   phase 1 (Y-slab y=s), per x point p:   t = Sx u, tx = SDx u along k, then
//            w = Sz t, wz = SDz t, wx = Sz tx  -> shared (z, y=s, p)
//   phase 2 (Z-slab z=s), per x point p:   dx = Sy wx, dy = SDy w, dz = Sy wz at (., p),
//            f = G grad u, a += SDx(.,p)^T (Sy^T fx) + Sx(.,p)^T (SDy^T fy);  fz -> shared
//            (in place over the consumed column of wx), then c = Sy^T Sx^T fz
//   phase 3 (Y-slab), per x node i:        out = Sz^T a + SDz^T c, scatter
// Each lane overwrites only its own slab's region of the buffers between the two
// exchanges, so only the two exchanges (and the end of a group) need a __syncwarp.
template <int N> struct Stride {
  // per-cell stride of the exchange buffers, padded where that lowers bank conflicts of
  // the two exchange patterns (offsets N*s and N*N*s within a cell)
  static constexpr int CELL = N * N * N + ((N == 3 || N == 5) ? 0 : 1);
};

// Inverse-Jacobian formulation (geo = [group][x point p][y point q][10][LANES]: J^{-1} row by
// row, then JxW): the physical gradient J^{-T} grad_ref, times JxW, and back with J^{-1}
// (include/kernels/portable_local_laplace_operator.h:329-347).
template <int N, typename T>
__device__ __forceinline__ void invjac_flux(const T *__restrict__ geo, int64_t g, int lane, int q, int p,
                                            uint64_t pol, T dx, T dy, T dz, T (&f)[3]) {
  constexpr int LANES = Layout<N>::LANES, N2 = Layout<N>::N2;
  const T *gp = geo + g * (N2 * 10 * LANES) + (p * N + q) * 10 * LANES + lane;
  T iv[9];
#pragma unroll
  for (int m = 0; m < 9; ++m) iv[m] = ld_stream(gp + m * LANES, pol);
  const T jw = ld_stream(gp + 9 * LANES, pol);
  T gx[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) gx[k] = jw * (iv[k] * dx + iv[3 + k] * dy + iv[6 + k] * dz);
#pragma unroll
  for (int d = 0; d < 3; ++d) f[d] = iv[3 * d] * gx[0] + iv[3 * d + 1] * gx[1] + iv[3 * d + 2] * gx[2];
}

// the six components of the tensor at point (p, q, r) of cell c
template <int N, typename T, int GEOM>
__device__ __forceinline__ void load_g6(const T *__restrict__ geo, const T *__restrict__ coef, const Tab<N, T> &tab,
                                        int64_t cell, int r, int q, int p, T wr, T (&c)[6]) {
  using CD = CellData<N, line_layout(N, GEOM)>;
  if (GEOM == 0) {
#pragma unroll
    for (int m = 0; m < 6; ++m) c[m] = __ldg(geo + CD::template geo<T>(cell, p, q, r, m, 6));
  } else {
    T w = wr * tab.W[q] * tab.W[p];
    if (GEOM == 2) w *= __ldg(coef + CD::point(cell, p, q, r));
#pragma unroll
    for (int m = 0; m < 6; ++m) c[m] = w * __ldg(geo + cell * 8 + m);
  }
}

// Shared memory per warp of vmult_slab_kernel: 3 exchange buffers, plus (SMEM_G) the
// geometry column ring and its two mbarriers, plus (PIPE) one group's index block.
template <int N, typename T, bool SMEM_G, int PIPE = 0> struct SlabSmem {
  static constexpr size_t XCHG = size_t(3) * Layout<N>::CPW * Stride<N>::CELL * sizeof(T);
  static constexpr size_t CHUNK = size_t(N) * 6 * Layout<N>::LANES * sizeof(T); // one x column
  static constexpr size_t GEO = SMEM_G ? 2 * CHUNK : 0;                         // two-slot ring
  static constexpr size_t IDX = PIPE ? size_t(Layout<N>::N2) * Layout<N>::LANES * 4 : 0; // one index block
  static constexpr size_t OFF_IDX = ((GEO + XCHG + 15) / 16) * 16;
  static constexpr size_t PER_WARP = OFF_IDX + ((IDX + 15) / 16) * 16 + (SMEM_G ? 16 : 0);
};

// SMEM_G: the x columns of each group's geometry (contiguous chunks) stream through a
// two-slot shared-memory ring; the copy of the next column (or of the next group's first
// column) is issued when a column starts, so it overlaps with that column's work.
// Warps share nothing (each has its own ring, barriers and buffers): any warps per block.
// PIPE 1: the next group's index block is copied into shared memory one group ahead by
// per-thread cp.async copies (each lane copies exactly the entries it later reads, so
// cp.async.wait_group alone orders them).
template <int N, typename T, int GEOM, bool SMEM_G, int PIPE = 0>
__global__ void __launch_bounds__(SMEM_G ? 256 : 128, (SMEM_G ? 1 : (sizeof(T) == 8 && !(GEOM == 2 && N == 3) ? 3 : 2)))
    vmult_slab_kernel(const __grid_constant__ Tab<N, T> tab, const T *__restrict__ src, T *__restrict__ dst,
                      const uint32_t *__restrict__ idx, const T *__restrict__ geo,
                      const T *__restrict__ coef, int64_t n_groups, unsigned int *err) {
  static_assert(N == 2 || N == 3, "degrees 1 and 2; line_kernels.cuh has the others");
  static_assert(GEOM == 0 || GEOM == 2 || GEOM == 3, "axis-aligned cells without a coefficient: vmult_box_kernel");
  using Lo = Layout<N>;
  constexpr int CPW = Lo::CPW, LANES = Lo::LANES, N2 = Lo::N2;
  constexpr int CS = Stride<N>::CELL;
  constexpr unsigned MASK = Lo::MASK;
  // even/odd contractions where they measured faster on B200 (N = 2 gains nothing, the FP64
  // runtime-loop variants spill); outer streaming loops in runtime form for FP64 direct loads
  constexpr bool EO = N == 3 && (SMEM_G || sizeof(T) == 4 || GEOM == 2);
  constexpr int UNR = (SMEM_G || sizeof(T) == 4 || EO) ? N : 1;
  using SM = SlabSmem<N, T, SMEM_G, PIPE>;
  constexpr int NCOMP = GEOM == 3 ? 10 : 6; // geometry values per quadrature point
  pdl_trigger();
  pdl_wait();
  src = pdl_after(src);
  geo = pdl_after(geo);
  coef = pdl_after(coef);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  if (lane >= LANES) return;
  const int e = lane / N;
  const int s = lane - e * N;
  unsigned char *wsm = smem_raw + (threadIdx.x >> 5) * SM::PER_WARP;
  T *ring = reinterpret_cast<T *>(wsm);                     // geometry column ring (SMEM_G)
  T *bufW = reinterpret_cast<T *>(wsm + SM::GEO) + e * CS;  // exchange buffers
  T *bufZ = bufW + CPW * CS;
  T *bufX = bufZ + CPW * CS;
  uint64_t *bars = reinterpret_cast<uint64_t *>(wsm + SM::PER_WARP - 16);
  uint32_t *ibuf = reinterpret_cast<uint32_t *>(wsm + SM::OFF_IDX) + lane; // [N2][LANES]
  constexpr int CHUNK_ELEMS = N * 6 * LANES;
  uint32_t chunk = 0; // columns consumed so far; slot = chunk & 1, parity = (chunk >> 1) & 1
  const int64_t warp0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  if (SMEM_G && GEOM == 0) {
    if (lane == 0) {
      mbar_init(&bars[0], 1);
      mbar_init(&bars[1], 1);
      if (warp0 < n_groups)
        bulk_load(ring, geo + warp0 * (N2 * 6 * LANES), CHUNK_ELEMS * sizeof(T), &bars[0], pol_first);
    }
    __syncwarp(MASK);
  }
  const T wr = line_weight<N, T>(tab.W, s); // Gauss weight of this lane's z point (coefficient geometry)

  // copy the index block of group gg; every call commits exactly one cp.async group
  auto issue_idx = [&](int64_t gg) {
    if (gg < n_groups) {
      const uint32_t *ip = idx + gg * (N2 * LANES) + lane;
#pragma unroll
      for (int a = 0; a < N2; ++a) cp_async(ibuf + a * LANES, ip + a * LANES, 4, 4, pol_first);
    }
    cp_async_commit();
  };
  if (PIPE == 1) issue_idx(warp0);

  for (int64_t g = warp0; g < n_groups; g += nwarps) {
    // the ring streams each column ahead already: an L2 prefetch as well only added traffic
    // (FP32 Q2 at 128^3 398 against 381 us)
    if ((GEOM == 0 || GEOM == 3) && !SMEM_G && lane == 0 && g + nwarps < n_groups)
      prefetch_l2(geo + (g + nwarps) * (N2 * NCOMP * LANES), N2 * NCOMP * LANES * sizeof(T), pol_first);
    const uint32_t *ig = idx + g * (N2 * LANES) + lane;

    // ---- phase 1: gather the Y-slab y = s, u[k][i] = src at node (i, s, k) ----
    {
      T u[N][N];
      if (PIPE == 1) cp_async_wait<0>(); // this group's index block
#pragma unroll
      for (int k = 0; k < N; ++k)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const uint32_t id = PIPE == 1 ? ibuf[(k * N + i) * LANES] : ld_stream(ig + (k * N + i) * LANES, pol_first);
          u[k][i] = (id != kInvalidIdx) ? ld_keep(src + id, pol_last) : T(0);
        }
      if constexpr (EO) {
        // x contractions t = Sx u, tx = SDx u by mirrored pairs of points (p, N-1-p): the
        // sums and differences of mirrored nodes replace u in place (u[k][i] = e_i and
        // u[k][N-1-i] = o_i for i < H)
        constexpr int H = N / 2, Q = (N + 1) / 2;
        // z contraction of one x point p in even/odd form: w = Sz t, wz = SDz t, wx = Sz tx
        auto zstore = [&](int p, const T(&t)[N], const T(&tx)[N]) {
          eo_apply<N, T, 1>(tab.eS, t, [&](int r, T v) { bufW[(r * N + s) * N + p] = v; });
          eo_apply<N, T, -1>(tab.eSD, t, [&](int r, T v) { bufZ[(r * N + s) * N + p] = v; });
          eo_apply<N, T, 1>(tab.eS, tx, [&](int r, T v) { bufX[(r * N + s) * N + p] = v; });
        };
#pragma unroll
        for (int k = 0; k < N; ++k)
#pragma unroll
          for (int i = 0; i < H; ++i) {
            const T a = u[k][i], b = u[k][N - 1 - i];
            u[k][i] = a + b;
            u[k][N - 1 - i] = a - b;
          }
#pragma unroll
        for (int p = 0; p < H; ++p) {
          T tp[N], tm[N], xp[N], xm[N];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            T es = (N & 1) ? tab.eS.C[p] * u[k][H] : T(0), os = T(0);
            T ed = (N & 1) ? tab.eSD.C[p] * u[k][H] : T(0), od = T(0);
#pragma unroll
            for (int i = 0; i < H; ++i) {
              es = fma(tab.eS.A[i * Q + p], u[k][i], es);
              os = fma(tab.eS.B[i * Q + p], u[k][N - 1 - i], os);
              ed = fma(tab.eSD.A[i * Q + p], u[k][i], ed);
              od = fma(tab.eSD.B[i * Q + p], u[k][N - 1 - i], od);
            }
            tp[k] = es + os;
            tm[k] = es - os;
            xp[k] = ed + od;
            xm[k] = od - ed;
          }
          zstore(p, tp, xp);
          zstore(N - 1 - p, tm, xm);
        }
        if (N & 1) {
          T t[N], tx[N];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            T a = tab.eS.C[H] * u[k][H], b = T(0);
#pragma unroll
            for (int i = 0; i < H; ++i) {
              a = fma(tab.eS.A[i * Q + H], u[k][i], a);
              b = fma(tab.eSD.B[i * Q + H], u[k][N - 1 - i], b);
            }
            t[k] = a;
            tx[k] = b;
          }
          zstore(H, t, tx);
        }
      } else {
#pragma unroll UNR
        for (int p = 0; p < N; ++p) {
          T t[N], tx[N];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            T a = T(0), b = T(0);
#pragma unroll
            for (int i = 0; i < N; ++i) {
              a = fma(tab.S[i * N + p], u[k][i], a);
              b = fma(tab.SD[i * N + p], u[k][i], b);
            }
            t[k] = a;
            tx[k] = b;
          }
          // z contraction: w = Sz t, wz = SDz t, wx = Sz tx at (z = r, y = s, x = p)
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
              bufW[o] = w;
              bufZ[o] = wz;
              bufX[o] = wx;
            }
        }
      }
    }
    if (PIPE == 1) issue_idx(g + nwarps); // the index block is consumed: refill it for the next group
    __syncwarp(MASK);

    // ---- phase 2: Z-slab z = s, streamed over the x point p ----
    T cd0 = T(0), cd3 = T(0), cd5 = T(0); // diagonal of the affine cell tensor
    if (GEOM == 2) {
      const T *cg = geo + (g * CPW + e) * 8;
      cd0 = __ldg(cg);
      cd3 = __ldg(cg + 3);
      cd5 = __ldg(cg + 5);
    }
    {
      T a[N][N]; // [j][i]
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) a[j][i] = T(0);
#pragma unroll UNR
      for (int p = 0; p < N; ++p) {
        const T *gcol = nullptr;
        if (SMEM_G && GEOM == 0) {
          // issue the next column (this group's p+1, or the next group's column 0) into the
          // other slot, whose previous column every lane finished with at the last syncwarp
          if (lane == 0) {
            const T *next = nullptr;
            if (p + 1 < N) next = geo + g * (N2 * 6 * LANES) + (p + 1) * CHUNK_ELEMS;
            else if (g + nwarps < n_groups) next = geo + (g + nwarps) * (N2 * 6 * LANES);
            if (next)
              bulk_load(ring + ((chunk + 1) & 1) * CHUNK_ELEMS, next, CHUNK_ELEMS * sizeof(T),
                        &bars[(chunk + 1) & 1], pol_first);
          }
          if (!mbar_wait_bounded(&bars[chunk & 1], (chunk >> 1) & 1, err, 1u << 24)) {
            if (lane == 0) mbar_wait_bounded(&bars[(chunk + 1) & 1], ((chunk + 1) >> 1) & 1, err, 1u << 24);
            if (PIPE == 1) cp_async_wait<0>();
            return; // the error flag is set; let copies in flight land before leaving
          }
          gcol = ring + (chunk & 1) * CHUNK_ELEMS;
        }
        T Wc[N], Zc[N], Xc[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const int o = (s * N + j) * N + p;
          Wc[j] = bufW[o];
          Zc[j] = bufZ[o];
          Xc[j] = bufX[o];
        }
        T fx[N], fy[N];
        if constexpr (EO) {
          // f = G grad u at the point (p, q) of this slab: fx, fy kept, fz -> own bufX region
          auto point = [&](int q, T dx, T dy, T dz) {
            if (GEOM == 0) {
              T gc[6];
              const T *gp = SMEM_G ? gcol + q * 6 * LANES + lane // the staged x column p
                                   : geo + g * (N2 * 6 * LANES) + (p * N + q) * 6 * LANES + lane;
#pragma unroll
              for (int m = 0; m < 6; ++m) gc[m] = SMEM_G ? gp[m * LANES] : ld_stream(gp + m * LANES, pol_first);
              fx[q] = gc[0] * dx + gc[1] * dy + gc[2] * dz;
              fy[q] = gc[1] * dx + gc[3] * dy + gc[4] * dz;
              bufX[(s * N + q) * N + p] = gc[2] * dx + gc[4] * dy + gc[5] * dz; // fz
            } else if (GEOM == 3) {
              T f3[3];
              invjac_flux<N, T>(geo, g, lane, q, p, pol_first, dx, dy, dz, f3);
              fx[q] = f3[0];
              fy[q] = f3[1];
              bufX[(s * N + q) * N + p] = f3[2]; // fz
            } else {
              // affine cells are axis-aligned boxes: the cell tensor is diagonal (rr, ss, tt)
              T w = wr * tab.W[q] * tab.W[p];
              w *= ld_stream(coef + g * (N2 * LANES) + (q * N + p) * LANES + lane, pol_first);
              fx[q] = (w * cd0) * dx;
              fy[q] = (w * cd3) * dy;
              bufX[(s * N + q) * N + p] = (w * cd5) * dz; // fz
            }
          };
          // dx = Sy wx, dy = SDy w, dz = Sy wz along the column; y1 = Sy^T fx, y2 = SDy^T fy
          T dxv[N], dyv[N], dzv[N], y1v[N], y2v[N];
          eo_apply<N, T, 1>(tab.eS, Xc, [&](int q, T v) { dxv[q] = v; });
          eo_apply<N, T, -1>(tab.eSD, Wc, [&](int q, T v) { dyv[q] = v; });
          eo_apply<N, T, 1>(tab.eS, Zc, [&](int q, T v) { dzv[q] = v; });
#pragma unroll
          for (int q = 0; q < N; ++q) point(q, dxv[q], dyv[q], dzv[q]);
          eo_apply<N, T, 1>(tab.eST, fx, [&](int j, T v) { y1v[j] = v; });
          eo_apply<N, T, -1>(tab.eSDT, fy, [&](int j, T v) { y2v[j] = v; });
#pragma unroll
          for (int j = 0; j < N; ++j)
#pragma unroll
            for (int i = 0; i < N; ++i) {
              a[j][i] = fma(tab.SD[i * N + p], y1v[j], a[j][i]);
              a[j][i] = fma(tab.S[i * N + p], y2v[j], a[j][i]);
            }
        } else {
#pragma unroll
          for (int q = 0; q < N; ++q) {
            T dx = T(0), dy = T(0), dz = T(0);
#pragma unroll
            for (int j = 0; j < N; ++j) {
              dx = fma(tab.S[j * N + q], Xc[j], dx);
              dy = fma(tab.SD[j * N + q], Wc[j], dy);
              dz = fma(tab.S[j * N + q], Zc[j], dz);
            }
            // f = G grad u at the point (p, q) of this slab: fx, fy kept, fz -> own bufX region
            if (GEOM == 0) {
              T gc[6];
              const T *gp = SMEM_G ? gcol + q * 6 * LANES + lane // the staged x column p
                                   : geo + g * (N2 * 6 * LANES) + (p * N + q) * 6 * LANES + lane;
#pragma unroll
              for (int m = 0; m < 6; ++m) gc[m] = SMEM_G ? gp[m * LANES] : ld_stream(gp + m * LANES, pol_first);
              fx[q] = gc[0] * dx + gc[1] * dy + gc[2] * dz;
              fy[q] = gc[1] * dx + gc[3] * dy + gc[4] * dz;
              bufX[(s * N + q) * N + p] = gc[2] * dx + gc[4] * dy + gc[5] * dz; // fz
            } else if (GEOM == 3) {
              T f3[3];
              invjac_flux<N, T>(geo, g, lane, q, p, pol_first, dx, dy, dz, f3);
              fx[q] = f3[0];
              fy[q] = f3[1];
              bufX[(s * N + q) * N + p] = f3[2]; // fz
            } else {
              T w = wr * tab.W[q] * tab.W[p];
              w *= ld_stream(coef + g * (N2 * LANES) + (q * N + p) * LANES + lane, pol_first);
              fx[q] = (w * cd0) * dx;
              fy[q] = (w * cd3) * dy;
              bufX[(s * N + q) * N + p] = (w * cd5) * dz; // fz
            }
          }
#pragma unroll
          for (int j = 0; j < N; ++j) {
            T y1 = T(0), y2 = T(0);
#pragma unroll
            for (int q = 0; q < N; ++q) {
              y1 = fma(tab.S[j * N + q], fx[q], y1);
              y2 = fma(tab.SD[j * N + q], fy[q], y2);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) {
              a[j][i] = fma(tab.SD[i * N + p], y1, a[j][i]);
              a[j][i] = fma(tab.S[i * N + p], y2, a[j][i]);
            }
          }
        }
        if (SMEM_G && GEOM == 0) {
          __syncwarp(MASK); // this slot may be refilled from the next column on
          ++chunk;
        }
      }
      // a -> own slab region of bufW (all of this lane's reads of it are done)
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) bufW[(s * N + j) * N + i] = a[j][i];
    }
    {
      // c = Sy^T Sx^T fz from this lane's fz region, into its own region of bufZ
      T c[N][N];
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) c[j][i] = T(0);
#pragma unroll UNR
      for (int q = 0; q < N; ++q) {
        T fz[N];
#pragma unroll
        for (int p = 0; p < N; ++p) fz[p] = bufX[(s * N + q) * N + p];
        if constexpr (EO) {
          T x3v[N]; // x3 = Sx^T fz along this row
          eo_apply<N, T, 1>(tab.eST, fz, [&](int i, T v) { x3v[i] = v; });
#pragma unroll
          for (int i = 0; i < N; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) c[j][i] = fma(tab.S[j * N + q], x3v[i], c[j][i]);
        } else {
#pragma unroll
          for (int i = 0; i < N; ++i) {
            T x3 = T(0);
#pragma unroll
            for (int p = 0; p < N; ++p) x3 = fma(tab.S[i * N + p], fz[p], x3);
#pragma unroll
            for (int j = 0; j < N; ++j) c[j][i] = fma(tab.S[j * N + q], x3, c[j][i]);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < N; ++j)
#pragma unroll
        for (int i = 0; i < N; ++i) bufZ[(s * N + j) * N + i] = c[j][i];
    }
    __syncwarp(MASK);

    // ---- phase 3: Y-slab y = s, out = Sz^T a + SDz^T c, scatter ----
#pragma unroll UNR
    for (int i = 0; i < N; ++i) {
      T A[N], Cc[N];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        A[r] = bufW[(r * N + s) * N + i];
        Cc[r] = bufZ[(r * N + s) * N + i];
      }
      // out = Sz^T a + SDz^T c
      T v[N];
      if constexpr (EO) {
        eo_apply<N, T, 1>(tab.eST, A, [&](int k, T x) { v[k] = x; });
        eo_apply<N, T, -1>(tab.eSDT, Cc, [&](int k, T x) { v[k] += x; });
      } else {
#pragma unroll
        for (int k = 0; k < N; ++k) {
          v[k] = T(0);
#pragma unroll
          for (int r = 0; r < N; ++r) {
            v[k] = fma(tab.S[k * N + r], A[r], v[k]);
            v[k] = fma(tab.SD[k * N + r], Cc[r], v[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < N; ++k) {
        const uint32_t id = ld_stream(ig + (k * N + i) * LANES, pol_first);
        if (id != kInvalidIdx) red_keep(dst + id, v[k], pol_last);
      }
    }
    __syncwarp(MASK); // buffers are rewritten by the next group
  }
  if (PIPE == 1) cp_async_wait<0>(); // no copy may land after the warp has left
}

// Diagonal of the cell operator summed into diag (atomic), same layout and slab scheme:
// diag(i,j,k) = sum_q sum_{d1,d2} G_{d1 d2}(q) d_{d1}phi_ijk(q) d_{d2}phi_ijk(q), factored
// by the z-factor of each component pair (S^2 for xx, xy, yy; S*SD for xz, yz; SD^2 for zz).
template <int N, typename T, int GEOM>
__global__ void __launch_bounds__(128) diag_slab_kernel(const Tab2<N, T> tab,
                                                        T *__restrict__ diag,
                                                        const uint32_t *__restrict__ idx,
                                                        const T *__restrict__ geo,
                                                        const T *__restrict__ coef,
                                                        int64_t n_groups) {
  using Lo = Layout<N>;
  using CD = CellData<N, line_layout(N, GEOM)>;
  constexpr int CPW = Lo::CPW, LANES = Lo::LANES, N3 = Lo::N3;
  constexpr unsigned MASK = Lo::MASK;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  if (lane >= LANES) return;
  const int e = lane / N;
  const int s = lane - e * N;
  T *b0 = reinterpret_cast<T *>(smem_raw) + (threadIdx.x >> 5) * (3 * CPW * N3) + e * N3;
  T *b1 = b0 + CPW * N3;
  T *b2 = b1 + CPW * N3;
  const int64_t warp0 = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = (int64_t(gridDim.x) * blockDim.x) >> 5;
  const T *S2 = tab.S2, *SS = tab.SS, *D2 = tab.D2;
  T wr = tab.W[0];
#pragma unroll
  for (int r = 1; r < N; ++r)
    if (s == r) wr = tab.W[r];
  for (int64_t g = warp0; g < n_groups; g += nwarps) {
    // Z-slab (z = s): G at the points of the slab
    T gxx[N][N], gxy[N][N], gyy[N][N], gxz[N][N], gyz[N][N], gzz[N][N];
#pragma unroll
    for (int q = 0; q < N; ++q)
#pragma unroll
      for (int p = 0; p < N; ++p) {
        T c[6];
        if (GEOM == 0) {
#pragma unroll
          for (int m = 0; m < 6; ++m) c[m] = __ldg(geo + CD::template geo<T>(g * CPW + e, p, q, s, m, 6));
        } else if (GEOM == 3) {
          // G = JxW J^{-1} J^{-T} from the inverse-Jacobian layout, in the order of G
          T iv[9];
#pragma unroll
          for (int m = 0; m < 9; ++m) iv[m] = __ldg(geo + CD::template geo<T>(g * CPW + e, p, q, s, m, 10));
          const T jw = __ldg(geo + CD::template geo<T>(g * CPW + e, p, q, s, 9, 10));
          int m = 0;
#pragma unroll
          for (int d1 = 0; d1 < 3; ++d1)
#pragma unroll
            for (int d2 = d1; d2 < 3; ++d2)
              c[m++] = jw * (iv[3 * d1] * iv[3 * d2] + iv[3 * d1 + 1] * iv[3 * d2 + 1] + iv[3 * d1 + 2] * iv[3 * d2 + 2]);
        } else {
          const T *cg = geo + (g * CPW + e) * 8;
          T w = wr * tab.W[q] * tab.W[p];
          if (GEOM == 2) w *= __ldg(coef + CD::point(g * CPW + e, p, q, s));
#pragma unroll
          for (int m = 0; m < 6; ++m) c[m] = w * __ldg(cg + m);
        }
        gxx[q][p] = c[0];
        gxy[q][p] = T(2) * c[1];
        gxz[q][p] = T(2) * c[2];
        gyy[q][p] = c[3];
        gyz[q][p] = T(2) * c[4];
        gzz[q][p] = c[5];
      }
    // x then y contractions, grouped by the z factor
#pragma unroll
    for (int i = 0; i < N; ++i) {
      T ua[N], ub[N], uc[N], va[N], vb[N], wc[N]; // per q
#pragma unroll
      for (int q = 0; q < N; ++q) {
        T a = 0, b = 0, c = 0, d = 0, f = 0, h = 0;
#pragma unroll
        for (int p = 0; p < N; ++p) {
          a = fma(D2[i * N + p], gxx[q][p], a);
          b = fma(SS[i * N + p], gxy[q][p], b);
          c = fma(S2[i * N + p], gyy[q][p], c);
          d = fma(SS[i * N + p], gxz[q][p], d);
          f = fma(S2[i * N + p], gyz[q][p], f);
          h = fma(S2[i * N + p], gzz[q][p], h);
        }
        ua[q] = a; ub[q] = b; uc[q] = c; va[q] = d; vb[q] = f; wc[q] = h;
      }
#pragma unroll
      for (int j = 0; j < N; ++j) {
        T A = 0, B = 0, Cz = 0;
#pragma unroll
        for (int q = 0; q < N; ++q) {
          A = fma(S2[j * N + q], ua[q], A);
          A = fma(SS[j * N + q], ub[q], A);
          A = fma(D2[j * N + q], uc[q], A);
          B = fma(S2[j * N + q], va[q], B);
          B = fma(SS[j * N + q], vb[q], B);
          Cz = fma(S2[j * N + q], wc[q], Cz);
        }
        b0[(s * N + j) * N + i] = A;
        b1[(s * N + j) * N + i] = B;
        b2[(s * N + j) * N + i] = Cz;
      }
    }
    __syncwarp(MASK);
    // Y-slab (y = s): z contraction and scatter
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        T v = 0;
#pragma unroll
        for (int r = 0; r < N; ++r) {
          v = fma(S2[k * N + r], b0[(r * N + s) * N + i], v);
          v = fma(SS[k * N + r], b1[(r * N + s) * N + i], v);
          v = fma(D2[k * N + r], b2[(r * N + s) * N + i], v);
        }
        const uint32_t id = __ldg(idx + CD::idx(g * CPW + e, i, s, k));
        if (id != kInvalidIdx) atomic_add(diag + id, v);
      }
    __syncwarp(MASK);
  }
}

} // namespace kern

// host-side launchers, one translation unit per degree (laplace_p<degree>.cu)
struct SlabLaunch {
  const void *src;
  void *dst;
  const uint32_t *idx;
  const uint32_t *patch_idx; // null: apply the cells one by one
  const void *geo;
  const void *coef;
  int64_t n_groups, n_cells;
  int geom; // 0 full, 1 affine, 2 affine + coefficient, 3 inverse Jacobian
  double affine[3]; // diagonal of the affine cell tensor (geom 1 and 2)
  int dtype;
  int64_t resident_warps; // warps of the diagonal kernel resident on the whole device
  unsigned int *err; // device flag set when a bounded wait gives up
  cudaStream_t stream;
  const double *S, *SD, *D, *W; // host tables (double), converted to the kernel type
  int64_t *units, *launched; // if set: receive the vmult's work units and the warps (blocks) sharing them
};
void launch_vmult_p1(const SlabLaunch &);
void launch_vmult_p2(const SlabLaunch &);
void launch_vmult_p3(const SlabLaunch &);
void launch_vmult_p4(const SlabLaunch &);
void launch_vmult_p5(const SlabLaunch &);
void launch_vmult_p6(const SlabLaunch &);
void launch_diag_p1(const SlabLaunch &);
void launch_diag_p2(const SlabLaunch &);
void launch_diag_p3(const SlabLaunch &);
void launch_diag_p4(const SlabLaunch &);
void launch_diag_p5(const SlabLaunch &);
void launch_diag_p6(const SlabLaunch &);
// resident warps per SM of the diagonal kernels
int occupancy_diag_p1(int dtype, int geom);
int occupancy_diag_p2(int dtype, int geom);
int occupancy_diag_p3(int dtype, int geom);
int occupancy_diag_p4(int dtype, int geom);
int occupancy_diag_p5(int dtype, int geom);
int occupancy_diag_p6(int dtype, int geom);

} // namespace pmg
