// Cell kernel of the axis-aligned Q_p Laplace operators without a coefficient on patches of 2 x 2 x 2
// cells, one thread per line of a patch: what vmult_box_kernel (line_kernels.cuh) computes for the eight
// cells, with the nodes that the cells share gathered, exchanged and added to the result once.
//
// That kernel is bound by the load/store pipe, half of whose work is the gather and the scatter (FP32
// Q4: 59 of 125 wavefronts per cell).  A patch has (2p+1)^3 nodes where its cells have 8 (p+1)^3 (Q4 729
// for 1000, Q6 2197 for 2744), and its lines, over eight cells that follow one another in the numbering,
// lie closer together in memory: 79 wavefronts per cell, of which 38 are gather and scatter.  A line is
// contracted cell by cell with the tables of a cell, and the results at its middle node are added.
//
// The steps are those of vmult_box_kernel.  Every value stays in the place of its node and a thread
// writes only the line that it has read, so the exchanges need two buffers and a barrier each.
#pragma once

#include "line_kernels.cuh"

namespace pmg {
namespace kern {

// out = the sum of the two cells' M(i, q) in_i along a line of a patch; f(q, .) is called once for every node q
template <int N, typename T, typename F>
__device__ __forceinline__ void eo_patch(const EvenOdd<N, T> &m, const T (&in)[2 * N - 1], F &&f) {
  T l[N], mid = T(0);
#pragma unroll
  for (int i = 0; i < N; ++i) l[i] = in[i];
  eo_apply<N, T, 1>(m, l, [&](int q, T v) {
    if (q == N - 1) mid = v;
    else f(q, v);
  });
#pragma unroll
  for (int i = 0; i < N; ++i) l[i] = in[N - 1 + i];
  eo_apply<N, T, 1>(m, l, [&](int q, T v) {
    if (q == 0) f(N - 1, mid + v);
    else f(N - 1 + q, v);
  });
}

// Buffer strides: node (i, j, k) of patch e at e*CS + i*I + j*J + k*K, those with the fewest bank
// conflicts of an exhaustive search over permuted, padded strides for the accesses along z (lanes
// over i, then j), y (lanes over i, then k; over k, then i where YK) and x (lanes over j, then k; over
// k, then j where XK).
template <int I_, int J_, int K_, int CS_, int YK_, int XK_> struct PLayout {
  static constexpr int I = I_, J = J_, K = K_, CS = CS_, YK = YK_, XK = XK_;
};
template <int N, typename T> struct PatchLayout;
template <> struct PatchLayout<3, float> : PLayout<1, 56, 5, 249, 0, 0> {};
template <> struct PatchLayout<3, double> : PLayout<1, 9, 53, 253, 0, 1> {};
template <> struct PatchLayout<4, float> : PLayout<1, 8, 71, 481, 0, 1> {};
template <> struct PatchLayout<4, double> : PLayout<1, 8, 71, 481, 0, 1> {};
template <> struct PatchLayout<5, float> : PLayout<1, 81, 9, 729, 0, 1> {};
template <> struct PatchLayout<5, double> : PLayout<1, 81, 9, 729, 1, 1> {};
template <> struct PatchLayout<6, float> : PLayout<1, 11, 131, 1431, 1, 0> {};
template <> struct PatchLayout<6, double> : PLayout<1, 11, 123, 1351, 0, 0> {};
template <> struct PatchLayout<7, float> : PLayout<1, 13, 197, 2533, 1, 0> {};
template <> struct PatchLayout<7, double> : PLayout<1, 13, 173, 2245, 0, 0> {};

// PPB patches per block, registers allocated for MINB blocks per SM
template <int PPB_, int MINB_> struct PatchShape {
  static constexpr int PPB = PPB_, MINB = MINB_;
};
template <int N, typename SH> constexpr int patch_threads() {
  return (SH::PPB * (2 * N - 1) * (2 * N - 1) + 31) / 32 * 32;
}
template <int N, typename T, typename SH> constexpr size_t patch_smem() {
  return size_t(2) * SH::PPB * PatchLayout<N, T>::CS * sizeof(T);
}

// no coefficient: (cx, cy, cz) = vol / h^2 per direction
template <int N, typename T, typename SH>
__global__ void __launch_bounds__(patch_threads<N, SH>(), SH::MINB)
    vmult_box_patch_kernel(const __grid_constant__ BoxTab<N, T> tab, const T *__restrict__ src, T *__restrict__ dst,
                           const uint32_t *__restrict__ idx, T cx, T cy, T cz, int64_t n_patches) {
  using L = PatchLayout<N, T>;
  constexpr int n1 = 2 * N - 1, PPB = SH::PPB;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T *A0 = reinterpret_cast<T *>(smem_raw), *A1 = A0 + PPB * L::CS;
  const int e = threadIdx.x / (n1 * n1), r = threadIdx.x - e * (n1 * n1), ra = r % n1, rb = r / n1, o0 = e * L::CS;
  const bool active = e < PPB;
  const int64_t p = int64_t(blockIdx.x) * PPB + e;
  const int z = o0 + ra * L::I + rb * L::J;
  const uint64_t pol_first = policy_evict_first(), pol_last = policy_evict_last();
  uint32_t id[n1];
  {
    const uint32_t *ip = idx + p * (n1 * n1 * n1) + r; // (fixed at setup: read before the wait)
#pragma unroll
    for (int k = 0; k < n1; ++k) id[k] = active && p < n_patches ? ld_keep_early(ip + k * (n1 * n1), pol_first) : kInvalidIdx;
  }
  pdl_wait();
  src = pdl_after(src);
  if (active) {
    T u[n1];
#pragma unroll
    for (int k = 0; k < n1; ++k) u[k] = id[k] != kInvalidIdx ? ld_keep(src + id[k], pol_last) : T(0);
    eo_patch<N, T>(tab.eM, u, [&](int q, T v) { A0[z + q * L::K] = v; });
    eo_patch<N, T>(tab.eK, u, [&](int q, T v) { A1[z + q * L::K] = cz * v; });
  }
  __syncthreads();
  if (active) {
    const int y = o0 + (L::YK ? rb * L::I + ra * L::K : ra * L::I + rb * L::K);
    T a[n1], o[n1];
#pragma unroll
    for (int j = 0; j < n1; ++j) a[j] = A0[y + j * L::J];
    eo_patch<N, T>(tab.eM, a, [&](int q, T v) { A0[y + q * L::J] = v; });
    eo_patch<N, T>(tab.eK, a, [&](int q, T v) { o[q] = v; });
#pragma unroll
    for (int j = 0; j < n1; ++j) a[j] = A1[y + j * L::J];
    eo_patch<N, T>(tab.eM, a, [&](int q, T v) { A1[y + q * L::J] = fma(cy, o[q], v); });
  }
  __syncthreads();
  if (active) {
    const int x = o0 + (L::XK ? rb * L::J + ra * L::K : ra * L::J + rb * L::K);
    T a[n1], o[n1];
#pragma unroll
    for (int i = 0; i < n1; ++i) a[i] = A0[x + i * L::I];
    eo_patch<N, T>(tab.eK, a, [&](int q, T v) { o[q] = v; });
#pragma unroll
    for (int i = 0; i < n1; ++i) a[i] = A1[x + i * L::I];
    eo_patch<N, T>(tab.eM, a, [&](int q, T v) { A0[x + q * L::I] = fma(cx, o[q], v); });
  }
  __syncthreads();
  if (active) {
#pragma unroll
    for (int k = 0; k < n1; ++k)
      if (id[k] != kInvalidIdx) red_keep(dst + id[k], A0[z + k * L::K], pol_last);
  }
}

} // namespace kern
} // namespace pmg
