// Launchers of the vmult and diagonal kernels for one polynomial degree.  Included by
// laplace_p<d>.cu with PMG_DEGREE defined, so each degree compiles as its own translation unit.
#pragma once

#include <algorithm>
#include <map>
#include <mutex>
#include <set>
#include <utility>

#include "fields.hpp"
#include "laplace_kernels.cuh"
#include "line_kernels.cuh"
#include "line_tables.hpp"
#include "patch_kernels.cuh"
#include "pdl.cuh"
#include "pmg_internal.hpp"

#ifndef PMG_DEGREE
#error "define PMG_DEGREE before including laplace_launch.cuh"
#endif

#define PMG_CAT2(a, b) a##b
#define PMG_CAT(a, b) PMG_CAT2(a, b)

namespace pmg {
namespace {

constexpr int kN = PMG_DEGREE + 1;
constexpr int kWarpsPerBlock = 4;

template <typename T> kern::Tab<kN, T> make_tab(const SlabLaunch &L) {
  kern::Tab<kN, T> t;
  for (int a = 0; a < kN * kN; ++a) {
    t.S[a] = (T)L.S[a];
    t.SD[a] = (T)L.SD[a];
    t.D[a] = (T)L.D[a];
  }
  for (int a = 0; a < kN; ++a) t.W[a] = (T)L.W[a];
  kern::fill_even_odd<kN>(t, L.S, L.SD);
  return t;
}

template <typename T> kern::Tab2<kN, T> make_tab2(const SlabLaunch &L) {
  kern::Tab2<kN, T> t;
  for (int a = 0; a < kN * kN; ++a) {
    t.S2[a] = (T)(L.S[a] * L.S[a]);
    t.SS[a] = (T)(L.S[a] * L.SD[a]);
    t.D2[a] = (T)(L.SD[a] * L.SD[a]);
  }
  for (int a = 0; a < kN; ++a) t.W[a] = (T)L.W[a];
  return t;
}

template <typename T> constexpr size_t diag_smem() {
  return size_t(kWarpsPerBlock) * 3 * kern::Layout<kN>::CPW * kern::Layout<kN>::N3 * sizeof(T);
}

// cudaFuncSetAttribute for the dynamic shared memory, once per device and kernel
template <typename K> void allow_smem(K kernel, size_t bytes) {
  static std::mutex mu;
  static std::set<std::pair<int, const void *>> done;
  int dev = 0;
  PMG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(dev, reinterpret_cast<const void *>(kernel));
  if (done.count(key)) return;
  PMG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  done.insert(key);
}

// ---- line kernels ----
// Cells per block, cells per warp (0: lines follow one another across the warps of a block) and
// the blocks per SM that registers are allocated for.  The fastest of the shapes measured on
// B200 (64^3 cells, Q5 and Q6 32^3, Q6 with a coefficient 48^3; time in us with the shape next
// in line): one warp per pair of Q3 cells needs no block barrier (FP64 full geometry 163; Q4 has
// 25 lines, which leave 7 lanes of a warp idle: 381 against 376 in blocks of five cells); Q5 and Q6
// fill 3 cells' lines into 4 and 5 warps.  MINB trades registers for warps: FP64 Q4 full geometry at
// 4 / 6 / 7 blocks 423 / 376 / 405, Q6 with a coefficient at 4 / 6 blocks 339 / 328.
template <typename T, int GEOM> constexpr auto line_shape() {
  constexpr bool d = sizeof(T) == 8;
  using kern::LineShape;
  if constexpr (GEOM == 1) { // vmult_box_kernel
    if constexpr (kN == 2) return LineShape<32, 8, 12>{};
    else if constexpr (kN == 3) return LineShape<14, 0, 8>{};
    else if constexpr (kN == 4) return LineShape<16, 2, 5>{};
    else if constexpr (kN == 5) return LineShape<2, 1, 12>{};
    else if constexpr (kN == 6) return LineShape<3, 0, 9>{};
    else return LineShape<3, 0, 6>{};
  } else if constexpr (GEOM == 2) {
    if constexpr (kN == 2) return LineShape<16, 8, 20>{};
    else if constexpr (kN == 4) return LineShape<8, 2, 6>{};
    else if constexpr (kN == 5) return LineShape<2, 1, 12>{};
    else if constexpr (kN == 6) return LineShape<3, 0, 9>{};
    else return LineShape<3, 0, 6>{};
  } else {
    if constexpr (kN == 4 && d) return LineShape<2, 2, 24>{};
    else if constexpr (kN == 4) return LineShape<8, 2, 10>{};
    else if constexpr (kN == 5 && d) return LineShape<5, 0, 6>{};
    else if constexpr (kN == 5) return LineShape<2, 1, 10>{};
    else if constexpr (kN == 6) return LineShape<3, 0, d ? 6 : 8>{};
    else return LineShape<3, 0, d ? 4 : 7>{};
  }
}

// The same for FP32 in pairs of cells (CPB and WC count pairs), degrees 3 to 6.  Half the arithmetic
// instructions, and the exchanges move 8 bytes per lane.  us, pairs against single cells, 64^3 cells
// (Q5 32^3, Q6 48^3) with full geometry / a coefficient / neither: Q3 98 / 67 / 48 against 102 / 76 / 75,
// Q4 226 / 152 / 105 against 234 / 187 / 127, Q5 53 / 34 / 21 against 58 / 41 / 25, Q6 274 / 188 / 113
// against 285 / 213 / 123 (Q4 without a coefficient in blocks of ten pairs: 105 alone, but 59 against 53 at
// 64 x 64 x 32, between the updates of a smoother).  On 16^3 cells and fewer both take as long as a launch.
template <int GEOM> constexpr auto pair_shape() {
  using kern::LineShape;
  if constexpr (GEOM == 1) {
    if constexpr (kN == 4) return LineShape<4, 2, 10>{};
    else if constexpr (kN == 5) return LineShape<4, 1, 8>{};
    else if constexpr (kN == 6) return LineShape<3, 0, 5>{};
    else return LineShape<3, 0, 4>{};
  } else if constexpr (GEOM == 2) {
    if constexpr (kN == 4) return LineShape<4, 2, 10>{};
    else if constexpr (kN == 5) return LineShape<4, 1, 8>{};
    else if constexpr (kN == 6) return LineShape<8, 0, 2>{};
    else return LineShape<3, 0, 5>{};
  } else {
    if constexpr (kN == 4) return LineShape<2, 2, 20>{};
    else if constexpr (kN == 5) return LineShape<4, 1, 6>{};
    else if constexpr (kN == 6) return LineShape<3, 0, 5>{};
    else return LineShape<3, 0, 3>{};
  }
}

template <typename V, int GEOM, typename SH> void line_launch_as(const SlabLaunch &L) {
  using T = typename kern::Elem<V>::T;
  constexpr int cells = SH::CPB * kern::Elem<V>::CELLS;
  const int64_t blocks = (L.n_cells + cells - 1) / cells;
  constexpr int threads = kern::line_threads<kN, SH>();
  const T *src = static_cast<const T *>(L.src);
  T *dst = static_cast<T *>(L.dst);
  const V c0 = (V)L.affine[0], c1 = (V)L.affine[1], c2 = (V)L.affine[2];
  if constexpr (GEOM == 1) {
    constexpr size_t smem = kern::box_smem<kN, V, SH>();
    static_assert(smem <= 48 * 1024, "no opt-in for the dynamic shared memory");
    launch_dependent(kern::vmult_box_kernel<kN, V, SH>, (unsigned)blocks, threads, smem, L.stream, box_tables<kN, V>(), src,
                     dst, L.idx, c0, c1, c2, L.n_cells);
  } else {
    constexpr size_t smem = kern::line_smem<kN, V, SH>();
    static_assert(smem <= 48 * 1024, "no opt-in for the dynamic shared memory");
    launch_dependent(kern::vmult_line_kernel<kN, V, GEOM, SH>, (unsigned)blocks, threads, smem, L.stream,
                     line_tables<kN, V>(), src, dst, L.idx, static_cast<const T *>(L.geo),
                     static_cast<const T *>(L.coef), c0, c1, c2, L.n_cells);
  }
  if (L.units) *L.units = L.n_cells;
  if (L.launched) *L.launched = blocks;
}
// Patches per block (cubes of several small lines share one) and blocks per SM, the fastest measured; cells
// alone, us, patches against cells (FP64 / FP32; 64^3 cells, Q5 32^3, Q6 48^3): Q2 31 / 21 against 52 / 33,
// Q3 72 / 45 against 85 / 52, Q4 138 / 84 against 176 / 109, Q5 33 / 23 against 41 / 27, Q6 164 / 101 against
// 216 / 119.  With a coefficient per point only the nodes are shared: patches 4 % faster at Q4 (257 / 149
// against 267 / 156) and slower at Q6 (373 with spills / 196 against 335 / 194), not enough for a kernel
// of their own: cells.
template <typename T> constexpr auto patch_shape() {
  [[maybe_unused]] constexpr bool d = sizeof(T) == 8;
  using kern::PatchShape;
  if constexpr (kN == 3) return PatchShape<5, 6>{};
  else if constexpr (kN == 4) return PatchShape<5, d ? 5 : 4>{};
  else if constexpr (kN == 5) return PatchShape<1, d ? 10 : 8>{};
  else if constexpr (kN == 6) return PatchShape<1, 8>{};
  else return PatchShape<1, 4>{};
}
template <typename T> void patch_launch(const SlabLaunch &L) {
  using SH = decltype(patch_shape<T>());
  constexpr int threads = kern::patch_threads<kN, SH>();
  constexpr size_t smem = kern::patch_smem<kN, T, SH>();
  static_assert(smem <= 48 * 1024, "no opt-in for the dynamic shared memory");
  const int64_t n = L.n_cells / 8, blocks = (n + SH::PPB - 1) / SH::PPB;
  launch_dependent(kern::vmult_box_patch_kernel<kN, T, SH>, (unsigned)blocks, threads, smem, L.stream, box_tables<kN, T>(),
                   static_cast<const T *>(L.src), static_cast<T *>(L.dst), L.patch_idx, (T)L.affine[0], (T)L.affine[1],
                   (T)L.affine[2], n);
  if (L.units) *L.units = L.n_cells;
  if (L.launched) *L.launched = blocks;
}

template <typename T, int GEOM> void line_launch(const SlabLaunch &L) {
  if constexpr (kern::patch_layout(kN, GEOM)) {
    if (L.patch_idx) return patch_launch<T>(L);
  }
  if constexpr (sizeof(T) == 4 && GEOM != 3 && kN >= 4) line_launch_as<kern::F2, GEOM, decltype(pair_shape<GEOM>())>(L);
  else line_launch_as<T, GEOM, decltype(line_shape<T, GEOM>())>(L);
}

// ---- slab kernels (degrees 1 and 2) ----
// Full geometry streams through the shared-memory column ring (TMA), except FP32 degree 1,
// whose unrolled direct loads hide the latency at 8 warps/SM; the ring variant's index block is
// copied one group ahead for FP64 degree 2 (677 -> 657 us at 128^3).
template <typename T, int GEOM> constexpr bool use_ring() { return GEOM == 0 && (sizeof(T) == 8 || kN == 3); }
template <typename T, int GEOM> constexpr int use_pipe() {
  return (use_ring<T, GEOM>() && sizeof(T) == 8 && kN == 3) ? 1 : 0;
}

// Block shape of a slab vmult on the current device: warps per block and resident warps
// per SM.  The direct variant takes four warps; the ring variant, whose warps share nothing,
// takes the block size (1..8 warps) that fits the most warps per SM.
struct VmultShape {
  int wpb = 1, warps_per_sm = 1;
};
template <typename T, int GEOM> VmultShape slab_shape() {
  constexpr bool SG = use_ring<T, GEOM>();
  constexpr int PIPE = use_pipe<T, GEOM>();
  static std::mutex mu;
  static std::map<int, VmultShape> cache; // device -> shape
  int dev = 0;
  PMG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return it->second;
  auto k = kern::vmult_slab_kernel<kN, T, GEOM, SG, PIPE>;
  constexpr size_t per_warp = kern::SlabSmem<kN, T, SG, PIPE>::PER_WARP;
  VmultShape best;
  const int lo = SG ? 1 : kWarpsPerBlock, hi = SG ? 8 : kWarpsPerBlock;
  PMG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(hi * per_warp)));
  best.warps_per_sm = 0;
  for (int w = lo; w <= hi; ++w) {
    int nb = 0;
    PMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, 32 * w, w * per_warp));
    if (nb * w > best.warps_per_sm) {
      best.wpb = w;
      best.warps_per_sm = nb * w;
    }
  }
  best.warps_per_sm = std::max(1, best.warps_per_sm);
  cache.emplace(dev, best);
  return best;
}

template <typename T, int GEOM> void slab_launch(const SlabLaunch &L) {
  constexpr bool SG = use_ring<T, GEOM>();
  constexpr int PIPE = use_pipe<T, GEOM>();
  auto k = kern::vmult_slab_kernel<kN, T, GEOM, SG, PIPE>;
  const VmultShape sh = slab_shape<T, GEOM>();
  int sms = 0, dev = 0;
  PMG_CUDA(cudaGetDevice(&dev));
  PMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t want = (L.n_groups + sh.wpb - 1) / sh.wpb;
  const int64_t resident_blocks = (int64_t)sh.warps_per_sm * sms / sh.wpb;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, resident_blocks));
  const size_t smem = (size_t)sh.wpb * kern::SlabSmem<kN, T, SG, PIPE>::PER_WARP;
  launch_dependent(k, grid, 32 * sh.wpb, smem, L.stream, make_tab<T>(L), static_cast<const T *>(L.src),
                   static_cast<T *>(L.dst), L.idx, static_cast<const T *>(L.geo), static_cast<const T *>(L.coef),
                   L.n_groups, L.err);
  if (L.units) *L.units = L.n_groups;
  if (L.launched) *L.launched = (int64_t)grid * sh.wpb;
}

template <typename T, int GEOM> void vmult_geom(const SlabLaunch &L) {
  if constexpr (kern::line_layout(kN, GEOM)) line_launch<T, GEOM>(L);
  else slab_launch<T, GEOM>(L);
}

template <typename T, int GEOM> void diag_geom(const SlabLaunch &L) {
  auto k = kern::diag_slab_kernel<kN, T, GEOM>;
  allow_smem(k, diag_smem<T>());
  const int64_t want = (L.n_groups + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(want, L.resident_warps / kWarpsPerBlock));
  k<<<grid, 32 * kWarpsPerBlock, diag_smem<T>(), L.stream>>>(
      make_tab2<T>(L), static_cast<T *>(L.dst), L.idx, static_cast<const T *>(L.geo),
      static_cast<const T *>(L.coef), L.n_groups);
  PMG_LAUNCH_CHECK();
}

template <typename T> void vmult_type(const SlabLaunch &L) {
  if (L.geom == 0) vmult_geom<T, 0>(L);
  else if (L.geom == 1) vmult_geom<T, 1>(L);
  else if (L.geom == 3) vmult_geom<T, 3>(L);
  else vmult_geom<T, 2>(L);
}

template <typename T> void diag_type(const SlabLaunch &L) {
  if (L.geom == 0) diag_geom<T, 0>(L);
  else if (L.geom == 1) diag_geom<T, 1>(L);
  else if (L.geom == 3) diag_geom<T, 3>(L);
  else diag_geom<T, 2>(L);
}

template <typename T, int GEOM> int occ_diag() {
  auto k = kern::diag_slab_kernel<kN, T, GEOM>;
  allow_smem(k, diag_smem<T>());
  int nb = 0;
  PMG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k, 32 * kWarpsPerBlock, diag_smem<T>()));
  return nb * kWarpsPerBlock; // resident warps per SM
}
template <typename T> int occ_diag_geom(int geom) {
  switch (geom) {
  case 0: return occ_diag<T, 0>();
  case 1: return occ_diag<T, 1>();
  case 3: return occ_diag<T, 3>();
  default: return occ_diag<T, 2>();
  }
}

} // namespace

void PMG_CAT(launch_vmult_p, PMG_DEGREE)(const SlabLaunch &L) {
  if (L.dtype == PMG_F64) vmult_type<double>(L);
  else vmult_type<float>(L);
}

void PMG_CAT(launch_diag_p, PMG_DEGREE)(const SlabLaunch &L) {
  if (L.dtype == PMG_F64) diag_type<double>(L);
  else diag_type<float>(L);
}

int PMG_CAT(occupancy_diag_p, PMG_DEGREE)(int dtype, int geom) {
  return dtype == PMG_F64 ? occ_diag_geom<double>(geom) : occ_diag_geom<float>(geom);
}

} // namespace pmg
