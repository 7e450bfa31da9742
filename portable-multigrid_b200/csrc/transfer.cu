// Multigrid transfers between levels: polynomial (same mesh, degree pc -> pf;
// include/multigrid/portable_polynomial_transfer.h + BK1 batched kernels
// include/kernels/bk1_kokkos_kernels.h:462-1051) and geometric (same degree, one global
// refinement; include/multigrid/portable_geometric_transfer.h).  Both are "patch"
// transfers: every patch (fine cell for p, coarse cell for h) maps its coarse DoFs
// (Dirichlet entries dropped) through the tensor product of a 1D matrix onto its fine
// DoFs.  On the caller's maps each fine entry is scaled by its weight, 1/(number of patches
// holding it) by default and 0 when constrained.  On box meshes the patches that hold a fine DoF
// interpolate the same value there (the coarse function is continuous), so the first of them
// alone stands for the DoF and the others skip it: no weights, and about half of the fine entries
// of a patch are neither read nor added to.
#include <algorithm>

#include "pdl.cuh"
#include "pmg_internal.hpp"
#include "transfer.hpp"

namespace pmg {
namespace {

// One thread per line of a patch's fine nodes, NF^2 threads per patch; coarse -> fine takes the
// lines x, y, z, fine -> coarse z, y, x, so that lines along z gather or scatter the fine nodes:
// neighbouring lanes hold neighbouring fine DoFs.  DIR 0: prolongation, 1: restriction, 2: restriction of
// src - Ax, which zeroes Ax (no weights: every fine entry is read by one patch).  fidx: the sentinel for an entry that another
// patch stands for; w: weights, or null.
template <int NC, int NF, typename T> struct TMat {
  T m[NC * NF]; // m[i_c * NF + j_f]
};

template <int NC, int NF> struct PatchShape {
  static constexpr int NF2 = NF * NF;
  // patches per block: lines of several patches fill its warps (at least 94 % of the lanes; one patch
  // of 13^2 lines 88 %)
  static constexpr int PPB = NF == 3 ? 14 : NF == 4 ? 8 : NF == 5 ? 5 : NF == 6 ? 7 : NF == 7 ? 5 : NF == 9 ? 3 : NF == 11 ? 2 : 1;
  static constexpr int THREADS = (PPB * NF2 + 31) / 32 * 32;
  static constexpr int ROW = NF | 1;                 // x lines of the first exchange, odd stride
  static constexpr int A = NC * NC * ROW, B = NC * NF2; // the exchanges between x and y, y and z
  static constexpr int ELEMS = (A + B) | 1;
};

template <typename T, int NC, int NF, int DIR>
__global__ void __launch_bounds__(PatchShape<NC, NF>::THREADS)
    transfer_line_kernel(const __grid_constant__ TMat<NC, NF, T> P, const T *src, T *Ax, T *dst,
                         const uint32_t *__restrict__ cidx, const uint32_t *__restrict__ fidx,
                         const T *__restrict__ w, int64_t n_patches) {
  using Sh = PatchShape<NC, NF>;
  constexpr int NF2 = NF * NF, NF3 = NF2 * NF, NC2 = NC * NC, NC3 = NC2 * NC, ROW = Sh::ROW;
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int e = threadIdx.x / NF2, r = threadIdx.x - e * NF2;
  T *A = reinterpret_cast<T *>(smem_raw) + e * Sh::ELEMS, *B = A + Sh::A;
  const int64_t patch = int64_t(blockIdx.x) * Sh::PPB + e;
  const bool in = e < Sh::PPB && patch < n_patches;
  // the maps are fixed at setup: read before the wait
  uint32_t f[NF], c[NC];
#pragma unroll
  for (int k = 0; k < NF; ++k) f[k] = in ? __ldg(fidx + patch * NF3 + k * NF2 + r) : kInvalid;
  const bool xline = in && r < NC2;      // x line (j, k): r = k*NC + j
  const bool yline = in && r < NC * NF;  // y line (i, k): r = k*NF + i
  const int yk = r / NF, yi = r - yk * NF;
#pragma unroll
  for (int i = 0; i < NC; ++i) c[i] = xline ? __ldg(cidx + patch * NC3 + r * NC + i) : kInvalid;
  pdl_wait();
  src = pdl_after(src);
  Ax = pdl_after(Ax);
  if (DIR == 0) {
    if (xline) {
      T u[NC];
#pragma unroll
      for (int i = 0; i < NC; ++i) u[i] = c[i] != kInvalid ? src[c[i]] : T(0);
#pragma unroll
      for (int x = 0; x < NF; ++x) {
        T v = T(0);
#pragma unroll
        for (int i = 0; i < NC; ++i) v = fma(P.m[i * NF + x], u[i], v);
        A[r * ROW + x] = v;
      }
    }
    __syncthreads();
    if (yline) {
      T u[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) u[j] = A[(yk * NC + j) * ROW + yi];
#pragma unroll
      for (int y = 0; y < NF; ++y) {
        T v = T(0);
#pragma unroll
        for (int j = 0; j < NC; ++j) v = fma(P.m[j * NF + y], u[j], v);
        B[yk * NF2 + y * NF + yi] = v;
      }
    }
    __syncthreads();
    if (in) {
      T u[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) u[k] = B[k * NF2 + r];
#pragma unroll
      for (int z = 0; z < NF; ++z) {
        T v = T(0);
#pragma unroll
        for (int k = 0; k < NC; ++k) v = fma(P.m[k * NF + z], u[k], v);
        if (w) v *= __ldg(w + patch * NF3 + z * NF2 + r);
        if (f[z] != kInvalid) atomicAdd(dst + f[z], v);
      }
    }
  } else {
    if (in) {
      T u[NF];
#pragma unroll
      for (int z = 0; z < NF; ++z) u[z] = f[z] != kInvalid ? src[f[z]] : T(0);
      if (DIR == 2) {
        T a[NF];
#pragma unroll
        for (int z = 0; z < NF; ++z) a[z] = f[z] != kInvalid ? Ax[f[z]] : T(0);
#pragma unroll
        for (int z = 0; z < NF; ++z) u[z] -= a[z];
      } else if (w) {
#pragma unroll
        for (int z = 0; z < NF; ++z) u[z] *= __ldg(w + patch * NF3 + z * NF2 + r);
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        T v = T(0);
#pragma unroll
        for (int z = 0; z < NF; ++z) v = fma(P.m[k * NF + z], u[z], v);
        B[k * NF2 + r] = v;
      }
      if (DIR == 2) { // (after the loads have returned: a store to a line still being read waits)
#pragma unroll
        for (int z = 0; z < NF; ++z)
          if (f[z] != kInvalid) Ax[f[z]] = T(0);
      }
    }
    __syncthreads();
    if (yline) {
      T u[NF];
#pragma unroll
      for (int y = 0; y < NF; ++y) u[y] = B[yk * NF2 + y * NF + yi];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        T v = T(0);
#pragma unroll
        for (int y = 0; y < NF; ++y) v = fma(P.m[j * NF + y], u[y], v);
        A[(yk * NC + j) * ROW + yi] = v;
      }
    }
    __syncthreads();
    if (xline) {
      T u[NF];
#pragma unroll
      for (int x = 0; x < NF; ++x) u[x] = A[r * ROW + x];
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        T v = T(0);
#pragma unroll
        for (int x = 0; x < NF; ++x) v = fma(P.m[i * NF + x], u[x], v);
        if (c[i] != kInvalid) atomicAdd(dst + c[i], v);
      }
    }
  }
}

// DG <-> CG at equal degree: the 1D matrix is the identity and every fine (DG) entry is
// listed once, so the transfer is an entry-wise gather / scatter-add.
template <typename T, int DIR>
__global__ void transfer_identity_kernel(const T *src, T *dst,
                                         const uint32_t *__restrict__ cidx, const uint32_t *__restrict__ fidx,
                                         const T *__restrict__ w, int64_t n_entries) {
  pdl_trigger();
  pdl_wait();
  src = pdl_after(src);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_entries;
       e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t id = __ldg(cidx + e);
    if (DIR == 0) {
      const uint32_t f = __ldg(fidx + e);
      dst[f] += (id != kInvalid) ? __ldg(w + e) * src[id] : T(0);
    } else if (id != kInvalid) {
      atomicAdd(dst + id, __ldg(w + e) * src[__ldg(fidx + e)]);
    }
  }
}

template <typename T, int NC, int NF, int DIR>
void patch_launch(const pmg_transfer &t, void *dst, const void *src, void *Ax, cudaStream_t s) {
  using Sh = PatchShape<NC, NF>;
  constexpr size_t smem = size_t(Sh::PPB) * Sh::ELEMS * sizeof(T);
  static_assert(smem <= 48 * 1024, "no opt-in for the dynamic shared memory");
  TMat<NC, NF, T> P;
  for (int i = 0; i < NC * NF; ++i) P.m[i] = (T)t.P_host[i];
  const int64_t blocks = (t.n_patches + Sh::PPB - 1) / Sh::PPB;
  t.launch_units = t.n_patches;
  t.launch_par = blocks;
  launch_dependent(transfer_line_kernel<T, NC, NF, DIR>, (unsigned)blocks, Sh::THREADS, smem, s, P,
                   static_cast<const T *>(src), static_cast<T *>(Ax), static_cast<T *>(dst), t.coarse_idx.as<uint32_t>(),
                   t.fine_idx.as<uint32_t>(), t.weights.as<T>(), t.n_patches);
}

// runtime (nc, nf) -> compiled pair; false if the pair has no compiled form
template <typename T, int DIR, int NC, int NF> bool try_pair(const pmg_transfer &t, void *dst, const void *src,
                                                           void *Ax, cudaStream_t s) {
  if (t.nc != NC || t.nf != NF) return false;
  patch_launch<T, NC, NF, DIR>(t, dst, src, Ax, s);
  return true;
}
template <typename T, int DIR> bool patch_dispatch(const pmg_transfer &t, void *dst, const void *src, void *Ax, cudaStream_t s) {
  return try_pair<T, DIR, 2, 3>(t, dst, src, Ax, s) || try_pair<T, DIR, 2, 4>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 2, 5>(t, dst, src, Ax, s) || try_pair<T, DIR, 2, 6>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 2, 7>(t, dst, src, Ax, s) || try_pair<T, DIR, 3, 4>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 3, 5>(t, dst, src, Ax, s) || try_pair<T, DIR, 3, 6>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 3, 7>(t, dst, src, Ax, s) || try_pair<T, DIR, 4, 5>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 4, 6>(t, dst, src, Ax, s) || try_pair<T, DIR, 4, 7>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 5, 6>(t, dst, src, Ax, s) || try_pair<T, DIR, 5, 7>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 6, 7>(t, dst, src, Ax, s) || try_pair<T, DIR, 5, 9>(t, dst, src, Ax, s) ||
         try_pair<T, DIR, 6, 11>(t, dst, src, Ax, s) || try_pair<T, DIR, 7, 13>(t, dst, src, Ax, s);
}

template <typename T> std::vector<T> cast(const std::vector<double> &v) {
  return std::vector<T>(v.begin(), v.end());
}

bool same_box_geometry(const pmg_box &a, const pmg_box &b) {
  for (int d = 0; d < 3; ++d)
    if (a.coarse[d] != b.coarse[d] || a.lo[d] != b.lo[d] || a.hi[d] != b.hi[d]) return false;
  return a.deform == b.deform && a.amp == b.amp && a.dirichlet_mask == b.dirichlet_mask;
}

// ---- transfer maps and weights on the device (setup) ----
// out[e] = the sentinel where plain[e] is one or a constrained DoF, else plain[e]
__global__ void sentinel_map_kernel(const uint32_t *__restrict__ plain, const uint8_t *__restrict__ cons, int64_t n,
                                    uint32_t *__restrict__ out) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t d = plain[e];
    out[e] = (d == kInvalid || cons[d]) ? kInvalid : d;
  }
}

// h-transfer patch of coarse cell c: the (2p+1)^3 fine nodes from 2p * (cell coordinates) on
__global__ void h_patch_kernel(const int32_t *__restrict__ coarse_xyz, int64_t n_patches, int p,
                               const uint32_t *__restrict__ fine_lattice, int64_t L0, int64_t L1,
                               uint32_t *__restrict__ fidx) {
  const int nf = 2 * p + 1, nf3 = nf * nf * nf;
  const int64_t total = n_patches * nf3;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = t / nf3;
    const int l = (int)(t - c * nf3);
    const int i = l % nf, j = (l / nf) % nf, k = l / (nf * nf);
    const int64_t x = 2LL * p * coarse_xyz[3 * c] + i, y = 2LL * p * coarse_xyz[3 * c + 1] + j,
                  z = 2LL * p * coarse_xyz[3 * c + 2] + k;
    fidx[t] = fine_lattice[(z * L1 + y) * L0 + x];
  }
}

__global__ void multiplicity_kernel(const uint32_t *__restrict__ fidx, int64_t n, uint32_t *__restrict__ cnt) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    atomicAdd(cnt + fidx[e], 1u);
}

// w[e] = 1 / (patches holding fine DoF fidx[e]), 0 on constrained fine DoFs
template <typename T>
__global__ void weights_kernel(const uint32_t *__restrict__ fidx, int64_t n, const uint32_t *__restrict__ cnt,
                               const uint8_t *__restrict__ cons, T *__restrict__ w) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t d = fidx[e];
    const uint32_t m = cnt[d];
    w[e] = (cons[d] || m == 0) ? T(0) : (T)(1.0 / (double)m);
  }
}

// the first patch that holds each fine DoF (owner: all ones before), and the map without the entries
// of other patches and of constrained DoFs
__global__ void first_patch_kernel(const uint32_t *__restrict__ fidx, int64_t n, int nf3, uint32_t *__restrict__ owner) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    atomicMin(owner + fidx[e], (uint32_t)(e / nf3));
}
__global__ void keep_first_kernel(uint32_t *__restrict__ fidx, int64_t n, int nf3, const uint32_t *__restrict__ owner,
                                  const uint8_t *__restrict__ cons) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t d = fidx[e];
    if (cons[d] || owner[d] != (uint32_t)(e / nf3)) fidx[e] = kInvalid;
  }
}

int setup_grid(int64_t n, int sms) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)sms * 32));
}

// the 1D matrix and, on box meshes (`nested`), the fine map without repeated entries; else the
// weights (1 / multiplicity of the fine DoF over all patches, 0 when constrained, unless given).
// t.coarse_idx and t.fine_idx are set
void transfer_finish(pmg_transfer &t, const pmg_operator &fine, const std::vector<double> &P,
                     const double *given_weights, bool nested) {
  int sms = 0;
  PMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, t.device));
  t.sms = sms;
  const int64_t nf3 = (int64_t)t.nf * t.nf * t.nf, n_w = t.n_patches * nf3;
  t.P_host = P;
  if (nested) {
    if (n_w > 0) {
      DeviceBuffer owner(sizeof(uint32_t) * std::max<int64_t>(1, t.n_fine));
      PMG_CUDA(cudaMemset(owner.get(), 0xFF, owner.bytes()));
      first_patch_kernel<<<setup_grid(n_w, sms), 256>>>(t.fine_idx.as<uint32_t>(), n_w, (int)nf3, owner.as<uint32_t>());
      PMG_LAUNCH_CHECK();
      keep_first_kernel<<<setup_grid(n_w, sms), 256>>>(t.fine_idx.as<uint32_t>(), n_w, (int)nf3, owner.as<uint32_t>(),
                                                       fine.dcons.as<uint8_t>());
      PMG_LAUNCH_CHECK();
      PMG_CUDA(cudaDeviceSynchronize()); // owner is freed on return
    }
  } else if (given_weights) {
    std::vector<double> w(given_weights, given_weights + n_w);
    if (t.dtype == PMG_F64) t.weights = upload(w);
    else t.weights = upload(cast<float>(w));
  } else {
    t.weights.allocate(dtype_size(t.dtype) * std::max<int64_t>(1, n_w));
    if (n_w > 0) {
      DeviceBuffer cnt(sizeof(uint32_t) * std::max<int64_t>(1, t.n_fine));
      PMG_CUDA(cudaMemset(cnt.get(), 0, cnt.bytes()));
      multiplicity_kernel<<<setup_grid(n_w, sms), 256>>>(t.fine_idx.as<uint32_t>(), n_w, cnt.as<uint32_t>());
      PMG_LAUNCH_CHECK();
      if (t.dtype == PMG_F64)
        weights_kernel<double><<<setup_grid(n_w, sms), 256>>>(t.fine_idx.as<uint32_t>(), n_w, cnt.as<uint32_t>(),
                                                              fine.dcons.as<uint8_t>(), t.weights.as<double>());
      else
        weights_kernel<float><<<setup_grid(n_w, sms), 256>>>(t.fine_idx.as<uint32_t>(), n_w, cnt.as<uint32_t>(),
                                                             fine.dcons.as<uint8_t>(), t.weights.as<float>());
      PMG_LAUNCH_CHECK();
      PMG_CUDA(cudaDeviceSynchronize()); // cnt is freed on return
    }
  }
}

// coarse map with the sentinel from the coarse operator's device numbering
void coarse_map_from(pmg_transfer &t, const pmg_operator &coarse, const uint32_t *plain, int64_t n) {
  t.coarse_idx.allocate(sizeof(uint32_t) * std::max<int64_t>(1, n));
  if (n == 0) return;
  sentinel_map_kernel<<<setup_grid(n, t.sms > 0 ? t.sms : 148), 256>>>(plain, coarse.dcons.as<uint8_t>(), n,
                                                                      t.coarse_idx.as<uint32_t>());
  PMG_LAUNCH_CHECK();
}

} // namespace

void transfer_setup_from_maps(pmg_transfer &t, const pmg_operator &coarse, const pmg_operator &fine,
                              const pmg_transfer_maps &m) {
  PMG_REQUIRE(coarse.dtype == fine.dtype, "transfer levels must have the same dtype");
  PMG_REQUIRE(coarse.device == fine.device, "transfer levels must live on one device");
  PMG_REQUIRE(m.n_patches >= 0, "negative patch count");
  PMG_REQUIRE(m.n_patches == 0 || (m.coarse_indices && m.fine_indices), "null index map");
  PMG_CUDA(cudaSetDevice(fine.device));
  t.device = fine.device;
  t.dtype = fine.dtype;
  t.n_coarse = coarse.n_dofs;
  t.n_fine = fine.n_dofs;
  t.n_patches = m.n_patches;
  PMG_CUDA(cudaDeviceGetAttribute(&t.sms, cudaDevAttrMultiProcessorCount, t.device));
  const int pc = coarse.degree, pf = fine.degree;
  std::vector<double> P;
  if (m.kind == PMG_TRANSFER_POLYNOMIAL) {
    PMG_REQUIRE(pc < pf, "polynomial transfer needs degree_coarse < degree_fine");
    t.kind = 0;
    t.nc = pc + 1;
    t.nf = pf + 1;
    P = p_transfer_matrix(pc, pf);
  } else if (m.kind == PMG_TRANSFER_GEOMETRIC) {
    PMG_REQUIRE(pc == pf, "geometric transfer needs equal degrees");
    t.kind = 1;
    t.nc = pc + 1;
    t.nf = 2 * pc + 1;
    P = h_transfer_matrix(pc);
  } else if (m.kind == PMG_TRANSFER_DG_CG) {
    PMG_REQUIRE(pc == pf, "DG <-> CG transfer needs equal degrees");
    t.kind = 2;
    t.nc = t.nf = pc + 1;
    P.assign(t.nc * t.nf, 0.0);
    for (int i = 0; i < t.nc; ++i) P[i * t.nf + i] = 1.0;
  } else {
    fail(PMG_EINVAL, "kind must be PMG_TRANSFER_POLYNOMIAL, _GEOMETRIC or _DG_CG");
  }
  const size_t nc3 = (size_t)t.nc * t.nc * t.nc, nf3 = (size_t)t.nf * t.nf * t.nf;
  const size_t n_c = (size_t)m.n_patches * nc3, n_f = (size_t)m.n_patches * nf3;
  for (size_t e = 0; e < n_c; ++e) {
    const uint32_t d = m.coarse_indices[e];
    if (d != kInvalid && (int64_t)d >= t.n_coarse)
      fail(PMG_EBOUNDS, "coarse_indices[" + std::to_string(e) + "] = " + std::to_string(d) + " >= " +
                            std::to_string(t.n_coarse));
  }
  for (size_t e = 0; e < n_f; ++e)
    if ((int64_t)m.fine_indices[e] >= t.n_fine)
      fail(PMG_EBOUNDS, "fine_indices[" + std::to_string(e) + "] = " + std::to_string(m.fine_indices[e]) + " >= " +
                            std::to_string(t.n_fine));
  // caller maps: coarse entries naming constrained coarse DoFs become the sentinel
  DeviceBuffer craw = upload(std::vector<uint32_t>(m.coarse_indices, m.coarse_indices + n_c));
  coarse_map_from(t, coarse, craw.as<uint32_t>(), (int64_t)n_c);
  t.fine_idx = upload(std::vector<uint32_t>(m.fine_indices, m.fine_indices + n_f));
  PMG_CUDA(cudaDeviceSynchronize()); // craw is freed on return
  transfer_finish(t, fine, P, m.weights, false);
}

void transfer_setup(pmg_transfer &t, const pmg_operator &coarse, const pmg_operator &fine) {
  PMG_REQUIRE(!coarse.from_maps && !fine.from_maps,
              "operators built from caller maps take their transfers from pmg_transfer_create_from_maps");
  PMG_REQUIRE(coarse.dtype == fine.dtype, "transfer levels must have the same dtype");
  PMG_REQUIRE(coarse.device == fine.device, "transfer levels must live on one device");
  PMG_REQUIRE(same_box_geometry(coarse.mesh.box, fine.mesh.box), "levels must discretise the same box");
  PMG_CUDA(cudaSetDevice(fine.device));
  t.device = fine.device;
  t.dtype = fine.dtype;
  t.n_coarse = coarse.n_dofs;
  t.n_fine = fine.n_dofs;
  PMG_CUDA(cudaDeviceGetAttribute(&t.sms, cudaDevAttrMultiProcessorCount, t.device));
  const int pc = coarse.degree, pf = fine.degree;
  const int64_t cnm3 = (int64_t)(pc + 1) * (pc + 1) * (pc + 1);
  std::vector<double> P;
  if (fine.kind == PMG_OP_DG_SIPG || coarse.mesh.box.refine == fine.mesh.box.refine) {
    if (fine.kind == PMG_OP_DG_SIPG) {
      // DG <-> CG at equal degree (ContinuousTransfer): identity on every cell
      PMG_REQUIRE(coarse.kind == PMG_OP_LAPLACE, "the coarse level of a DG transfer must be continuous");
      PMG_REQUIRE(pc == pf && coarse.mesh.box.refine == fine.mesh.box.refine,
                  "DG <-> CG transfer needs equal degrees on the same mesh");
      t.kind = 2;
      t.nc = t.nf = pc + 1;
      P.assign(t.nc * t.nf, 0.0);
      for (int i = 0; i < t.nc; ++i) P[i * t.nf + i] = 1.0;
    } else {
      PMG_REQUIRE(coarse.kind == PMG_OP_LAPLACE, "a DG level can only be the finest level of a transfer");
      PMG_REQUIRE(pc < pf, "polynomial transfer needs degree_coarse < degree_fine");
      t.kind = 0;
      t.nc = pc + 1;
      t.nf = pf + 1;
      P = p_transfer_matrix(pc, pf);
    }
    // one patch per cell of the common mesh: the coarse map with the sentinel, the fine map
    t.n_patches = fine.n_cells;
    coarse_map_from(t, coarse, coarse.dplain.as<uint32_t>(), t.n_patches * cnm3);
    const int64_t n_f = t.n_patches * t.nf * t.nf * t.nf;
    t.fine_idx.allocate(sizeof(uint32_t) * std::max<int64_t>(1, n_f));
    if (n_f > 0)
      PMG_CUDA(cudaMemcpy(t.fine_idx.get(), fine.dplain.get(), sizeof(uint32_t) * n_f, cudaMemcpyDeviceToDevice));
  } else {
    PMG_REQUIRE(fine.mesh.box.refine == coarse.mesh.box.refine + 1,
                "geometric transfer needs the fine mesh refined exactly once more");
    PMG_REQUIRE(pc == pf, "geometric transfer needs equal degrees");
    PMG_REQUIRE(fine.dlattice.get() != nullptr, "fine operator has no node lattice");
    const int p = pc;
    t.kind = 1;
    t.nc = p + 1;
    t.nf = 2 * p + 1;
    t.n_patches = coarse.n_cells;
    P = h_transfer_matrix(p);
    coarse_map_from(t, coarse, coarse.dplain.as<uint32_t>(), t.n_patches * cnm3);
    const int64_t n_f = t.n_patches * t.nf * t.nf * t.nf;
    t.fine_idx.allocate(sizeof(uint32_t) * std::max<int64_t>(1, n_f));
    if (n_f > 0) {
      h_patch_kernel<<<setup_grid(n_f, t.sms), 256>>>(coarse.cell_xyz.as<int32_t>(), t.n_patches, p,
                                                       fine.dlattice.as<uint32_t>(), fine.num.L[0], fine.num.L[1],
                                                       t.fine_idx.as<uint32_t>());
      PMG_LAUNCH_CHECK();
    }
  }
  transfer_finish(t, fine, P, nullptr, t.kind != 2);
}

void transfer_apply(const pmg_transfer &t, int dir, void *dst, const void *src, cudaStream_t s) {
  PMG_REQUIRE(dst && src, "null vector");
  if (t.n_patches == 0) return;
  prof::Scope scope(dir == 0 ? "transfer_prolongate" : "transfer_restrict", s);
  if (t.kind == 2) {
    const int64_t n = t.n_patches * t.nf * t.nf * t.nf;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)t.sms * 16));
    t.launch_units = n;
    t.launch_par = (int64_t)grid * 256;
    auto go = [&](auto kernel, auto zero) {
      using T = decltype(zero);
      launch_dependent(kernel, grid, 256, 0, s, static_cast<const T *>(src), static_cast<T *>(dst),
                       t.coarse_idx.as<uint32_t>(), t.fine_idx.as<uint32_t>(), t.weights.as<T>(), n);
    };
    if (t.dtype == PMG_F64) dir == 0 ? go(transfer_identity_kernel<double, 0>, 0.0) : go(transfer_identity_kernel<double, 1>, 0.0);
    else dir == 0 ? go(transfer_identity_kernel<float, 0>, 0.0f) : go(transfer_identity_kernel<float, 1>, 0.0f);
    return;
  }
  bool done = false;
  if (t.dtype == PMG_F64) done = dir == 0 ? patch_dispatch<double, 0>(t, dst, src, nullptr, s) : patch_dispatch<double, 1>(t, dst, src, nullptr, s);
  else done = dir == 0 ? patch_dispatch<float, 0>(t, dst, src, nullptr, s) : patch_dispatch<float, 1>(t, dst, src, nullptr, s);
  PMG_REQUIRE(done, "no transfer kernel for these degrees");
}

namespace {
__global__ void owned_kernel(const uint32_t *__restrict__ fidx, int64_t n, uint8_t *__restrict__ owned) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    if (fidx[e] != kInvalid) owned[fidx[e]] = 1;
}
__global__ void free_unowned_kernel(const uint8_t *__restrict__ owned, const uint8_t *__restrict__ cons, int64_t n,
                                    unsigned int *__restrict__ bad) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (owned[i] == cons[i]) atomicOr(bad, 1u); // free and not read, or constrained and read
}
} // namespace

// Where every free DoF of the fine operator is read by one patch (box meshes), the restriction of a V-cycle
// takes def - A sol itself and leaves the product zero: a launch, the residual's vector and a pass over the
// product less (V-cycle on 32^3 cells of degree 4, FP32: 513 -> 502 us; 48^3 solve of degree 6 28.8 -> 28.5 ms).
bool transfer_restricts_residual(const pmg_transfer &t, const pmg_operator &fine) {
  if (t.kind == 2 || t.weights.get() || t.n_patches == 0 || t.dtype != fine.dtype || t.n_fine != fine.n_dofs) return false;
  DeviceBuffer owned(std::max<int64_t>(1, t.n_fine)), flag(sizeof(unsigned int));
  PMG_CUDA(cudaMemset(owned.get(), 0, owned.bytes()));
  PMG_CUDA(cudaMemset(flag.get(), 0, flag.bytes()));
  const int64_t entries = t.n_patches * t.nf * t.nf * t.nf;
  owned_kernel<<<(unsigned)std::min<int64_t>((entries + 255) / 256, t.sms * 16), 256>>>(t.fine_idx.as<uint32_t>(), entries,
                                                                                       owned.as<uint8_t>());
  PMG_LAUNCH_CHECK();
  free_unowned_kernel<<<(unsigned)std::min<int64_t>((t.n_fine + 255) / 256, t.sms * 16), 256>>>(
      owned.as<uint8_t>(), fine.dcons.as<uint8_t>(), t.n_fine, flag.as<unsigned int>());
  PMG_LAUNCH_CHECK();
  unsigned int bad = 0;
  PMG_CUDA(cudaMemcpy(&bad, flag.get(), sizeof(bad), cudaMemcpyDeviceToHost));
  return !bad;
}

void transfer_restrict_residual(const pmg_transfer &t, void *dst, const void *def, void *Ax, cudaStream_t s) {
  prof::Scope scope("transfer_restrict", s);
  const bool done = t.dtype == PMG_F64 ? patch_dispatch<double, 2>(t, dst, def, Ax, s) : patch_dispatch<float, 2>(t, dst, def, Ax, s);
  PMG_REQUIRE(done, "no transfer kernel for these degrees");
}

} // namespace pmg
