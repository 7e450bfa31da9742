// The coarse levels of a V-cycle in one kernel of one block, all vectors in shared memory.
//
// A V-cycle ends in levels of a few to a few hundred DoFs, each about two dozen dependent steps
// (smoother products and updates, residual, transfers) that take a few hundred cycles of work but a
// launch of 1.3 us each: on the Q4 32^3 hierarchy the four levels below 1,000 DoFs took about 100 of
// 658 us.  Here the block runs them with block barriers.  The chain of latencies bounds it, so a
// thread keeps its DoFs and its cell's indices in registers through a smoothing sweep.  A product is two phases: every cell's
// A_K u into an array, then every DoF sums what its cells hold for it (in a fixed order, no atomics)
// and takes the Chebyshev step at once, so A x is never stored.  At degree 1 a thread applies a cell
// in registers, at degree 2 a line of one (as vmult_box_kernel).  Transfers work the same way:
// a patch is a coarse cell, so the coarse level's own lists sum what the patches hold.
//
// The steps and their arithmetic are those of chebyshev_apply and mg_vcycle (solver.cu).
// Degree 2 with a coefficient or full geometry, and degrees above, run in launches: a line of such a cell
// needs three exchange arrays more, and what they would gain has not been measured.
// (Larger levels on a cluster of 16 blocks with vectors in L2 and atomics were measured as well: 60
// to 90 us per level of 4,913 DoFs against 58 us in separate launches.)
#include "mg_tail.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "line_tables.hpp"
#include "pdl.cuh"
#include "solver.hpp"
#include "transfer.hpp"

namespace pmg {

constexpr int kTailLevels = 8;         // levels of one launch
constexpr int kTailDegree = 24;        // Chebyshev iterates per level
// threads: a cell each at degree 1, a line of a cell (9 per cell) at degree 2
template <int N> constexpr int kTailThreads = N == 2 ? 512 : 640;
constexpr int kTailSmem = 200 * 1024;
constexpr uint16_t kNoEntry = 0xFFFF;  // end of a DoF's list; a Dirichlet entry of a cell
constexpr uint16_t kFixedDof = 0xFFFE; // first entry of a Dirichlet DoF's list

// One level's maps in the plan, in 16-bit units from the plan's start (each a multiple of 16 bytes):
// idx [cell][N^3] nodes, gmap [DoF][8] places in the cells' results (Tail::place), fidx [patch][NF^3]
// the fine DoF a patch entry stands for, from [DoF] that entry
struct TailMaps {
  int idx = 0, gmap = 0, fidx = 0, from = 0;
  int n_cells = 0, n_dofs = 0, n_patches = 0;
};
struct TailPlan {
  int N = 0, geom = 0, dtype = 0, levels = 0;
  TailMaps maps[kTailLevels];
  int units[kTailLevels] = {0}; // 16-bit units of the maps of levels 0 .. l
  DeviceBuffer data;
};

namespace {

template <typename T> struct TailLevel {
  const T *geo, *coef, *invd;
  T c0, c1, c2;                    // diagonal of the affine cell tensor
  T scale, f1[kTailDegree], f2[kTailDegree];
  int degree;                      // Chebyshev iterates
  int sol, def, xo, di;            // offsets of the level's vectors in shared memory
  TailMaps m;
};
template <int N, typename T> struct TailTables { // indexed at compile time: constant bank
  kern::LineTab<N, T> line;
  kern::BoxTab<N, T> box;
};
template <int N, typename T> struct TailParams { // indexed by level and lane: copied to shared memory
  T P[N * (2 * N - 1)]; // [coarse node][fine node]
  TailLevel<T> level[kTailLevels];
  const uint4 *plan;
  const T *def; // of the finest level
  T *sol;
  int n_levels, maps_bytes, work; // work: offset of the cells' results, then of the exchange buffers
};

// out = M in along direction D (0: x) of a cell's N^3 values, even/odd
template <int N, typename T, int SIG, int D, typename F>
__device__ __forceinline__ void apply_dir(const kern::EvenOdd<N, T> &m, const T (&in)[N * N * N], F &&f) {
  constexpr int ST = D == 0 ? 1 : (D == 1 ? N : N * N), S1 = D == 0 ? N : 1, S2 = D == 2 ? N : N * N;
#pragma unroll
  for (int a = 0; a < N; ++a)
#pragma unroll
    for (int b = 0; b < N; ++b) {
      const int o = a * S2 + b * S1;
      T l[N];
#pragma unroll
      for (int i = 0; i < N; ++i) l[i] = in[o + i * ST];
      kern::eo_apply<N, T, SIG>(m, l, [&](int q, T v) { f(o + q * ST, v); });
    }
}

// u := A_K u for one cell (GEOM 0 full geometry, 1 axis-aligned, 2 with a coefficient)
template <int N, typename T, int GEOM>
__device__ __forceinline__ void cell_matrix(const TailTables<N, T> &p, const TailLevel<T> &lv, int64_t c,
                                            T (&u)[N * N * N]) {
  constexpr int N3 = N * N * N;
  if constexpr (GEOM == 1) { // K x M x M + M x K x M + M x M x K (vmult_box_kernel)
    T a[N3], b[N3], v[N3];
    apply_dir<N, T, 1, 2>(p.box.eM, u, [&](int o, T x) { a[o] = x; });
    apply_dir<N, T, 1, 2>(p.box.eK, u, [&](int o, T x) { b[o] = lv.c2 * x; });
    apply_dir<N, T, 1, 1>(p.box.eM, a, [&](int o, T x) { v[o] = x; });
    apply_dir<N, T, 1, 1>(p.box.eK, a, [&](int o, T x) { u[o] = lv.c1 * x; });
    apply_dir<N, T, 1, 1>(p.box.eM, b, [&](int o, T x) { u[o] += x; });
    apply_dir<N, T, 1, 0>(p.box.eK, v, [&](int o, T x) { a[o] = lv.c0 * x; });
    apply_dir<N, T, 1, 0>(p.box.eM, u, [&](int o, T x) { b[o] = a[o] + x; });
#pragma unroll
    for (int l = 0; l < N3; ++l) u[l] = b[l];
  } else {
    using CD = kern::CellData<N, kern::line_layout(N, GEOM)>;
    T t[N3], tz[N3], w[N3], wy[N3], wz[N3];
    apply_dir<N, T, 1, 2>(p.line.eS, u, [&](int o, T x) { t[o] = x; });
    apply_dir<N, T, -1, 2>(p.line.eSD, u, [&](int o, T x) { tz[o] = x; });
    apply_dir<N, T, 1, 1>(p.line.eS, t, [&](int o, T x) { w[o] = x; });
    apply_dir<N, T, -1, 1>(p.line.eSD, t, [&](int o, T x) { wy[o] = x; });
    apply_dir<N, T, 1, 1>(p.line.eS, tz, [&](int o, T x) { wz[o] = x; });
    apply_dir<N, T, -1, 0>(p.line.eSD, w, [&](int o, T x) { t[o] = x; });
    apply_dir<N, T, 1, 0>(p.line.eS, wy, [&](int o, T x) { tz[o] = x; });
    apply_dir<N, T, 1, 0>(p.line.eS, wz, [&](int o, T x) { u[o] = x; });
#pragma unroll
    for (int r = 0; r < N; ++r)
#pragma unroll
      for (int q = 0; q < N; ++q)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const int o = (r * N + q) * N + i;
          const T x = t[o], y = tz[o], z = u[o];
          if constexpr (GEOM == 0) {
            T g[6];
#pragma unroll
            for (int m = 0; m < 6; ++m) g[m] = lv.geo[CD::template geo<T>(c, i, q, r, m, 6)];
            t[o] = g[0] * x + g[1] * y + g[2] * z;
            tz[o] = g[1] * x + g[3] * y + g[4] * z;
            u[o] = g[2] * x + g[4] * y + g[5] * z;
          } else {
            const T f = p.line.W[i] * p.line.W[q] * p.line.W[r] * lv.coef[CD::point(c, i, q, r)];
            t[o] = (f * lv.c0) * x;
            tz[o] = (f * lv.c1) * y;
            u[o] = (f * lv.c2) * z;
          }
        }
    apply_dir<N, T, -1, 0>(p.line.eSDT, t, [&](int o, T x) { w[o] = x; });
    apply_dir<N, T, 1, 0>(p.line.eST, tz, [&](int o, T x) { wy[o] = x; });
    apply_dir<N, T, 1, 0>(p.line.eST, u, [&](int o, T x) { wz[o] = x; });
    apply_dir<N, T, 1, 1>(p.line.eST, w, [&](int o, T x) { t[o] = x; });
    apply_dir<N, T, -1, 1>(p.line.eSDT, wy, [&](int o, T x) { t[o] += x; });
    apply_dir<N, T, 1, 1>(p.line.eST, wz, [&](int o, T x) { tz[o] = x; });
    apply_dir<N, T, 1, 2>(p.line.eST, t, [&](int o, T x) { u[o] = x; });
    apply_dir<N, T, -1, 2>(p.line.eSDT, tz, [&](int o, T x) { u[o] += x; });
  }
}

// What a thread keeps of a level while it works on it: the nodes of its cell (degree 1) or line of a
// cell (degree 2), and its DoFs (t and t + threads) with their lists, right-hand side, inverse
// diagonal and last two iterates.  Shared memory holds the current iterate, which cells gather.
template <int N, typename T> struct Own {
  static constexpr int D = 2; // DoFs per thread
  uint16_t id[N == 2 ? 8 : 3];
  bool cell;
  uint16_t list[D][8];
  bool on[D];
  T b[D], di[D], x[D], xp[D];
};

template <int N, typename T> struct Tail {
  const TailTables<N, T> &tab;
  const TailParams<N, T> &p;
  unsigned char *smem;
  static constexpr int N2 = N * N, N3 = N2 * N, NF = 2 * N - 1, NF2 = NF * NF, NF3 = NF2 * NF;
  static constexpr int TH = kTailThreads<N>, D = Own<N, T>::D;
  __device__ __forceinline__ T *vec(int offset) const { return reinterpret_cast<T *>(smem + offset); }
  __device__ __forceinline__ const uint16_t *map(int units) const { return reinterpret_cast<const uint16_t *>(smem) + units; }
  __device__ __forceinline__ T *results() const { return vec(p.work); }
  // the place of node l of cell c (of n) among the results: lanes hold cells at degree 1, lines at 2
  __device__ __forceinline__ static int place(int c, int l, int n) { return N == 2 ? l * n + c : c * N3 + l; }

  __device__ __forceinline__ void own(const TailLevel<T> &lv, Own<N, T> &o) const {
    const uint16_t *idx = map(lv.m.idx);
    const int t = threadIdx.x;
    if constexpr (N == 2) {
      o.cell = t < lv.m.n_cells;
      if (o.cell) memcpy(o.id, idx + t * 8, 16);
    } else {
      o.cell = t < lv.m.n_cells * N2;
      if (o.cell) {
        const int c = t / N2, r = t - c * N2;
#pragma unroll
        for (int k = 0; k < N; ++k) o.id[k] = idx[c * N3 + k * N2 + r];
      }
    }
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const int i = t + j * TH;
      o.on[j] = i < lv.m.n_dofs;
      if (o.on[j]) {
        memcpy(o.list[j], map(lv.m.gmap) + i * 8, 16);
        o.b[j] = vec(lv.def)[i];
        o.di[j] = vec(lv.di)[i];
      }
    }
  }

  // every cell's A_K x into results(); ends in a barrier
  template <int GEOM> __device__ __forceinline__ void cells(const TailLevel<T> &lv, const Own<N, T> &o, const T *x) const {
    T *val = results();
    const int nc = lv.m.n_cells, t = threadIdx.x;
    if constexpr (N == 2) {
      if (o.cell) {
        T u[N3];
#pragma unroll
        for (int l = 0; l < N3; ++l) u[l] = o.id[l] != kNoEntry ? x[o.id[l]] : T(0);
        cell_matrix<N, T, GEOM>(tab, lv, t, u);
#pragma unroll
        for (int l = 0; l < N3; ++l) val[place(t, l, nc)] = u[l];
      }
    } else { // a line of a cell per thread (GEOM 1); node l of cell c at c*N3 + l everywhere
      T *A = val + N3 * nc, *B = A + N3 * nc, *V = B + N3 * nc, *W = V + N3 * nc;
      const int c = t / N2, r = t - c * N2;
      if (o.cell) {
        const int at = c * N3 + r;
        T u[N];
#pragma unroll
        for (int k = 0; k < N; ++k) u[k] = o.id[k] != kNoEntry ? x[o.id[k]] : T(0);
        kern::eo_apply<N, T, 1>(tab.box.eM, u, [&](int q, T v) { A[at + q * N2] = v; });
        kern::eo_apply<N, T, 1>(tab.box.eK, u, [&](int q, T v) { B[at + q * N2] = lv.c2 * v; });
      }
      __syncthreads();
      if (o.cell) {
        const int at = c * N3 + (r / N) * N2 + r % N;
        T a[N], b[N], g[N];
#pragma unroll
        for (int j = 0; j < N; ++j) {
          a[j] = A[at + j * N];
          b[j] = B[at + j * N];
        }
        kern::eo_apply<N, T, 1>(tab.box.eM, a, [&](int q, T v) { V[at + q * N] = v; });
        kern::eo_apply<N, T, 1>(tab.box.eK, a, [&](int q, T v) { g[q] = lv.c1 * v; });
        kern::eo_apply<N, T, 1>(tab.box.eM, b, [&](int q, T v) { W[at + q * N] = g[q] + v; });
      }
      __syncthreads();
      if (o.cell) {
        const int at = c * N3 + r * N;
        T a[N], b[N], g[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
          a[i] = V[at + i];
          b[i] = W[at + i];
        }
        kern::eo_apply<N, T, 1>(tab.box.eK, a, [&](int q, T v) { g[q] = lv.c0 * v; });
        kern::eo_apply<N, T, 1>(tab.box.eM, b, [&](int q, T v) { val[at + q] = g[q] + v; });
      }
    }
    __syncthreads();
  }
  // what a list names in results(); x on a Dirichlet DoF
  __device__ __forceinline__ T sum(const uint16_t (&e)[8], T x) const {
    const T *val = results();
    if (e[0] == kFixedDof) return x;
    T v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = e[k] != kNoEntry ? val[e[k]] : T(0);
    return ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
  }
  __device__ __forceinline__ void publish(const Own<N, T> &o, T *x) const {
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (o.on[j]) x[threadIdx.x + j * TH] = o.x[j];
    __syncthreads();
  }

  // the Chebyshev iterates after the first, x_1 = o.x from x_0 = o.xp, into sol
  template <int GEOM> __device__ __forceinline__ void iterate(const TailLevel<T> &lv, Own<N, T> &o) const {
    T *const sol = vec(lv.sol);
    publish(o, sol);
    for (int k = 1; k < lv.degree; ++k) {
      const T f1 = lv.f1[k], f2 = lv.f2[k];
      cells<GEOM>(lv, o, sol);
#pragma unroll
      for (int j = 0; j < D; ++j)
        if (o.on[j]) {
          const T x = o.x[j];
          o.x[j] = x + f1 * (x - o.xp[j]) + f2 * o.di[j] * (o.b[j] - sum(o.list[j], x));
          o.xp[j] = x;
        }
      publish(o, sol);
    }
  }

  // pre-smoothing of level l from zero, and for l > 0 def of level l-1 = P^T (def - A sol)
  template <int GEOM> __device__ __forceinline__ void down(int l) const {
    const TailLevel<T> &lv = p.level[l];
    Own<N, T> o;
    own(lv, o);
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (o.on[j]) {
        o.x[j] = lv.scale * o.di[j] * o.b[j];
        o.xp[j] = T(0);
      }
    iterate<GEOM>(lv, o);
    if (l == 0) return;
    const TailLevel<T> &co = p.level[l - 1];
    T *t = vec(lv.xo), *val = results();
    cells<GEOM>(lv, o, vec(lv.sol));
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (o.on[j]) t[threadIdx.x + j * TH] = o.b[j] - sum(o.list[j], o.x[j]);
    __syncthreads();
    const uint16_t *f = map(lv.m.fidx);
    const int np = lv.m.n_patches;
    for (int e = threadIdx.x; e < np * N3; e += TH) { // coarse node (i, j, k) of a patch
      const int patch = e / N3, a = e - patch * N3, i = a % N, j = (a / N) % N, k = a / N2;
      T px[NF];
#pragma unroll
      for (int x = 0; x < NF; ++x) px[x] = p.P[i * NF + x];
      T s = T(0);
      for (int z = 0; z < NF; ++z) {
        T sy = T(0);
#pragma unroll
        for (int y = 0; y < NF; ++y) {
          T sx = T(0);
#pragma unroll
          for (int x = 0; x < NF; ++x) {
            const uint16_t d = f[patch * NF3 + (z * NF + y) * NF + x];
            sx = fma(px[x], d != kNoEntry ? t[d] : T(0), sx);
          }
          sy = fma(p.P[j * NF + y], sx, sy);
        }
        s = fma(p.P[k * NF + z], sy, s);
      }
      val[place(patch, a, np)] = s;
    }
    __syncthreads();
    T *dc = vec(co.def);
    for (int i = threadIdx.x; i < co.m.n_dofs; i += TH) {
      uint16_t e[8];
      memcpy(e, map(co.m.gmap) + i * 8, 16);
      dc[i] = sum(e, T(0));
    }
    __syncthreads();
  }

  // sol of level l += P sol of level l-1, then post-smoothing
  template <int GEOM> __device__ __forceinline__ void up(int l) const {
    const TailLevel<T> &lv = p.level[l], &co = p.level[l - 1];
    Own<N, T> o;
    own(lv, o);
    T *sol = vec(lv.sol);
    const T *sc = vec(co.sol);
    const uint16_t *c = map(co.m.idx), *from = map(lv.m.from);
#pragma unroll
    for (int j = 0; j < D; ++j) {
      if (!o.on[j]) continue;
      const int i = threadIdx.x + j * TH;
      o.x[j] = sol[i];
      const uint16_t e = from[i]; // the patch entry that stands for this DoF
      if (e == kNoEntry) continue;
      const int patch = e / NF3, a = e - patch * NF3, x = a % NF, y = (a / NF) % NF, z = a / NF2;
      T s = T(0);
#pragma unroll
      for (int k = 0; k < N; ++k) {
        T sy = T(0);
#pragma unroll
        for (int m = 0; m < N; ++m) {
          T sx = T(0);
#pragma unroll
          for (int n = 0; n < N; ++n) {
            const uint16_t q = c[patch * N3 + (k * N + m) * N + n];
            sx = fma(p.P[n * NF + x], q != kNoEntry ? sc[q] : T(0), sx);
          }
          sy = fma(p.P[m * NF + y], sx, sy);
        }
        s = fma(p.P[k * NF + z], sy, s);
      }
      o.x[j] += s;
    }
    publish(o, sol);
    cells<GEOM>(lv, o, sol);
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (o.on[j]) {
        const T x = o.x[j];
        o.x[j] = x + lv.scale * o.di[j] * (o.b[j] - sum(o.list[j], x));
        o.xp[j] = x;
      }
    iterate<GEOM>(lv, o);
  }
};

template <int N, typename T, int GEOM>
__global__ void __launch_bounds__(kTailThreads<N>, 1) mg_tail_kernel(const __grid_constant__ TailTables<N, T> tab, const __grid_constant__ TailParams<N, T> in) {
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char tail_smem[];
  __shared__ TailParams<N, T> p;
  for (int i = threadIdx.x; i < (int)(sizeof(p) / 4); i += kTailThreads<N>)
    reinterpret_cast<uint32_t *>(&p)[i] = reinterpret_cast<const uint32_t *>(&in)[i];
  for (int i = threadIdx.x; i < in.maps_bytes / 16; i += kTailThreads<N>) // the maps, fixed at setup
    reinterpret_cast<uint4 *>(tail_smem)[i] = __ldg(in.plan + i);
  pdl_wait();
  __syncthreads();
  const Tail<N, T> t{tab, p, tail_smem};
  const int top = p.n_levels - 1;
  for (int l = 0; l <= top; ++l) {
    const T *invd = pdl_after(p.level[l].invd);
    T *di = t.vec(p.level[l].di);
    for (int i = threadIdx.x; i < p.level[l].m.n_dofs; i += kTailThreads<N>) di[i] = invd[i];
  }
  {
    const T *from = pdl_after(p.def);
    T *def = t.vec(p.level[top].def);
    for (int i = threadIdx.x; i < p.level[top].m.n_dofs; i += kTailThreads<N>) def[i] = from[i];
  }
  __syncthreads();
  for (int l = top; l >= 0; --l) t.template down<GEOM>(l);
  for (int l = 1; l <= top; ++l) t.template up<GEOM>(l);
  const T *sol = t.vec(p.level[top].sol);
  for (int i = threadIdx.x; i < p.level[top].m.n_dofs; i += kTailThreads<N>) p.sol[i] = sol[i];
}

int geom_of(const pmg_operator &op) {
  if (op.geometry == PMG_GEOMETRY_FULL) return 0;
  if (op.geometry == PMG_GEOMETRY_AFFINE) return op.has_coeff_values ? 2 : 1;
  return 3;
}

// bytes of shared memory beyond the maps for levels 0 .. top of a plan, and the vectors' offsets
size_t layout(const TailPlan &plan, int top, int *vectors, int *work) {
  const size_t ts = dtype_size(plan.dtype);
  const int n3 = plan.N * plan.N * plan.N;
  size_t at = (size_t)plan.units[top] * 2, cells = 0;
  for (int l = 0; l <= top; ++l) {
    if (vectors) vectors[l] = (int)at;
    at += 4 * ((plan.maps[l].n_dofs * ts + 15) / 16 * 16);
    cells = std::max(cells, (size_t)plan.maps[l].n_cells);
  }
  if (work) *work = (int)at;
  return at + cells * n3 * ts * (plan.N == 2 ? 1 : 5);
}

} // namespace

std::shared_ptr<TailPlan> mg_tail_plan(const pmg_mg &mg) {
  const pmg_operator &first = *mg.levels[0];
  const int N = first.nm, geom = geom_of(first), n3 = N * N * N, nf = 2 * N - 1, nf3 = nf * nf * nf;
  if (!((N == 2 && geom <= 2) || (N == 3 && geom == 1))) return nullptr;
  auto plan = std::make_shared<TailPlan>();
  plan->N = N;
  plan->geom = geom;
  plan->dtype = first.dtype;
  const int threads = N == 2 ? kTailThreads<2> : kTailThreads<3>;
  std::vector<uint16_t> data;
  auto pad = [&] { data.resize((data.size() + 7) / 8 * 8, 0); }; // 16 bytes
  for (int l = 0; l < (int)mg.levels.size() && l < kTailLevels; ++l) {
    const pmg_operator &op = *mg.levels[l];
    if (op.kind != PMG_OP_LAPLACE || op.from_maps || op.nm != N || geom_of(op) != geom || op.dtype != first.dtype ||
        op.device != first.device || op.n_dofs == 0 || op.n_cells == 0 || op.n_dofs > 2 * threads ||
        op.n_cells * (N == 2 ? 1 : N * N) > threads)
      break;
    TailMaps &m = plan->maps[l];
    m.n_cells = (int)op.n_cells;
    m.n_dofs = (int)op.n_dofs;
    if (l > 0) {
      const pmg_transfer &t = *mg.transfers[l];
      if (t.kind != 1 || t.nc != N || t.nf != nf || t.weights.get() || t.n_patches != plan->maps[l - 1].n_cells) break;
      m.n_patches = (int)t.n_patches;
    }
    const size_t start = data.size();
    const Numbering &num = host_numbering(op);
    m.idx = (int)data.size();
    for (int64_t e = 0; e < op.n_cells * n3; ++e) {
      const uint32_t d = num.plain[e];
      data.push_back(d == kInvalid || num.constrained[d] ? kNoEntry : (uint16_t)d);
    }
    pad();
    m.gmap = (int)data.size();
    data.resize(data.size() + 8 * (size_t)m.n_dofs, kNoEntry);
    bool fits = true;
    std::vector<uint8_t> used(m.n_dofs, 0);
    for (int64_t e = 0; e < op.n_cells * n3 && fits; ++e) {
      const uint16_t d = data[m.idx + e];
      if (d == kNoEntry) continue;
      if (used[d] == 8) fits = false;
      else data[m.gmap + (size_t)d * 8 + used[d]++] = (uint16_t)(N == 2 ? (e % n3) * m.n_cells + e / n3 : e);
    }
    for (int d = 0; d < m.n_dofs; ++d)
      if (num.constrained[d]) data[m.gmap + (size_t)d * 8] = kFixedDof;
    pad();
    m.fidx = (int)data.size();
    if (l > 0 && fits) {
      std::vector<uint32_t> f((size_t)m.n_patches * nf3);
      PMG_CUDA(cudaMemcpy(f.data(), mg.transfers[l]->fine_idx.get(), f.size() * 4, cudaMemcpyDeviceToHost));
      for (uint32_t d : f) data.push_back(d == kInvalid ? kNoEntry : (uint16_t)d);
      pad();
      m.from = (int)data.size();
      data.resize(data.size() + m.n_dofs, kNoEntry);
      for (size_t e = 0; e < f.size(); ++e)
        if (f[e] != kInvalid) data[m.from + f[e]] = (uint16_t)e;
    }
    pad();
    plan->units[l] = (int)data.size();
    if (!fits || layout(*plan, l, nullptr, nullptr) > (size_t)kTailSmem) {
      data.resize(start);
      break;
    }
    plan->levels = l + 1;
  }
  if (plan->levels == 0) return nullptr;
  plan->data = upload(data);
  return plan;
}

int mg_tail_top(const pmg_mg &mg) {
  if (!mg.tail) return -1;
  int top = -1;
  for (int l = 0; l < mg.tail->levels; ++l) {
    if (mg.levels[l]->tensor_cores || mg.smoothers[l]->degree > kTailDegree) break;
    top = l;
  }
  return top;
}

namespace {

template <int N, typename T, int GEOM> void launch(pmg_mg &mg, int top, cudaStream_t s) {
  const TailPlan &plan = *mg.tail;
  const TailTables<N, T> tab{line_tables<N, T>(), box_tables<N, T>()};
  TailParams<N, T> p{};
  if (top > 0)
    for (int a = 0; a < N * (2 * N - 1); ++a) p.P[a] = (T)mg.transfers[1]->P_host[a];
  p.n_levels = top + 1;
  p.plan = plan.data.as<uint4>();
  p.maps_bytes = plan.units[top] * 2;
  p.def = mg.def[top].as<T>();
  p.sol = mg.sol[top].as<T>();
  int vectors[kTailLevels];
  const size_t smem = layout(plan, top, vectors, &p.work);
  for (int l = 0; l <= top; ++l) {
    const pmg_operator &op = *mg.levels[l];
    const pmg_chebyshev &c = *mg.smoothers[l];
    TailLevel<T> &lv = p.level[l];
    lv.geo = op.geo.as<T>();
    lv.coef = op.coef.as<T>();
    lv.invd = op.inv_diag.as<T>();
    lv.c0 = (T)op.affine[0];
    lv.c1 = (T)op.affine[1];
    lv.c2 = (T)op.affine[2];
    lv.m = plan.maps[l];
    const int step = (int)((lv.m.n_dofs * sizeof(T) + 15) / 16 * 16);
    lv.sol = vectors[l];
    lv.def = lv.sol + step;
    lv.xo = lv.def + step;
    lv.di = lv.xo + step;
    lv.degree = (c.degree < 2 || std::fabs(c.delta) < 1e-40) ? 1 : c.degree;
    lv.scale = (T)(1.0 / c.theta);
    double rhok = c.delta / c.theta;
    for (int k = 1; k < lv.degree; ++k) {
      const double rhokp = 1.0 / (2.0 * (c.theta / c.delta) - rhok);
      lv.f1[k] = (T)(rhokp * rhok);
      lv.f2[k] = (T)(2.0 * rhokp / c.delta);
      rhok = rhokp;
    }
  }
  auto k = mg_tail_kernel<N, T, GEOM>;
  PMG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem));
  launch_dependent(k, 1, kTailThreads<N>, smem, s, tab, p);
}

} // namespace

void mg_tail(pmg_mg &mg, int top, cudaStream_t s) {
  prof::Scope scope("mg_tail", s);
  const TailPlan &plan = *mg.tail;
  if (plan.dtype == PMG_F64) {
    if (plan.N == 3) launch<3, double, 1>(mg, top, s);
    else if (plan.geom == 0) launch<2, double, 0>(mg, top, s);
    else if (plan.geom == 1) launch<2, double, 1>(mg, top, s);
    else launch<2, double, 2>(mg, top, s);
  } else {
    if (plan.N == 3) launch<3, float, 1>(mg, top, s);
    else if (plan.geom == 0) launch<2, float, 0>(mg, top, s);
    else if (plan.geom == 1) launch<2, float, 1>(mg, top, s);
    else launch<2, float, 2>(mg, top, s);
  }
}

} // namespace pmg
