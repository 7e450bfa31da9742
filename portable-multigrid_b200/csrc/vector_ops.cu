// Vector kernels of the Chebyshev smoother, the V-cycle and CG: fused updates (one pass
// over HBM per update instead of deal.II's chain of sadd/add/DiagonalMatrix::vmult calls)
// and deterministic dot products accumulated in FP64 whatever the vector type.
//
// All are bound by memory: every thread moves 16 bytes per vector and step where the vectors allow
// it (all 16-byte aligned), else one entry.
#include <cmath>
#include <mutex>
#include <vector>

#include "pdl.cuh"
#include "pmg_internal.hpp"
#include "vector_ops.hpp"

namespace pmg {
namespace vec {
namespace {

constexpr int kBlock = 256;
constexpr int kMaxPartials = 1024;

// SM count of the current device (cached per device)
int current_sms() {
  static std::mutex mu;
  static int sms[64] = {0};
  int dev = 0;
  PMG_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  int &n = sms[dev & 63];
  if (n == 0) PMG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
  return n;
}

// grid of a grid-stride kernel over `items`: eight 256-thread blocks per SM at most
inline int grid_for(int64_t items) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((items + kBlock - 1) / kBlock, 8 * (int64_t)current_sms()));
}
inline int reduce_grid(int64_t items) {
  return (int)std::min<int64_t>(kMaxPartials, std::max<int64_t>(1, (items + kBlock - 1) / kBlock));
}

inline bool aligned16() { return true; }
template <typename... P> bool aligned16(const void *p, P... rest) {
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && aligned16(rest...);
}

// W consecutive entries of a vector
template <typename T, int W> struct Pack {
  T v[W];
};
template <int W, typename T> __device__ __forceinline__ Pack<T, W> load(const T *p) {
  Pack<T, W> r;
  constexpr int bytes = W * (int)sizeof(T);
  if constexpr (bytes % 16 == 0) {
#pragma unroll
    for (int b = 0; b < bytes / 16; ++b) {
      const uint4 q = reinterpret_cast<const uint4 *>(p)[b];
      memcpy(reinterpret_cast<char *>(r.v) + 16 * b, &q, 16);
    }
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = p[k];
  }
  return r;
}
template <int W, typename T> __device__ __forceinline__ void store(T *p, const Pack<T, W> &r) {
  constexpr int bytes = W * (int)sizeof(T);
  if constexpr (bytes % 16 == 0) {
#pragma unroll
    for (int b = 0; b < bytes / 16; ++b) {
      uint4 q;
      memcpy(&q, reinterpret_cast<const char *>(r.v) + 16 * b, 16);
      reinterpret_cast<uint4 *>(p)[b] = q;
    }
  } else {
#pragma unroll
    for (int k = 0; k < W; ++k) p[k] = r.v[k];
  }
}

// f.template run<W>(i) for the entries i .. i+W-1 of every pack, run<1> for the tail
template <int W, typename F> __device__ __forceinline__ void for_packs(int64_t n, F &f) {
  const int64_t id = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  const int64_t m = n / W;
  for (int64_t i = id; i < m; i += step) f.template run<W>(i * W);
  if (W > 1 && id < n - m * W) f.template run<1>(m * W + id);
}
template <int W, typename F> __global__ void __launch_bounds__(kBlock) map_k(F f, int64_t n) {
  pdl_trigger();
  pdl_wait();
  for_packs<W>(n, f);
}
// W: entries of a 16-byte pack of the widest type, if `wide`
template <int W, typename F> void map(const F &f, int64_t n, bool wide, cudaStream_t s) {
  if (wide) launch_dependent(map_k<W, F>, grid_for((n + W - 1) / W), kBlock, 0, s, f, n);
  else launch_dependent(map_k<1, F>, grid_for(n), kBlock, 0, s, f, n);
}
template <typename T> constexpr int kW = 16 / (int)sizeof(T);

template <typename T> struct FillMod11 {
  T *x;
  double mean;
  template <int W> __device__ void run(int64_t i) {
    Pack<T, W> r;
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = (T)((double)((i + k) % 11) - mean);
    store<W>(x + i, r);
  }
};

template <typename TD, typename TS> struct Convert {
  TD *d;
  const TS *s;
  template <int W> __device__ void run(int64_t i) {
    const auto a = load<W>(s + i);
    Pack<TD, W> r;
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = (TD)a.v[k];
    store<W>(d + i, r);
  }
};

template <typename T> struct ChebInit {
  T *dst;
  const T *src, *invd;
  T scale;
  template <int W> __device__ void run(int64_t i) {
    const auto b = load<W>(src + i), di = load<W>(invd + i);
    Pack<T, W> r;
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = scale * di.v[k] * b.v[k];
    store<W>(dst + i, r);
  }
};

// entries i .. of the product with the identity rows of x; zero afterwards if `clear`
template <typename T> struct Consumed {
  T *Ax;
  const uint32_t *bits;
  bool clear;
  template <int W> __device__ Pack<T, W> take(int64_t i, const Pack<T, W> &x) const {
    Pack<T, W> a = load<W>(Ax + i);
    if (bits) { // (W divides 32: one word)
      const uint32_t w = __ldg(bits + (i >> 5)) >> (i & 31);
#pragma unroll
      for (int k = 0; k < W; ++k)
        if ((w >> k) & 1u) a.v[k] = x.v[k];
    }
    return a;
  }
  // called once the entries have been used: a store to a line whose load is still in flight stalls the
  // load pipe (8.5M FP32 entries: an update that cleared first took 138 us, 37 without clearing)
  template <int W> __device__ void done(int64_t i) const {
    if (clear) store<W>(Ax + i, Pack<T, W>{});
  }
};

template <typename T> struct InitProduct {
  T *dst;
  const T *src;
  const uint32_t *bits;
  template <int W> __device__ void run(int64_t i) {
    Pack<T, W> r{};
    const uint32_t w = __ldg(bits + (i >> 5)) >> (i & 31);
#pragma unroll
    for (int k = 0; k < W; ++k)
      if ((w >> k) & 1u) r.v[k] = src[i + k];
    store<W>(dst + i, r);
  }
};

template <typename T, bool KEEP> struct ChebFirst {
  T *out, *keep;
  const T *x0, *src;
  Consumed<T> p;
  const T *invd;
  T scale;
  template <int W> __device__ void run(int64_t i) {
    const auto x = load<W>(x0 + i), b = load<W>(src + i), di = load<W>(invd + i), a = p.template take<W>(i, x);
    Pack<T, W> r;
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = x.v[k] + scale * di.v[k] * (b.v[k] - a.v[k]);
    if (KEEP) store<W>(keep + i, x);
    store<W>(out + i, r);
    p.template done<W>(i);
  }
};

template <typename T, bool PREV> struct ChebUpdate {
  T *out;
  const T *cur, *prev, *src;
  Consumed<T> p;
  const T *invd;
  T f1, f2;
  template <int W> __device__ void run(int64_t i) {
    const auto x = load<W>(cur + i), b = load<W>(src + i), di = load<W>(invd + i), a = p.template take<W>(i, x);
    Pack<T, W> xo{}, r;
    if (PREV) xo = load<W>(prev + i);
#pragma unroll
    for (int k = 0; k < W; ++k)
      r.v[k] = x.v[k] + f1 * (x.v[k] - xo.v[k]) + f2 * di.v[k] * (b.v[k] - a.v[k]);
    store<W>(out + i, r);
    p.template done<W>(i);
  }
};

template <typename T> struct Residual {
  T *t;
  const T *def, *x;
  Consumed<T> p;
  template <int W> __device__ void run(int64_t i) {
    Pack<T, W> xv{};
    if (p.bits) xv = load<W>(x + i);
    const auto b = load<W>(def + i), a = p.template take<W>(i, xv);
    Pack<T, W> r;
#pragma unroll
    for (int k = 0; k < W; ++k) r.v[k] = b.v[k] - a.v[k];
    store<W>(t + i, r);
    p.template done<W>(i);
  }
};
template <typename T> struct Zero {
  T *p;
  template <int W> __device__ void run(int64_t i) { store<W>(p + i, Pack<T, W>{}); }
};
// f over n entries and zeros over n_zero others
template <int W, typename T, typename F>
__global__ void __launch_bounds__(kBlock) map_zero_k(F f, int64_t n, Zero<T> z, int64_t n_zero) {
  pdl_trigger();
  pdl_wait();
  for_packs<W>(n, f);
  for_packs<W>(n_zero, z);
}
template <typename T, typename F>
void map_zero(const F &f, int64_t n, void *zero, int64_t n_zero, bool wide, cudaStream_t s) {
  const Zero<T> z{static_cast<T *>(zero)};
  if (!zero) n_zero = 0;
  if (wide) launch_dependent(map_zero_k<kW<T>, T, F>, grid_for((std::max(n, n_zero) + kW<T> - 1) / kW<T>), kBlock, 0, s, f, n, z, n_zero);
  else launch_dependent(map_zero_k<1, T, F>, grid_for(std::max(n, n_zero)), kBlock, 0, s, f, n, z, n_zero);
}

template <typename T> struct Jacobi {
  T *z;
  const T *invd, *r;
  template <int W> __device__ void run(int64_t i) {
    const auto d = load<W>(invd + i), a = load<W>(r + i);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) v.v[k] = d.v[k] * a.v[k];
    store<W>(z + i, v);
  }
};
template <typename T> struct Xpay {
  T *p;
  const T *z;
  T beta;
  template <int W> __device__ void run(int64_t i) {
    const auto a = load<W>(z + i), b = load<W>(p + i);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) v.v[k] = a.v[k] + beta * b.v[k];
    store<W>(p + i, v);
  }
};
// p = z + (rho / rho_old) p with the scalars from device memory; rho_old null: p = z
template <typename T, typename TZ> struct CgDirection {
  T *p;
  const TZ *z;
  const double *rho, *rho_old;
  T beta;
  template <int W> __device__ void run(int64_t i) {
    const auto a = load<W>(z + i);
    Pack<T, W> v;
    if (rho_old) {
      v = load<W>(p + i);
#pragma unroll
      for (int k = 0; k < W; ++k) v.v[k] = (T)a.v[k] + beta * v.v[k];
    } else {
#pragma unroll
      for (int k = 0; k < W; ++k) v.v[k] = (T)a.v[k];
    }
    store<W>(p + i, v);
  }
};
template <int W, typename F> __global__ void __launch_bounds__(kBlock) cg_direction_k(F f, int64_t n) {
  pdl_trigger();
  pdl_wait();
  if (f.rho_old) f.beta = static_cast<decltype(f.beta)>(*f.rho / *f.rho_old);
  for_packs<W>(n, f);
}
template <typename T> struct Axpy {
  T *y;
  const T *x;
  T alpha;
  template <int W> __device__ void run(int64_t i) {
    const auto a = load<W>(x + i), b = load<W>(y + i);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) v.v[k] = b.v[k] + alpha * a.v[k];
    store<W>(y + i, v);
  }
};

// ---- reductions: every block stores its partial sums (NS of them) and the last block to arrive adds
// the partials in a fixed order (deterministic), into device memory and into host-visible memory ----
struct Sum {
  double *partials;       // [NS][kMaxPartials]
  unsigned int *arrived;  // 0 between kernels
  double *device[2], *host[2]; // the results' places
};

__device__ __forceinline__ double block_sum(double v) { // valid in thread 0
  __shared__ double red[kBlock / 32];
  __syncthreads();
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = threadIdx.x < kBlock / 32 ? red[threadIdx.x] : 0.0;
  for (int o = kBlock / 64; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
template <int NS> __device__ __forceinline__ void finish_sum(const double (&acc)[NS], const Sum &sum) {
  __shared__ bool last;
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    const double v = block_sum(acc[k]);
    if (threadIdx.x == 0) __stcg(sum.partials + k * kMaxPartials + blockIdx.x, v);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicInc(sum.arrived, gridDim.x - 1) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < NS; ++k) {
    double w = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kBlock) w += __ldcg(sum.partials + k * kMaxPartials + i);
    w = block_sum(w);
    if (threadIdx.x == 0) {
      *sum.device[k] = w;
      *sum.host[k] = w;
    }
  }
}
template <int W, typename F> __global__ void __launch_bounds__(kBlock) reduce_k(F f, int64_t n, Sum sum) {
  pdl_trigger();
  pdl_wait();
  f.begin();
  for_packs<W>(n, f);
  finish_sum(f.acc, sum);
}
template <int W, typename F> void reduce(const F &f, int64_t n, bool wide, const Sum &sum, cudaStream_t s) {
  if (wide) launch_dependent(reduce_k<W, F>, reduce_grid((n + W - 1) / W), kBlock, 0, s, f, n, sum);
  else launch_dependent(reduce_k<1, F>, reduce_grid(n), kBlock, 0, s, f, n, sum);
}

template <typename T, typename TB> struct Dot {
  const T *a;
  const TB *b;
  double acc[1];
  __device__ void begin() {}
  template <int W> __device__ void run(int64_t i) {
    const auto x = load<W>(a + i);
    const auto y = load<W>(b + i);
#pragma unroll
    for (int k = 0; k < W; ++k) acc[0] += (double)x.v[k] * (double)(T)y.v[k];
  }
};
template <typename T> struct DotProduct {
  const T *p;
  Consumed<T> Ap;
  double acc[1];
  __device__ void begin() {}
  template <int W> __device__ void run(int64_t i) {
    const auto x = load<W>(p + i), y = Ap.template take<W>(i, x);
#pragma unroll
    for (int k = 0; k < W; ++k) acc[0] += (double)x.v[k] * (double)y.v[k];
  }
};
// a copy of a vector in another type, written beside it
template <typename T, typename TC> struct Copy {
  TC *to; // null: none
  template <int W> __device__ void put(int64_t i, const Pack<T, W> &v) const {
    if (!to) return;
    Pack<TC, W> c;
#pragma unroll
    for (int k = 0; k < W; ++k) c.v[k] = (TC)v.v[k];
    store<W>(to + i, c);
  }
};
__device__ __forceinline__ bool cg_step(const double *rho, const double *pv, double &alpha) {
  const double a = *rho, b = *pv;
  alpha = a / b;
  return isfinite(a) && isfinite(b) && b > 0.0;
}
// The updates of a CG iteration read the operator's product before its identity rows are set and leave
// it zero, write the residual in the V-cycle's type too and read its result in that type: with a V-cycle
// three launches less per iteration (two conversions and the product's first pass), 15 instead of 18
// vectors moved.  Solves with a V-cycle: 16^3 cells of degree 2, FP64, 952 -> 855 us; 48^3 of degree 6,
// FP64 CG on FP32 levels, 30.4 -> 30.0 ms.  Eigenvalue estimates (CgUpdateJacobi: no iterate, the two sums
// in one pass; four launches per iteration instead of six) of the eight levels below 32^3 cells of degree
// 4: 2.3 -> 1.8 ms.
template <typename T, typename TC> struct CgUpdate {
  T *x, *r;
  const T *p;
  Consumed<T> Ap;
  Copy<T, TC> copy;
  const double *rho, *pv;
  double acc[1];
  T alpha;
  bool step;
  __device__ void begin() {
    double a;
    step = cg_step(rho, pv, a);
    alpha = (T)a;
  }
  template <int W> __device__ void run(int64_t i) {
    Pack<T, W> rv = load<W>(r + i);
    const auto pp = load<W>(p + i), vv = Ap.template take<W>(i, pp);
    if (step) {
      auto xv = load<W>(x + i);
#pragma unroll
      for (int k = 0; k < W; ++k) {
        xv.v[k] += alpha * pp.v[k];
        rv.v[k] = rv.v[k] - alpha * vv.v[k];
      }
      store<W>(x + i, xv);
      store<W>(r + i, rv);
    }
    copy.template put<W>(i, rv);
#pragma unroll
    for (int k = 0; k < W; ++k) acc[0] += (double)rv.v[k] * (double)rv.v[k];
    Ap.template done<W>(i);
  }
};
// The step of an eigenvalue estimate is taken whatever the signs: with an indefinite operator (a DG penalty
// below the coercive one) or a negative one p.Ap < 0 is a step of the Lanczos run like any other.  (CG itself
// stops there.)
template <typename T> struct CgUpdateJacobi {
  T *r, *z;
  const T *invd, *p;
  Consumed<T> Ap;
  const double *rho, *pv;
  double acc[2]; // r.r, r.z
  T alpha;
  __device__ void begin() { alpha = (T)(*rho / *pv); }
  template <int W> __device__ void run(int64_t i) {
    Pack<T, W> rv = load<W>(r + i), zv;
    const auto pp = load<W>(p + i), vv = Ap.template take<W>(i, pp), di = load<W>(invd + i);
#pragma unroll
    for (int k = 0; k < W; ++k) {
      rv.v[k] = rv.v[k] - alpha * vv.v[k];
      zv.v[k] = di.v[k] * rv.v[k];
      acc[0] += (double)rv.v[k] * (double)rv.v[k];
      acc[1] += (double)rv.v[k] * (double)zv.v[k];
    }
    store<W>(r + i, rv);
    store<W>(z + i, zv);
    Ap.template done<W>(i);
  }
};
// r = b - A x and r.r
template <typename T, typename TC> struct ResidualDot {
  T *r;
  const T *b, *x;
  Consumed<T> Ax;
  Copy<T, TC> copy;
  double acc[1];
  __device__ void begin() {}
  template <int W> __device__ void run(int64_t i) {
    const auto xv = load<W>(x + i), bv = load<W>(b + i), a = Ax.template take<W>(i, xv);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      v.v[k] = bv.v[k] - a.v[k];
      acc[0] += (double)v.v[k] * (double)v.v[k];
    }
    store<W>(r + i, v);
    copy.template put<W>(i, v);
    Ax.template done<W>(i);
  }
};
// z = invd * r and r.z
template <typename T> struct JacobiDot {
  T *z;
  const T *invd, *r;
  double acc[1];
  __device__ void begin() {}
  template <int W> __device__ void run(int64_t i) {
    const auto d = load<W>(invd + i), a = load<W>(r + i);
    Pack<T, W> v;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      v.v[k] = d.v[k] * a.v[k];
      acc[0] += (double)a.v[k] * (double)v.v[k];
    }
    store<W>(z + i, v);
  }
};

} // namespace

// device and host-visible memory of one user of reductions; kept in a pool per device between
// uses (at most kPool idle ones), so that concurrent users have memory of their own
struct ScalarSpace {
  int device = 0;
  DeviceBuffer partials; // 2 kMaxPartials partial sums, kSlots results, the arrival counter
  double *host = nullptr;
  ScalarSpace() = default;
  ~ScalarSpace() {
    if (host && cudaFreeHost(host) != cudaSuccess) (void)cudaGetLastError();
  }
  Sum sum(int slot, int second = 0) {
    double *p = partials.as<double>(), *v = p + 2 * kMaxPartials;
    return Sum{p, reinterpret_cast<unsigned int *>(v + Scalars::kSlots), {v + slot, v + second}, {host + slot, host + second}};
  }
  const double *value(int slot) { return partials.as<double>() + 2 * kMaxPartials + slot; }
};
namespace {
constexpr size_t kPool = 4;
struct Pool {
  std::mutex mu;
  std::vector<std::unique_ptr<ScalarSpace>> idle;
};
Pool &pool() {
  static Pool *p = new Pool; // never destroyed: the CUDA context may be gone by then
  return *p;
}
} // namespace

Scalars::Scalars(cudaStream_t s) : s_(s) {
  int dev = 0;
  PMG_CUDA(cudaGetDevice(&dev));
  {
    Pool &p = pool();
    std::lock_guard<std::mutex> lock(p.mu);
    for (auto &w : p.idle)
      if (w->device == dev) {
        w_ = std::move(w);
        std::swap(w, p.idle.back());
        p.idle.pop_back();
        return;
      }
  }
  w_ = std::make_unique<ScalarSpace>();
  w_->device = dev;
  w_->partials.allocate(sizeof(double) * (2 * kMaxPartials + kSlots + 1));
  PMG_CUDA(cudaMemset(w_->partials.get(), 0, w_->partials.bytes()));
  PMG_CUDA(cudaDeviceSynchronize());
  PMG_CUDA(cudaMallocHost(&w_->host, sizeof(double) * kSlots));
}
// the memory goes back to the pool only once no kernel uses it
Scalars::~Scalars() {
  bool unused = cudaStreamSynchronize(s_) == cudaSuccess;
  if (!unused) {
    (void)cudaGetLastError(); // raised where it arose: the checks of the next call must not find it again
    // refused because the stream is being captured: the capture is void, and nothing of it runs
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    unused = cudaStreamIsCapturing(s_, &st) == cudaSuccess && st != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();
  }
  Pool &p = pool();
  std::lock_guard<std::mutex> lock(p.mu);
  if (unused && p.idle.size() < kPool) p.idle.push_back(std::move(w_));
}
void Scalars::sync() { PMG_CUDA(cudaStreamSynchronize(s_)); }
double Scalars::operator[](int slot) const { return w_->host[slot]; }

#define DISPATCH(dtype, ...)                                                                  \
  do {                                                                                        \
    if ((dtype) == PMG_F64) {                                                                 \
      using T = double;                                                                       \
      __VA_ARGS__;                                                                            \
    } else {                                                                                  \
      using T = float;                                                                        \
      __VA_ARGS__;                                                                            \
    }                                                                                         \
  } while (0)

namespace {
template <typename T> const T *in(const void *p) { return static_cast<const T *>(p); }
template <typename T> T *io(void *p) { return static_cast<T *>(p); }
template <typename T> Consumed<T> consumed(const Product &p) { return Consumed<T>{io<T>(p.Ax), p.bits, p.clear}; }
} // namespace

void fill_mod11(void *x, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  // mean of (i mod 11) over i < n, exactly
  const int64_t full = n / 11, rem = n % 11;
  const double sum = double(full) * 55.0 + double(rem * (rem - 1) / 2);
  const double mean = n > 0 ? sum / double(n) : 0.0;
  DISPATCH(dtype, map<kW<T>>(FillMod11<T>{io<T>(x), mean}, n, aligned16(x), s));
}

void convert(void *dst, int dt_dst, const void *src, int dt_src, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  if (dt_dst == dt_src) {
    PMG_CUDA(cudaMemcpyAsync(dst, src, dtype_size(dt_dst) * n, cudaMemcpyDeviceToDevice, s));
    return;
  }
  const bool wide = aligned16(dst, src);
  if (dt_dst == PMG_F32) map<4>(Convert<float, double>{io<float>(dst), in<double>(src)}, n, wide, s);
  else map<4>(Convert<double, float>{io<double>(dst), in<float>(src)}, n, wide, s);
}

void init_product(void *dst, const void *src, const uint32_t *bits, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vmult_init", s);
  DISPATCH(dtype, map<kW<T>>(InitProduct<T>{io<T>(dst), in<T>(src), bits}, n, aligned16(dst), s));
}

void cheb_init(void *dst, const void *src, const void *invd, double scale, void *zero, int64_t n_zero, int dtype,
               int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  DISPATCH(dtype, map_zero<T>(ChebInit<T>{io<T>(dst), in<T>(src), in<T>(invd), (T)scale}, n, zero, n_zero,
                              aligned16(dst, src, invd, zero), s));
}

void cheb_first_step(void *out, void *keep, const void *x0, const void *src, const Product &p, const void *invd,
                     double scale, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  const bool wide = aligned16(out, keep, x0, src, p.Ax, invd);
  if (keep)
    DISPATCH(dtype, map<kW<T>>(ChebFirst<T, true>{io<T>(out), io<T>(keep), in<T>(x0), in<T>(src), consumed<T>(p),
                                                  in<T>(invd), (T)scale}, n, wide, s));
  else
    DISPATCH(dtype, map<kW<T>>(ChebFirst<T, false>{io<T>(out), nullptr, in<T>(x0), in<T>(src), consumed<T>(p),
                                                   in<T>(invd), (T)scale}, n, wide, s));
}

void cheb_update(void *out, const void *cur, const void *prev, const void *src, const Product &p, const void *invd,
                 double f1, double f2, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  const bool wide = aligned16(out, cur, prev, src, p.Ax, invd);
  if (prev)
    DISPATCH(dtype, map<kW<T>>(ChebUpdate<T, true>{io<T>(out), in<T>(cur), in<T>(prev), in<T>(src), consumed<T>(p),
                                                   in<T>(invd), (T)f1, (T)f2}, n, wide, s));
  else
    DISPATCH(dtype, map<kW<T>>(ChebUpdate<T, false>{io<T>(out), in<T>(cur), nullptr, in<T>(src), consumed<T>(p),
                                                    in<T>(invd), (T)f1, (T)f2}, n, wide, s));
}

void residual(void *t, const void *def, const void *x, const Product &p, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  DISPATCH(dtype, map<kW<T>>(Residual<T>{io<T>(t), in<T>(def), in<T>(x), consumed<T>(p)}, n, aligned16(t, def, x, p.Ax), s));
}

void jacobi(void *z, const void *invd, const void *r, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  DISPATCH(dtype, map<kW<T>>(Jacobi<T>{io<T>(z), in<T>(invd), in<T>(r)}, n, aligned16(z, invd, r), s));
}

void xpay(void *p, const void *z, double beta, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  DISPATCH(dtype, map<kW<T>>(Xpay<T>{io<T>(p), in<T>(z), (T)beta}, n, aligned16(p, z), s));
}

void axpy(void *y, const void *x, double alpha, int dtype, int64_t n, cudaStream_t s) {
  prof::Scope scope_("vector_update", s);
  DISPATCH(dtype, map<kW<T>>(Axpy<T>{io<T>(y), in<T>(x), (T)alpha}, n, aligned16(y, x), s));
}

double dot(const void *a, const void *b, int dtype, int64_t n, cudaStream_t s) {
  Scalars v(s);
  v.dot(0, a, b, dtype, n);
  v.sync();
  return v[0];
}

// f(T, T2) for the types of dtype and dtype2
#define DISPATCH2(dtype, dtype2, ...)                                                         \
  DISPATCH(dtype, {                                                                           \
    if ((dtype2) == PMG_F64) {                                                                \
      using T2 = double;                                                                      \
      __VA_ARGS__;                                                                            \
    } else {                                                                                  \
      using T2 = float;                                                                       \
      __VA_ARGS__;                                                                            \
    }                                                                                         \
  })
// entries per pack where vectors of both types are moved
namespace {
template <typename T, typename T2> constexpr int kW2 = (sizeof(T) == 8 && sizeof(T2) == 8) ? 2 : 4;
}

void Scalars::dot(int slot, const void *a, const void *b, int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH(dtype, reduce<kW<T>>(Dot<T, T>{in<T>(a), in<T>(b), {0.0}}, n, aligned16(a, b), w_->sum(slot), s_));
}

void Scalars::dot_converted(int slot, const void *a, int dt_a, const void *b, int dt_b, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH2(dt_a, dt_b, reduce<kW2<T, T2>>(Dot<T, T2>{in<T>(a), in<T2>(b), {0.0}}, n, aligned16(a, b), w_->sum(slot), s_));
}

void Scalars::dot_product(int slot, const void *p, const Product &Ap, int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH(dtype, reduce<kW<T>>(DotProduct<T>{in<T>(p), consumed<T>(Ap), {0.0}}, n, aligned16(p, Ap.Ax), w_->sum(slot), s_));
}

void Scalars::cg_update(int slot, void *x, void *r, const void *p, const Product &Ap, int rho, int pv, void *copy,
                        int dt_copy, int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH2(dtype, dt_copy,
            reduce<kW2<T, T2>>(CgUpdate<T, T2>{io<T>(x), io<T>(r), in<T>(p), consumed<T>(Ap), Copy<T, T2>{io<T2>(copy)},
                                               w_->value(rho), w_->value(pv), {0.0}, T(0), false}, n,
                               aligned16(x, r, p, Ap.Ax, copy), w_->sum(slot), s_));
}

void Scalars::cg_update_jacobi(int slot_rr, int slot_rz, void *r, void *z, const void *invd, const void *p,
                               const Product &Ap, int rho, int pv, int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH(dtype, reduce<kW<T>>(CgUpdateJacobi<T>{io<T>(r), io<T>(z), in<T>(invd), in<T>(p), consumed<T>(Ap), w_->value(rho),
                                                  w_->value(pv), {0.0, 0.0}, T(0)}, n, aligned16(r, z, invd, p, Ap.Ax),
                                w_->sum(slot_rr, slot_rz), s_));
}

void Scalars::residual_dot(int slot, void *r, const void *b, const void *x, const Product &Ax, void *copy, int dt_copy,
                           int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH2(dtype, dt_copy,
            reduce<kW2<T, T2>>(ResidualDot<T, T2>{io<T>(r), in<T>(b), in<T>(x), consumed<T>(Ax), Copy<T, T2>{io<T2>(copy)},
                                                  {0.0}}, n, aligned16(r, b, x, Ax.Ax, copy), w_->sum(slot), s_));
}

void Scalars::jacobi_dot(int slot, void *z, const void *invd, const void *r, int dtype, int64_t n) {
  prof::Scope scope_("vector_reduce", s_);
  DISPATCH(dtype, reduce<kW<T>>(JacobiDot<T>{io<T>(z), in<T>(invd), in<T>(r), {0.0}}, n, aligned16(z, invd, r), w_->sum(slot), s_));
}

void Scalars::xpay(void *p, int dtype, const void *z, int dt_z, int rho, int rho_old, int64_t n) {
  prof::Scope scope_("vector_update", s_);
  DISPATCH2(dtype, dt_z, {
    constexpr int W = kW2<T, T2>;
    const CgDirection<T, T2> f{io<T>(p), in<T2>(z), w_->value(rho), rho_old < 0 ? nullptr : w_->value(rho_old), T(0)};
    if (aligned16(p, z)) launch_dependent(cg_direction_k<W, CgDirection<T, T2>>, grid_for((n + W - 1) / W), kBlock, 0, s_, f, n);
    else launch_dependent(cg_direction_k<1, CgDirection<T, T2>>, grid_for(n), kBlock, 0, s_, f, n);
  });
}

} // namespace vec
} // namespace pmg
