// Vector kernels used by the smoother, the V-cycle and CG (vector_ops.cu).  Every function
// enqueues on `s`; the ones returning a double synchronise `s` to read the reduction.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>

namespace pmg {
namespace vec {

void fill_mod11(void *x, int dtype, int64_t n, cudaStream_t s);
void convert(void *dst, int dt_dst, const void *src, int dt_src, int64_t n, cudaStream_t s);

// A product A x that an update consumes: the cells' sum, to which the identity rows of the
// constrained DoFs (bit i of `bits`; null: none) are added as it is read, and which is left zero
// for the next product (clear) -- so no launch zeroes it.
struct Product {
  void *Ax;
  const uint32_t *bits = nullptr;
  bool clear = false;
};
// dst = 0 with the identity rows dst_i = src_i of the constrained DoFs
void init_product(void *dst, const void *src, const uint32_t *bits, int dtype, int64_t n, cudaStream_t s);
// Chebyshev vector steps (x_{k+1} = x_k + f1 (x_k - x_{k-1}) + f2 D^{-1} (b - A x_k)):
// cheb_init: dst = scale D^{-1} src; zero (null: none) [n_zero] is set to zero in the same launch
void cheb_init(void *dst, const void *src, const void *invd, double scale, void *zero, int64_t n_zero, int dtype,
               int64_t n, cudaStream_t s);
// cheb_first_step: out = x0 + scale D^{-1} (src - A x0), and keep = x0 unless null (keep != x0;
// out == x0 allowed)
void cheb_first_step(void *out, void *keep, const void *x0, const void *src, const Product &p, const void *invd,
                     double scale, int dtype, int64_t n, cudaStream_t s);
// cheb_update: out = the update from cur and prev (null: zero), out == prev allowed
void cheb_update(void *out, const void *cur, const void *prev, const void *src, const Product &p, const void *invd,
                 double f1, double f2, int dtype, int64_t n, cudaStream_t s);
// t = def - A x
void residual(void *t, const void *def, const void *x, const Product &p, int dtype, int64_t n, cudaStream_t s);
void jacobi(void *z, const void *invd, const void *r, int dtype, int64_t n, cudaStream_t s);
void xpay(void *p, const void *z, double beta, int dtype, int64_t n, cudaStream_t s);
void axpy(void *y, const void *x, double alpha, int dtype, int64_t n, cudaStream_t s); // y += alpha x
double dot(const void *a, const void *b, int dtype, int64_t n, cudaStream_t s);

// Reductions whose results stay on the device, where later kernels of the same stream take the CG
// step lengths from them; the host reads them after sync().  Slots 0 .. kSlots-1.
struct ScalarSpace;
class Scalars {
public:
  static constexpr int kSlots = 64;
  explicit Scalars(cudaStream_t s);
  ~Scalars();
  Scalars(const Scalars &) = delete;
  Scalars &operator=(const Scalars &) = delete;
  void dot(int slot, const void *a, const void *b, int dtype, int64_t n);
  // the same with b of type dt_b, each entry converted to a's type first
  void dot_converted(int slot, const void *a, int dt_a, const void *b, int dt_b, int64_t n);
  void dot_product(int slot, const void *p, const Product &Ap, int dtype, int64_t n); // p.(A p), nothing cleared
  void jacobi_dot(int slot, void *z, const void *invd, const void *r, int dtype, int64_t n); // z = invd r; r.z
  // r = b - A x; r.r; copy (null: none): r in type dt_copy
  void residual_dot(int slot, void *r, const void *b, const void *x, const Product &Ax, void *copy, int dt_copy,
                    int dtype, int64_t n);
  // alpha = rho / pv: x += alpha p, r -= alpha (A p); r.r; copy as above.  Where rho or pv is not
  // finite or pv <= 0, x and r stay as they are.
  void cg_update(int slot, void *x, void *r, const void *p, const Product &Ap, int rho, int pv, void *copy, int dt_copy,
                 int dtype, int64_t n);
  // the same without x and with every step taken, and z = invd r; r.r and r.z
  void cg_update_jacobi(int slot_rr, int slot_rz, void *r, void *z, const void *invd, const void *p, const Product &Ap,
                        int rho, int pv, int dtype, int64_t n);
  // p = z + (rho / rho_old) p with z of type dt_z; rho_old < 0: p = z
  void xpay(void *p, int dtype, const void *z, int dt_z, int rho, int rho_old, int64_t n);
  void sync();                  // waits for the stream
  double operator[](int slot) const; // valid after sync()

private:
  cudaStream_t s_;
  std::unique_ptr<ScalarSpace> w_;
};

} // namespace vec
} // namespace pmg
