// af_blas.h -- BLAS-1 / Krylov helpers (see af_blas.cu).
#pragma once

#include <cuda_runtime.h>

namespace af {

constexpr int kMaxPartials = 1184;  // 8 x 148 SMs

// Leading dimension of a stored Krylov basis of length-n FP64 vectors: n rounded up to even,
// so that every basis vector starts on a 16-byte boundary (the operator entry points and the
// cell kernel's bulk copies need that) when n is odd, e.g. 1 x 3 cells at degree 4.
constexpr long krylov_stride(long n) { return (n + 1) & ~1L; }

// Device-resident Krylov scalars.  status: 0 ok, 1 iteration cap, 2 breakdown, 3 NaN/Inf.
struct KrylovState {
  double rr, rz, rr0, tol2, pAp, alpha, beta;
  int its, done, status, pad;
};

int reduce_blocks(long n);
// out (device) = x.y (y == null: x.x); partial needs reduce_blocks(n) doubles
cudaError_t dot(const double* x, const double* y, long n, double* partial, double* out, cudaStream_t st);
// y = a x + b y
cudaError_t axpby(double a, const double* x, double b, double* y, long n, cudaStream_t st);

// Preconditioned CG in pieces (x is the initial guess; Ax = A x, or null when x == 0):
//   cg_start(...)                     r = b - Ax, z = invd r, p = z, tolerance, done flag
//   loop: Ap = A p ; cg_after_apply   alpha, x/r/z update, beta, p = z + beta p
// part needs 2 * kMaxPartials doubles.  tol2 is preset in the state unless rel_to_initial,
// in which case tol = rel_tol * |r0|.
cudaError_t cg_start(KrylovState* s, const double* b, const double* Ax, const double* invd, double* r, double* z,
                     double* p, long n, double* part, double rel_tol, int rel_to_initial, cudaStream_t st);
cudaError_t cg_after_apply(KrylovState* s, double* x, double* r, double* z, double* p, const double* Ap,
                           const double* invd, long n, double* part, int maxit, cudaStream_t st);

// ---- Krylov basis kernels.  One KrylovWork per operator handle, shared by its solvers (a handle is not
// re-entrant): reduction partials, the block counter of the finishing block, the results on the
// device and, in mapped pinned memory, on the host (read after a stream synchronisation, no copy).
constexpr int kKrylovMax = 64;      // basis vectors
constexpr int kKrylovBlocks = 444;  // 3 per SM of a B200 (148); FP64 IMEX step at 256x128 71.7 ms, with 592 72.5, with 740 74.8
struct KrylovWork {
  static constexpr int kHostSlots = 8;
  static constexpr size_t kDevDoubles = (size_t)kKrylovBlocks * kKrylovMax + 2 * kKrylovMax + 2 + 1;
  static constexpr size_t kHostDoubles = kKrylovMax + kHostSlots;
  double* dev = nullptr;       // partials, h1[kKrylovMax], h2[kKrylovMax], norm^2 (slot 0, 1), the counter (0)
  double* host = nullptr;      // h[kKrylovMax], then kHostSlots scalars
  double* host_dev = nullptr;  // the same memory as the device sees it
  double h(int j) const { return static_cast<const volatile double*>(host)[j]; }
  double slot(int s) const { return static_cast<const volatile double*>(host)[kKrylovMax + s]; }
  double* slot_dev(int s) const { return host_dev + kKrylovMax + s; }
};
// w orthogonalised against V_0 .. V_{k-1} (V_j = V + j*ldv; k <= kKrylovMax) by classical Gram-Schmidt
// applied twice, w = pre .* w first when pre is given; then w scaled by 1/|w| (when |w| > 0).  Host:
// h(j) = the sum of both passes' coefficients, slot(0) = |w|^2 before the scaling.
cudaError_t gram_schmidt(const KrylovWork& kw, const double* V, long ldv, int k, double* w, const double* pre, long n,
                         cudaStream_t st);
constexpr int kGramSchmidtLaunches = 4;
// r = b - r (pre .* (b - r) when pre is given);  v = r / |r| (when |r| > 0);  slot(1) = |r|^2
cudaError_t residual_start(const KrylovWork& kw, const double* b, double* r, const double* pre, double* v, long n,
                           cudaStream_t st);
// slot(s) = |x|^2, s >= 2
cudaError_t norm2_host(const KrylovWork& kw, const double* x, long n, int s, cudaStream_t st);
cudaError_t mcombine(const double* V, long ldv, int k, const double* y_host, double* x, long n,
                     cudaStream_t st);  // x += V y
cudaError_t dmul(const double* d, const double* x, double* z, long n, cudaStream_t st);  // z = d .* x
// out[0] = max|x|, out[1] = max|x - y| (0 when y is null); partial needs 2*kMaxPartials doubles
cudaError_t maxabs2(const double* x, const double* y, long n, double* partial, double* out, cudaStream_t st);
// state->tol2 = eps^2 * bb[0]  (bb a device scalar, e.g. |b|^2 from dot)
cudaError_t cg_set_abs_tol(KrylovState* s, const double* bb, double eps, cudaStream_t st);

}  // namespace af
