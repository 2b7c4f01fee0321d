// af_blas.cu -- BLAS-1 and Krylov helper kernels (FP64), device-resident scalars.
//
// Reductions are deterministic: a fixed grid (a function of n only) produces per-block
// partial sums in a fixed order, and one block adds the partials in a fixed order.
// Krylov scalars live in a device KrylovState so iterations can be queued without host
// round trips; every update kernel returns early once state->done is set, which lets the
// host enqueue a batch of iterations and test convergence once per batch.
#include <cuda_runtime.h>

#include <algorithm>

#include "af_blas.h"
#include "af_cellop.cuh"

namespace af {

constexpr int RB = 256;  // threads per reduction block

__device__ __forceinline__ double block_sum(double v, double* sh) {
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
#pragma unroll
  for (int s = RB / 2; s > 0; s >>= 1) {
    if (t < s) sh[t] += sh[t + s];
    __syncthreads();
  }
  return sh[0];
}

int reduce_blocks(long n) {
  long b = (n + RB * 4 - 1) / (RB * 4);
  if (b > kMaxPartials) b = kMaxPartials;
  if (b < 1) b = 1;
  return (int)b;
}

// partial[b] = sum over the block's grid-stride range of x*y (y == null: x*x)
__global__ void k_dot_partial(const double* __restrict__ x, const double* __restrict__ y, long n,
                              double* __restrict__ partial) {
  __shared__ double sh[RB];
  double s = 0.0;
  const long stride = (long)gridDim.x * RB;
  for (long i = (long)blockIdx.x * RB + threadIdx.x; i < n; i += stride) s = fma(x[i], y ? y[i] : x[i], s);
  const double b = block_sum(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = b;
}

// out = sum(partial[0..nb)) ; optional: also writes sqrt into out_sqrt
__global__ void k_sum_partials(const double* __restrict__ partial, int nb, double* out) {
  __shared__ double sh[RB];
  double s = 0.0;
  for (int i = threadIdx.x; i < nb; i += RB) s += partial[i];
  const double b = block_sum(s, sh);
  if (threadIdx.x == 0) *out = b;
}

cudaError_t dot(const double* x, const double* y, long n, double* partial, double* out, cudaStream_t st) {
  const int nb = reduce_blocks(n);
  k_dot_partial<<<nb, RB, 0, st>>>(x, y, n, partial);
  k_sum_partials<<<1, RB, 0, st>>>(partial, nb, out);
  return cudaGetLastError();
}

__global__ void k_axpby(double a, const double* __restrict__ x, double b, double* __restrict__ y, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] = fma(a, x[i], b * y[i]);
}

cudaError_t axpby(double a, const double* x, double b, double* y, long n, cudaStream_t st) {
  const int bs = 256;
  k_axpby<<<(unsigned)((n + bs - 1) / bs), bs, 0, st>>>(a, x, b, y, n);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ CG pieces
// state layout: see KrylovState in af_blas.h

// r = b - Ax (or r = b when x == 0), z = invd * r, p = z; partials of r.r and r.z
__global__ void k_cg_init(const double* __restrict__ b, const double* __restrict__ Ax, const double* __restrict__ invd,
                          double* __restrict__ r, double* __restrict__ z, double* __restrict__ p, long n,
                          double* __restrict__ part_rr, double* __restrict__ part_rz) {
  __shared__ double sh[RB];
  double rr = 0.0, rz = 0.0;
  const long stride = (long)gridDim.x * RB;
  for (long i = (long)blockIdx.x * RB + threadIdx.x; i < n; i += stride) {
    const double ri = Ax ? b[i] - Ax[i] : b[i];
    const double zi = invd ? invd[i] * ri : ri;
    r[i] = ri;
    z[i] = zi;
    p[i] = zi;
    rr = fma(ri, ri, rr);
    rz = fma(ri, zi, rz);
  }
  double v = block_sum(rr, sh);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = v;
  __syncthreads();
  v = block_sum(rz, sh);
  if (threadIdx.x == 0) part_rz[blockIdx.x] = v;
}

// finalise: rr, rz from partials; tol2 = (rel * sqrt(bb))^2 given bb = rr at start when
// rel_to_initial, else tol2 preset; done if rr <= tol2
__global__ void k_cg_start(KrylovState* s, const double* __restrict__ part_rr, const double* __restrict__ part_rz,
                           int nb, double rel_tol, int rel_to_initial) {
  __shared__ double sh[RB];
  double a = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < nb; i += RB) { a += part_rr[i]; c += part_rz[i]; }
  const double rr = block_sum(a, sh);
  __syncthreads();
  const double rz = block_sum(c, sh);
  if (threadIdx.x == 0) {
    s->rr = rr;
    s->rz = rz;
    s->rr0 = rr;
    if (rel_to_initial) s->tol2 = rel_tol * rel_tol * rr;
    s->its = 0;
    s->done = (rr <= s->tol2) ? 1 : 0;
    s->status = 0;
  }
}

__global__ void k_pAp_partial(const KrylovState* s, const double* __restrict__ p, const double* __restrict__ Ap,
                              long n, double* __restrict__ part) {
  if (s->done) return;
  __shared__ double sh[RB];
  double v = 0.0;
  const long stride = (long)gridDim.x * RB;
  for (long i = (long)blockIdx.x * RB + threadIdx.x; i < n; i += stride) v = fma(p[i], Ap[i], v);
  v = block_sum(v, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = v;
}

__global__ void k_cg_alpha(KrylovState* s, const double* __restrict__ part, int nb) {
  if (s->done) return;
  __shared__ double sh[RB];
  double a = 0.0;
  for (int i = threadIdx.x; i < nb; i += RB) a += part[i];
  const double pAp = block_sum(a, sh);
  if (threadIdx.x == 0) {
    s->pAp = pAp;
    s->alpha = s->rz / pAp;
    if (!(pAp > 0.0) || !isfinite(s->alpha)) { s->status = 2; s->done = 1; }
  }
}

// x += alpha p, r -= alpha Ap, z = invd r ; partials of r.r and r.z
__global__ void k_cg_update(const KrylovState* s, double* __restrict__ x, double* __restrict__ r,
                            double* __restrict__ z, const double* __restrict__ p, const double* __restrict__ Ap,
                            const double* __restrict__ invd, long n, double* __restrict__ part_rr,
                            double* __restrict__ part_rz) {
  if (s->done) return;
  __shared__ double sh[RB];
  const double alpha = s->alpha;
  double rr = 0.0, rz = 0.0;
  const long stride = (long)gridDim.x * RB;
  for (long i = (long)blockIdx.x * RB + threadIdx.x; i < n; i += stride) {
    x[i] = fma(alpha, p[i], x[i]);
    const double ri = fma(-alpha, Ap[i], r[i]);
    r[i] = ri;
    const double zi = invd ? invd[i] * ri : ri;
    z[i] = zi;
    rr = fma(ri, ri, rr);
    rz = fma(ri, zi, rz);
  }
  double v = block_sum(rr, sh);
  if (threadIdx.x == 0) part_rr[blockIdx.x] = v;
  __syncthreads();
  v = block_sum(rz, sh);
  if (threadIdx.x == 0) part_rz[blockIdx.x] = v;
}

__global__ void k_cg_beta(KrylovState* s, const double* __restrict__ part_rr, const double* __restrict__ part_rz,
                          int nb, int maxit) {
  if (s->done) return;
  __shared__ double sh[RB];
  double a = 0.0, c = 0.0;
  for (int i = threadIdx.x; i < nb; i += RB) { a += part_rr[i]; c += part_rz[i]; }
  const double rr = block_sum(a, sh);
  __syncthreads();
  const double rz = block_sum(c, sh);
  if (threadIdx.x == 0) {
    s->its += 1;
    s->rr = rr;
    s->beta = rz / s->rz;
    s->rz = rz;
    if (!isfinite(rr)) { s->status = 3; s->done = 1; }
    else if (rr <= s->tol2) s->done = 1;
    else if (s->its >= maxit) { s->status = 1; s->done = 1; }
  }
}

__global__ void k_cg_dir(const KrylovState* s, double* __restrict__ p, const double* __restrict__ z, long n) {
  if (s->done) return;
  const double beta = s->beta;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = fma(beta, p[i], z[i]);
}

cudaError_t cg_start(KrylovState* s, const double* b, const double* Ax, const double* invd, double* r, double* z,
                     double* p, long n, double* part, double rel_tol, int rel_to_initial, cudaStream_t st) {
  const int nb = reduce_blocks(n);
  k_cg_init<<<nb, RB, 0, st>>>(b, Ax, invd, r, z, p, n, part, part + kMaxPartials);
  k_cg_start<<<1, RB, 0, st>>>(s, part, part + kMaxPartials, nb, rel_tol, rel_to_initial);
  return cudaGetLastError();
}

cudaError_t cg_after_apply(KrylovState* s, double* x, double* r, double* z, double* p, const double* Ap,
                           const double* invd, long n, double* part, int maxit, cudaStream_t st) {
  const int nb = reduce_blocks(n);
  k_pAp_partial<<<nb, RB, 0, st>>>(s, p, Ap, n, part);
  k_cg_alpha<<<1, RB, 0, st>>>(s, part, nb);
  k_cg_update<<<nb, RB, 0, st>>>(s, x, r, z, p, Ap, invd, n, part, part + kMaxPartials);
  k_cg_beta<<<1, RB, 0, st>>>(s, part, part + kMaxPartials, nb, maxit);
  k_cg_dir<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(s, p, z, n);
  return cudaGetLastError();
}

}  // namespace af

// ---------------------------------------------------------------- FP64 peak probe
// 8 independent FMA chains per thread, enough warps to fill every SM: the measured
// DFMA throughput is the denominator of the FP64 roofline reported by bench.py.
namespace af {
__global__ void k_dfma_peak(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-7, x1 = x0 + 1e-9, x2 = x0 + 2e-9, x3 = x0 + 3e-9;
  double x4 = x0 + 4e-9, x5 = x0 + 5e-9, x6 = x0 + 6e-9, x7 = x0 + 7e-9;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
      x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
    }
  }
  const double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
  if (s == 12345.678) out[0] = s;  // keeps the chains alive
}
}  // namespace af

extern "C" int af_measure_fp64_peak(double* tflops) {
  if (!tflops) return 1;
  int dev = 0, nsm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 2;
  double* d = nullptr;
  if (cudaMalloc(&d, sizeof(double)) != cudaSuccess) return 2;
  const int blocks = nsm * 8, threads = 256, iters = 2048;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  af::k_dfma_peak<<<blocks, threads>>>(d, 64, 0.999999, 1e-9);  // warm-up
  float best = 1e30f;
  for (int r = 0; r < 5; ++r) {
    cudaEventRecord(e0);
    af::k_dfma_peak<<<blocks, threads>>>(d, iters, 0.999999, 1e-9);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) best = ms;
  }
  const double flops = 2.0 * 8 * 16 * (double)iters * blocks * threads;
  *tflops = flops / (best * 1e-3) / 1e12;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(d);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// ------------------------------------------------------------------ GMRES / IMEX pieces
namespace af {

// Gram-Schmidt and residual passes over the Krylov basis.  They are bound by memory: the basis is
// read once per pass, three times in all (both dot products of the second pass and the update of the
// first share one read: a chunk of 1024 elements of every V_j is read again while it is in cache),
// with 16-byte loads and four basis vectors in flight per thread.  Each thread owns its elements of a
// chunk in registers and one partial sum per basis vector in shared memory; block partials are added
// in a fixed order by the block that finishes last, which also hands the coefficients to the next
// pass and, with the norm, to the host through mapped memory.  Measured, all four launches: 15
// vectors of 3.3 M elements 247 us (5.4 TB/s), of 0.8 M 67 us, of 0.2 M 35 us.  Before: eight
// launches, four reads of the basis with 8-byte loads, and two pageable copies per iteration; the FP64
// IMEX step at 256x128 (456 iterations) 95.0 -> 74.2 ms, the small 40x16 step 1.17 -> 0.84 ms.  The
// second pass takes the chunks from the last to the first, so that the end of the basis is read from L2
// by it and the beginning by the third (FP64 step 73.9 -> 71.7 ms).
constexpr int KT = 256, KC = 4 * KT;  // threads per block, elements per chunk
constexpr int KJ = 4;                 // basis vectors loaded together (6, 8: 5 % faster at k = 28, 10-20 % slower at k = 4)

int krylov_blocks(long n) { return (int)std::min<long>((n + KC - 1) / KC, kKrylovBlocks); }

struct KrylovDev {
  double* part;
  double *h1, *h2, *n2;
  unsigned* count;
  double* host;
};
KrylovDev krylov_dev(const KrylovWork& k) {
  double* h1 = k.dev + (size_t)kKrylovBlocks * kKrylovMax;
  return {k.dev, h1, h1 + kKrylovMax, h1 + 2 * kKrylovMax, reinterpret_cast<unsigned*>(h1 + 2 * kKrylovMax + 2), k.host_dev};
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// elements i, i+1 of x (i even; the second one 0 past the end)
__device__ __forceinline__ double2 load2(const double* x, long i, long n) {
  if (i + 1 < n) return *reinterpret_cast<const double2*>(x + i);
  return make_double2(i < n ? x[i] : 0.0, 0.0);
}
// the same where x may be off a 16-byte boundary (a caller's right-hand side)
__device__ __forceinline__ double2 load2_any(const double* x, long i, long n) {
  if ((reinterpret_cast<size_t>(x) & 15) == 0) return load2(x, i, n);
  return make_double2(i < n ? x[i] : 0.0, i + 1 < n ? x[i + 1] : 0.0);
}
__device__ __forceinline__ void store2(double* x, long i, long n, double2 v) {
  if (i + 1 < n) *reinterpret_cast<double2*>(x + i) = v;
  else if (i < n) x[i] = v.x;
}

// whether this block is the last of the grid to arrive (its partials written before)
__device__ __forceinline__ bool last_block(unsigned* count) {
  __shared__ bool s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(count, 1u) == gridDim.x - 1;
    if (s_last) *count = 0u;
  }
  __syncthreads();
  __threadfence();
  return s_last;
}
// sum of the block's per-thread values, in thread 0
__device__ __forceinline__ double block_total(double v) {
  __shared__ double sh[KT / 32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
#pragma unroll
    for (int i = 0; i < KT / 32; ++i) t += sh[i];
  __syncthreads();
  return t;
}

// MODE 0: (w = pre .* w,) h1 = V^T w;  1: w -= V h1, h2 = V^T w;  2: w -= V h2, n2 = |w|^2, host results
template <int MODE>
__global__ void __launch_bounds__(KT)
    k_gram_schmidt(const double* V, const long ldv, const int k, double* w, const double* pre, const long n,
                   const KrylovDev kd) {
  extern __shared__ double acc[];  // [k][KT]
  __shared__ double s_h[kKrylovMax + KJ];  // 0 past the k-th
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  pdl_allow_next();
  pdl_wait_previous();
  if (MODE > 0 && t < kKrylovMax + KJ) s_h[t] = t < k ? (MODE == 1 ? kd.h1 : kd.h2)[t] : 0.0;
  if (MODE < 2)
    for (int j = 0; j < k; ++j) acc[j * KT + t] = 0.0;
  __syncthreads();
  double nn = 0.0;
  // a chunk wholly inside the vectors loads without checks, so that the loads of several basis
  // vectors are issued together; the last chunk checks every element
  auto chunk = [&](const long c, auto whole) {
    const long i0 = c * KC + 2 * t, i1 = i0 + 2 * KT;
    auto load = [&](const double* x, long i) {
      if constexpr (decltype(whole)::value) return *reinterpret_cast<const double2*>(x + i);
      else return load2(x, i, n);
    };
    // the elements of KJ basis vectors from the j-th on (past the k-th: the k-th again)
    auto batch = [&](int j, long i0, long i1, double2* p, double2* q) {
#pragma unroll
      for (int e = 0; e < KJ; ++e) {
        const double* v = V + (long)min(j + e, k - 1) * ldv;
        p[e] = load(v, i0);
        q[e] = load(v, i1);
      }
    };
    double2 a = load(w, i0), b = load(w, i1);
    if (MODE == 0 && pre) {
      const double2 p = load(pre, i0), q = load(pre, i1);
      a.x *= p.x; a.y *= p.y; b.x *= q.x; b.y *= q.y;
    }
    if constexpr (MODE > 0) {
      double2 s = make_double2(0.0, 0.0), u = s;
      for (int j = 0; j < k; j += KJ) {
        double2 p[KJ], q[KJ];
        batch(j, i0, i1, p, q);
#pragma unroll
        for (int e = 0; e < KJ; ++e) {
          const double h = s_h[j + e];
          s.x = fma(h, p[e].x, s.x); s.y = fma(h, p[e].y, s.y);
          u.x = fma(h, q[e].x, u.x); u.y = fma(h, q[e].y, u.y);
        }
      }
      a.x -= s.x; a.y -= s.y; b.x -= u.x; b.y -= u.y;
    }
    if (MODE > 0 || pre) {
      store2(w, i0, n, a);
      store2(w, i1, n, b);
    }
    if constexpr (MODE < 2) {
      for (int j = 0; j < k; j += KJ) {
        double2 p[KJ], q[KJ];
        batch(j, i0, i1, p, q);
#pragma unroll
        for (int e = 0; e < KJ; ++e)
          if (j + e < k) acc[(j + e) * KT + t] += fma(p[e].x, a.x, p[e].y * a.y) + fma(q[e].x, b.x, q[e].y * b.y);
      }
    } else {
      nn += fma(a.x, a.x, a.y * a.y) + fma(b.x, b.x, b.y * b.y);
    }
  };
  const long nc = (n + KC - 1) / KC;
  for (long b = blockIdx.x; b < nc; b += gridDim.x) {
    const long c = MODE == 1 ? nc - 1 - b : b;  // backwards: what the pass before read last is still in L2
    if ((c + 1) * KC <= n) chunk(c, std::true_type{});
    else chunk(c, std::false_type{});
  }
  const int nb = gridDim.x;
  if constexpr (MODE < 2) {
    __syncthreads();
    for (int j = warp; j < k; j += KT / 32) {
      double v = 0.0;
#pragma unroll
      for (int i = 0; i < KT / 32; ++i) v += acc[j * KT + i * 32 + lane];
      v = warp_sum(v);
      if (lane == 0) kd.part[j * nb + blockIdx.x] = v;
    }
    if (!last_block(kd.count)) return;
    for (int j = warp; j < k; j += KT / 32) {
      double v = 0.0;
      for (int i = lane; i < nb; i += 32) v += __ldcg(kd.part + j * nb + i);
      v = warp_sum(v);
      if (lane == 0) (MODE == 0 ? kd.h1 : kd.h2)[j] = v;
    }
  } else {
    nn = block_total(nn);
    if (t == 0) kd.part[blockIdx.x] = nn;
    if (!last_block(kd.count)) return;
    double v = 0.0;
    for (int i = t; i < nb; i += KT) v += __ldcg(kd.part + i);
    v = block_total(v);
    if (t < k) kd.host[t] = kd.h1[t] + kd.h2[t];
    if (t == 0) {
      kd.n2[0] = v;
      kd.host[kKrylovMax] = v;
    }
    __threadfence_system();
  }
}

// r = b - r (pre .* (b - r)), n2[1] and host slot 1 = |r|^2
__global__ void __launch_bounds__(KT)
    k_residual(const double* b, double* r, const double* pre, const long n, const KrylovDev kd) {
  const int t = threadIdx.x;
  pdl_allow_next();
  pdl_wait_previous();
  double nn = 0.0;
  for (long c = blockIdx.x; c * KC < n; c += gridDim.x)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const long i = c * KC + 2 * t + e * 2 * KT;
      const double2 x = load2_any(b, i, n), y = load2(r, i, n);
      double2 v = make_double2(x.x - y.x, x.y - y.y);
      if (pre) {
        const double2 p = load2(pre, i, n);
        v.x *= p.x;
        v.y *= p.y;
      }
      store2(r, i, n, v);
      nn += fma(v.x, v.x, v.y * v.y);
    }
  nn = block_total(nn);
  if (t == 0) kd.part[blockIdx.x] = nn;
  if (!last_block(kd.count)) return;
  double v = 0.0;
  for (int i = t; i < (int)gridDim.x; i += KT) v += __ldcg(kd.part + i);
  v = block_total(v);
  if (t == 0) {
    kd.n2[1] = v;
    kd.host[kKrylovMax + 1] = v;
    __threadfence_system();
  }
}

// host slot s = |x|^2
__global__ void __launch_bounds__(KT) k_norm2_host(const double* x, const long n, const int s, const KrylovDev kd) {
  const int t = threadIdx.x;
  pdl_allow_next();
  pdl_wait_previous();
  double nn = 0.0;
  for (long c = blockIdx.x; c * KC < n; c += gridDim.x)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const double2 v = load2_any(x, c * KC + 2 * t + e * 2 * KT, n);
      nn += fma(v.x, v.x, v.y * v.y);
    }
  nn = block_total(nn);
  if (t == 0) kd.part[blockIdx.x] = nn;
  if (!last_block(kd.count)) return;
  double v = 0.0;
  for (int i = t; i < (int)gridDim.x; i += KT) v += __ldcg(kd.part + i);
  v = block_total(v);
  if (t == 0) {
    kd.host[kKrylovMax + s] = v;
    __threadfence_system();
  }
}

// y = x / sqrt(n2) (left alone unless the norm is positive); x and y may be one array
__global__ void __launch_bounds__(KT) k_normalise(const double* x, double* y, const long n, const double* n2) {
  pdl_allow_next();
  pdl_wait_previous();
  const double r = sqrt(*n2);
  if (!(r > 0.0)) return;
  const double a = 1.0 / r;
  const long i = 2 * ((long)blockIdx.x * KT + threadIdx.x);
  if (i >= n) return;
  const double2 v = load2(x, i, n);
  store2(y, i, n, make_double2(a * v.x, a * v.y));
}

namespace {
template <class K, class... A>
cudaError_t launch_k(K kernel, int blocks, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(KT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = kPDL ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
cudaError_t normalise(const double* x, double* y, long n, const double* n2, cudaStream_t st) {
  return launch_k(k_normalise, (int)((n + 2 * KT - 1) / (2 * KT)), 0, st, x, y, n, n2);
}
}  // namespace

cudaError_t gram_schmidt(const KrylovWork& kw, const double* V, long ldv, int k, double* w, const double* pre, long n,
                         cudaStream_t st) {
  if (k < 1 || k > kKrylovMax || (ldv & 1) || ((reinterpret_cast<size_t>(V) | reinterpret_cast<size_t>(w) |
                                                reinterpret_cast<size_t>(pre)) & 15))
    return cudaErrorInvalidValue;
  const KrylovDev kd = krylov_dev(kw);
  const int nb = krylov_blocks(n);
  const size_t smem = sizeof(double) * (size_t)k * KT;
  static std::atomic<unsigned long long> configured[2]{};
  constexpr size_t most = sizeof(double) * kKrylovMax * KT;
  cudaError_t e = allow_smem(k_gram_schmidt<0>, most, configured[0]);
  if (e == cudaSuccess) e = allow_smem(k_gram_schmidt<1>, most, configured[1]);
  if (e == cudaSuccess) e = launch_k(k_gram_schmidt<0>, nb, smem, st, V, ldv, k, w, pre, n, kd);
  if (e == cudaSuccess) e = launch_k(k_gram_schmidt<1>, nb, smem, st, V, ldv, k, w, (const double*)nullptr, n, kd);
  if (e == cudaSuccess) e = launch_k(k_gram_schmidt<2>, nb, 0, st, V, ldv, k, w, (const double*)nullptr, n, kd);
  if (e == cudaSuccess) e = normalise(w, w, n, kd.n2, st);
  return e;
}

cudaError_t residual_start(const KrylovWork& kw, const double* b, double* r, const double* pre, double* v, long n,
                           cudaStream_t st) {
  if ((reinterpret_cast<size_t>(r) | reinterpret_cast<size_t>(v) | reinterpret_cast<size_t>(pre)) & 15)
    return cudaErrorInvalidValue;
  const KrylovDev kd = krylov_dev(kw);
  cudaError_t e = launch_k(k_residual, krylov_blocks(n), 0, st, b, r, pre, n, kd);
  if (e == cudaSuccess) e = normalise(r, v, n, kd.n2 + 1, st);
  return e;
}

cudaError_t norm2_host(const KrylovWork& kw, const double* x, long n, int s, cudaStream_t st) {
  return launch_k(k_norm2_host, krylov_blocks(n), 0, st, x, n, s, krylov_dev(kw));
}

// x += sum_{j<k} y[j] V_j  (y passed by value, k <= 64)
struct SmallVec { double v[64]; };
__global__ void k_mcombine(const double* __restrict__ V, long ldv, int k, const SmallVec y, double* __restrict__ x,
                           long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int j = 0; j < k; ++j) s = fma(y.v[j], V[(long)j * ldv + i], s);
  x[i] += s;
}

cudaError_t mcombine(const double* V, long ldv, int k, const double* y_host, double* x, long n, cudaStream_t st) {
  if (k > 64) return cudaErrorInvalidValue;
  SmallVec y{};
  for (int j = 0; j < k; ++j) y.v[j] = y_host[j];
  k_mcombine<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(V, ldv, k, y, x, n);
  return cudaGetLastError();
}

// z = d .* x
__global__ void k_dmul(const double* __restrict__ d, const double* __restrict__ x, double* __restrict__ z, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) z[i] = d[i] * x[i];
}
cudaError_t dmul(const double* d, const double* x, double* z, long n, cudaStream_t st) {
  k_dmul<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, x, z, n);
  return cudaGetLastError();
}
// out[0] = max |x| ; out[1] = max |x - y| (y may be null -> only out[0])
__device__ __forceinline__ double block_max(double v, double* sh) {
  const int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
#pragma unroll
  for (int s = RB / 2; s > 0; s >>= 1) {
    if (t < s) sh[t] = fmax(sh[t], sh[t + s]);
    __syncthreads();
  }
  return sh[0];
}
__global__ void k_maxabs2_partial(const double* __restrict__ x, const double* __restrict__ y, long n,
                                  double* __restrict__ partial) {
  __shared__ double sh[RB];
  double a = 0.0, b = 0.0;
  const long stride = (long)gridDim.x * RB;
  for (long i = (long)blockIdx.x * RB + threadIdx.x; i < n; i += stride) {
    a = fmax(a, fabs(x[i]));
    if (y) b = fmax(b, fabs(x[i] - y[i]));
  }
  double v = block_max(a, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = v;
  __syncthreads();
  v = block_max(b, sh);
  if (threadIdx.x == 0) partial[kMaxPartials + blockIdx.x] = v;
}
__global__ void k_maxabs2_final(const double* __restrict__ partial, int nb, double* out) {
  __shared__ double sh[RB];
  double a = 0.0, b = 0.0;
  for (int i = threadIdx.x; i < nb; i += RB) { a = fmax(a, partial[i]); b = fmax(b, partial[kMaxPartials + i]); }
  const double ma = block_max(a, sh);
  __syncthreads();
  const double mb = block_max(b, sh);
  if (threadIdx.x == 0) { out[0] = ma; out[1] = mb; }
}
cudaError_t maxabs2(const double* x, const double* y, long n, double* partial, double* out, cudaStream_t st) {
  const int nb = reduce_blocks(n);
  k_maxabs2_partial<<<nb, RB, 0, st>>>(x, y, n, partial);
  k_maxabs2_final<<<1, RB, 0, st>>>(partial, nb, out);
  return cudaGetLastError();
}

__global__ void k_cg_set_tol(KrylovState* s, const double* bb, double eps) { s->tol2 = eps * eps * bb[0]; }
cudaError_t cg_set_abs_tol(KrylovState* s, const double* bb, double eps, cudaStream_t st) {
  k_cg_set_tol<<<1, 1, 0, st>>>(s, bb, eps);
  return cudaGetLastError();
}

}  // namespace af
