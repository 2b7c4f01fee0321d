// The Krylov basis kernels (csrc/af_blas.h) against long double sums on the host, at vector lengths
// around a chunk (1024 elements) and above what one trip of every block covers (444 chunks): whole and
// partial last chunks, a partial chunk on a block's second and third trip, basis counts around the
// batches of four and the largest.  Built and run by tests/test_gpu_krylov_kernels.py; prints "OK".
//
// Tolerance: a thread's chain of additions, the block's and the last block's are together below 100
// terms, so a dot product is within 100 u |x||y| (1e-14); two passes over up to 64 vectors: 1e-12.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "af_blas.h"

#define REQUIRE(c)                                                                                       \
  do {                                                                                                   \
    if (!(c)) {                                                                                          \
      std::printf("FAILED %s at line %d (n = %ld, k = %d, pre = %d)\n", #c, __LINE__, n, k, (int)pre);   \
      return false;                                                                                      \
    }                                                                                                    \
  } while (0)

namespace {
constexpr double kTol = 1e-12;
cudaStream_t st;
af::KrylovWork kw;

double* device(const std::vector<double>& h) {
  double* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(double)) != cudaSuccess) return nullptr;
  cudaMemcpy(d, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice);
  return d;
}

bool check(long n, int k, bool pre) {
  const long ld = af::krylov_stride(n);
  std::mt19937_64 gen(17 * n + k);
  std::normal_distribution<double> dist;
  std::vector<double> V((size_t)ld * k), w(n), p(n), b(n + 1);
  const double a = 1.0 / std::sqrt((double)n);
  for (auto& v : V) v = a * dist(gen);
  for (auto& v : w) v = dist(gen);
  for (auto& v : p) v = 1.0 + 0.5 * dist(gen) * dist(gen);
  for (auto& v : b) v = dist(gen);
  double *dV = device(V), *dw = device(w), *dp = device(p), *db = device(b), *dv = device(w);
  REQUIRE(dV && dw && dp && db && dv);
  const double* gp = pre ? dp : nullptr;

  std::vector<double> got(n), x(w);
  REQUIRE(af::gram_schmidt(kw, dV, ld, k, dw, gp, n, st) == cudaSuccess);
  REQUIRE(cudaStreamSynchronize(st) == cudaSuccess);
  cudaMemcpy(got.data(), dw, n * sizeof(double), cudaMemcpyDeviceToHost);
  if (pre)
    for (long i = 0; i < n; ++i) x[i] *= p[i];
  long double size = 0;
  for (double v : x) size += (long double)v * v;
  size = sqrtl(size);
  std::vector<long double> y(x.begin(), x.end()), h(k, 0);
  for (int pass = 0; pass < 2; ++pass) {
    std::vector<long double> c(k, 0);
    for (int j = 0; j < k; ++j)
      for (long i = 0; i < n; ++i) c[j] += V[(size_t)j * ld + i] * y[i];
    for (int j = 0; j < k; ++j) {
      for (long i = 0; i < n; ++i) y[i] -= c[j] * V[(size_t)j * ld + i];
      h[j] += c[j];
    }
  }
  long double nn = 0, err = 0;
  for (long double v : y) nn += v * v;
  for (int j = 0; j < k; ++j) REQUIRE(fabsl(kw.h(j) - h[j]) <= kTol * size);
  REQUIRE(fabsl(sqrtl(kw.slot(0)) - sqrtl(nn)) <= kTol * size);
  // the last vector may be nearly dependent (n <= k): compare before the scaling
  for (long i = 0; i < n; ++i) {
    const long double d = got[i] * sqrtl(kw.slot(0)) - y[i];
    err += d * d;
  }
  REQUIRE(sqrtl(err) <= kTol * size);

  // residual: r = b - r, |r|, v = r / |r|, with b off a 16-byte boundary; then a norm alone
  cudaMemcpy(dw, w.data(), n * sizeof(double), cudaMemcpyHostToDevice);
  REQUIRE(af::residual_start(kw, db + 1, dw, gp, dv, n, st) == cudaSuccess);
  REQUIRE(af::norm2_host(kw, db + 1, n, 5, st) == cudaSuccess);
  REQUIRE(cudaStreamSynchronize(st) == cudaSuccess);
  cudaMemcpy(got.data(), dv, n * sizeof(double), cudaMemcpyDeviceToHost);
  long double rr = 0, bb = 0;
  for (long i = 0; i < n; ++i) {
    y[i] = ((long double)b[i + 1] - w[i]) * (pre ? p[i] : 1.0);
    rr += y[i] * y[i];
    bb += (long double)b[i + 1] * b[i + 1];
  }
  REQUIRE(fabsl(kw.slot(1) - rr) <= kTol * rr);
  REQUIRE(fabsl(kw.slot(5) - bb) <= kTol * bb);
  for (long i = 0; i < n; ++i) REQUIRE(fabsl(got[i] * sqrtl(rr) - y[i]) <= kTol * sqrtl(rr));
  for (double* d : {dV, dw, dp, db, dv}) cudaFree(d);
  return true;
}
}  // namespace

int main() {
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return 1;
  if (cudaMalloc(&kw.dev, af::KrylovWork::kDevDoubles * sizeof(double)) != cudaSuccess) return 1;
  if (cudaMemset(kw.dev, 0, af::KrylovWork::kDevDoubles * sizeof(double)) != cudaSuccess) return 1;
  if (cudaHostAlloc((void**)&kw.host, af::KrylovWork::kHostDoubles * sizeof(double), cudaHostAllocMapped) != cudaSuccess)
    return 1;
  if (cudaHostGetDevicePointer((void**)&kw.host_dev, kw.host, 0) != cudaSuccess) return 1;
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  const long trip = (long)af::kKrylovBlocks * 1024;
  for (bool pre : {false, true}) {
    for (long n : {255L, 1023L, 1024L, 1025L, 5L * 1024 + 511, trip - 1, trip, trip + 1, 2 * trip + 777})
      for (int k : {1, 3, 4, 5})
        if (!check(n, k, pre)) return 1;
    for (int k : {63, 64})
      for (long n : {1025L, trip + 1023})
        if (!check(n, k, pre)) return 1;
  }
  std::printf("OK\n");
  return 0;
}
