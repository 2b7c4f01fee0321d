// af_kern.cu -- per-degree kernel instantiations.  Compiled once per polynomial degree
// with -DAF_P=<p>; each object registers its entry points in the degree table used by
// the C ABI (af_capi.cu).
#include <cstdint>
#include <cstdio>

#include "af_adjoint.cuh"
#include "af_gauss.cuh"
#include "af_internal.h"

#ifndef AF_P
#error "compile with -DAF_P=<degree>"
#endif

namespace af {

static __constant__ Tab<AF_P> c_tab;
static __constant__ TabT<AF_P, float> c_tabf;
static __constant__ TabT<AF_P, float, AF_P + 1> c_tabfr;  // reduced quadrature (preconditioner)
static __constant__ TabT<AF_P, double, AF_P + 1> c_tabr;  // reduced quadrature (exact B)
static __constant__ TransT<AF_P, double> c_tr;
static __constant__ TransT<AF_P, float> c_trf;
static __constant__ CobT<AF_P, double> c_cob;
static __constant__ CobT<AF_P, float> c_cobf;

template <>
__device__ __forceinline__ const Tab<AF_P>& tabr<AF_P, double>() {
  return c_tab;
}
template <>
__device__ __forceinline__ const TabT<AF_P, float>& tabr<AF_P, float>() {
  return c_tabf;
}
template <>
__device__ __forceinline__ const TabT<AF_P, float, AF_P + 1>& tabr<AF_P, float, AF_P + 1>() {
  return c_tabfr;
}
template <>
__device__ __forceinline__ const TabT<AF_P, double, AF_P + 1>& tabr<AF_P, double, AF_P + 1>() {
  return c_tabr;
}
template <>
__device__ __forceinline__ const CobT<AF_P, double>& cobr<AF_P, double>() {
  return c_cob;
}
template <>
__device__ __forceinline__ const CobT<AF_P, float>& cobr<AF_P, float>() {
  return c_cobf;
}

namespace {

constexpr int P = AF_P;
// Cells per CTA of the reduced-quadrature (P+1 points) B kernel: its CTAs have NQ = P+1 threads per cell,
// about half of the full-quadrature kernel's.  Measured, us at 128x64 and 512x256 cells:
//   p=1  64: 3.6, 12.1;  32: 3.5, 12.3      p=2  32: 3.5, 15.3;  42: 3.7, 16.0
//   p=3  8: 6.9, 37.5;  16: 5.3 to 9, 41.8;  24: 9.1, 39.5;  32: 9.4, 40.8;  64: 9.3, 42.5
//   p=4  32: 5.5, 34.8;  16: 5.7, 39.8      p=5  8: 7.4, 61.2;  20: 9.0, 64.0     p=6  18: 6.9, 68.6;  8: 6.6, 71.4
constexpr int kReducedCB = P == 1 ? 64 : (P == 2 ? 32 : (P == 3 ? 8 : (P == 4 ? 32 : (P == 5 ? 8 : 18))));

constexpr int kND = (P + 1) * (P + 1);
constexpr int kNPK = kND * (kND + 1) / 2;
constexpr int kNQ = 2 * P + 1, kNPair = (P + 1) * (P + 2) / 2;
constexpr int kInvRows = (kND + 1) / 2;         // threads per cell, two rows each
constexpr int kInvCells = 128 / kInvRows;
constexpr int kInvThreads = 128;
// products of basis values: [pair i <= j, pair = j (j+1)/2 + i][point]
struct PairTab {
  double ss[kNPair][kNQ];
};
static __constant__ PairTab c_pair;
__host__ __device__ constexpr int pair_of(int i, int j) { return i <= j ? j * (j + 1) / 2 + i : i * (i + 1) / 2 + j; }

cudaError_t upload_tables() {
  static const Tab<P> t = host::make_tab<P>();
  static const TabT<P, float> tf = host::make_tab<P, float>();
  static const TabT<P, float, P + 1> tfr = host::make_tab<P, float, P + 1>();
  static const TabT<P, double, P + 1> tr1 = host::make_tab<P, double, P + 1>();
  static const TransT<P, double> tr = host::make_trans<P, double>();
  static const TransT<P, float> trf = host::make_trans<P, float>();
  static const CobT<P, double> cob = host::make_cob<P, double>();
  static const CobT<P, float> cobf = host::make_cob<P, float>();
  static const PairTab pt = [] {
    PairTab p{};
    std::vector<host::LD> nd = host::gll(P), x, w;
    host::gauss(kNQ, x, w);
    for (int j = 0; j <= P; ++j)
      for (int i = 0; i <= j; ++i)
        for (int q = 0; q < kNQ; ++q)
          p.ss[pair_of(i, j)][q] = (double)(host::lag(nd, i, x[q]) * host::lag(nd, j, x[q]));
    return p;
  }();
  cudaError_t e = cudaMemcpyToSymbol(c_tab, &t, sizeof(t));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_pair, &pt, sizeof(pt));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_cob, &cob, sizeof(cob));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_cobf, &cobf, sizeof(cobf));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tabf, &tf, sizeof(tf));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tabfr, &tfr, sizeof(tfr));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tabr, &tr1, sizeof(tr1));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_tr, &tr, sizeof(tr));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_trf, &trf, sizeof(trf));
  return e;
}

template <int STAGE, int MASK, bool GEN>
cudaError_t rhs_mask(const MeshDev& mesh, const RhsSources& s, const RhsParams& prm, double* o_rho, double* o_u,
                     double* o_p, int ncell, cudaStream_t st) {
  using Ph = RhsPhys<STAGE, MASK, GEN>;
  ArgPtrs<PhysInfo<Ph>::NARR_TOTAL, Ph::NOUT_ARR> a{};
  int k = 0;
  for (int j = 0; j < STAGE; ++j) {
    a.in[k++] = s.rho[j];
    a.in[k++] = s.u[j];
    if (Ph::VEL || Ph::PRES) a.in[k++] = s.p[j];
    if (Ph::quirk_group(j)) a.in[k++] = s.u[0];
  }
  if (Ph::HAS_I) {
    a.in[k++] = s.rho_c;
    if (Ph::PRES) a.in[k++] = s.u_fix;
  }
  int o = 0;
  if (Ph::RHO) a.out[o++] = o_rho;
  if (Ph::VEL) a.out[o++] = o_u;
  if (Ph::PRES) a.out[o++] = o_p;
  for (int i = 0; i < k; ++i)
    if (!a.in[i]) return cudaErrorInvalidValue;
  for (int i = 0; i < o; ++i)
    if (!a.out[i]) return cudaErrorInvalidValue;
  return launch_cellop<P, Ph>(mesh, a, prm, ncell, st);
}

template <int STAGE, bool GEN>
cudaError_t rhs_stage(const MeshDev& mesh, int mask, const RhsSources& s, const RhsParams& prm, double* o_rho,
                      double* o_u, double* o_p, int ncell, cudaStream_t st) {
  switch (mask) {
    case 1: return rhs_mask<STAGE, 1, GEN>(mesh, s, prm, o_rho, o_u, o_p, ncell, st);
    case 2: return rhs_mask<STAGE, 2, GEN>(mesh, s, prm, o_rho, o_u, o_p, ncell, st);
    case 4: return rhs_mask<STAGE, 4, GEN>(mesh, s, prm, o_rho, o_u, o_p, ncell, st);
    case 6: return rhs_mask<STAGE, 6, GEN>(mesh, s, prm, o_rho, o_u, o_p, ncell, st);
    case 7: return rhs_mask<STAGE, 7, GEN>(mesh, s, prm, o_rho, o_u, o_p, ncell, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t rhs(const MeshDev& mesh, int stage, int mask, const RhsSources& s, const RhsParams& prm, double* o_rho,
                double* o_u, double* o_p, int ncell, cudaStream_t st) {
  const bool gen = prm.radial || prm.sponge;
  auto run = [&](auto sc) {
    constexpr int S = decltype(sc)::value;
    return gen ? rhs_stage<S, true>(mesh, mask, s, prm, o_rho, o_u, o_p, ncell, st)
               : rhs_stage<S, false>(mesh, mask, s, prm, o_rho, o_u, o_p, ncell, st);
  };
  switch (stage) {
    case 1: return run(std::integral_constant<int, 1>{});
    case 2: return run(std::integral_constant<int, 2>{});
    case 3: return run(std::integral_constant<int, 3>{});
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t mass(const MeshDev& mesh, int ncomp, const double* src, const double* weight, double scale, double* dst,
                 int ncell, cudaStream_t st) {
  MassParams prm{scale};
  if (weight) {
    if (ncomp == 2) {
      ArgPtrs<2, 1> a{{src, weight}, {dst}};
      return launch_cellop<P, MassPhys<2, true>>(mesh, a, prm, ncell, st);
    }
    ArgPtrs<2, 1> a{{src, weight}, {dst}};
    return launch_cellop<P, MassPhys<1, true>>(mesh, a, prm, ncell, st);
  }
  if (ncomp == 2) {
    ArgPtrs<1, 1> a{{src}, {dst}};
    return launch_cellop<P, MassPhys<2, false>>(mesh, a, prm, ncell, st);
  }
  ArgPtrs<1, 1> a{{src}, {dst}};
  return launch_cellop<P, MassPhys<1, false>>(mesh, a, prm, ncell, st);
}

cudaError_t op_B(const MeshDev& mesh, const double* p, double c, double* u, int ncell, cudaStream_t st) {
  ArgPtrs<1, 1> a{{p}, {u}};
  return launch_cellop<P, BPhysExactReduced, kReducedCB>(mesh, a, BParams{c}, ncell, st);
}

cudaError_t op_C(const MeshDev& mesh, const double* w, const double* pf, const double* p, const CParams& prm,
                 double* dst, int ncell, cudaStream_t st) {
  if (p) {
    ArgPtrs<3, 1> a{{p, w, pf}, {dst}};
    return launch_cellop<P, CPhys<true, -1>>(mesh, a, prm, ncell, st);
  }
  ArgPtrs<2, 1> a{{w, pf}, {dst}};
  return launch_cellop<P, CPhys<false, 1>>(mesh, a, prm, ncell, st);
}

// Diagonal of the (weighted) mass matrix, inverted:
//   diag_i = sum_q l_i(x_q)^2 l_j(z_q)^2 w(q) JxW(q)   (what the reference's unit-vector
//   probing in assemble_diagonal_cell_term_* computes, euler_operator.h:2458-2586)
__global__ void k_inv_diag(const MeshDev mesh, const double* __restrict__ weight, const double scale,
                           double* __restrict__ dst, const int ncomp, const int ncell) {
  using T = Tab<P>;
  constexpr int P1 = T::P1, NQ = T::NQ, ND = P1 * P1;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const Tab<P>& tb = c_tab;
  const int i = c % mesh.nx, j = c / mesh.nx, W = mesh.nx + 1;
  const double2 v0 = mesh.vtx[j * W + i], v1 = mesh.vtx[j * W + i + 1];
  const double2 v2 = mesh.vtx[(j + 1) * W + i], v3 = mesh.vtx[(j + 1) * W + i + 1];
  const double Ax = v1.x - v0.x, Az = v1.y - v0.y, Cx = v2.x - v0.x, Cz = v2.y - v0.y;
  const double Bx = v3.x - v2.x - v1.x + v0.x, Bz = v3.y - v2.y - v1.y + v0.y;
  double wn[ND];
  if (weight) {
#pragma unroll
    for (int k = 0; k < ND; ++k) wn[k] = weight[(size_t)c * ND + k];
  }
  double dz[P1][NQ];
#pragma unroll
  for (int iz = 0; iz < P1; ++iz)
#pragma unroll
    for (int qx = 0; qx < NQ; ++qx) dz[iz][qx] = 0.0;
  for (int qx = 0; qx < NQ; ++qx) {
    double tx[P1];
    if (weight) {
#pragma unroll
      for (int iz = 0; iz < P1; ++iz) {
        double s = 0.0;
#pragma unroll
        for (int ix = 0; ix < P1; ++ix) s = fma(tb.S[qx][ix], wn[iz * P1 + ix], s);
        tx[iz] = s;
      }
    }
    const double xi = tb.x[qx];
    const double J01 = fma(Bx, xi, Cx), J11 = fma(Bz, xi, Cz);
#pragma unroll
    for (int qz = 0; qz < NQ; ++qz) {
      const double eta = tb.x[qz];
      const double J00 = fma(Bx, eta, Ax), J10 = fma(Bz, eta, Az);
      double f = (J00 * J11 - J01 * J10) * tb.w[qx] * tb.w[qz];
      if (weight) {
        double wv = 0.0;
#pragma unroll
        for (int iz = 0; iz < P1; ++iz) wv = fma(tb.S[qz][iz], tx[iz], wv);
        f *= wv;
      } else {
        f *= scale;
      }
#pragma unroll
      for (int iz = 0; iz < P1; ++iz) dz[iz][qx] = fma(tb.S[qz][iz] * tb.S[qz][iz], f, dz[iz][qx]);
    }
  }
#pragma unroll
  for (int iz = 0; iz < P1; ++iz)
#pragma unroll
    for (int ix = 0; ix < P1; ++ix) {
      double s = 0.0;
#pragma unroll
      for (int qx = 0; qx < NQ; ++qx) s = fma(tb.S[qx][ix] * tb.S[qx][ix], dz[iz][qx], s);
      const double inv = 1.0 / s;
      for (int d = 0; d < ncomp; ++d) dst[((size_t)c * ncomp + d) * ND + iz * P1 + ix] = inv;
    }
}

cudaError_t inv_diag(const MeshDev& mesh, int ncomp, const double* weight, double scale, double* dst, int ncell,
                     cudaStream_t st) {
  const int bs = 128;
  k_inv_diag<<<(ncell + bs - 1) / bs, bs, 0, st>>>(mesh, weight, scale, dst, ncomp, ncell);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- exact cell inverse
// Cell mass matrix  M_K[I][J] = sum_q w(q) JxW(q) phi_I(q) phi_J(q)  (w = 1 or a density) and its
// inverse, stored as the packed lower triangle (row-major) cell-major, Minv[c * NPK + k], so that the
// apply kernel reads a cell's inverse as one contiguous block.
//
// One CTA forms kInvCells cells, one thread per two rows of a cell (117 of 128 threads at degree 4, 125
// at degree 6):
//   F(q) = w(q) JxW(q) at the Gauss points, w by sum factorisation;
//   T(qz)[ix <= jx] = sum_qx S[qx][ix] S[qx][jx] F(qz, qx),  thread = (cell, qz);
//   Q[iz <= jz][ix <= jx] = sum_qz S[qz][iz] S[qz][jz] T(qz)[ix][jx],  thread = (cell, ix <= jx)
// (the products S S from constant memory: each value is loaded once per thread and multiplied by
// compile-time constants), which holds every entry of the matrix once: M[(iz, ix)][(jz, jx)] =
// Q[iz, jz][ix, jx].  The inverse by the symmetric sweep operator (M is symmetric positive definite,
// no pivoting): sweeping pivot k maps a_kk -> -1/a_kk, a_rk = a_kr -> a_rk/a_kk and, for r, j != k,
// a_rj -> a_rj - (a_rk/a_kk) a_kj; sweeping every pivot leaves -M^{-1}.  A thread keeps two rows
// in registers, rotated so that the pivot column comes first: every pivot runs the same code (a loop,
// not ND unrolled copies) and writes a[j] from a[j+1].  The pivot row is the column of the threads'
// first elements, published in shared memory (twice in a row, so that the rotated row is contiguous),
// one barrier per pivot.
//
// Bound by the broadcast loads of the pivot row and FP64 issue (ND^3 multiply-adds a cell); two rows
// per thread share a load (one row per thread: degree 4 720 us with the shared-memory data path at
// 96 %, degree 6 980 us), and the loads are of 8 bytes: a 16-byte load of a warp takes four wavefronts
// even when its lanes read two addresses (degree 6 845 us with them).  Measured: degree 4, 131072 cells 610 us (one warp per cell with lane = row, two exchanges per
// pivot and all pivots unrolled: 889 us); degree 6, 32385 cells 823 us (Cholesky of the packed matrix in
// shared memory, one warp per cell: 5085 us).
struct InvShape {  // shared memory of one cell, in doubles
  static constexpr int F = 0, T = F + kNQ * kNQ, Q = T + kNQ * kNPair, W = Q + kNPair * kNPair, X = W + kND,
                       END = X + (P + 1) * kNQ;
  static constexpr int BASE = END > kNPK ? END : kNPK;  // the packed inverse takes their place
  static constexpr int RL = 2 * kND;                    // the pivot row, twice
  static constexpr int R = BASE, ID = R + 2 * RL, GEO = ID + 2;
  static constexpr int CELL = (GEO + 6) | 1;  // odd: the loads of two cells in a warp meet different banks
  static constexpr size_t BYTES = sizeof(double) * CELL * kInvCells;
};

__global__ void __launch_bounds__(kInvThreads, P <= 4 ? 4 : 2)
    k_mass_inverse(const MeshDev mesh, const double* __restrict__ weight, double* __restrict__ Lg, const int ncell) {
  using S = InvShape;
  constexpr int P1 = P + 1, NQ = kNQ, ND = kND, NT = kInvThreads, NC = kInvCells;
  extern __shared__ __align__(16) double sm[];
  const Tab<P>& tb = c_tab;
  const int t = threadIdx.x, c0 = blockIdx.x * NC, nc = min(NC, ncell - c0);
  // nodal weights and the bilinear maps
  if (weight)
    for (int e = t; e < nc * ND; e += NT) sm[(e / ND) * S::CELL + S::W + e % ND] = weight[(size_t)c0 * ND + e];
  if (t < nc) {
    const int c = c0 + t, i = c % mesh.nx, j = c / mesh.nx, W = mesh.nx + 1;
    const double2* v = mesh.vtx + (size_t)j * W + i;
    const double2 v0 = v[0], v1 = v[1], v2 = v[W], v3 = v[W + 1];
    double* g = sm + t * S::CELL + S::GEO;
    g[0] = v1.x - v0.x; g[1] = v1.y - v0.y;
    g[2] = v2.x - v0.x; g[3] = v2.y - v0.y;
    g[4] = v3.x - v2.x - v1.x + v0.x; g[5] = v3.y - v2.y - v1.y + v0.y;
  }
  __syncthreads();
  if (weight) {  // rows of the weight at the x points: thread = (cell, row)
    for (int e = t; e < nc * P1; e += NT) {
      double* s = sm + (e / P1) * S::CELL;
      const int iz = e % P1;
      double r[P1];
#pragma unroll
      for (int i = 0; i < P1; ++i) r[i] = s[S::W + iz * P1 + i];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        double a = 0.0;
#pragma unroll
        for (int i = 0; i < P1; ++i) a = fma(tb.S[q][i], r[i], a);
        s[S::X + iz * NQ + q] = a;
      }
    }
    __syncthreads();
  }
  for (int e = t; e < nc * NQ; e += NT) {  // F: thread = (cell, column qx)
    double* s = sm + (e / NQ) * S::CELL;
    const double* g = s + S::GEO;
    const int qx = e % NQ;
    const double xi = tb.x[qx], wx = tb.w[qx], J01 = fma(g[4], xi, g[2]), J11 = fma(g[5], xi, g[3]);
    double r[P1];
    if (weight)
#pragma unroll
      for (int i = 0; i < P1; ++i) r[i] = s[S::X + i * NQ + qx];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double J00 = fma(g[4], tb.x[q], g[0]), J10 = fma(g[5], tb.x[q], g[1]);
      double f = (J00 * J11 - J01 * J10) * wx * tb.w[q];
      if (weight) {
        double a = 0.0;
#pragma unroll
        for (int i = 0; i < P1; ++i) a = fma(tb.S[q][i], r[i], a);
        f *= a;
      }
      s[S::F + q * NQ + qx] = f;
    }
  }
  __syncthreads();
  for (int e = t; e < nc * NQ; e += NT) {  // T: thread = (cell, qz)
    double* s = sm + (e / NQ) * S::CELL;
    const int qz = e % NQ;
    double f[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) f[q] = s[S::F + qz * NQ + q];
#pragma unroll
    for (int p = 0; p < kNPair; ++p) {
      double a = 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) a = fma(c_pair.ss[p][q], f[q], a);
      s[S::T + qz * kNPair + p] = a;
    }
  }
  __syncthreads();
  for (int e = t; e < nc * kNPair; e += NT) {  // Q: thread = (cell, ix <= jx)
    double* s = sm + (e / kNPair) * S::CELL;
    const int px = e % kNPair;
    double f[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) f[q] = s[S::T + q * kNPair + px];
#pragma unroll
    for (int p = 0; p < kNPair; ++p) {
      double a = 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) a = fma(c_pair.ss[p][q], f[q], a);
      s[S::Q + p * kNPair + px] = a;
    }
  }
  __syncthreads();
  // rows 2i, 2i + 1 of cell cc (a row past the last repeats it and publishes nothing; so do threads
  // past the last cell)
  const int cc = min(t / kInvRows, nc - 1), i2 = 2 * (t % kInvRows);
  const bool own = t / kInvRows < nc;
  double* s = sm + cc * S::CELL;
  double a[2][ND];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = min(i2 + h, ND - 1), rz = r / P1, rx = r % P1;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const int jz = j / P1, jx = j % P1;
      const int pz = rz <= jz ? jz * (jz + 1) / 2 + rz : rz * (rz + 1) / 2 + jz;
      const int px = rx <= jx ? jx * (jx + 1) / 2 + rx : rx * (rx + 1) / 2 + jx;
      a[h][j] = s[S::Q + pz * kNPair + px];
    }
  }
  const bool own1 = own && i2 + 1 < ND;
#pragma unroll 1
  for (int k = 0; k < ND; ++k) {
    // buffers alternate: the reads of pivot k-1 need no barrier before these writes, and those of
    // pivot k-2 lie behind the last one
    double* W = s + S::R + (k & 1) * S::RL;
    if (own) {
      W[i2] = a[0][0];
      W[i2 + ND] = a[0][0];
    }
    if (own1) {
      W[i2 + 1] = a[1][0];
      W[i2 + 1 + ND] = a[1][0];
    }
    if (own && (k & ~1) == i2) s[S::ID + (k & 1)] = 1.0 / ((k & 1) ? a[1][0] : a[0][0]);
    __syncthreads();
    const double id = s[S::ID + (k & 1)];
    double g0 = a[0][0] * id, g1 = a[1][0] * id, m0 = -g0, m1 = -g1;
    if (i2 == k) {
      m0 = id;
      g0 = -id;
#pragma unroll
      for (int j = 1; j < ND; ++j) a[0][j] = 0.0;
    } else if (i2 + 1 == k) {
      m1 = id;
      g1 = -id;
#pragma unroll
      for (int j = 1; j < ND; ++j) a[1][j] = 0.0;
    }
    const double* v = W + k + 1;
#pragma unroll
    for (int j = 0; j + 1 < ND; ++j) {
      a[0][j] = fma(m0, v[j], a[0][j + 1]);
      a[1][j] = fma(m1, v[j], a[1][j + 1]);
    }
    a[0][ND - 1] = g0;
    a[1][ND - 1] = g1;
  }
  __syncthreads();  // the forming arrays are long consumed; the packed inverse takes their place
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int r = i2 + h;
    if (h == 0 ? own : own1)
#pragma unroll
      for (int j = 0; j < ND; ++j)
        if (j <= r) s[r * (r + 1) / 2 + j] = -a[h][j];
  }
  __syncthreads();
  for (int e = t; e < nc * kNPK; e += NT) Lg[(size_t)c0 * kNPK + e] = sm[(e / kNPK) * S::CELL + e % kNPK];
}

cudaError_t mass_factor(const MeshDev& mesh, const double* weight, double* L, int ncell, cudaStream_t st) {
  static std::atomic<unsigned long long> configured{0};
  const cudaError_t e = allow_smem(k_mass_inverse, InvShape::BYTES, configured);
  if (e != cudaSuccess) return e;
  k_mass_inverse<<<(ncell + kInvCells - 1) / kInvCells, kInvThreads, InvShape::BYTES, st>>>(mesh, weight, L, ncell);
  return cudaGetLastError();
}

// x = scale * M_K^{-1} b per cell and component: one warp per cell stages the cell's packed
// symmetric inverse (contiguous, coalesced) and its right-hand sides in shared memory by
// asynchronous copies, then lane i forms row i.  One load round trip per cell, so small
// grids are not latency-bound.
// MODE 1 is the Chebyshev update of the multigrid smoother: with y = M_K^{-1} b,
// d = alpha d + scale y (d not read when alpha == 0), then x = d (first step) or x += d.
constexpr int kSolveWarps = 4;
template <class R, int MODE>
__global__ void __launch_bounds__(32 * kSolveWarps)
    k_mass_solve(const R* __restrict__ Minv, const R* __restrict__ b, R* __restrict__ x, R* __restrict__ dv,
                 const R scale, const R alpha, const int first, const int ncomp, const int ncell, int* status) {
  constexpr int ND = kND, NPK = kNPK;
  __shared__ alignas(16) R sM[kSolveWarps * NPK];
  __shared__ alignas(16) R sb[kSolveWarps * 2 * ND];
  __shared__ alignas(8) unsigned long long s_bar;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * kSolveWarps, c = c0 + warp;
  // A full block's inverses and right-hand sides are contiguous: one bulk copy (TMA) each when
  // the chunks are 16-byte multiples, else per-element asynchronous copies per warp.
  const size_t mbytes = sizeof(R) * (size_t)kSolveWarps * NPK, bbytes = sizeof(R) * (size_t)kSolveWarps * ncomp * ND;
  const bool bulk = c0 + kSolveWarps <= ncell && mbytes % 16 == 0 && bbytes % 16 == 0 &&
                    (reinterpret_cast<uintptr_t>(Minv + (size_t)c0 * NPK) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(b + (size_t)c0 * ncomp * ND) & 15) == 0;
  if (bulk) {
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&s_bar);
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"((unsigned)(mbytes + bbytes))
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(sM)),
                   "l"(Minv + (size_t)c0 * NPK), "r"((unsigned)mbytes), "r"(bar)
                   : "memory");
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                       (unsigned)__cvta_generic_to_shared(sb)),
                   "l"(b + (size_t)c0 * ncomp * ND), "r"((unsigned)bbytes), "r"(bar)
                   : "memory");
    }
    __syncthreads();  // barrier initialised before anyone waits on it
    const bool ok = mbar_wait(bar, 0);
    if (!ok) report_status(status, kStatusStageTimeout);
    if (__syncthreads_or(!ok)) {  // never expected; every thread leaves together
      if (threadIdx.x == 0) mbar_wait(bar, 0);  // (bounded) for the copies still in flight
      return;
    }
  } else {
    if (c >= ncell) return;  // whole warps only; no block-wide barrier on this path
    const R* mp = Minv + (size_t)c * NPK;
    for (int k = lane; k < NPK; k += 32) cp_async_el(&sM[warp * NPK + k], mp + k);
    const R* bp = b + (size_t)c * ncomp * ND;
    for (int k = lane; k < ncomp * ND; k += 32) cp_async_el(&sb[warp * ncomp * ND + k], bp + k);
    cp_async_wait_all();
    __syncwarp();
  }
  const R* M = sM + warp * NPK;
  const R* bb = sb + warp * ncomp * ND;
  for (int i = lane; i < ND; i += 32) {
    const int ri = i * (i + 1) / 2;
    R y0 = R(0), y1 = R(0);  // both components share each matrix load
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const R m = M[j <= i ? ri + j : j * (j + 1) / 2 + i];
      y0 = fmaR(m, bb[j], y0);
      if (ncomp == 2) y1 = fmaR(m, bb[ND + j], y1);
    }
    for (int d = 0; d < ncomp; ++d) {
      const R y = d == 0 ? y0 : y1;
      const size_t o = ((size_t)c * ncomp + d) * ND + i;
      if constexpr (MODE == 0) {
        x[o] = scale * y;
      } else {
        const R nd = (alpha != R(0) ? alpha * dv[o] : R(0)) + scale * y;
        dv[o] = nd;
        x[o] = first ? nd : x[o] + nd;
      }
    }
  }
}

template <class R, int MODE>
cudaError_t launch_mass_solve(const R* L, int ncomp, const R* b, R scale, R* x, R* d, R alpha, int first, int ncell,
                              int* status, cudaStream_t st) {
  if (ncomp < 1 || ncomp > 2) return cudaErrorInvalidValue;
  k_mass_solve<R, MODE><<<(ncell + kSolveWarps - 1) / kSolveWarps, 32 * kSolveWarps, 0, st>>>(L, b, x, d, scale, alpha,
                                                                                             first, ncomp, ncell, status);
  return cudaGetLastError();
}

cudaError_t mass_solve(const double* L, int ncomp, const double* b, double scale, double* x, int ncell, int* status,
                       cudaStream_t st) {
  return launch_mass_solve<double, 0>(L, ncomp, b, scale, x, nullptr, 0.0, 0, ncell, status, st);
}

// ------------------------------------------------------------------ multigrid kernels
// r += C0 w - D p: CPhys with SIGN +1 gives +C0 w; the D term enters with -g1
template <class R>
cudaError_t mg_res(const MeshDev& mesh, const R* w, const R* pf, const R* p, const CParamsT<R>& prm, R* r, int ncell,
                   cudaStream_t st) {
  ArgPtrs<3, 1, R> a{{p, w, pf}, {r}};
  CParamsT<R> q = prm;
  q.g1 = -prm.g1;
  return launch_cellop<P, CPhys<true, 1, R, false, true>>(mesh, a, q, ncell, st);
}

template <class R>
cudaError_t cheb(const R* L, const R* r, R alpha, R s, R* d, R* x, int first, int ncell, int* status,
                 cudaStream_t st) {
  return launch_mass_solve<R, 1>(L, 1, r, s, x, d, alpha, first, ncell, status, st);
}

template <class R>
__device__ __forceinline__ const TransT<P, R>& trans();
template <>
__device__ __forceinline__ const TransT<P, double>& trans<double>() {
  return c_tr;
}
template <>
__device__ __forceinline__ const TransT<P, float>& trans<float>() {
  return c_trf;
}

// One thread per fine node: xf[k] += sum_j Pz[kz][jz] Px[kx][jx] xc[j] over the parent cell.
template <class R>
__global__ void k_prolong(const R* __restrict__ xc, R* __restrict__ xf, const int nxc, const int nzc) {
  constexpr int P1 = P + 1, ND = P1 * P1;
  __shared__ R sP[2][P1][P1];
  for (int k = threadIdx.x; k < 2 * P1 * P1; k += blockDim.x) (&sP[0][0][0])[k] = (&trans<R>().Pm[0][0][0])[k];
  __syncthreads();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long total = 4L * nxc * nzc * ND;
  if (idx >= total) return;
  const int cf = (int)(idx / ND), k = (int)(idx % ND);
  const int nxf = 2 * nxc, i_f = cf % nxf, j_f = cf / nxf;
  const int ox = i_f & 1, oz = j_f & 1, cc = (j_f >> 1) * nxc + (i_f >> 1);
  const int kx = k % P1, kz = k / P1;
  const R* x = xc + (size_t)cc * ND;
  R s = 0;
#pragma unroll
  for (int jz = 0; jz < P1; ++jz) {
    R t = 0;
#pragma unroll
    for (int jx = 0; jx < P1; ++jx) t = fmaR(sP[ox][kx][jx], x[jz * P1 + jx], t);
    s = fmaR(sP[oz][kz][jz], t, s);
  }
  xf[idx] += s;
}

// One thread per coarse node: rc[k] = sum over children and child nodes of P^T rf.
template <class R>
__global__ void k_restrict(const R* __restrict__ rf, R* __restrict__ rc, const int nxc, const int nzc) {
  constexpr int P1 = P + 1, ND = P1 * P1;
  __shared__ R sP[2][P1][P1];
  for (int k = threadIdx.x; k < 2 * P1 * P1; k += blockDim.x) (&sP[0][0][0])[k] = (&trans<R>().Pm[0][0][0])[k];
  __syncthreads();
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long total = (long)nxc * nzc * ND;
  if (idx >= total) return;
  const int cc = (int)(idx / ND), k = (int)(idx % ND);
  const int ic = cc % nxc, jc = cc / nxc, nxf = 2 * nxc;
  const int kx = k % P1, kz = k / P1;
  R s = 0;
#pragma unroll
  for (int oz = 0; oz < 2; ++oz)
#pragma unroll
    for (int ox = 0; ox < 2; ++ox) {
      const R* r = rf + (size_t)((2 * jc + oz) * nxf + 2 * ic + ox) * ND;
#pragma unroll
      for (int iz = 0; iz < P1; ++iz) {
        R t = 0;
#pragma unroll
        for (int ix = 0; ix < P1; ++ix) t = fmaR(sP[ox][ix][kx], r[iz * P1 + ix], t);
        s = fmaR(sP[oz][iz][kz], t, s);
      }
    }
  rc[idx] = s;
}

// One thread per coarse node: value of the child polynomial containing the node.
__global__ void k_inject(const double* __restrict__ ff, double* __restrict__ fc, const int nxc, const int nzc) {
  constexpr int P1 = P + 1, ND = P1 * P1;
  const long idx = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long total = (long)nxc * nzc * ND;
  if (idx >= total) return;
  const TransT<P, double>& tr = c_tr;
  const int cc = (int)(idx / ND), k = (int)(idx % ND);
  const int ic = cc % nxc, jc = cc / nxc, nxf = 2 * nxc;
  const int kx = k % P1, kz = k / P1;
  const int ox = tr.ch[kx], oz = tr.ch[kz];
  const double* f = ff + (size_t)((2 * jc + oz) * nxf + 2 * ic + ox) * ND;
  double s = 0.0;
  for (int jz = 0; jz < P1; ++jz) {
    double t = 0.0;
    for (int jx = 0; jx < P1; ++jx) t = fma(tr.E[kx][jx], f[jz * P1 + jx], t);
    s = fma(tr.E[kz][jz], t, s);
  }
  fc[idx] = s;
}

// ------------------------------------------------------------------ adjoint
// Cells per CTA of the tangents and adjoints (fit_cells takes fewer where two CTAs would not share an
// SM): whole warps up to degree 3.  Measured, us of the stage-1 backward at 128x64 and 512x256 cells:
//   p=1  21: 10.9, 104;  16: 14.8, 114;  32: 14.2, 114;  42: 11.2, 106 (at 160x80 cells 18.0, 14.9, 14.4, 18.2:
//        the remainder of CTAs per SM)
//   p=2  12: 19.4, 183;  16: 22.9, 230;  19: 20.9, 249      p=3  9: 32.8, 393;  8: 33.6, 436;  13: 34.9, 428;  10: 40.0, 522
//   p=4  10: 41.9, 575;  7: 39.4, 590 (the tangent 535 and 744)
//   p=5  10 (6 by fit_cells): 84.3, 1188;  5: 90.4, 1348      p=6  10 (4 by fit_cells): 112, 1728
constexpr int kAdjCells = P == 1 ? 21 : (P == 2 ? 12 : (P == 3 ? 9 : 10));
cudaError_t rhs_adjoint1(const MeshDev& mesh, const double* const* in, const double* const* ybar,
                         double* const* xbar, const RhsParams& prm, int ncell, cudaStream_t st) {
  ArgPtrs<8, 5> a{{in[0], in[1], in[2], in[3], in[4], ybar[0], ybar[1], ybar[2]},
                  {xbar[0], xbar[1], xbar[2], xbar[3], xbar[4]}};
  return launch_cellop<P, RhsAdj1Phys, fit_cells<P, RhsAdj1Phys, kAdjCells>()>(mesh, a, prm, ncell, st);
}

cudaError_t rhs_tangent1(const MeshDev& mesh, const double* const* in, const double* const* din, double* const* dy,
                         const RhsParams& prm, int ncell, cudaStream_t st) {
  ArgPtrs<10, 3> a{{in[0], in[1], in[2], in[3], in[4], din[0], din[1], din[2], din[3], din[4]}, {dy[0], dy[1], dy[2]}};
  return launch_cellop<P, RhsTlm1Phys, fit_cells<P, RhsTlm1Phys, kAdjCells>()>(mesh, a, prm, ncell, st);
}

// ---- automatic tangents and adjoints of the fused rhs triple of any stage (dual numbers).
// Vectors in the fused order: rho_j, u_j, p_j for each explicit stage j, then rho_c, u_fixed.
template <int STAGE>
cudaError_t rhs_tangent_s(const MeshDev& mesh, const double* const* in, const double* const* din, double* const* dy,
                          const RhsParams& prm, int ncell, cudaStream_t st) {
  using Ph = RhsTanPhys<STAGE>;
  using B = RhsPhys<STAGE, 7>;
  ArgPtrs<PhysInfo<Ph>::NARR_TOTAL, 3> a{};
  int k = 0;
  for (int j = 0; j < STAGE; ++j) {
    for (int c = 0; c < 3; ++c) a.in[k++] = in[3 * j + c];
    for (int c = 0; c < 3; ++c) a.in[k++] = din[3 * j + c];
    if (B::quirk_group(j)) {  // u_old of the stage-2 kinetic jump
      a.in[k++] = in[1];
      a.in[k++] = din[1];
    }
  }
  a.in[k++] = in[3 * STAGE];
  a.in[k++] = in[3 * STAGE + 1];
  a.in[k++] = din[3 * STAGE];
  a.in[k++] = din[3 * STAGE + 1];
  a.out[0] = dy[0];
  a.out[1] = dy[1];
  a.out[2] = dy[2];
  for (int i = 0; i < k; ++i)
    if (!a.in[i]) return cudaErrorInvalidValue;
  return launch_cellop<P, Ph, fit_cells<P, Ph, kAdjCells>()>(mesh, a, prm, ncell, st);
}

template <int STAGE, int G>
cudaError_t rhs_adj_group(const MeshDev& mesh, const double* const* in, const double* const* ybar, double* const* xbar,
                          double* scratch, const RhsParams& prm, int ncell, cudaStream_t st) {
  using Ph = RhsAdjGPhys<STAGE, G>;
  ArgPtrs<Ph::NB + 3, Ph::NB> a{};
  const int base = 3 * G;  // the group's first vector in the fused order (implicit group: 3 STAGE)
  for (int i = 0; i < Ph::NBC; ++i) {
    a.in[i] = in[base + i];
    a.out[i] = xbar[base + i];
  }
  a.in[Ph::NBC] = ybar[0];
  a.in[Ph::NBC + 1] = ybar[1];
  a.in[Ph::NBC + 2] = ybar[2];
  if constexpr (Ph::Q) {  // u_old: its cotangent goes to scratch, added to u_0's by the caller
    a.in[Ph::NBC + 3] = in[1];
    a.out[Ph::NBC] = scratch;
  }
  return launch_cellop<P, Ph, fit_cells<P, Ph, kAdjCells>()>(mesh, a, prm, ncell, st);
}

__global__ void k_add(const double* __restrict__ x, double* __restrict__ y, const long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) y[i] += x[i];
}

// host-side compile-time loop (sfor is device-only)
template <class F, int... I>
void host_for_impl(F& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
void host_for(F&& f) {
  host_for_impl(f, std::make_integer_sequence<int, N>{});
}

template <int STAGE>
cudaError_t rhs_adjoint_s(const MeshDev& mesh, const double* const* in, const double* const* ybar, double* const* xbar,
                          double* scratch, const RhsParams& prm, int ncell, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  host_for<STAGE + 1>([&](auto gc) {
    constexpr int G = decltype(gc)::value;
    if (e == cudaSuccess) e = rhs_adj_group<STAGE, G>(mesh, in, ybar, xbar, scratch, prm, ncell, st);
  });
  if (e != cudaSuccess) return e;
  if constexpr (RhsPhys<STAGE, 7>::quirk_group(1)) {
    const long n = 2L * ncell * kND;
    k_add<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(scratch, xbar[1], n);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t rhs_tangent(const MeshDev& mesh, int stage, const double* const* in, const double* const* din,
                        double* const* dy, const RhsParams& prm, int ncell, cudaStream_t st) {
  switch (stage) {
    case 1: return rhs_tangent_s<1>(mesh, in, din, dy, prm, ncell, st);
    case 2: return rhs_tangent_s<2>(mesh, in, din, dy, prm, ncell, st);
    case 3: return rhs_tangent_s<3>(mesh, in, din, dy, prm, ncell, st);
    default: return cudaErrorInvalidValue;
  }
}
cudaError_t rhs_adjoint(const MeshDev& mesh, int stage, const double* const* in, const double* const* ybar,
                        double* const* xbar, double* scratch, const RhsParams& prm, int ncell, cudaStream_t st) {
  switch (stage) {
    case 1: return rhs_adjoint_s<1>(mesh, in, ybar, xbar, scratch, prm, ncell, st);
    case 2: return rhs_adjoint_s<2>(mesh, in, ybar, xbar, scratch, prm, ncell, st);
    case 3: return rhs_adjoint_s<3>(mesh, in, ybar, xbar, scratch, prm, ncell, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t op_BT(const MeshDev& mesh, const double* ubar, double c, double* pbar, int ncell, cudaStream_t st) {
  ArgPtrs<1, 1> a{{ubar}, {pbar}};
  return launch_cellop<P, BTPhys>(mesh, a, BParams{c}, ncell, st);
}
cudaError_t op_C_tangent(const MeshDev& mesh, const double* w, const double* dw, const double* pf,
                         const CParams& prm, double* dst, int ncell, cudaStream_t st) {
  ArgPtrs<3, 1> a{{w, dw, pf}, {dst}};
  return launch_cellop<P, CTlmPhys>(mesh, a, prm, ncell, st);
}
cudaError_t op_CT(const MeshDev& mesh, const double* w, const double* pf, const double* pbar, const CParams& prm,
                  double* wbar, int ncell, cudaStream_t st) {
  ArgPtrs<3, 1> a{{w, pf, pbar}, {wbar}};
  return launch_cellop<P, CTPhys>(mesh, a, prm, ncell, st);
}

// ------------------------------------------------------------------ change-of-basis inverses
// Gauss-point inverse weights of a cell's mass matrix: W[c][qz (P+1) + qx] = 1 / (rho JxW) at
// the (P+1)-point Gauss points (rho = 1 when null), for the sum-factorised inverse
// M_K^{-1} = Vi diag(W) Vi^T of CobT (exact for the plain mass matrix on bilinear cells).
template <class R>
__global__ void k_cob_weights(const MeshDev mesh, const double* __restrict__ rho, R* __restrict__ W, const int ncell) {
  constexpr int P1 = P + 1, ND = P1 * P1;
  const long e = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long)ncell * ND) return;
  const int c = (int)(e / ND), q = (int)(e % ND), qx = q % P1, qz = q / P1;
  const CobT<P, double>& cb = c_cob;
  const int i = c % mesh.nx, j = c / mesh.nx, Wd = mesh.nx + 1;
  const double2 v0 = mesh.vtx[j * Wd + i], v1 = mesh.vtx[j * Wd + i + 1];
  const double2 v2 = mesh.vtx[(j + 1) * Wd + i], v3 = mesh.vtx[(j + 1) * Wd + i + 1];
  const double Ax = v1.x - v0.x, Az = v1.y - v0.y, Cx = v2.x - v0.x, Cz = v2.y - v0.y;
  const double Bx = v3.x - v2.x - v1.x + v0.x, Bz = v3.y - v2.y - v1.y + v0.y;
  const double xi = cb.g[qx], eta = cb.g[qz];
  const double J00 = fma(Bx, eta, Ax), J10 = fma(Bz, eta, Az), J01 = fma(Bx, xi, Cx), J11 = fma(Bz, xi, Cz);
  double f = (J00 * J11 - J01 * J10) * cb.w[qx] * cb.w[qz];
  if (rho) {
    const double* rc = rho + (size_t)c * ND;
    double rv = 0.0;
#pragma unroll
    for (int iz = 0; iz < P1; ++iz) {
      double t = 0.0;
#pragma unroll
      for (int ix = 0; ix < P1; ++ix) t = fma(cb.V[qx][ix], rc[iz * P1 + ix], t);
      rv = fma(cb.V[qz][iz], t, rv);
    }
    f *= rv;
  }
  W[e] = (R)(1.0 / f);
}

// x = scale M_K^{-1} b per cell and component by the change of basis (MODE 0), or the
// Chebyshev update d = alpha d + scale M_K^{-1} b, x = d (first) or x += d (MODE 1, ncomp 1).
// Tasks are (component, cell, line) over three passes in shared memory.
constexpr int kCobCells = 32;
template <class R, int MODE>
__global__ void __launch_bounds__(128)
    k_cob_solve(const R* __restrict__ W, const R* __restrict__ b, R* __restrict__ x, R* __restrict__ dv,
                const R scale, const R alpha, const int first, const int ncomp, const int ncell) {
  constexpr int P1 = P + 1, ND = P1 * P1;
  __shared__ R sy[kCobCells * 2 * ND];
  __shared__ R sw[kCobCells * ND];
  const CobT<P, R>& cb = cobr<P, R>();
  const int c0 = blockIdx.x * kCobCells, ncb = min(kCobCells, ncell - c0);
  for (int e = threadIdx.x; e < ncb * ncomp * ND; e += blockDim.x) sy[e] = b[(size_t)c0 * ncomp * ND + e];
  for (int e = threadIdx.x; e < ncb * ND; e += blockDim.x) sw[e] = W[(size_t)c0 * ND + e];
  __syncthreads();
  const int nt = ncomp * ncb * P1;  // tasks (cell, component, line); sy is [cell][comp][node]
  for (int e = threadIdx.x; e < nt; e += blockDim.x) {  // along x, in place per row
    R* row = sy + (e / P1) * ND + (e % P1) * P1;
    R y[P1];
#pragma unroll
    for (int ix = 0; ix < P1; ++ix) y[ix] = row[ix];
#pragma unroll
    for (int qx = 0; qx < P1; ++qx) {
      R t = R(0);
#pragma unroll
      for (int ix = 0; ix < P1; ++ix) t = fmaR(cb.Vi[ix][qx], y[ix], t);
      row[qx] = t;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nt; e += blockDim.x) {  // along z per column, weights, back
    const int cc = e / (ncomp * P1), qx = e % P1;
    R* col = sy + (e / P1) * ND + qx;
    R u[P1], t[P1];
#pragma unroll
    for (int iz = 0; iz < P1; ++iz) u[iz] = col[iz * P1];
#pragma unroll
    for (int qz = 0; qz < P1; ++qz) {
      R a = R(0);
#pragma unroll
      for (int iz = 0; iz < P1; ++iz) a = fmaR(cb.Vi[iz][qz], u[iz], a);
      t[qz] = a * sw[cc * ND + qz * P1 + qx];
    }
#pragma unroll
    for (int iz = 0; iz < P1; ++iz) {
      R a = R(0);
#pragma unroll
      for (int qz = 0; qz < P1; ++qz) a = fmaR(cb.Vi[iz][qz], t[qz], a);
      col[iz * P1] = a;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nt; e += blockDim.x) {  // along x, then the store or update
    const R* row = sy + (e / P1) * ND + (e % P1) * P1;
    R v[P1];
#pragma unroll
    for (int qx = 0; qx < P1; ++qx) v[qx] = row[qx];
#pragma unroll
    for (int ix = 0; ix < P1; ++ix) {
      R y = R(0);
#pragma unroll
      for (int qx = 0; qx < P1; ++qx) y = fmaR(cb.Vi[ix][qx], v[qx], y);
      const size_t g = (size_t)c0 * ncomp * ND + (size_t)(e / P1) * ND + (e % P1) * P1 + ix;
      if constexpr (MODE == 0) {
        x[g] = scale * y;
      } else {
        const R nd = (alpha != R(0) ? alpha * dv[g] : R(0)) + scale * y;
        dv[g] = nd;
        x[g] = first ? nd : x[g] + nd;
      }
    }
  }
}

template <class R>
cudaError_t cob_weights(const MeshDev& mesh, const double* rho, R* W, int ncell, cudaStream_t st) {
  const long n = (long)ncell * kND;
  k_cob_weights<R><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(mesh, rho, W, ncell);
  return cudaGetLastError();
}
template <class R>
cudaError_t cob_solve(const R* W, int ncomp, const R* b, R scale, R* x, int ncell, cudaStream_t st) {
  if (ncomp < 1 || ncomp > 2) return cudaErrorInvalidValue;
  k_cob_solve<R, 0><<<(ncell + kCobCells - 1) / kCobCells, 128, 0, st>>>(W, b, x, nullptr, scale, R(0), 0, ncomp,
                                                                         ncell);
  return cudaGetLastError();
}
template <class R>
cudaError_t cob_cheb(const R* W, const R* r, R alpha, R s, R* d, R* x, int first, int ncell, cudaStream_t st) {
  k_cob_solve<R, 1><<<(ncell + kCobCells - 1) / kCobCells, 128, 0, st>>>(W, r, x, d, s, alpha, first, 1, ncell);
  return cudaGetLastError();
}

// ------------------------------------------------------------------ fused epilogues
// Launch shapes of the nodal FP32 smoother's kernels (cells per CTA; CTAs per SM asked of the compiler).
// Measured, us of the degree-16 polynomial with P+1 points per direction at 64x32, 256x128 and 512x256:
//   p=4  32: 162, 393, 1269;  16: 218, 435, 1424      p=3  16: 144, 334, 944;  32: 140, 334, 954 (with 2P+1
//   points 215, 434, 1477 and 155, 412, 1393; the multigrid solve at 256x128 18.6 and 19.2 ms)
// CTAs per SM at p = 4, (B with A^-1, residual): (3, 2) and (2, 3) the same times; p = 3, 16 cells, 3, 6
// and 8 the same solve.
constexpr int kFusedCB = P == 4 ? 32 : cells_per_block<P, float>();
constexpr int kFusedMinB = P == 3 || P == 5 ? 3 : 2;
constexpr int kBInvMinB = P == 4 ? 3 : kFusedMinB;
constexpr int kResChebMinB = kFusedMinB;
template <class R>
cudaError_t b_inv(const MeshDev& mesh, const R* p, R c, const R* WA, R scale, R* w, int ncell, cudaStream_t st) {
  ArgPtrs<1, 1, R> a{{p}, {w}};
  BInvParams<R> q;
  q.c = c;
  q.inv = WA;
  q.scale = scale;
  return launch_cellop<P, BInvPhys<R>, kFusedCB, kBInvMinB>(mesh, a, q, ncell, st);
}

template <class R>
cudaError_t res_cheb(const MeshDev& mesh, const R* w, const R* pf, const R* din, const CParamsT<R>& prm, const R* WM,
                     R alpha, R s, R* r, R* dout, R* x, int first, int ncell, cudaStream_t st) {
  if (din == dout) return cudaErrorInvalidValue;
  ArgPtrs<3, 1, R> a{{din, w, pf}, {r}};
  ResChebParams<R> q;
  static_cast<CParamsT<R>&>(q) = prm;
  q.g1 = -prm.g1;
  q.inv = WM;
  q.alpha = alpha;
  q.s = s;
  q.r = r;
  q.din = din;
  q.dout = dout;
  q.x = x;
  q.first = first;
  return launch_cellop<P, ResChebPhys<R>, kFusedCB, kResChebMinB>(mesh, a, q, ncell, st);
}

// reduced-quadrature (P+1 Gauss points) counterparts of mg_res, b_inv and res_cheb in FP32
cudaError_t mg_res_fr(const MeshDev& mesh, const float* w, const float* pf, const float* p, const CParamsT<float>& prm,
                      float* r, int ncell, cudaStream_t st) {
  ArgPtrs<3, 1, float> a{{p, w, pf}, {r}};
  CParamsT<float> q = prm;
  q.g1 = -prm.g1;
  return launch_cellop<P, CResRPhys<float>, kFusedCB, kResChebMinB>(mesh, a, q, ncell, st);
}
cudaError_t b_inv_fr(const MeshDev& mesh, const float* p, float c, const float* WA, float scale, float* w, int ncell,
                     cudaStream_t st) {
  ArgPtrs<1, 1, float> a{{p}, {w}};
  BInvParams<float> q;
  q.c = c;
  q.inv = WA;
  q.scale = scale;
  return launch_cellop<P, BInvRPhys<float>, kFusedCB, kBInvMinB>(mesh, a, q, ncell, st);
}
cudaError_t res_cheb_fr(const MeshDev& mesh, const float* w, const float* pf, const float* din,
                        const CParamsT<float>& prm, const float* WM, float alpha, float s, float* r, float* dout,
                        float* x, int first, int ncell, cudaStream_t st) {
  if (din == dout) return cudaErrorInvalidValue;
  ArgPtrs<3, 1, float> a{{din, w, pf}, {r}};
  ResChebParams<float> q;
  static_cast<CParamsT<float>&>(q) = prm;
  q.g1 = -prm.g1;
  q.inv = WM;
  q.alpha = alpha;
  q.s = s;
  q.r = r;
  q.din = din;
  q.dout = dout;
  q.x = x;
  q.first = first;
  return launch_cellop<P, ResChebRPhys<float>, kFusedCB, kResChebMinB>(mesh, a, q, ncell, st);
}

// the smoother step on the preconditioned residual z (ResChebZPhys): the kernel evaluates C0 w
// alone; full (2P+1) or reduced (P+1) Gauss points per direction
template <class Phys>
cudaError_t res_chebz_launch(const MeshDev& mesh, const float* w, const float* pf, const float* din,
                             const CParamsT<float>& prm, const float* WM, float g, float alpha, float s, float* z,
                             float* dout, float* x, int first, int ncell, cudaStream_t st) {
  if (din == dout) return cudaErrorInvalidValue;
  ArgPtrs<2, 1, float> a{{w, pf}, {z}};
  ResChebZParams<float> q;
  static_cast<CParamsT<float>&>(q) = prm;
  q.inv = WM;
  q.g = g;
  q.alpha = alpha;
  q.s = s;
  q.r = z;
  q.din = din;
  q.dout = dout;
  q.x = x;
  q.first = first;
  return launch_cellop<P, Phys, kFusedCB, kResChebMinB>(mesh, a, q, ncell, st);
}
cudaError_t res_chebz_f(const MeshDev& mesh, const float* w, const float* pf, const float* din,
                        const CParamsT<float>& prm, const float* WM, float g, float alpha, float s, float* z,
                        float* dout, float* x, int first, int reduced, int ncell, cudaStream_t st) {
  return reduced ? res_chebz_launch<ResChebZRPhys<float>>(mesh, w, pf, din, prm, WM, g, alpha, s, z, dout, x, first,
                                                          ncell, st)
                 : res_chebz_launch<ResChebZPhys<float>>(mesh, w, pf, din, prm, WM, g, alpha, s, z, dout, x, first,
                                                         ncell, st);
}

// ------------------------------------------------------------------ Gauss-point smoother
template <class K, class... A>
cudaError_t launch_gs(K kernel, int ncell, cudaStream_t st, bool pdl, A... args) {
  const int nblk = (ncell + kGsTile - 1) / kGsTile;
  if (ncell <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)nblk);
  cfg.blockDim = dim3((unsigned)GsShape<P>::NT);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = (kPDL && pdl) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
GsMesh gs_mesh(const MeshDev& m, const GsGeo& geo, int ncell) {
  return {geo.map, geo.det, FastDiv::make(m.nx), m.nz, m.periodic_x, ncell, m.status, m.test_wait_polls};
}
// words of one of the two face arrays of k_gs_chain (the mark of a given-up wait follows the second)
size_t gs_words(int ncell) { return (size_t)(ncell + kGsTile - 1) / kGsTile * kGsTile * 4 * (P + 1); }
cudaError_t gs_geo(const MeshDev& mesh, GsGeo geo, int ncell, cudaStream_t st) {
  k_gs_geo<<<(ncell + 255) / 256, 256, 0, st>>>(mesh, geo.map, geo.det, ncell);
  return cudaGetLastError();
}
cudaError_t gs_entry(const MeshDev& mesh, const GsGeo& geo, const double* v, float sc, float theta, float* z, float* d,
                     float* x, float* dtr, unsigned long long* words, int ncell, cudaStream_t st) {
  return launch_gs(k_gs_entry<P>, ncell, st, true, gs_mesh(mesh, geo, ncell), v, sc, theta, z, d, x, dtr, words,
                   words ? words + gs_words(ncell) : nullptr, words ? words + 2 * gs_words(ncell) : nullptr);
}
int gs_chain_tiles(int device) {
  int sms = 0, per = 0, coop = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_gs_chain<P>, GsShape<P>::NT, 0) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return coop ? sms * per : 0;
}
cudaError_t gs_chain(const MeshDev& mesh, const GsGeo& geo, const float* coef, int n, float cB, float cgg, float g,
                     const float* WA, const float* pg, const float* ptr, float* z, float* d, float* x, float* dtr,
                     unsigned long long* words, int ncell, cudaStream_t st, int* launched) {
  *launched = 0;
  if (ncell <= 0) return cudaSuccess;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)((ncell + kGsTile - 1) / kGsTile));
  cfg.blockDim = dim3((unsigned)GsShape<P>::NT);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  for (int k = 0; k < n; k += kGsSteps) {
    GsSteps s{};
    s.n = n - k < kGsSteps ? n - k : kGsSteps;
    for (int i = 0; i < s.n; ++i) {
      s.alpha[i] = coef[2 * (k + i)];
      s.s[i] = coef[2 * (k + i) + 1];
    }
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_gs_chain<P>, gs_mesh(mesh, geo, ncell), s, cB, cgg, g, WA, pg, ptr,
                                             z, d, x, dtr, words, words + gs_words(ncell), words + 2 * gs_words(ncell), 2 * k,
                                             k + s.n < n ? 1 : 0);
    if (e != cudaSuccess) return e;
    ++*launched;
  }
  return cudaSuccess;
}
cudaError_t gs_binv(const MeshDev& mesh, const GsGeo& geo, const float* d, const float* dtr, float cB, const float* WA,
                    const float* pg, const float* ptr, float cgg, float* fx, float* fe, float* gf, int ncell,
                    cudaStream_t st) {
  return launch_gs(k_gs_binv<P>, ncell, st, true, gs_mesh(mesh, geo, ncell), d, dtr, cB, WA, pg, ptr, cgg, fx, fe, gf);
}
cudaError_t gs_zstep(const MeshDev& mesh, const GsGeo& geo, const float* fx, const float* fe, const float* gf, float g,
                     float alpha, float s, float* z, float* d, float* x, int xmode, float* dtr, int ncell,
                     cudaStream_t st) {
  return launch_gs(k_gs_zstep<P>, ncell, st, true, gs_mesh(mesh, geo, ncell), fx, fe, gf, g, alpha, s, z, d, x, xmode,
                   dtr);
}
cudaError_t gs_exit(const float* x, double* out, const unsigned long long* words, int ncell, cudaStream_t st) {
  return launch_gs(k_gs_exit<P>, ncell, st, true, x, out, words ? words + 2 * gs_words(ncell) : nullptr, ncell);
}
cudaError_t gs_values(const MeshDev& mesh, const double* p, const double* rho, float* pg, float* ptr, float* WA,
                      int ncell, cudaStream_t st) {
  return launch_gs(k_gs_values<P>, ncell, st, false, mesh, p, rho, pg, ptr, WA, ncell);
}

cudaError_t op_A_rho_T(const MeshDev& mesh, const double* x, const double* y, double* rhobar, int ncell,
                       cudaStream_t st) {
  ArgPtrs<2, 1> a{{x, y}, {rhobar}};
  return launch_cellop<P, MassRhoTPhys>(mesh, a, MassParams{1.0}, ncell, st);
}
cudaError_t op_C_pf_T(const MeshDev& mesh, const double* w, const double* pbar, const CParams& prm, double* pfbar,
                      int ncell, cudaStream_t st) {
  ArgPtrs<2, 1> a{{w, pbar}, {pfbar}};
  return launch_cellop<P, CPfTPhys>(mesh, a, prm, ncell, st);
}

constexpr int kTransferThreads = 256;

template <class R>
cudaError_t prolong(const R* xc, R* xf, int nxc, int nzc, cudaStream_t st) {
  const long n = 4L * nxc * nzc * kND;
  k_prolong<R><<<(unsigned)((n + kTransferThreads - 1) / kTransferThreads), kTransferThreads, 0, st>>>(xc, xf, nxc, nzc);
  return cudaGetLastError();
}
template <class R>
cudaError_t restrict_(const R* rf, R* rc, int nxc, int nzc, cudaStream_t st) {
  const long n = (long)nxc * nzc * kND;
  k_restrict<R><<<(unsigned)((n + kTransferThreads - 1) / kTransferThreads), kTransferThreads, 0, st>>>(rf, rc, nxc, nzc);
  return cudaGetLastError();
}
cudaError_t inject(const double* ff, double* fc, int nxc, int nzc, cudaStream_t st) {
  const long n = (long)nxc * nzc * kND;
  k_inject<<<(unsigned)((n + kTransferThreads - 1) / kTransferThreads), kTransferThreads, 0, st>>>(ff, fc, nxc, nzc);
  return cudaGetLastError();
}

const DegreeOps kOps = {upload_tables,     rhs,
                        mass,              op_B,
                        op_C,              inv_diag,
                        mass_factor,       mass_solve,
                        kND % 2 ? 2 : 1, kNPK,
                        mg_res<double>,    mg_res<float>,
                        cheb<double>,
                        prolong<double>,   prolong<float>,
                        restrict_<double>, restrict_<float>,
                        inject,            rhs_adjoint1,
                        rhs_tangent1,      op_BT,
                        op_C_tangent,      op_CT,
                        cob_weights<float>, cob_weights<double>,
                        cob_solve<float>,  cob_solve<double>,
                        cob_cheb<float>,   b_inv<float>,
                        res_cheb<float>,   mg_res_fr,
                        b_inv_fr,          res_cheb_fr,
                        op_A_rho_T,        op_C_pf_T,
                        rhs_tangent,       rhs_adjoint,
                        res_chebz_f,       gs_geo,
                        gs_entry,          gs_binv,
                        gs_zstep,          gs_exit,
                        gs_values,         gs_chain_tiles,
                        gs_chain};

}  // namespace

void register_degree(int p, const DegreeOps* ops);

namespace {
struct Registrar {
  Registrar() { register_degree(P, &kOps); }
} registrar;
}  // namespace

}  // namespace af
