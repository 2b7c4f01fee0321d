// af_gauss.cuh -- the FP32 Chebyshev smoother of the Schur preconditioner in the Gauss-point
// basis (reduced quadrature: P+1 Gauss points per direction).
//
// The polynomial preconditioner iterates on D^{-1} S0, S0 = D - C0 A^{-1} B (the linearised
// Schur operator).  With P+1 Gauss points per direction, M, D and (approximately) A are
// V^T diag(.) V in the nodal (Gauss-Lobatto) basis, V[q][i] = l_i(g_q) square and invertible.
// In the basis of the Lagrange polynomials L_i of the Gauss points (coefficients = values at
// the Gauss points, u_g = (V x V) u) the three mass-type matrices are diagonal:
//   w_g  = diag(1 / (rho JxW)) B_g d_g         (w = A^{-1} B d)
//   (D^{-1} C0 w)_g = g diag(1 / JxW) C0_g w_g  (D^{-1} = g M^{-1})
// where B_g, C0_g are B and C0 with the L_i as test functions and the Gauss-point values as
// trial coefficients: (B d)_nodal = (V x V)^T B_g (V x V) d.  So the whole Chebyshev
// recurrence runs in the Gauss basis with element-wise inverses; only its input (the
// residual: z0 = g diag(1/JxW) (V x V)^{-T} r) and its output (x = (V x V)^{-1} x_g) change
// basis, once per preconditioner application.  In exact arithmetic this is the same
// preconditioner as the nodal reduced-quadrature smoother; the FP32 rounding differs.
//
// Per cell, the operators need the values of their inputs at the volume points (the
// coefficients themselves: no contraction) and their traces on the faces; test functions
// enter through Dg[q][i] = L_i'(g_q) (volume gradients) and L_i(0), L_i(1) (faces).  A face
// trace is an extrapolation along the normal line: u(0, g_q) = sum_i L_i(0) u_g[q][i].
//
// Layout: every array of the recurrence is tiled by 32 consecutive cells, the cell fastest:
//   field  v[(tile * ND + node) * 32 + lane],  node = qz (P+1) + qx
//   faces  t[((tile * 4 + face) * (P+1) + point) * 32 + lane]
// faces 0 (xi = 0), 1 (xi = 1), 2 (eta = 0), 3 (eta = 1); the point runs along the face, so a face
// and the neighbour's opposite face share point indices.  A CTA is one tile, lane = cell, warp m =
// column qx = m of the cells: every load and store of a warp is one aligned line of 32 cells, there
// is no index arithmetic per element, the column's work stays in registers, the tables are indexed
// by warp-uniform values, and only the contraction along x passes through shared memory (cell
// fastest: no bank conflicts).  The edge vectors of a face serve as its normal (the fluxes are
// linear in it).  Geometry is formed once per mesh, in FP64 from the vertices: the four edges of a cell,
// each rounded once, so that both sides of a face take the same bits for its normal (between opposite
// edges the map's derivatives are interpolated), and the determinant as three doubles.  On a bilinear
// cell it is affine, d0 + d1 xi + d2 eta (the product of the map's bilinear term with itself vanishes),
// so JxW at a point takes two FP64 operations and one rounding; products formed in FP32 cancel on sheared
// cells.
//
// The kernels pass between them what the next one needs and no more: k_gs_binv does not write w but
// the two mapped fluxes of C0 at the points (p_f w contracted with adj(J)) and one value per face
// point, p_f (w . n), so k_gs_zstep reads neither p_f nor the traces of w: its face flux is the own
// value minus the neighbour's.  x takes two directions every second step.
//
// The kernels of the chain overlap by programmatic dependent launch and read what the kernel before
// wrote, so none of their arrays is declared const __restrict__: such loads count as invariant over
// the kernel and the compiler may move them above griddepcontrol.wait (small meshes then read the
// previous step's values).
//
// Measured at 512x256, p = 4 (131072 cells), us per launch in a chain, before (cell-major arrays,
// element-wise copies through shared memory: 21.7 M and 26.6 M warp instructions) and now:
//   k_gs_binv 32.9 -> 23.8, k_gs_zstep 46.9 -> 21.0 (the mixed IMEX step 70.2 -> 45.5 ms)
// The step moves about 250 MB through L2 (164 MB of it DRAM) at 1024x256 in 37 us, 6.8 TB/s: it is
// bound by memory; k_gs_binv (200 MB, 41 us) by issue (0.66 of the cycles) and latency.
#pragma once

#include "af_cellop.cuh"
#include "af_internal.h"

namespace af {


// n / d for 0 <= n < 2^31 by one multiplication (Granlund and Montgomery, "Division by invariant
// integers using multiplication", 1994): m = floor(2^(31+l) / d) + 1, l = ceil(log2 d)
struct FastDiv {
  unsigned m;
  int l, d;
  static FastDiv make(int d) {
    int l = 0;
    while ((1LL << l) < d) ++l;
    return {(unsigned)((1ULL << (31 + l)) / (unsigned)d + 1), l, d};
  }
  __device__ __forceinline__ int div(int n) const { return (int)(__umulhi((unsigned)n << 1, m) >> l); }
};

struct GsMesh {
  const float* geo;   // [tile][kGsGeo][32]
  const double* det;  // [tile][kGsDet][32]
  FastDiv nx;
  int nz, periodic_x, ncell;
  int* status;          // as in MeshDev
  int test_wait_polls;  // as in MeshDev: k_gs_chain waits for a step that nobody reaches
};

// the coefficients of consecutive Chebyshev steps
constexpr int kGsSteps = 64;  // even: x takes two directions every second step
struct GsSteps {
  int n;
  float alpha[kGsSteps], s[kGsSteps];
};

template <int P>
struct GsShape {
  static constexpr int P1 = P + 1, ND = P1 * P1, NT = kGsTile * P1;
  // CTAs per SM asked of the compiler.  Degree 4, (k_gs_binv, k_gs_zstep), the mixed IMEX step at
  // 512x256: (4, 6) 46.3 ms, (5, 6) 45.4, (5, 7) 45.2, (6, 6) 46.8 (k_gs_binv spills at 64 registers).
  // Degree 3, 6 / 7 of k_gs_binv (80, 72 registers), us a degree-20 polynomial: 320x160 cells 191, 193;
  // 512x256 433, 422;  640x256 588, 569;  1024x256 1045, 1016.
  static constexpr int CTAS_B = (P == 3 ? 900 : 800) / NT, CTAS_Z = (P <= 4 ? 1120 : 900) / NT;
  // k_gs_chain: more CTAs per SM take larger meshes.  Degree-20 polynomial, degree 4, 3 / 4 / 5 per SM (128,
  // 96, 80 registers; 0, 164, 356 bytes of spill loads): 256 tiles 58, 62, 72 us, 440 tiles 64, 70, 92, 550
  // tiles (165 by the pairs) 165, 79, 107; degree 2, 5 / 8 per SM: 256 tiles 45, 48 us, 1024 tiles (122 by
  // the pairs) 122, 63
  static constexpr int CTAS_C = (P <= 2 ? 800 : 640) / NT;
  // the thread's element of node or point 0 .. and the strides between its nodes (column m) and faces
  __device__ __forceinline__ static size_t column(int tile, int m, int lane) {
    return (size_t)tile * (ND * kGsTile) + (m * kGsTile + lane);
  }
  static constexpr int SN = P1 * kGsTile, SF = P1 * kGsTile;
  __device__ __forceinline__ static size_t point(int tile, int m, int lane) {
    return (size_t)tile * (4 * P1 * kGsTile) + (m * kGsTile + lane);
  }
};

// what a thread knows of its cell and column
template <int P>
struct GsThread {
  int lane, m, tile, c;
  bool live;
  float Ax, Az, Cx, Cz, Rx, Rz, Tx, Tz;  // edges of the faces eta = 0, xi = 0, xi = 1, eta = 1
  float Bx, Bz, Dx, Dz;                  // R - C, T - A
  int nb[4];
  __device__ __forceinline__ explicit GsThread(const GsMesh& g) {
    lane = threadIdx.x & 31;
    m = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // warp-uniform
    tile = blockIdx.x;
    c = tile * kGsTile + lane;
    live = c < g.ncell;
  }
  __device__ __forceinline__ void geometry(const GsMesh& g) {
    const float* s = g.geo + (size_t)tile * kGsGeo * kGsTile + lane;
    Ax = s[0]; Az = s[kGsTile]; Cx = s[2 * kGsTile]; Cz = s[3 * kGsTile]; Rx = s[4 * kGsTile]; Rz = s[5 * kGsTile]; Tx = s[6 * kGsTile]; Tz = s[7 * kGsTile];
    Bx = Rx - Cx; Bz = Rz - Cz; Dx = Tx - Ax; Dz = Tz - Az;
  }
  __device__ __forceinline__ void neighbours(const GsMesh& g) {  // -1: wall (and past the last cell)
    const int nx = g.nx.d, j = g.nx.div(c), i = c - j * nx;
    nb[0] = i > 0 ? c - 1 : (g.periodic_x ? c + nx - 1 : -1);
    nb[1] = i < nx - 1 ? c + 1 : (g.periodic_x ? c - nx + 1 : -1);
    nb[2] = j > 0 ? c - nx : -1;
    nb[3] = j < g.nz - 1 ? c + nx : -1;
#pragma unroll
    for (int f = 0; f < 4; ++f) nb[f] = live ? nb[f] : -1;
  }
  __device__ __forceinline__ float J01(float xi) const { return fmaf(Bx, xi, Cx); }
  __device__ __forceinline__ float J11(float xi) const { return fmaf(Bz, xi, Cz); }
  __device__ __forceinline__ float J00(float eta) const { return fmaf(Dx, eta, Ax); }
  __device__ __forceinline__ float J10(float eta) const { return fmaf(Dz, eta, Az); }
  // outward normal times length of face f: (-tz, tx) of the edge on faces 0 and 3, (tz, -tx) on 1, 2
  __device__ __forceinline__ void normal(int f, float& n0, float& n1) const {
    const float tx = f == 0 ? Cx : (f == 1 ? Rx : (f == 2 ? Ax : Tx));
    const float tz = f == 0 ? Cz : (f == 1 ? Rz : (f == 2 ? Az : Tz));
    const float s = (f == 0 || f == 3) ? 1.f : -1.f;
    n0 = -s * tz;
    n1 = s * tx;
  }
};

// neighbour's value of a face array at this thread's point (own: what a wall takes)
template <int P>
__device__ __forceinline__ float gs_other(const float* t, const GsThread<P>& th, int f, float own) {
  const int nb = th.nb[f];
  return nb >= 0 ? t[GsShape<P>::point(nb >> 5, th.m, nb & 31) + (f ^ 1) * GsShape<P>::SF] : own;
}

// the traces on faces 2 and 3 of a column, at its point
template <int P>
__device__ __forceinline__ void gs_ends(const float* col, float& lo, float& hi) {
  const CobT<P, float>& cb = cobr<P, float>();
  lo = cb.lo[0] * col[0];
  hi = cb.hi[0] * col[0];
#pragma unroll
  for (int i = 1; i <= P; ++i) {
    lo = fmaf(cb.lo[i], col[i], lo);
    hi = fmaf(cb.hi[i], col[i], hi);
  }
}
// the traces on faces 0 and 1 at point m from the rows of a field in shared memory [node][lane]
template <int P>
__device__ __forceinline__ void gs_row_ends(const float* s, int m, int lane, float& lo, float& hi) {
  float row[P + 1];
#pragma unroll
  for (int i = 0; i <= P; ++i) row[i] = s[(m * (P + 1) + i) * kGsTile + lane];
  gs_ends<P>(row, lo, hi);
}

// the geometry block of a mesh (thread = cell)
static __global__ void k_gs_geo(const MeshDev mesh, float* __restrict__ geo, double* __restrict__ det, const int ncell) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (ncell + kGsTile - 1) / kGsTile * kGsTile) return;
  const int c = min(e, ncell - 1), i = c % mesh.nx, j = c / mesh.nx, W = mesh.nx + 1;
  const double2* v = mesh.vtx + (size_t)j * W + i;
  const double2 v0 = v[0], v1 = v[1], v2 = v[W], v3 = v[W + 1];
  const double G[kGsGeo] = {v1.x - v0.x, v1.y - v0.y, v2.x - v0.x, v2.y - v0.y,
                            v3.x - v1.x, v3.y - v1.y, v3.x - v2.x, v3.y - v2.y};
  const double Bx = v3.x - v2.x - v1.x + v0.x, Bz = v3.y - v2.y - v1.y + v0.y;
  float* g = geo + (size_t)(e / kGsTile) * kGsGeo * kGsTile + e % kGsTile;
#pragma unroll
  for (int k = 0; k < kGsGeo; ++k) g[k * kGsTile] = (float)G[k];
  double* d = det + (size_t)(e / kGsTile) * kGsDet * kGsTile + e % kGsTile;
  d[0] = G[0] * G[3] - G[2] * G[1];
  d[kGsTile] = G[0] * Bz - Bx * G[1];      // A x B
  d[2 * kGsTile] = Bx * G[3] - G[2] * Bz;  // B x C
}

// JxW at the points of column m of the thread's cell, and its inverse (one Newton step from the
// approximate quotient: FP32 rounding)
template <int P>
struct GsJxW {
  double dx, dz;
  __device__ __forceinline__ GsJxW(const GsMesh& g, const GsThread<P>& th) {
    const CobT<P, double>& cb = cobr<P, double>();
    const double* d = g.det + (size_t)th.tile * kGsDet * kGsTile + th.lane;
    const double wx = cb.w[th.m];
    dx = wx * fma(d[kGsTile], cb.g[th.m], d[0]);
    dz = wx * d[2 * kGsTile];
  }
  __device__ __forceinline__ float inv(int q) const {
    const float a = (*this)(q), r = __fdividef(1.f, a);
    return fmaf(r, fmaf(-a, r, 1.f), r);
  }
  __device__ __forceinline__ float operator()(int q) const {
    const CobT<P, double>& cb = cobr<P, double>();
    return (float)(fma(dz, cb.g[q], dx) * cb.w[q]);
  }
};

// ------------------------------------------- w = A^{-1} B d, handed on as the fluxes of C0 w
// d_g and its traces dtr -> w_g = diag(WA) B_g d_g, then at the points the mapped fluxes of C0,
//   (fx, fe) = -cdt gg p_f w_q (J11 w0 - J01 w1, J00 w1 - J10 w0),
// and at the face points gf = cdt gg/2 p_f (w . n) w_q with the cell's outward normal.
// B with coefficient cB (euler_operator.h:1536, 1574-1577, 1611-1613): volume
// -cB d div(phi), face cB {{d}} phi . n, wall cB d+ phi . n.
// C0 (euler_operator.h:1444, 1494-1502 without the wave-speed term): volume
// -cdt gg p_f w . grad(q), face cdt gg/2 (p_f+ w+ . n + p_f- w- . n) q, no wall term.
template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT, GsShape<P>::CTAS_B)
    k_gs_binv(const GsMesh mesh, const float* d, const float* dtr, const float cB,
              const float* WA, const float* pg, const float* ptr,
              const float cgg, float* fx, float* fe, float* gf) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND;
  __shared__ float s_sw[ND * kGsTile];        // weighted values of -cB d
  __shared__ float s_xf[4 * P1 * kGsTile];    // x-face fluxes of B [face][component][point][lane]
  __shared__ float s_w[2 * ND * kGsTile];     // w [component][node][lane]
  pdl_allow_next();
  const CobT<P, float>& cb = cobr<P, float>();
  GsThread<P> th(mesh);
  th.geometry(mesh);
  th.neighbours(mesh);
  const int lane = th.lane, m = th.m;
  pdl_wait_previous();
  const size_t oc = S::column(th.tile, m, lane), op = S::point(th.tile, m, lane);
  const float *dB = d + oc, *wB = WA + oc, *pB = pg + oc, *tB = dtr + op, *qB = ptr + op;
  float *fxB = fx + oc, *feB = fe + oc, *gB = gf + op;
  float dc[P1], wa[P1], pc[P1], tm[4], tp[4], pt[4];
#pragma unroll
  for (int q = 0; q < P1; ++q) dc[q] = dB[q * S::SN];
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    tp[f] = tB[f * S::SF];
    pt[f] = qB[f * S::SF];
  }
  gs_ends<P>(dc, tp[2], tp[3]);
#pragma unroll
  for (int f = 0; f < 4; ++f) tm[f] = gs_other<P>(dtr, th, f, tp[f]);
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    wa[q] = wB[q * S::SN];
    pc[q] = pB[q * S::SN];
  }
  const float wx = cb.w[m];
  float a0[P1], a1[P1];
  {
    float e0[P1], e1[P1];
#pragma unroll
    for (int q = 0; q < P1; ++q) {
      const float sw = -cB * dc[q] * (wx * cb.w[q]);
      s_sw[(q * P1 + m) * kGsTile + lane] = sw;
      e0[q] = -th.J10(cb.g[q]) * sw;
      e1[q] = th.J00(cb.g[q]) * sw;
    }
#pragma unroll
    for (int i = 0; i < P1; ++i) {
      a0[i] = cb.Dg[0][i] * e0[0];
      a1[i] = cb.Dg[0][i] * e1[0];
#pragma unroll
      for (int q = 1; q < P1; ++q) {
        a0[i] = fmaf(cb.Dg[q][i], e0[q], a0[i]);
        a1[i] = fmaf(cb.Dg[q][i], e1[q], a1[i]);
      }
    }
  }
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    float n0, n1;
    th.normal(f, n0, n1);
    const float a = cB * 0.5f * (tp[f] + tm[f]) * wx;
    const float F0 = a * n0, F1 = a * n1;
    if (f < 2) {
      s_xf[((f * 2 + 0) * P1 + m) * kGsTile + lane] = F0;
      s_xf[((f * 2 + 1) * P1 + m) * kGsTile + lane] = F1;
    } else {
#pragma unroll
      for (int i = 0; i < P1; ++i) {
        const float e = f == 2 ? cb.lo[i] : cb.hi[i];
        a0[i] = fmaf(e, F0, a0[i]);
        a1[i] = fmaf(e, F1, a1[i]);
      }
    }
  }
  __syncthreads();
  // node (i, m): the x-derivative test along row i (adj(J)'s x part depends on qx alone), the
  // x-face terms, A^{-1}; then the mapped fluxes of C0 at the point
  {
    float k0[P1], k1[P1];
#pragma unroll
    for (int q = 0; q < P1; ++q) {
      const float dg = cb.Dg[q][m];
      k0[q] = dg * th.J11(cb.g[q]);
      k1[q] = -dg * th.J01(cb.g[q]);
    }
    const float lo = cb.lo[m], hi = cb.hi[m];
    const float J01 = th.J01(cb.g[m]), J11 = th.J11(cb.g[m]);
#pragma unroll
    for (int i = 0; i < P1; ++i) {
      float v0 = a0[i], v1 = a1[i];
#pragma unroll
      for (int q = 0; q < P1; ++q) {
        const float sw = s_sw[(i * P1 + q) * kGsTile + lane];
        v0 = fmaf(k0[q], sw, v0);
        v1 = fmaf(k1[q], sw, v1);
      }
      v0 = fmaf(lo, s_xf[(0 * P1 + i) * kGsTile + lane], v0);
      v1 = fmaf(lo, s_xf[(1 * P1 + i) * kGsTile + lane], v1);
      v0 = fmaf(hi, s_xf[(2 * P1 + i) * kGsTile + lane], v0);
      v1 = fmaf(hi, s_xf[(3 * P1 + i) * kGsTile + lane], v1);
      const float w0 = wa[i] * v0, w1 = wa[i] * v1;
      a0[i] = w0;
      a1[i] = w1;
      s_w[(i * P1 + m) * kGsTile + lane] = w0;
      s_w[(ND + i * P1 + m) * kGsTile + lane] = w1;
      const float sv = -cgg * pc[i] * (wx * cb.w[i]);
      fxB[i * S::SN] = sv * (J11 * w0 - J01 * w1);
      feB[i * S::SN] = sv * (th.J00(cb.g[i]) * w1 - th.J10(cb.g[i]) * w0);
    }
  }
  gs_ends<P>(pc, pt[2], pt[3]);
  float t0[4], t1[4];
  gs_ends<P>(a0, t0[2], t0[3]);
  gs_ends<P>(a1, t1[2], t1[3]);
  __syncthreads();
  gs_row_ends<P>(s_w, m, lane, t0[0], t0[1]);
  gs_row_ends<P>(s_w + ND * kGsTile, m, lane, t1[0], t1[1]);
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    float n0, n1;
    th.normal(f, n0, n1);
    gB[f * S::SF] = 0.5f * cgg * wx * pt[f] * (t0[f] * n0 + t1[f] * n1);
  }
}

// ------------------------------------------------- the Chebyshev step on z = D^{-1} r
// The fluxes of C0 w (fx, fe at the points, gf at the face points) -> y = C0_g w_g, then per node
//   z' = z + g y / JxW - d,  d' = alpha d + s z',
// and the traces of d'.  xmode 0: x stays (its direction is added by the next step), 1: x += d + d',
// 2: x += d'.  In place: each CTA reads only its own cells of z, d and x.
template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT, GsShape<P>::CTAS_Z)
    k_gs_zstep(const GsMesh mesh, const float* fx, const float* fe,
               const float* gf, const float gfac, const float alpha, const float s,
               float* z, float* d, float* x, const int xmode,
               float* dtr) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND;
  __shared__ float s_fx[ND * kGsTile], s_d[ND * kGsTile], s_xf[2 * P1 * kGsTile];
  pdl_allow_next();
  const CobT<P, float>& cb = cobr<P, float>();
  GsThread<P> th(mesh);
  th.neighbours(mesh);
  const int lane = th.lane, m = th.m;
  const size_t oc = S::column(th.tile, m, lane), op = S::point(th.tile, m, lane);
  const GsJxW<P> jxw(mesh, th);
  pdl_wait_previous();
  const float *fxB = fx + oc, *feB = fe + oc, *gB = gf + op;
  float *zB = z + oc, *dB = d + oc, *xB = x + oc, *tB = dtr + op;
  float ec[P1], zc[P1], dc[P1], xc[P1], F[4];
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    s_fx[(q * P1 + m) * kGsTile + lane] = fxB[q * S::SN];
    ec[q] = feB[q * S::SN];
  }
#pragma unroll
  for (int f = 0; f < 4; ++f) {  // own minus the neighbour's (whose normal is the opposite); none at walls
    const float own = gB[f * S::SF];
    F[f] = own - gs_other<P>(gf, th, f, own);
  }
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    zc[q] = zB[q * S::SN];
    dc[q] = dB[q * S::SN];
    xc[q] = xmode ? xB[q * S::SN] : 0.f;
  }
  s_xf[m * kGsTile + lane] = F[0];
  s_xf[(P1 + m) * kGsTile + lane] = F[1];
  float a[P1];
#pragma unroll
  for (int i = 0; i < P1; ++i) {
    a[i] = fmaf(cb.hi[i], F[3], cb.lo[i] * F[2]);
#pragma unroll
    for (int q = 0; q < P1; ++q) a[i] = fmaf(cb.Dg[q][i], ec[q], a[i]);
  }
  __syncthreads();
  const float lo = cb.lo[m], hi = cb.hi[m];
#pragma unroll
  for (int i = 0; i < P1; ++i) {
    float y = a[i];
#pragma unroll
    for (int q = 0; q < P1; ++q) y = fmaf(cb.Dg[q][m], s_fx[(i * P1 + q) * kGsTile + lane], y);
    y = fmaf(lo, s_xf[i * kGsTile + lane], y);
    y = fmaf(hi, s_xf[(P1 + i) * kGsTile + lane], y);
    const float zn = zc[i] + gfac * y * jxw.inv(i) - dc[i];
    const float nd = alpha * dc[i] + s * zn;
    zB[i * S::SN] = zn;
    dB[i * S::SN] = nd;
    if (xmode == 1) xB[i * S::SN] = (xc[i] + dc[i]) + nd;
    else if (xmode == 2) xB[i * S::SN] = xc[i] + nd;
    s_d[(i * P1 + m) * kGsTile + lane] = nd;
    dc[i] = nd;
  }
  float t[4];
  gs_ends<P>(dc, t[2], t[3]);
  __syncthreads();
  gs_row_ends<P>(s_d, m, lane, t[0], t[1]);
#pragma unroll
  for (int f = 0; f < 4; ++f) tB[f * S::SF] = t[f];
}

// ------------------------------------------------- all steps in one launch, small meshes
// The pairs (k_gs_binv, k_gs_zstep) of st.n steps by CTAs that stay: one tile each, all resident at the
// same time (a cooperative launch; gs_chain_tiles), with z, d, x and the coefficients in registers and
// the fluxes of w in shared memory.  Between half steps only the face values pass through memory, each
// in one 8-byte word with the count of its half step: a thread reads the words of its four neighbour
// points until they carry the count that it needs, with no flag, fence or barrier in between, and forms
// meanwhile what its own tile contributes.  A value is overwritten only after the thread that reads it
// has published its own next one (the threads of a face point read each other's).  k_gs_entry writes
// the first words and clears the others; counts go on over the launches of one application.  Waits
// are bounded: a CTA that gives up reports it, marks the application in *gave_up (cleared by k_gs_entry)
// and leaves, and so do those that wait for it; k_gs_exit then writes nothing.
// What bounds it: latency.  Degree-20 polynomial, us, the pairs (one launch per half step) / with
// flags per tile, fences and barriers / now:
//   degree 4  256 tiles 123 / 97 / 62, 440 tiles 166 / 106 / 70;  degree 6, 96 tiles 167 / 94 / 60
//   (a step and its adjoint at 128x64: 49.9 / 46.6 / 38.8 ms)
constexpr int kGsWaitPolls = 1 << 19;
using GsWord = unsigned long long;  // a face value and its count
__device__ __forceinline__ GsWord gs_word(float v, int count) {
  return (GsWord)(unsigned)count << 32 | (GsWord)__float_as_uint(v);
}
__device__ __forceinline__ void gs_put(GsWord* w, float v, int count) {
  *reinterpret_cast<volatile GsWord*>(w) = gs_word(v, count);
}

template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT, GsShape<P>::CTAS_C)
    k_gs_chain(const __grid_constant__ GsMesh mesh, const __grid_constant__ GsSteps st, const float cB, const float cgg,
               const float gfac, const float* WA, const float* pg, const float* ptr, float* z, float* d, float* x,
               float* dtr, GsWord* wd, GsWord* wg, GsWord* gave_up, const int base, const int more) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND;
  __shared__ float s_sw[ND * kGsTile];      // weighted values of -cB d
  __shared__ float s_xf[4 * P1 * kGsTile];  // x-face fluxes of B [face][component][point][lane]
  __shared__ float s_w[2 * ND * kGsTile];   // w [component][node][lane]
  __shared__ float s_fx[ND * kGsTile], s_d[ND * kGsTile], s_xf2[2 * P1 * kGsTile];
  constexpr bool SHARED_EDGES = P >= 2 && P <= 5;
  __shared__ float s_rt[SHARED_EDGES ? 4 * kGsTile : 1];  // edges of the faces xi = 1 and eta = 1
  __shared__ float s_wm[ND * kGsTile];      // g / JxW; each thread reads its own column
  if (base > 0 && *gave_up) return;  // an earlier launch of this application
  const CobT<P, float>& cb = cobr<P, float>();
  GsThread<P> th(mesh);
  th.geometry(mesh);
  th.neighbours(mesh);
  const int lane = th.lane, m = th.m;
  const size_t oc = S::column(th.tile, m, lane), op = S::point(th.tile, m, lane);
  float zc[P1], dc[P1], xc[P1], wa[P1], pc[P1], pt[4], tp[4];
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    zc[q] = z[oc + q * S::SN];
    dc[q] = d[oc + q * S::SN];
    xc[q] = x[oc + q * S::SN];
    wa[q] = WA[oc + q * S::SN];
    pc[q] = pg[oc + q * S::SN];
  }
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    tp[f] = dtr[op + f * S::SF];
    pt[f] = ptr[op + f * S::SF];
  }
  gs_ends<P>(pc, pt[2], pt[3]);
  gs_ends<P>(dc, tp[2], tp[3]);
  // the far edges' normals come from shared memory at degrees 2 to 5 (in a trace, degree 4, 256 tiles: 59.9 us a
  // polynomial with them in registers, 56.7 us so; degree 6, 96 tiles: 60.5 and 71.9 us, nothing spills there;
  // degree 1, 256 and 437 tiles: 38.1 and 39.7 us in registers, 38.6 and 40.1 us so)
  if (SHARED_EDGES && m == 0) {
    s_rt[lane] = th.Rx;
    s_rt[kGsTile + lane] = th.Rz;
    s_rt[2 * kGsTile + lane] = th.Tx;
    s_rt[3 * kGsTile + lane] = th.Tz;
  }
  auto normal = [&](int f, float& n0, float& n1) {
    if (SHARED_EDGES && (f & 1)) {
      const float s = f == 3 ? 1.f : -1.f;
      n0 = -s * s_rt[f * kGsTile + lane];
      n1 = s * s_rt[(f - 1) * kGsTile + lane];
    } else {
      th.normal(f, n0, n1);
    }
  };
  // the neighbours' values of that count (a wall takes the own one); false when the bound was reached
  const bool hook = mesh.test_wait_polls > 0;
  const int polls = hook ? mesh.test_wait_polls : kGsWaitPolls;
  unsigned src[4];  // few tiles: 32 bits hold the offsets
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const int nb = th.nb[f] < 0 ? 0 : th.nb[f];
    src[f] = (unsigned)S::point(nb >> 5, m, nb & 31) + (f ^ 1) * S::SF;
  }
  auto others = [&](const GsWord* w, int count, const float* own, float* v) {
    if (hook) count = -1;
    bool ok = false;
    for (int it = 0; it < polls && !ok; ++it) {
      GsWord a[4];
#pragma unroll
      for (int f = 0; f < 4; ++f)
        a[f] = th.nb[f] >= 0 ? *reinterpret_cast<const volatile GsWord*>(w + src[f]) : gs_word(own[f], count);
      ok = true;
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        ok = ok && (int)(a[f] >> 32) == count;
        v[f] = __uint_as_float((unsigned)a[f]);
      }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (!ok && lane == 0) {
      *reinterpret_cast<volatile GsWord*>(gave_up) = 1;
      report_status(mesh.status, kStatusStageTimeout);
    }
    return ok;
  };

  const float wx = cb.w[m], lo = cb.lo[m], hi = cb.hi[m];
  const float J01 = th.J01(cb.g[m]), J11 = th.J11(cb.g[m]);
  const GsJxW<P> jxw(mesh, th);
#pragma unroll
  for (int q = 0; q < P1; ++q) s_wm[(q * P1 + m) * kGsTile + lane] = gfac * jxw.inv(q);
#pragma unroll
  for (int q = 0; q < P1; ++q) s_sw[(q * P1 + m) * kGsTile + lane] = -cB * dc[q] * (wx * cb.w[q]);
  __syncthreads();
#pragma unroll 1
  for (int it = 1; it <= st.n; ++it) {
    // ---- k_gs_binv: what the own tile gives, while the neighbours arrive
    float tm[4], ec[P1], g[4], a0[P1], a1[P1];
    {
      float e0[P1], e1[P1];
#pragma unroll
      for (int q = 0; q < P1; ++q) {
        const float sw = -cB * dc[q] * (wx * cb.w[q]);
        e0[q] = -th.J10(cb.g[q]) * sw;
        e1[q] = th.J00(cb.g[q]) * sw;
      }
#pragma unroll
      for (int i = 0; i < P1; ++i) {
        a0[i] = cb.Dg[0][i] * e0[0];
        a1[i] = cb.Dg[0][i] * e1[0];
#pragma unroll
        for (int q = 1; q < P1; ++q) {
          a0[i] = fmaf(cb.Dg[q][i], e0[q], a0[i]);
          a1[i] = fmaf(cb.Dg[q][i], e1[q], a1[i]);
        }
      }
#pragma unroll
      for (int q = 0; q < P1; ++q) {
        const float dg = cb.Dg[q][m], k0 = dg * th.J11(cb.g[q]), k1 = -dg * th.J01(cb.g[q]);
#pragma unroll
        for (int i = 0; i < P1; ++i) {
          const float sw = s_sw[(i * P1 + q) * kGsTile + lane];
          a0[i] = fmaf(k0, sw, a0[i]);
          a1[i] = fmaf(k1, sw, a1[i]);
        }
      }
    }
    const bool okd = others(wd, base + 2 * it - 2, tp, tm);
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      float n0, n1;
      normal(f, n0, n1);
      const float a = cB * 0.5f * (tp[f] + tm[f]) * wx;
      const float F0 = a * n0, F1 = a * n1;
      if (f < 2) {
        s_xf[((f * 2 + 0) * P1 + m) * kGsTile + lane] = F0;
        s_xf[((f * 2 + 1) * P1 + m) * kGsTile + lane] = F1;
      } else {
#pragma unroll
        for (int i = 0; i < P1; ++i) {
          const float e = f == 2 ? cb.lo[i] : cb.hi[i];
          a0[i] = fmaf(e, F0, a0[i]);
          a1[i] = fmaf(e, F1, a1[i]);
        }
      }
    }
    if (__syncthreads_or(!okd)) return;
#pragma unroll
    for (int i = 0; i < P1; ++i) {
      float v0 = a0[i], v1 = a1[i];
      v0 = fmaf(lo, s_xf[(0 * P1 + i) * kGsTile + lane], v0);
      v1 = fmaf(lo, s_xf[(1 * P1 + i) * kGsTile + lane], v1);
      v0 = fmaf(hi, s_xf[(2 * P1 + i) * kGsTile + lane], v0);
      v1 = fmaf(hi, s_xf[(3 * P1 + i) * kGsTile + lane], v1);
      const float w0 = wa[i] * v0, w1 = wa[i] * v1;
      a0[i] = w0;
      a1[i] = w1;
      s_w[(i * P1 + m) * kGsTile + lane] = w0;
      s_w[(ND + i * P1 + m) * kGsTile + lane] = w1;
      const float sv = -cgg * pc[i] * (wx * cb.w[i]);
      s_fx[(i * P1 + m) * kGsTile + lane] = sv * (J11 * w0 - J01 * w1);
      ec[i] = sv * (th.J00(cb.g[i]) * w1 - th.J10(cb.g[i]) * w0);
    }
    {
      float t0[4], t1[4];
      gs_ends<P>(a0, t0[2], t0[3]);
      gs_ends<P>(a1, t1[2], t1[3]);
      __syncthreads();
      gs_row_ends<P>(s_w, m, lane, t0[0], t0[1]);
      gs_row_ends<P>(s_w + ND * kGsTile, m, lane, t1[0], t1[1]);
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        float n0, n1;
        normal(f, n0, n1);
        g[f] = 0.5f * cgg * wx * pt[f] * (t0[f] * n0 + t1[f] * n1);
        gs_put(wg + op + f * S::SF, g[f], base + 2 * it - 1);
      }
    }
    // ---- k_gs_zstep
    float F[4], a[P1];
#pragma unroll
    for (int i = 0; i < P1; ++i) {
      a[i] = cb.Dg[0][i] * ec[0];
#pragma unroll
      for (int q = 1; q < P1; ++q) a[i] = fmaf(cb.Dg[q][i], ec[q], a[i]);
#pragma unroll
      for (int q = 0; q < P1; ++q) a[i] = fmaf(cb.Dg[q][m], s_fx[(i * P1 + q) * kGsTile + lane], a[i]);
    }
    const bool okg = others(wg, base + 2 * it - 1, g, F);
#pragma unroll
    for (int f = 0; f < 4; ++f) F[f] = g[f] - F[f];
    s_xf2[m * kGsTile + lane] = F[0];
    s_xf2[(P1 + m) * kGsTile + lane] = F[1];
#pragma unroll
    for (int i = 0; i < P1; ++i) a[i] = fmaf(cb.hi[i], F[3], fmaf(cb.lo[i], F[2], a[i]));
    if (__syncthreads_or(!okg)) return;
    const float alpha = st.alpha[it - 1], s = st.s[it - 1];
#pragma unroll
    for (int i = 0; i < P1; ++i) {
      float y = a[i];
      y = fmaf(lo, s_xf2[i * kGsTile + lane], y);
      y = fmaf(hi, s_xf2[(P1 + i) * kGsTile + lane], y);
      const float zn = zc[i] + s_wm[(i * P1 + m) * kGsTile + lane] * y - dc[i];
      const float nd = alpha * dc[i] + s * zn;
      if (it % 2 == 0) xc[i] = (xc[i] + dc[i]) + nd;
      else if (it == st.n) xc[i] = xc[i] + nd;
      s_d[(i * P1 + m) * kGsTile + lane] = nd;
      s_sw[(i * P1 + m) * kGsTile + lane] = -cB * nd * (wx * cb.w[i]);
      zc[i] = zn;
      dc[i] = nd;
    }
    if (it == st.n && !more) break;
    gs_ends<P>(dc, tp[2], tp[3]);
    __syncthreads();
    gs_row_ends<P>(s_d, m, lane, tp[0], tp[1]);
#pragma unroll
    for (int f = 0; f < 4; ++f) gs_put(wd + op + f * S::SF, tp[f], base + 2 * it);
  }
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    x[oc + q * S::SN] = xc[q];
    if (more) {
      z[oc + q * S::SN] = zc[q];
      d[oc + q * S::SN] = dc[q];
    }
  }
  if (more)
#pragma unroll
    for (int f = 0; f < 2; ++f) dtr[op + f * S::SF] = tp[f];
}

// ------------------------------------------------------------ basis changes
// The preconditioner's input: v (FP64, a residual: dual, nodal) -> b_g = (Vi x Vi)^T v,
// d = x = sc b_g / JxW, z = theta d and the traces of d, for k_gs_chain also as words of count 0 (wd; wg and the
// mark *gave_up cleared).
template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT)
    k_gs_entry(const GsMesh mesh, const double* v, const float sc, const float theta,
               float* z, float* d, float* x, float* dtr, GsWord* wd, GsWord* wg, GsWord* gave_up) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND, NDS = ND | 1;
  __shared__ float s_v[kGsTile * NDS], s_t[ND * kGsTile];
  pdl_allow_next();
  const CobT<P, float>& cb = cobr<P, float>();
  GsThread<P> th(mesh);
  const int lane = th.lane, m = th.m;
  const int n = min(kGsTile, mesh.ncell - th.tile * kGsTile) * ND;
  const size_t oc = S::column(th.tile, m, lane);
  float *zB = z + oc, *dB = d + oc, *xB = x + oc, *tB = dtr + S::point(th.tile, m, lane);
  const GsJxW<P> jxw(mesh, th);
  pdl_wait_previous();
  for (int e = threadIdx.x; e < n; e += S::NT) s_v[(e / ND) * NDS + e % ND] = (float)v[(size_t)th.tile * kGsTile * ND + e];
  __syncthreads();
#pragma unroll
  for (int qx = 0; qx < P1; ++qx) {  // along x on row m
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < P1; ++i) t = fmaf(cb.Vi[i][qx], s_v[lane * NDS + m * P1 + i], t);
    s_t[(m * P1 + qx) * kGsTile + lane] = t;
  }
  __syncthreads();
  float u[P1], dc[P1];
#pragma unroll
  for (int i = 0; i < P1; ++i) u[i] = s_t[(i * P1 + m) * kGsTile + lane];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < P1; ++q) {  // along z on column m, then the weights
    float b = 0.f;
#pragma unroll
    for (int i = 0; i < P1; ++i) b = fmaf(cb.Vi[i][q], u[i], b);
    dc[q] = sc * b * jxw.inv(q);
    dB[q * S::SN] = dc[q];
    xB[q * S::SN] = dc[q];
    zB[q * S::SN] = theta * dc[q];
    s_t[(q * P1 + m) * kGsTile + lane] = dc[q];
  }
  float t[4];
  gs_ends<P>(dc, t[2], t[3]);
  __syncthreads();
  gs_row_ends<P>(s_t, m, lane, t[0], t[1]);
#pragma unroll
  for (int f = 0; f < 4; ++f) tB[f * S::SF] = t[f];
  if (wd)
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const size_t o = S::point(th.tile, m, lane) + f * S::SF;
      wd[o] = gs_word(t[f], 0);
      wg[o] = 0;
    }
  if (wd && blockIdx.x == 0 && threadIdx.x == 0) *gave_up = 0;
}

// The preconditioner's output: x = (Vi x Vi) x_g (nodal, FP64); nothing when k_gs_chain gave up (gave_up:
// null where it did not run).
template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT)
    k_gs_exit(const float* xg, double* out, const GsWord* gave_up, const int ncell) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND, NDS = ND | 1;
  __shared__ float s_v[kGsTile * NDS], s_t[ND * kGsTile];
  pdl_allow_next();
  const CobT<P, float>& cb = cobr<P, float>();
  const int lane = threadIdx.x & 31, m = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), tile = blockIdx.x;
  const int n = min(kGsTile, ncell - tile * kGsTile) * ND;
  pdl_wait_previous();
  const bool skip = gave_up && *gave_up;  // looked at with the store: its load overlaps the others
  float u[P1];
#pragma unroll
  for (int q = 0; q < P1; ++q) u[q] = xg[S::column(tile, m, lane) + q * S::SN];
#pragma unroll
  for (int i = 0; i < P1; ++i) {  // along z on column m
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < P1; ++q) t = fmaf(cb.Vi[i][q], u[q], t);
    s_t[(i * P1 + m) * kGsTile + lane] = t;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < P1; ++q) u[q] = s_t[(m * P1 + q) * kGsTile + lane];
#pragma unroll
  for (int i = 0; i < P1; ++i) {  // along x on row m
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < P1; ++q) t = fmaf(cb.Vi[i][q], u[q], t);
    s_v[lane * NDS + m * P1 + i] = t;
  }
  __syncthreads();
  if (skip) return;
  for (int e = threadIdx.x; e < n; e += S::NT)
    out[(size_t)tile * kGsTile * ND + e] = (double)s_v[(e / ND) * NDS + e % ND];
}

// A coefficient field (FP64, nodal) at the Gauss points, pg = (V x V) p, and its traces on faces 0, 1
// (those on faces 2 and 3 are formed from the columns where they are used); and, given rho, the
// Gauss-point inverse weights of A, WA = 1 / (rho JxW).
template <int P>
__global__ void __launch_bounds__(GsShape<P>::NT)
    k_gs_values(const MeshDev mesh, const double* __restrict__ p, const double* __restrict__ rho,
                float* __restrict__ pg, float* __restrict__ ptr, float* __restrict__ WA, const int ncell) {
  using S = GsShape<P>;
  constexpr int P1 = S::P1, ND = S::ND, NDS = ND | 1;
  __shared__ double s_v[kGsTile * NDS], s_t[ND * kGsTile];
  const CobT<P, double>& cb = cobr<P, double>();
  const int lane = threadIdx.x & 31, m = threadIdx.x >> 5, tile = blockIdx.x;
  const int n = min(kGsTile, ncell - tile * kGsTile) * ND;
  const int c = min(tile * kGsTile + lane, ncell - 1);
  // the values of a nodal field at the points of column m
  auto values = [&](const double* __restrict__ v, double* u) {
    for (int e = threadIdx.x; e < n; e += S::NT) s_v[(e / ND) * NDS + e % ND] = v[(size_t)tile * kGsTile * ND + e];
    __syncthreads();
    double r[P1];
#pragma unroll
    for (int i = 0; i < P1; ++i) r[i] = s_v[lane * NDS + m * P1 + i];
#pragma unroll
    for (int q = 0; q < P1; ++q) {  // along x on row m
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < P1; ++i) t = fma(cb.V[q][i], r[i], t);
      s_t[(m * P1 + q) * kGsTile + lane] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < P1; ++i) r[i] = s_t[(i * P1 + m) * kGsTile + lane];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < P1; ++q) {  // along z on column m
      double t = 0.0;
#pragma unroll
      for (int i = 0; i < P1; ++i) t = fma(cb.V[q][i], r[i], t);
      u[q] = t;
    }
  };
  double u[P1];
  values(p, u);
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    pg[S::column(tile, m, lane) + q * S::SN] = (float)u[q];
    s_t[(q * P1 + m) * kGsTile + lane] = u[q];
  }
  __syncthreads();
  double lo = 0.0, hi = 0.0;
#pragma unroll
  for (int i = 0; i < P1; ++i) {
    lo = fma(cb.lo[i], s_t[(m * P1 + i) * kGsTile + lane], lo);
    hi = fma(cb.hi[i], s_t[(m * P1 + i) * kGsTile + lane], hi);
  }
  ptr[S::point(tile, m, lane)] = (float)lo;
  ptr[S::point(tile, m, lane) + S::SF] = (float)hi;
  __syncthreads();
  values(rho, u);
  const int i = c % mesh.nx, j = c / mesh.nx, W = mesh.nx + 1;
  const double2* v = mesh.vtx + (size_t)j * W + i;
  const double2 v0 = v[0], v1 = v[1], v2 = v[W], v3 = v[W + 1];
  const double Ax = v1.x - v0.x, Az = v1.y - v0.y, Cx = v2.x - v0.x, Cz = v2.y - v0.y;
  const double Bx = v3.x - v2.x - v1.x + v0.x, Bz = v3.y - v2.y - v1.y + v0.y;
  const double xi = cb.g[m], J01 = fma(Bx, xi, Cx), J11 = fma(Bz, xi, Cz);
#pragma unroll
  for (int q = 0; q < P1; ++q) {
    const double eta = cb.g[q], J00 = fma(Bx, eta, Ax), J10 = fma(Bz, eta, Az);
    WA[S::column(tile, m, lane) + q * S::SN] = (float)(1.0 / (u[q] * ((J00 * J11 - J01 * J10) * cb.w[m] * cb.w[q])));
  }
}

}  // namespace af
