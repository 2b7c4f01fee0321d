// af_cellop.cuh -- generic cell-centric, sum-factorised DG operator kernel for sm_100a.
//
// One CTA owns CB consecutive cells (deal.II active-cell order = DoF order) and NQ threads per
// cell.  Every operator of the reference's EULEROperator is a sum over "groups" of input fields
// of (cell integral) + (face integral) terms, so a Phys policy describes, per group, the input
// arrays, the pointwise integrand and the numerical flux; this kernel does the data movement and
// the tensor-product algebra:
//
//   per batch of groups (PhysInfo):
//     traces : 1D contractions of the neighbours' face nodes, read directly from global memory
//              while the own cells' nodes arrive by bulk copies
//     lines  : 1D contractions of the own nodes along x, rows (i, P-i) combined even/odd, and of
//              the own x-faces' nodes; one line per thread, consecutive threads on consecutive
//              cells
//     faces  : thread = face point; numerical flux from the traces of both sides
//     z pass : thread = quadrature column qx; points (qz, NQ-1-qz) in pairs, integrand, then the
//              test-function contraction along z accumulated in registers (even/odd split,
//              constant-memory coefficients)
//   then:      contraction along x of the accumulated rows, plus the face terms on the x-faces'
//              nodes -> shared memory -> bulk stores.
//
// Faces are evaluated from both sides (cell-centric): no atomics, deterministic, and both cells of
// a face form its normal from the same two vertices.  Boundary faces call Phys::boundary.
//
// What bounds it and why this split (FP64, degree 4, 512x256 cells, fused stage-1 right-hand sides):
// FP64 issue (68 M warp instructions, a 110 us floor at the pipe's rate, against 44 us of HBM
// traffic) and the shared-memory data path (39 M wavefronts).  402 us before this layout, 206 us with
// it.  What gave that:
// - 14 cells x 9 points fill 4 warps and three such CTAs an SM (168 registers, 74 KB); 16 cells left
//   half a warp idle and two CTAs an SM;
// - the face traces are 1D contractions done once per face line (even/odd, one thread) instead of at
//   each of the 9 face points, the x-neighbours' read from the own lines of the same CTA, and the
//   own z-face traces are sums of rows that the z pass needs anyway;
// - rows are laid out [row][cell][point], lines at an odd stride: no bank conflicts in the z pass;
// - fluxes are linear in the normal, so edge vectors replace unit normals (no square roots), and the
//   quadrature weights sit in the tables and in one factor per accumulator;
// - the three groups of stage 3 run in batches (below): 10.8 -> 3.8 ms at 2048x512.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <type_traits>
#include <utility>

#include "af_tables.cuh"

namespace af {

struct MeshDev {
  const double2* vtx;  // (nz+1)*(nx+1) vertices, row-major in (j, i)
  int nx, nz, periodic_x, gravity;
  double radial_a;
  int cell0;  // cell kernels: the first cell of the launch;
              // the launch covers [cell0, ncell).  0 for whole-mesh launches
  // Status word of the caller (host-visible; null: not reported).  A kernel that gives up a
  // bounded wait writes kStatusStageTimeout there and leaves without writing its outputs.
  int* status;
  // Test hook (0 in normal use): when > 0, each CTA of a cell kernel first waits on a barrier
  // phase that never completes and gives up after this many polls, before it issues any copy.
  int test_wait_polls;
};

// Codes a kernel leaves in MeshDev::status.
constexpr int kStatusStageTimeout = 1;

struct PointGeo {
  double X[2];  // physical position (valid when Phys::NEED_X)
  double J[4];  // Jacobian (x_xi, x_eta, z_xi, z_eta) (valid for policies with gradient fields)
};

// Policies may declare "gradient fields": the last nfg_of(G) cell fields of group G, whose
// reference-coordinate derivatives at the quadrature points are passed to their point
// function as well (point<G>(prm, v, deta, pg, val, gr): v holds the group's values, then
// d/dxi of the gradient fields; deta holds their d/deta).  Policies without nfg_of have none.
template <class Phys, class = void>
struct NfgOf {
  static constexpr bool any = false;
  static constexpr int get(int) { return 0; }
};
template <class Phys>
struct NfgOf<Phys, std::void_t<decltype(Phys::nfg_of(0))>> {
  static constexpr bool any = true;
  static constexpr int get(int g) { return Phys::nfg_of(g); }
};

// Policies may map their integrand to the reference cell themselves (Phys::MAPPED): their
// point_mapped<G>(prm, v, pg, A, dw, fv, fx, fe) adds, per output o, fv[o] = value * |J| and
// (fx[o], fe[o]) = (A0 g0 - A1 g1, A3 g1 - A2 g0) for the output's flux g, with
// A = (J11, J01, J10, J00) = adj(J) and dw = |J| (the kernel applies the quadrature weights).  A
// policy that knows the structure of its fluxes can share products of the Jacobian between outputs
// (contravariant velocities); the others return physical values and fluxes and the kernel maps them.
template <class Phys, class = void>
struct MappedOf {
  static constexpr bool value = false;
};
template <class Phys>
struct MappedOf<Phys, std::void_t<decltype(Phys::MAPPED)>> {
  static constexpr bool value = Phys::MAPPED;
};

// Whether a policy's point functions read the physical position: Phys::NEED_X, and for
// parameters that say so (needs_position()) only when they do (the vertical gravity of the hill
// needs no position, radial gravity and the sponge do).
template <class Prm, class = void>
struct PositionUse {
  __device__ static bool get(const Prm&) { return true; }
};
template <class Prm>
struct PositionUse<Prm, std::void_t<decltype(std::declval<const Prm&>().needs_position())>> {
  __device__ static bool get(const Prm& p) { return p.needs_position(); }
};

// Policies may declare a cell-local epilogue (Phys::EPI) that replaces the plain store.  Both
// apply a cell-wise inverse mass matrix by the change of basis to the Gauss points (CobT):
//   M_K^{-1} y = Vi (W_K (Vi^T y)),  W_K = prm.inv[cell][q] = 1 / (rho(g_q) JxW(g_q)),
//   1: out = scale * M_K^{-1} y per cell and component;
//   2: the Chebyshev step on a residual increment y:  r += y;  d' = alpha d + s M_K^{-1} r;
//      x = d' (first) or x += d'   (prm.r, prm.din, prm.dout, prm.x).  d' goes to its own
//      array: other CTAs still read d's face nodes when the operator's input is d.
//   3: the Chebyshev step on a preconditioned residual z (prm.r holds z):
//      z' = z + g M_K^{-1} y - d;  d' = alpha d + s z';  x = d' (first) or x += d'.
// The CTA's weights are brought in by a bulk copy issued at kernel start.
template <class Phys, class = void>
struct EpiOf {
  static constexpr int value = 0;
};
template <class Phys>
struct EpiOf<Phys, std::void_t<decltype(Phys::EPI)>> {
  static constexpr int value = Phys::EPI;
};

template <int N, class F, int... I>
__device__ __forceinline__ void sfor_impl(F& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void sfor(F&& f) {
  sfor_impl<N>(f, std::make_integer_sequence<int, N>{});
}

// 1D tables of degree P in precision R; each kernel translation unit defines the
// specialisations it uses (constant memory is per module).
template <int P, class R, int NQ = 2 * P + 1>
__device__ __forceinline__ const TabT<P, R, NQ>& tabr();
template <int P>
__device__ __forceinline__ const Tab<P>& tab() {
  return tabr<P, double>();
}
// change-of-basis tables (cell-wise inverse mass matrices without stored matrices)
template <int P, class R>
__device__ __forceinline__ const CobT<P, R>& cobr();

// Outputs that the integrands of batch B feed with values and with fluxes: those of the policy, or
// fewer where it says so (val_in(B, o), grad_in(B, o)).
template <class Phys, class = void>
struct TermsOf {
  static constexpr bool val(int, int o) { return Phys::has_val(o); }
  static constexpr bool grad(int, int o) { return Phys::has_grad(o); }
};
template <class Phys>
struct TermsOf<Phys, std::void_t<decltype(Phys::val_in(0, 0))>> {
  static constexpr bool val(int b, int o) { return Phys::has_val(o) && Phys::val_in(b, o); }
  static constexpr bool grad(int b, int o) { return Phys::has_grad(o) && Phys::grad_in(b, o); }
};

// Fused multiply-add in the working precision (no silent promotion of float operands).
__device__ __forceinline__ double fmaR(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fmaR(float a, float b, float c) { return __fmaf_rn(a, b, c); }

// Working precision of a Phys policy: Phys::real.
template <class Phys>
using RealOf = typename Phys::real;

// Asynchronous global -> shared copies (all of a group in flight, one wait).
__device__ __forceinline__ void cp_async_el(double* smem_dst, const double* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_el(float* smem_dst, const float* gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

constexpr int odd(int n) { return n | 1; }

// Programmatic dependent launch between consecutive cell-operator launches in a stream: every
// CTA allows the next launch at its entry (griddepcontrol.launch_dependents), so the next
// launch's CTAs start on the SMs this one frees and run their prologue while it finishes; they
// wait (griddepcontrol.wait: this grid complete, its writes visible) before they read or write
// anything a kernel can write.  Geometry-first prologue (the geometry before the wait, the
// own-cell copies after it) or wait-first (the copies issued at once, overlapping the
// geometry, as without the dependent launch): AF_PDL_GEO_FIRST 1 always, 0 never, 2 for the
// FP32 kernels only.  Measured, us without the dependent launch / geometry-first / wait-first, p = 4: the
// fused FP64 rhs at 512x256 207.6 / 208.4 / 206.5, at 64x32 10.5 / 8.4 / 8.4; the degree-16 nodal FP32
// polynomial (32 launches) at 512x256 1348 / 1269 / 1279, at 64x32 224 / 162 / 172.
#ifndef AF_PDL
#define AF_PDL 1
#endif
#ifndef AF_PDL_GEO_FIRST
#define AF_PDL_GEO_FIRST 2
#endif
constexpr bool kPDL = AF_PDL != 0;
template <class R>
constexpr bool pdl_geo_first() {
  return kPDL && (AF_PDL_GEO_FIRST == 1 || (AF_PDL_GEO_FIRST == 2 && sizeof(R) == 4));
}
__device__ __forceinline__ void pdl_allow_next() {
  if constexpr (kPDL) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}
__device__ __forceinline__ void pdl_wait_previous() {
  if constexpr (kPDL) asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// Bounded wait on a shared-memory mbarrier phase; false when the bound was reached.
constexpr int kStageWaitPolls = 1 << 20;
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned phase, int polls = kStageWaitPolls) {
  for (int it = 0; it < polls; ++it) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(phase)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Records a given-up wait in the caller's status word (mapped host memory or device memory;
// every CTA that gives up writes the same code, so a plain store is enough).
__device__ __forceinline__ void report_status(int* status, int code) {
  if (status) {
    *reinterpret_cast<volatile int*>(status) = code;
    __threadfence_system();
  }
}

// Cells per CTA, per degree: whole warps at 2P+1 threads a cell.  Small CTAs wait less for one another
// at the barriers, but more of their cells have neighbours outside.  Measured (us, 131072 cells; fused
// stage 1, stage 3, the three split calls of stage 3, C):
//   p=1 (262144 cells)  42 x 3 CTAs per SM 106, 242, 440, 36;  32 x 4: 100, 231, 436, 35;  21 x 6: 107, 253, 459, 37
//   p=2  24 x 3: 84, 195, 369, 32;  18 x 4: 86, 203, 391, 33;  12 x 6: 85, 208, 402, 35
//   p=3 (element copies)  9 x 6: 163, 352, 725, 63;  13 x 4: 176, 385, 771, 66;  18 x 3: 178, 376, 739, 62
//   p=4  14 x 3: 207, 481, 911, 82;  12 x 3: 229, 545, 1007, 91;  10 x 4: 221, 548, 1000, 87;  6 x 6: 232, 557, 1088, 101
//   p=5 (65536 cells)  11 x 2: 227, 515, 928, 66;  8 x 3: 217, 483, 825, 68 (stage 2 430, not 412);  5 x 4: 224, 545, 978, 67
//   p=6 (32768 cells)  8 x 2: 152, 327, 561, 44;  4 x 4: 151, 332, 587, 47
// Meshes of a few CTAs per SM take 10 to 15 percent more or less with the remainder of that count (p=3, C at
// 128x64 cells: 9 cells, 911 CTAs on 888 places, 8.4;  13 cells 8.0;  160x80: 8.3 and 10.1).
// An odd number of cells needs an even number of nodes a cell: the bulk copies start on 16 bytes.
template <int P, class R = double>
constexpr int cells_per_block() {
  if (sizeof(R) == 4) return P <= 1 ? 64 : (P == 2 ? 32 : (P <= 4 ? 16 : 8));
  return P <= 1 ? 32 : (P == 2 ? 24 : (P == 3 ? 9 : (P == 4 ? 14 : (P == 5 ? 11 : 8))));
}

template <int MAXARR, int MAXOUT, class R = double>
struct ArgPtrs {
  const R* in[MAXARR];
  R* out[MAXOUT];
};

// ----------------------------------------------------------------------------------
// compile-time helpers over a Phys policy
// ----------------------------------------------------------------------------------
template <class Phys, int G>
struct GroupInfo {
  using Gr = typename Phys::template Grp<G>;
  static constexpr int NARR = Gr::NARR;
  static constexpr bool FACE = Phys::FACES && Gr::FACE;
  static constexpr int NF = [] {
    int n = 0;
    for (int a = 0; a < NARR; ++a) n += Gr::ncomp(a);
    return n;
  }();
  static constexpr int NF_GRAD = NfgOf<Phys>::get(G);  // the last NF_GRAD cell fields
  static constexpr int NF_CELL = [] {  // fields used by cell integrals (face-only ones last)
    int n = 0;
    for (int a = 0; a < NARR; ++a)
      if (!Gr::face_only(a)) n += Gr::ncomp(a);
    return n;
  }();
  static constexpr int arr_of(int f) {  // array of field f
    int a = 0;
    for (int n = Gr::ncomp(0); f >= n; n += Gr::ncomp(a)) ++a;
    return a;
  }
  static constexpr int first_field(int a) {
    int n = 0;
    for (int k = 0; k < a; ++k) n += Gr::ncomp(k);
    return n;
  }
};

// Policies whose faces read only some fields of a group declare face_field(G, f); the others
// read all of them.
template <class Phys, class = void>
struct FaceFieldOf {
  static constexpr bool get(int, int) { return true; }
};
template <class Phys>
struct FaceFieldOf<Phys, std::void_t<decltype(Phys::face_field(0, 0))>> {
  static constexpr bool get(int g, int f) { return Phys::face_field(g, f); }
};

template <class Phys, int... G>
constexpr int arr_total(int upto, std::integer_sequence<int, G...>) {
  return ((G < upto ? GroupInfo<Phys, G>::NARR : 0) + ... + 0);
}

// The groups of a policy run in batches: one batch stages its groups' fields, contracts them
// along x and evaluates them together at the points, so that their integrands share one mapping
// and one test contraction.  A policy with one face group is one batch; with several (the stages
// with two and three explicit groups) each is its own batch and so is the implicit group after
// them: the batches' fields follow one another through the same shared memory, which keeps two or
// three CTAs on an SM (all of them at once left one CTA of 16 cells per SM at degree 4: the
// stage-3 right-hand sides at 2048x512 10.8 ms in the layout before, 3.8 ms now).
template <class Phys>
struct PhysInfo {
  using Seq = std::make_integer_sequence<int, Phys::NG>;
  static constexpr int NARR_TOTAL = arr_total<Phys>(Phys::NG, Seq{});
  static constexpr int arr_base(int G) { return arr_total<Phys>(G, Seq{}); }
  template <int... G>
  static constexpr int batch_of_impl(int g, std::integer_sequence<int, G...>) {
    const bool face[] = {GroupInfo<Phys, G>::FACE...};
    int b = 0, nface = 0;
    for (int k = 0; k < Phys::NG; ++k) nface += face[k] ? 1 : 0;
    bool has = false;
    for (int k = 0; k <= g; ++k) {
      if (has && (face[k] || nface > 1)) {
        ++b;
        has = false;
      }
      has = has || face[k];
    }
    return b;
  }
  static constexpr int batch_of(int g) { return batch_of_impl(g, Seq{}); }
  static constexpr int NB = batch_of(Phys::NG - 1) + 1;
  template <int... G>
  static constexpr int face_group_impl(int b, std::integer_sequence<int, G...>) {
    int r = -1;
    ((r = (GroupInfo<Phys, G>::FACE && batch_of(G) == b) ? G : r), ...);
    return r;
  }
  // the face group of batch b (-1: none)
  static constexpr int face_group(int b) { return face_group_impl(b, Seq{}); }
  // x-contracted slots before group G in its batch: per group its cell fields (contracted with
  // S), then its gradient fields again (contracted with D, for d/dxi)
  template <int... G>
  static constexpr int slots_impl(int g, int b, std::integer_sequence<int, G...>) {
    return ((G < g && batch_of(G) == b ? GroupInfo<Phys, G>::NF_CELL + GroupInfo<Phys, G>::NF_GRAD : 0) + ... + 0);
  }
  static constexpr int slot_offset(int g) { return slots_impl(g, batch_of(g), Seq{}); }
  static constexpr int slots(int b) { return slots_impl(Phys::NG, b, Seq{}); }
  template <int... G>
  static constexpr int grads_impl(int g, int b, std::integer_sequence<int, G...>) {
    return ((G < g && batch_of(G) == b ? GroupInfo<Phys, G>::NF_GRAD : 0) + ... + 0);
  }
  static constexpr int grad_offset(int g) { return grads_impl(g, batch_of(g), Seq{}); }
  static constexpr int grads(int b) { return grads_impl(Phys::NG, b, Seq{}); }
};

// The fields that the faces of group G read: count, and the k-th one; those that are face-only
// (no x-contracted rows) come last.
template <class Phys, int G>
struct FaceInfo {
  using Gi = GroupInfo<Phys, G < 0 ? 0 : G>;
  static constexpr int NF = [] {
    int n = 0;
    if (G >= 0)
      for (int f = 0; f < Gi::NF; ++f) n += FaceFieldOf<Phys>::get(G, f) ? 1 : 0;
    return n;
  }();
  static constexpr int NC = [] {  // of them with x-contracted rows
    int n = 0;
    if (G >= 0)
      for (int f = 0; f < Gi::NF_CELL; ++f) n += FaceFieldOf<Phys>::get(G, f) ? 1 : 0;
    return n;
  }();
  static constexpr int before(int f) {  // face fields before field f
    int n = 0;
    if (G >= 0)
      for (int i = 0; i < f; ++i) n += FaceFieldOf<Phys>::get(G, i) ? 1 : 0;
    return n;
  }
  static constexpr int field(int k) {
    int f = 0;
    for (;; ++f) {
      if (!FaceFieldOf<Phys>::get(G, f)) continue;
      if (k-- == 0) return f;
    }
  }
};

// Gauss points per direction of a policy: the operator's 2P+1, or P+1 for a policy that
// declares REDUCED_Q (preconditioner operators; exact for B, M and D on bilinear cells).
template <int P, class Phys, class = void>
struct NQOf {
  static constexpr int value = 2 * P + 1;
};
template <int P, class Phys>
struct NQOf<P, Phys, std::void_t<decltype(Phys::REDUCED_Q)>> {
  static constexpr int value = Phys::REDUCED_Q ? P + 1 : 2 * P + 1;
};

constexpr int imax(int a, int b) { return a > b ? a : b; }

template <int P, class Phys, int CB_ = cells_per_block<P, RealOf<Phys>>()>
struct Layout {
  using R = RealOf<Phys>;
  using I = PhysInfo<Phys>;
  using T = TabT<P, R, NQOf<P, Phys>::value>;
  static constexpr int P1 = T::P1, NQ = T::NQ, ND = P1 * P1;
  static constexpr int CB = CB_;
  static constexpr int NT = CB * NQ;
  static constexpr int NDP = odd(ND);
  static constexpr int NOUT = Phys::NOUT;
  static constexpr int NB = I::NB;
  // Rows: one value per (cell, point) of the CTA at stride NQP per cell.  A thread owns the
  // point m of cell cl at offset cl NQP + m, so a warp reads a row without bank conflicts, and a
  // line task writes or reads the NQ values of one cell at an odd stride between consecutive
  // cells, again without conflicts.
  static constexpr int NQP = odd(NQ);
  static constexpr int RS = CB * NQP;
  static constexpr int ALIGN = 16 / (int)sizeof(R);
  // The rows of one x-contracted slot, and the x-face traces of one field (up to two outer
  // neighbours per side), padded to 8 (mod 16) FP64 elements: the line tasks of a velocity
  // alternate between its components, whose results then fall on the two halves of the banks.
  static constexpr int half_banks(int n) { return n + (24 - n % 16) % 16; }
  static constexpr int SLS = half_banks(P1 * RS);
  static constexpr int TXS = half_banks((CB + 2) * NQP);
  static constexpr int up(int n) { return (n + ALIGN - 1) / ALIGN * ALIGN; }
  // Own-cell staging: the nodes of every (cell, component) of a batch's arrays form one list of
  // lines of ND nodes at stride LS, array after array, [cell][component] inside an array (the
  // global order).  With an odd number of nodes per cell the list is the arrays' image and arrives
  // by one bulk copy (TMA) per array; at degree 5 in FP64 by one bulk copy per line of 36 nodes, 16
  // bytes apart against bank conflicts (unpadded 748 us, padded 707 us for the fused right-hand
  // sides at 512x256); else by per-element copies of all threads.  At degree 3 a bulk copy of a line
  // of 16 nodes costs more than the elements (one warp issues 63 to 130 of them): stage 3 at 512x256
  // 405 -> 352 us with element copies, the split right-hand sides at 91x32 28.6 -> 19.4 us, C at 40x16
  // 5.2 -> 4.9 us.  Consecutive threads take consecutive lines, an odd number of elements apart.
  static constexpr bool BULK = (ND % 2 == 1 && (CB * ND * (int)sizeof(R)) % 16 == 0) || (ND % 2 == 0 && sizeof(R) == 8 && P >= 5);
  static constexpr int PADB = (BULK && ND % 2 == 0) ? ALIGN : 0;
  static constexpr int LS = BULK ? ND + PADB : odd(ND);
  static constexpr int ISSUE_LANES = PADB ? 32 : 1;  // threads that issue the copies
  // fields of the groups before G0 in its batch (G0 = NG: of batch b): cell fields, face-only fields
  template <int... G>
  static constexpr int cells_before(int g0, int b, std::integer_sequence<int, G...>) {
    return ((G < g0 && I::batch_of(G) == b ? GroupInfo<Phys, G>::NF_CELL : 0) + ... + 0);
  }
  template <int... G>
  static constexpr int only_before(int g0, int b, std::integer_sequence<int, G...>) {
    return ((G < g0 && I::batch_of(G) == b ? GroupInfo<Phys, G>::NF - GroupInfo<Phys, G>::NF_CELL : 0) + ... + 0);
  }
  // first line of array a of group G in its batch: the cell fields of all groups come first, then
  // the face-only ones
  template <int G>
  static constexpr int line_base(int a) {
    using Gi = GroupInfo<Phys, G>;
    using S = typename I::Seq;
    const int b = I::batch_of(G), f = Gi::first_field(a);
    if (f < Gi::NF_CELL) return CB * (cells_before(G, b, S{}) + f);
    return CB * (cells_before(Phys::NG, b, S{}) + only_before(G, b, S{}) + f - Gi::NF_CELL);
  }
  template <int G>
  static constexpr int group_size() {
    return CB * GroupInfo<Phys, G>::NF * LS;
  }
  template <int... G>
  static constexpr int batch_in(int b, std::integer_sequence<int, G...>) {
    return ((I::batch_of(G) == b ? group_size<G>() : 0) + ... + 0);
  }
  template <int B>
  struct Batch {
    static constexpr int FG = I::face_group(B);
    using F = FaceInfo<Phys, FG>;
    static constexpr int NS = I::slots(B), NG = I::grads(B);
    static constexpr int IN = batch_in(B, typename I::Seq{});
    // face traces: of the own x-faces (and up to two neighbours outside the CTA per side), of the
    // z-neighbours, and of the own z-faces for face-only fields
    static constexpr int NX = 2 * F::NF * TXS, NZ = 2 * F::NF * RS, NO = 2 * (F::NF - F::NC) * RS;
    static constexpr int TR = NX + NZ + NO;
    // lines of cell fields (they precede those of face-only fields), of gradient fields (the last
    // of them), of face fields
    static constexpr int NLC = (NS - NG) * CB, NLG = NG * CB, NLF = F::NF * CB;
  };
  template <class F, int... B>
  static constexpr int over(F f, std::integer_sequence<int, B...>) {
    int m = 0;
    ((m = imax(m, f(std::integral_constant<int, B>{}))), ...);
    return m;
  }
  using BSeq = std::make_integer_sequence<int, NB>;
  static constexpr int R_EO = up(over([](auto b) { return Batch<decltype(b)::value>::NS * SLS; }, BSeq{}));
  static constexpr int R_IN = up(over([](auto b) { return Batch<decltype(b)::value>::IN; }, BSeq{}));
  static constexpr int R_TR = up(over([](auto b) { return Batch<decltype(b)::value>::TR; }, BSeq{}));
  static constexpr int NTF = over([](auto b) { return Batch<decltype(b)::value>::F::NF; }, BSeq{});
  static constexpr int NTL = over([](auto b) { return Batch<decltype(b)::value>::NLC; }, BSeq{});
  static constexpr int NTT = imax(1, over([](auto b) { return Batch<decltype(b)::value>::NLF; }, BSeq{}));
  static_assert(NB == 1 || I::grads(0) == 0, "gradient fields in a policy of several batches");
  static_assert(imax(R_EO, imax(R_IN, R_TR)) < 65536, "offsets of the line tables");
  // x-face fluxes, then their z-contracted rows
  static constexpr int R_FX = Phys::FACES ? up(2 * NOUT * RS) : 0;
  // accumulators after the z pass: per output the rows tested with phi and with d/dxi phi, then
  // the contracted x-face fluxes [face][output][row][cell]
  static constexpr int O_XF = NOUT * (Phys::has_grad(0) ? 2 : 1) * P1 * RS;
  static constexpr int R_ACC = up(O_XF + (Phys::FACES ? 2 * NOUT * P1 * CB : 0));
  static constexpr int R_OUT = up(NOUT * CB * NDP);
  static constexpr int O_IN = R_EO, O_TR = O_IN + R_IN;
  // the x-face fluxes of a single batch take the place of its staged nodes, which the line tasks
  // have consumed; those of several batches are summed in a region of their own
  static constexpr int O_FX1 = imax(R_EO, R_ACC);
  static constexpr bool FX_IN = NB == 1 && O_FX1 + R_FX <= O_TR;
  static constexpr int O_FX = FX_IN ? O_FX1 : imax(O_TR + R_TR, R_ACC);
  static constexpr int O_OUT = R_ACC;
  static constexpr int BASE = imax(imax(O_TR + R_TR, O_FX + R_FX), O_OUT + R_OUT);
  // per cell: A, B, C (bilinear map), v0, edges of the faces xi = 1 and eta = 1 (two each)
  static constexpr int GS = 13;
  static constexpr int O_GEO = BASE;
  // region E (epilogue policies): the CTA's Gauss-point inverse weights, 16-byte aligned
  static constexpr int EPI = EpiOf<Phys>::value;
  // (EPI 2 and 3 also prefetch the residual (or z), the previous direction and the iterate of
  // their cells: NE chunks)
  static constexpr int NE = EPI >= 2 ? 4 : 1;
  static constexpr int OE = up(O_GEO + CB * GS);
  static constexpr int TOTAL = EPI ? OE + NE * CB * ND : O_GEO + CB * GS;
  // the epilogue's scratch (input rows and half-transformed values) lives in the accumulators' place
  static_assert(EPI == 0 || O_OUT >= (NOUT + 1) * CB * ND, "accumulator region too small for the epilogue");
  static constexpr size_t BYTES = sizeof(R) * TOTAL;
  // static shared memory: tables, neighbours, barriers (bound)
  static constexpr int STATIC = 2 * NB * (NTL + 2 * NTT) + 12 * NB * NTF + 16 * CB + 4 * NOUT + 64;
  static constexpr size_t MAX_BYTES = 225 * 1024;  // 227 KB per CTA, up to 2 KB of it static
  // CTAs per SM, the hint of __launch_bounds__: as many as the shared memory holds, at most 12 warps
  // (168 registers a thread; degrees 5 and 6 need more: 8 warps) or, with larger CTAs, three (two)
  static constexpr int FIT = (int)(228 * 1024 / (BYTES + 1024 + STATIC));
  static constexpr int WARPS = (NT + 31) / 32;
  static constexpr int MOST = P >= 5 ? imax(2, 8 / WARPS) : imax(3, 12 / WARPS);
  static constexpr int CTAS = FIT < 1 ? 1 : (FIT > MOST ? MOST : FIT);
};

// Cells per CTA of a policy launched without a choice of its own: cells_per_block, or the next smaller
// count with which the bulk copies stay aligned where the shared memory then holds one more CTA per SM.
// That is so for the fused stage-2 right-hand sides of degree 4 (12 cells: three CTAs, not two; 455 ->
// 411 us at 512x256) and degree 3 (8 cells: six, not five; 361 -> 340 us, 298 with element copies).
template <int P, class Phys>
constexpr int default_cells() {
  using R = RealOf<Phys>;
  constexpr int CB = cells_per_block<P, R>(), LESS = CB - ((P + 1) * (P + 1) % 2 ? 2 : 1);
  using L = Layout<P, Phys, CB>;
  if constexpr (sizeof(R) == 8 && L::FIT < L::MOST) {
    return Layout<P, Phys, LESS>::FIT > L::FIT ? LESS : CB;
  } else {
    return CB;
  }
}

// The most cells per CTA, from CB down in steps of two, with which two CTAs share an SM (one, when
// two do not fit even with two cells).
template <int P, class Phys, int CB>
constexpr int fit_cells() {
  constexpr size_t bytes = Layout<P, Phys, CB>::BYTES;
  if constexpr (2 * (bytes + 2048) <= 228 * 1024 || CB <= 2) return CB;
  else return fit_cells<P, Phys, CB - 2>();
}

// even/odd contraction of a P1-vector r along one direction to NQ values
template <int P, class R, int NQ>
__device__ __forceinline__ void contract_eo(const R* r, R* y) {
  using T = TabT<P, R, NQ>;
  const T& t = tabr<P, R, NQ>();
  R re[T::H > 0 ? T::H : 1], ro[T::H > 0 ? T::H : 1];
#pragma unroll
  for (int i = 0; i < T::H; ++i) {
    re[i] = r[i] + r[P - i];
    ro[i] = r[i] - r[P - i];
  }
  const R rm = T::MIDN ? r[P / 2] : 0.0;
#pragma unroll
  for (int k = 0; k < T::QH; ++k) {
    R e = T::MIDN ? t.Sm[k] * rm : t.Se[k][0] * re[0], o = t.So[k][0] * ro[0];
#pragma unroll
    for (int i = 0; i < T::H; ++i) {
      if (T::MIDN || i > 0) e = fmaR(t.Se[k][i], re[i], e);
      if (i > 0) o = fmaR(t.So[k][i], ro[i], o);
    }
    y[k] = e + o;
    y[T::NQ - 1 - k] = e - o;
  }
  if constexpr (T::QMID) {  // the middle point sees the even part only
    R e = T::MIDN ? t.Sm[T::QH] * rm : t.Se[T::QH][0] * re[0];
#pragma unroll
    for (int i = 0; i < T::H; ++i)
      if (T::MIDN || i > 0) e = fmaR(t.Se[T::QH][i], re[i], e);
    y[T::QH] = e;
  }
}

// derivative counterpart: y[q] = sum_i D[q][i] r[i] with D[NQ-1-q][i] = -D[q][P-i]
template <int P, class R, int NQ>
__device__ __forceinline__ void contract_eo_D(const R* r, R* y) {
  using T = TabT<P, R, NQ>;
  const T& t = tabr<P, R, NQ>();
  R re[T::H > 0 ? T::H : 1], ro[T::H > 0 ? T::H : 1];
#pragma unroll
  for (int i = 0; i < T::H; ++i) {
    re[i] = r[i] + r[P - i];
    ro[i] = r[i] - r[P - i];
  }
  const R rm = T::MIDN ? r[P / 2] : R(0);
#pragma unroll
  for (int k = 0; k < T::QE; ++k) {
    R e = 0.0, o = 0.0;
#pragma unroll
    for (int i = 0; i < T::H; ++i) {
      e = fmaR(t.De[k][i], re[i], e);
      o = fmaR(t.Do[k][i], ro[i], o);
    }
    if (T::MIDN) e = fmaR(t.Dm[k], rm, e);
    y[k] = e + o;
    if (k < T::QH) y[T::NQ - 1 - k] = o - e;
  }
}

// transposed contraction of NQ values f to P1 values y[i] = sum_q S[q][i] f[q]
template <int P, class R, int NQ>
__device__ __forceinline__ void contract_eo_T(const R* f, R* y) {
  using T = TabT<P, R, NQ>;
  const T& t = tabr<P, R, NQ>();
  R e[T::H > 0 ? T::H : 1], o[T::H > 0 ? T::H : 1], mid = R(0);
#pragma unroll
  for (int i = 0; i < T::H; ++i) {
    e[i] = T::QMID ? t.Se[T::QE - 1][i] * f[T::QE - 1] : R(0);
    o[i] = R(0);
  }
  if (T::MIDN && T::QMID) mid = t.Sm[T::QE - 1] * f[T::QE - 1];
#pragma unroll
  for (int k = 0; k < T::QH; ++k) {
    const R s = f[k] + f[NQ - 1 - k], d = f[k] - f[NQ - 1 - k];
#pragma unroll
    for (int i = 0; i < T::H; ++i) {
      e[i] = fmaR(t.Se[k][i], s, e[i]);
      o[i] = fmaR(t.So[k][i], d, o[i]);
    }
    if (T::MIDN) mid = fmaR(t.Sm[k], s, mid);
  }
#pragma unroll
  for (int i = 0; i < T::H; ++i) {
    y[i] = e[i] + o[i];
    y[P - i] = e[i] - o[i];
  }
  if (T::MIDN) y[P / 2] = mid;
}

// ----------------------------------------------------------------------------------
// the kernel
// ----------------------------------------------------------------------------------
template <int P, class Phys, int CB_ = default_cells<P, Phys>(), int MINB = Layout<P, Phys, CB_>::CTAS>
__global__ void __launch_bounds__(Layout<P, Phys, CB_>::NT, MINB)
    k_cellop(const __grid_constant__ MeshDev mesh,
             const __grid_constant__ ArgPtrs<PhysInfo<Phys>::NARR_TOTAL, Phys::NOUT_ARR, RealOf<Phys>> ptr,
             const __grid_constant__ typename Phys::Params prm, const int ncell) {
  using L = Layout<P, Phys, CB_>;
  using I = PhysInfo<Phys>;
  using R = RealOf<Phys>;
  using T = typename L::T;
  constexpr int P1 = L::P1, NQ = L::NQ, ND = L::ND, CB = L::CB, NT = L::NT, NQP = L::NQP, RS = L::RS;
  constexpr int H = T::H;
  constexpr bool MIDN = T::MIDN;
  constexpr int QH = T::QH;  // quadrature point pairs (q, NQ-1-q); middle point QH if T::QMID
  constexpr int NOUT = Phys::NOUT, NB = L::NB;
  const T& tb = tabr<P, R, NQ>();
  static_assert(L::BYTES <= L::MAX_BYTES, "shared memory of one CTA above the sm_100 limit");

  extern __shared__ __align__(16) unsigned char smem_raw[];
  R* const smem = reinterpret_cast<R*>(smem_raw);
  R* const s_eo = smem;              // x-contracted rows of the batch
  R* const s_acc = smem;             //   (after the z pass)
  R* const s_tr = smem + L::O_TR;    // face traces of the batch
  R* const s_fx = smem + L::O_FX;    // x-face fluxes
  R* const s_out = smem + L::O_OUT;  //   (after the z pass)
  R* const s_geo = smem + L::O_GEO;
  // neighbours of the CTA's cells: x-faces: the slot of the neighbour's trace (-1: wall), z-faces: 0 or -1
  __shared__ int s_nb[4 * CB];
  // line tables: per cell line its place in the x-contracted rows, per face line its place in the
  // input buffer and in the traces; per face field its global array and the array's components
  __shared__ unsigned short s_line[NB * L::NTL], s_tsrc[NB * L::NTT], s_tdst[NB * L::NTT];
  __shared__ int s_tc[Phys::FACES ? NB * L::NTF : 1];
  __shared__ const R* s_tp[Phys::FACES ? NB * L::NTF : 1];
  __shared__ int s_to[NOUT];
  // completion of the input buffer's bulk copies
  __shared__ alignas(8) unsigned long long s_bar;
  const unsigned bar = (unsigned)__cvta_generic_to_shared(&s_bar);
  pdl_allow_next();
  if (mesh.test_wait_polls > 0) {
    // test hook: the bounded wait gives up on a phase that nobody completes (s_bar is armed
    // with an arrival count of 1 and nobody arrives), then the CTA leaves as after a real
    // staging timeout; no copy has been issued yet
    bool ok = true;
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
      ok = mbar_wait(bar, 0, mesh.test_wait_polls);
      if (!ok) report_status(mesh.status, kStatusStageTimeout);
    }
    if (__syncthreads_or(!ok)) return;
  }
  const int tid = threadIdx.x;
  const int c0 = mesh.cell0 + blockIdx.x * CB;
  const int ncb = min(CB, ncell - c0);  // valid cells in this block
  // bulk staging when every chunk starts and ends on 16 bytes (uniform per CTA); a chunk starts
  // off a boundary only with an odd number of nodes per cell and an odd first cell
  const bool bulk = L::BULK && ((size_t)ncb * ND * sizeof(R)) % 16 == 0 && ((size_t)c0 * ND * sizeof(R)) % 16 == 0;
  // batch B's arrays into its input buffer, by warp 0 (lane 0 alone without padding)
  auto issue_batch = [&](auto bc) {
    constexpr int B = decltype(bc)::value;
    R* const buf = smem + L::O_IN;
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    if (tid == 0) {
      unsigned bytes = 0;
      sfor<Phys::NG>([&](auto gc) {
        constexpr int G = decltype(gc)::value;
        if constexpr (I::batch_of(G) == B) bytes += (unsigned)(ncb * GroupInfo<Phys, G>::NF * ND * sizeof(R));
      });
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
    }
    if constexpr (L::PADB > 0) __syncwarp();
    sfor<Phys::NG>([&](auto gc) {
      constexpr int G = decltype(gc)::value;
      if constexpr (I::batch_of(G) == B) {
        using Gi = GroupInfo<Phys, G>;
        sfor<Gi::NARR>([&](auto ac) {
          constexpr int A = decltype(ac)::value;
          constexpr int NC = Gi::Gr::ncomp(A);
          const R* src = ptr.in[I::arr_base(G) + A] + (size_t)c0 * NC * ND;
          const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + L::template line_base<G>(A) * L::LS);
          // one copy per array, or one per line (every chunk and slot a multiple of 16 bytes)
          for (int cc = tid; cc < (L::PADB ? ncb * NC : 1); cc += 32)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                    dst + (unsigned)(cc * L::LS * (int)sizeof(R))),
                "l"(src + (size_t)cc * ND), "r"((unsigned)((L::PADB ? 1 : ncb * NC) * ND * sizeof(R))), "r"(bar)
                : "memory");
        });
      }
    });
  };
  // the same by per-element copies of all threads (waited for with cp_async_wait_all), issued where the
  // bulk copies are; in a bulk layout, whose last CTA alone may need them, at the wait (issued early
  // there too, their code costs every CTA: the transposed C at 128x64, p = 4, 10.6 -> 11.2 us)
  auto copy_batch = [&](auto bc) {
    constexpr int B = decltype(bc)::value;
    sfor<Phys::NG>([&](auto gc) {
      constexpr int G = decltype(gc)::value;
      if constexpr (I::batch_of(G) == B) {
        using Gi = GroupInfo<Phys, G>;
        sfor<Gi::NARR>([&](auto ac) {
          constexpr int A = decltype(ac)::value;
          constexpr int NC = Gi::Gr::ncomp(A);
          const R* src = ptr.in[I::arr_base(G) + A] + (size_t)c0 * NC * ND;
          for (int e = tid; e < ncb * NC * ND; e += NT)
            cp_async_el(&smem[L::O_IN + (L::template line_base<G>(A) + e / ND) * L::LS + e % ND], src + e);
        });
      }
    });
  };
  // copies were issued and not yet waited for; their phase
  bool pending = L::BULK && bulk;
  unsigned phase = 0u;
  if constexpr (L::BULK) {
    if (tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar) : "memory");
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (L::PADB > 0 && tid < 32) __syncwarp();
  }

  bool abort = false;
  // epilogue policies: the CTA's inverse weights (and for EPI 2, 3: r, din, x), each
  // [cell][node] over the CTA's cells, copied from the start of the kernel on
  __shared__ alignas(8) unsigned long long s_bar_e;
  const unsigned bar_e = (unsigned)__cvta_generic_to_shared(&s_bar_e);
  R* s_minv = smem + L::OE;
  bool epi_bulk = false;
  const R* epi_src[4] = {nullptr, nullptr, nullptr, nullptr};
  size_t epi_bytes = 0;
  if constexpr (L::EPI != 0) {
    epi_bytes = sizeof(R) * (size_t)ncb * ND;
    epi_src[0] = prm.inv + (size_t)c0 * ND;
    if constexpr (L::EPI >= 2) {
      epi_src[1] = prm.r + (size_t)c0 * ND;
      epi_src[2] = prm.din + (size_t)c0 * ND;
      epi_src[3] = prm.x + (size_t)c0 * ND;
    }
    epi_bulk = epi_bytes % 16 == 0;
#pragma unroll
    for (int k = 0; k < L::NE; ++k) epi_bulk = epi_bulk && (reinterpret_cast<size_t>(epi_src[k]) & 15) == 0;
    if (epi_bulk && tid == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar_e) : "memory");
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
  }
  // the copies that read what earlier kernels wrote: batch 0 and the epilogue's chunks
  auto issue_inputs = [&]() {
    if constexpr (L::BULK) {
      if (tid < L::ISSUE_LANES && bulk) issue_batch(std::integral_constant<int, 0>{});
    }
    if constexpr (!L::BULK) copy_batch(std::integral_constant<int, 0>{});
    if constexpr (L::EPI != 0) {
      if (epi_bulk) {
        if (tid == 0) {
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar_e),
                       "r"((unsigned)(epi_bytes * L::NE))
                       : "memory");
#pragma unroll
          for (int k = 0; k < L::NE; ++k)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                    (unsigned)__cvta_generic_to_shared(s_minv + k * CB * ND)),
                "l"(epi_src[k]), "r"((unsigned)epi_bytes), "r"(bar_e)
                : "memory");
        }
      } else {
#pragma unroll
        for (int k = 0; k < L::NE; ++k)
          for (int e = tid; e < ncb * ND; e += NT) cp_async_el(&s_minv[k * CB * ND + e], epi_src[k] + e);
      }
    }
  };
  // without the geometry-first prologue the copies start at once and overlap the geometry
  constexpr bool GEO_FIRST = pdl_geo_first<R>();
  if constexpr (!GEO_FIRST) {
    pdl_wait_previous();
    issue_inputs();
  }

  // two maps of the threads: point map (cell cl, point m) of the z pass and the faces; line map
  // (cell ct, line mt + NQ k) of the 1D contractions, consecutive threads on consecutive cells
  const int cl = tid / NQ, m = tid % NQ;
  const int mt = tid / CB, ct = tid % CB;
  const int cg = c0 + (ct < ncb ? ct : ncb - 1);  // global index of cell ct
  const int gi = cg % mesh.nx, gj = cg / mesh.nx;
  const int clast = c0 + ncb - 1;

  // ---- per-cell geometry and neighbours (one row of the line map), tables of the line tasks
  if (mt == NQ - 1) {
    const int W = mesh.nx + 1;
    const double2* v = mesh.vtx + (size_t)gj * W + gi;
    const double2 v0 = v[0], v1 = v[1], v2 = v[W], v3 = v[W + 1];
    R* g = s_geo + ct * L::GS;
    g[0] = v1.x - v0.x; g[1] = v1.y - v0.y;                              // A = x_xi at eta = 0
    g[2] = v3.x - v2.x - v1.x + v0.x; g[3] = v3.y - v2.y - v1.y + v0.y;  // B (bilinear term)
    g[4] = v2.x - v0.x; g[5] = v2.y - v0.y;                              // C = x_eta at xi = 0
    g[6] = v0.x; g[7] = v0.y;
    // the edges of the faces xi = 1 and eta = 1; those of xi = 0 and eta = 0 are C and A.  A
    // face's normal is formed from its two vertices the same way by both cells.
    g[8] = v3.x - v1.x; g[9] = v3.y - v1.y;
    g[10] = v3.x - v2.x; g[11] = v3.y - v2.y;
    if constexpr (Phys::FACES) {
      // x-neighbours in the CTA: their own trace slot; outside it: two extra slots per side, the
      // first for the cell before (after) the CTA, the second for a periodic one
      const int nl = gi > 0 ? cg - 1 : (mesh.periodic_x ? cg + mesh.nx - 1 : -1);
      const int nr = gi < mesh.nx - 1 ? cg + 1 : (mesh.periodic_x ? cg - mesh.nx + 1 : -1);
      s_nb[4 * ct] = nl < 0 ? -1 : ((nl >= c0 && nl <= clast) ? nl - c0 : CB + (gi > 0 ? 0 : 1));
      s_nb[4 * ct + 1] = nr < 0 ? -1 : ((nr >= c0 && nr <= clast) ? nr - c0 : CB + (gi < mesh.nx - 1 ? 0 : 1));
      s_nb[4 * ct + 2] = gj > 0 ? 0 : -1;
      s_nb[4 * ct + 3] = gj < mesh.nz - 1 ? 0 : -1;
    }
  }
  sfor<Phys::NG>([&](auto gc) {
    constexpr int G = decltype(gc)::value, B = I::batch_of(G);
    using Gi = GroupInfo<Phys, G>;
    using F = FaceInfo<Phys, Gi::FACE ? G : -1>;
    sfor<Gi::NARR>([&](auto ac) {
      constexpr int A = decltype(ac)::value, NC = Gi::Gr::ncomp(A), f0 = Gi::first_field(A);
      constexpr bool cell_field = !Gi::Gr::face_only(A), face_field = Gi::FACE && FaceFieldOf<Phys>::get(G, f0);
      constexpr int k0 = F::before(f0);  // face fields before this array's
      static_assert(!cell_field || L::template line_base<G>(A) + CB * NC <= L::NTL, "line outside its table");
      static_assert(!face_field || k0 * CB + CB * NC <= L::NTT, "face line outside its table");
      for (int t = tid; t < CB * NC; t += NT) {
        const int cc = t / NC, d = t % NC, line = L::template line_base<G>(A) + t;
        if (cell_field) s_line[B * L::NTL + line] = (unsigned short)((I::slot_offset(G) + f0 + d) * L::SLS + cc * NQP);
        if (face_field) {
          s_tsrc[B * L::NTT + k0 * CB + t] = (unsigned short)(line * L::LS);
          s_tdst[B * L::NTT + k0 * CB + t] = (unsigned short)((k0 + d) * L::TXS + cc * NQP);
        }
      }
      if constexpr (face_field) {
        if (tid < NC) {
          s_tc[B * L::NTF + k0 + tid] = NC;
          s_tp[B * L::NTF + k0 + tid] = ptr.in[I::arr_base(G) + A] + tid * ND;
        }
      }
    });
  });
  if (tid < 32) {
    sfor<Phys::NOUT_ARR>([&](auto oc) {
      constexpr int OA = decltype(oc)::value, NC = Phys::out_ncomp(OA);
      constexpr int ob = [] { int b = 0; for (int a = 0; a < OA; ++a) b += Phys::out_ncomp(a); return b; }();
      sfor<NC>([&](auto dc) {
        constexpr int d = decltype(dc)::value;
        if (tid == ob + d) s_to[ob + d] = L::EPI ? ((ob + d) * CB * L::NDP) | (L::NDP << 20) : (ob * CB * ND + d * ND) | ((NC * ND) << 20);
      });
    });
  }
  // geometry-first prologue: everything above read only the mesh vertices and the constant
  // tables, which no kernel writes just before a cell-operator launch; from here on the
  // previous grid's writes are visible
  if constexpr (GEO_FIRST) {
    pdl_wait_previous();
    issue_inputs();
  }
  __syncthreads();  // geometry and tables visible

  // accumulators of the z pass (see below)
  constexpr int HE = H > 0 ? H : 1;
  R aE[NOUT][HE], aO[NOUT][HE], aM[NOUT], bE[NOUT][HE], bO[NOUT][HE], bM[NOUT];
#pragma unroll
  for (int o = 0; o < NOUT; ++o) {
#pragma unroll
    for (int i = 0; i < HE; ++i) aE[o][i] = aO[o][i] = bE[o][i] = bO[o][i] = R(0);
    aM[o] = bM[o] = R(0);
  }

  sfor<NB>([&](auto bc) {
    constexpr int B = decltype(bc)::value;
    using Bt = typename L::template Batch<B>;
    using F = typename Bt::F;
    constexpr int FG = Bt::FG, NFF = F::NF;
    R* const s_in = smem + L::O_IN;
    if (abort) return;
    if (B > 0) __syncthreads();  // the rows and traces of the batch before are free

    // ---- traces of the neighbours' faces, straight from their nodes (L2-resident): one line per
    //      (z-side, field, cell), and per field up to two cells on either side of the CTA
    if constexpr (FG >= 0) {
      constexpr int NZT = (2 * NFF + NQ - 1) / NQ;  // rounds of the z-sides' lines
      constexpr int NXT = (4 * NFF + NT - 1) / NT;  // rounds of the outer x-neighbours' lines
#pragma unroll 1
      for (int t = 0; t < NZT + NXT; ++t) {
        int k, nb = -1, start, stride;
        R* dst;
        if (t < NZT) {
          const int e = mt + t * NQ, top = e >= NFF ? 1 : 0;
          k = e - top * NFF;
          if (e < 2 * NFF) nb = top ? (gj < mesh.nz - 1 ? cg + mesh.nx : -1) : (gj > 0 ? cg - mesh.nx : -1);
          start = top ? 0 : P * P1;
          stride = 1;
          dst = s_tr + Bt::NX + (e * CB + ct) * NQP;
        } else {
          const int e = NT - 1 - tid + (t - NZT) * NT, x = e & 3;
          k = e >> 2;
          const int first = c0 - c0 % mesh.nx, lrow = clast - clast % mesh.nx;  // rows of the first and last cell
          if (e >= 4 * NFF) nb = -1;
          else if (x == 0) nb = c0 > first ? c0 - 1 : -1;
          else if (x == 1) nb = mesh.periodic_x && lrow >= c0 && lrow + mesh.nx - 1 > clast ? lrow + mesh.nx - 1 : -1;
          else if (x == 2) nb = clast < lrow + mesh.nx - 1 ? clast + 1 : -1;
          else nb = mesh.periodic_x && first + mesh.nx - 1 <= clast && first < c0 ? first : -1;
          start = x < 2 ? P : 0;  // a left neighbour's right face, a right neighbour's left face
          stride = P1;
          dst = s_tr + ((x < 2 ? 1 : 0) * NFF + k) * L::TXS + (CB + (x & 1)) * NQP;
        }
        if (nb >= 0) {
          const R* src = s_tp[B * L::NTF + k] + (size_t)nb * (s_tc[B * L::NTF + k] * ND) + start;
          R r[P1], y[NQ];
#pragma unroll
          for (int i = 0; i < P1; ++i) r[i] = src[i * stride];
          contract_eo<P, R, NQ>(r, y);
#pragma unroll
          for (int q = 0; q < NQ; ++q) dst[q] = y[q];
        }
      }
    }

    // ---- the own cells' nodes
    bool ok = true;
    if (bulk) {
      ok = mbar_wait(bar, phase);
      if (ok) {
        phase ^= 1u;
        pending = false;
      } else {
        report_status(mesh.status, kStatusStageTimeout);
      }
    } else {
      if constexpr (L::BULK) copy_batch(bc);  // (an odd last CTA)
      cp_async_wait_all();
      __syncthreads();
    }

    // ---- line tasks on them: the rows (k, P-k) of every line, even/odd, contracted along x
    auto load = [&](const R* src, int st, R* r) {
#pragma unroll
      for (int i = 0; i < P1; ++i) r[i] = src[i * st];
    };
    auto store = [&](R* dst, const R* y) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) dst[q] = y[q];
    };
    auto row_pair = [&](int line, int k, auto der) {
      R a[P1], b[P1], r[P1], y[NQ];
      load(s_in + line * L::LS + k * P1, 1, a);
      load(s_in + line * L::LS + (P - k) * P1, 1, b);
      R* dst = s_eo + s_line[B * L::NTL + line] + (decltype(der)::value ? Bt::NG * L::SLS : 0) + k * RS;
#pragma unroll
      for (int i = 0; i < P1; ++i) r[i] = a[i] + b[i];
      if constexpr (decltype(der)::value) contract_eo_D<P, R, NQ>(r, y);
      else contract_eo<P, R, NQ>(r, y);
      store(dst, y);
#pragma unroll
      for (int i = 0; i < P1; ++i) r[i] = a[i] - b[i];
      if constexpr (decltype(der)::value) contract_eo_D<P, R, NQ>(r, y);
      else contract_eo<P, R, NQ>(r, y);
      store(dst + H * RS, y);
    };
    for (int e = tid; e < H * Bt::NLC; e += NT) row_pair(e % Bt::NLC, e / Bt::NLC, std::false_type{});
    if constexpr (Bt::NG > 0) {
      for (int e = tid; e < H * Bt::NLG; e += NT)
        row_pair(Bt::NLC - Bt::NLG + e % Bt::NLG, e / Bt::NLG, std::true_type{});
    }
    //      the middle rows, the traces of the x-faces and of the z-faces of face-only fields (from the
    //      other end of the CTA, which has fewer row pairs)
    constexpr int NM = MIDN ? Bt::NLC : 0, NLO = (NFF - F::NC) * CB, NLX = Bt::NLF;
    for (int e = NT - 1 - tid; e < NM + 2 * NLX + 2 * NLO; e += NT) {
      const R* src;
      R* dst;
      int st = 1;
      if (e < NM) {
        src = s_in + e * L::LS + (P / 2) * P1;
        dst = s_eo + s_line[B * L::NTL + e] + 2 * H * RS;
      } else if (e < NM + 2 * NLX) {
        const int f = e >= NM + NLX ? 1 : 0, t = e - NM - f * NLX;
        src = s_in + s_tsrc[B * L::NTT + t] + f * P;
        dst = s_tr + s_tdst[B * L::NTT + t] + f * NFF * L::TXS;
        st = P1;
      } else {
        const int f = e >= NM + 2 * NLX + NLO ? 1 : 0, o = e - NM - 2 * NLX - f * NLO, t = NLX - NLO + o;
        const int p = s_tdst[B * L::NTT + t], k = p / L::TXS;  // face field of the line
        src = s_in + s_tsrc[B * L::NTT + t] + f * P * P1;
        dst = s_tr + Bt::NX + Bt::NZ + (f * (NFF - F::NC) + k - F::NC) * RS + (p - k * L::TXS);
      }
      R r[P1], y[NQ];
      load(src, st, r);
      contract_eo<P, R, NQ>(r, y);
      store(dst, y);
    }
    if constexpr (Bt::NG > 0 && MIDN) {
      for (int e = NT - 1 - tid; e < Bt::NLG; e += NT) {
        const int line = Bt::NLC - Bt::NLG + e;
        R r[P1], y[NQ];
        load(s_in + line * L::LS + (P / 2) * P1, 1, r);
        contract_eo_D<P, R, NQ>(r, y);
        store(s_eo + s_line[B * L::NTL + line] + Bt::NG * L::SLS + 2 * H * RS, y);
      }
    }
    if (__syncthreads_or(!ok)) {  // a staging wait gave up: every thread leaves together
      abort = true;
      return;
    }
    if constexpr (B + 1 < NB) {  // the line tasks have consumed the buffer: the next batch's nodes
      if (bulk) {
        if (tid < L::ISSUE_LANES) issue_batch(std::integral_constant<int, B + 1>{});
        pending = true;
      }
      if constexpr (!L::BULK) copy_batch(std::integral_constant<int, B + 1>{});
    }

    // ---- faces: numerical flux at face point m of cell cl.  The fluxes are linear in the normal's
    //      length, so the edge vector times the quadrature weight serves as normal times JxW.  The
    //      z-faces go into the accumulators of node rows 0 and P (whose weight is theirs, w_m), the
    //      x-faces to shared memory.
    const R* const g = s_geo + cl * L::GS;
    const int pt = cl * NQP + m;
    if constexpr (FG >= 0) {
      constexpr int NFG_ = GroupInfo<Phys, FG>::NF;
      const R wq = tb.w[m];
      R zb[NFF], zt[NFF];
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        if (f == 2) {  // the own traces on eta = 0 and 1: half the sum and difference of the rows 0 +- P
          sfor<NFF>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            if constexpr (k < F::NC) {
              const R* e = s_eo + (I::slot_offset(FG) + F::field(k)) * L::SLS + pt;
              const R a = R(0.5) * e[0], b = e[H * RS];
              zb[k] = fmaR(R(0.5), b, a);
              zt[k] = fmaR(R(-0.5), b, a);
            } else {
              const R* e = s_tr + Bt::NX + Bt::NZ + (k - F::NC) * RS + pt;
              zb[k] = e[0];
              zt[k] = e[(NFF - F::NC) * RS];
            }
          });
        }
        R vp[NFG_], vm[NFG_], fo[NOUT];
        const int nb = s_nb[4 * cl + f];
        if (f < 2) {
          const R* own = s_tr + f * NFF * L::TXS + pt;
          const R* oth = s_tr + (1 - f) * NFF * L::TXS + (nb < 0 ? 0 : nb) * NQP + m;
          sfor<NFF>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            vp[F::field(k)] = own[k * L::TXS];
            vm[F::field(k)] = oth[k * L::TXS];
          });
        } else {
          sfor<NFF>([&](auto kc) {
            constexpr int k = decltype(kc)::value;
            vp[F::field(k)] = f == 2 ? zb[k] : zt[k];
            vm[F::field(k)] = s_tr[Bt::NX + ((f - 2) * NFF + k) * RS + pt];
          });
        }
        constexpr int E0[4] = {4, 8, 0, 10};
        // outward: (-tz, tx) on faces 0 and 3
        const R sw = (f == 0 || f == 3 ? R(1) : R(-1)) * (f < 2 ? wq : R(1));
        const R n[2] = {-sw * g[E0[f] + 1], sw * g[E0[f]]};
#pragma unroll
        for (int o = 0; o < NOUT; ++o) fo[o] = R(0);
        if (nb >= 0) Phys::template face<FG>(prm, vp, vm, n, fo);
        else Phys::template boundary<FG>(prm, vp, n, fo);
#pragma unroll
        for (int o = 0; o < NOUT; ++o) {
          if (f < 2) {
            R* d = s_fx + (f * NOUT + o) * RS + pt;
            *d = B > 0 ? *d + fo[o] : fo[o];
          } else {
            aE[o][0] += R(0.5) * fo[o];
            aO[o][0] += (f == 2 ? R(0.5) : R(-0.5)) * fo[o];
          }
        }
        asm volatile("" ::: "memory");  // one face's traces at a time in registers
      }
    } else if constexpr (Phys::FACES && B == 0) {
#pragma unroll
      for (int o = 0; o < 2 * NOUT; ++o) s_fx[o * RS + pt] = R(0);
    }

    // ---- z pass: member = quadrature column qx = m.  All fields of the batch are evaluated at each
    // point, their integrands summed, and the sum is mapped to reference coordinates and
    // contracted along z once.  The contraction of a point pair (q, NQ-1-q) goes into even/odd
    // accumulators of the node pairs (i, P-i) (tables with the z weight folded in; the x weight
    // multiplies the accumulators at the end):
    //   S terms:  E_i += Se[q][i] (f1 + f2),  O_i += So[q][i] (f1 - f2),  mid += Sm[q] (f1 + f2)
    //   D terms:  E_i += De[q][i] (g1 - g2),  O_i += Do[q][i] (g1 + g2),  mid += Dm[q] (g1 - g2)
    // (S[NQ-1-q][i] = S[q][P-i], D[NQ-1-q][i] = -D[q][P-i]); node i gets E_i + O_i, node P-i
    // gets E_i - O_i.  A middle point is a pair with f2 = g2 = 0.
    {
      constexpr int NS = Bt::NS, NGR = Bt::NG;
      const R xi = tb.x[m];
      const R J01 = fmaR(g[2], xi, g[4]);  // x_eta (x component)
      const R J11 = fmaR(g[3], xi, g[5]);  // x_eta (z component)
      const bool need_x = Phys::NEED_X && PositionUse<typename Phys::Params>::get(prm);
      const R* const eo = s_eo + pt;
      // the mapped integrands of one point, up to the quadrature weights: fv (tested with phi), fx,
      // fe (with d/dxi, d/deta phi)
      auto integrand = [&](const R* v, const R* deta, const int qz, R* fvo, R* fxo, R* feo) {
        const R eta = tb.x[qz];
        const R a11 = fmaR(g[2], eta, g[0]), a10 = fmaR(g[3], eta, g[1]);  // x_xi, z_xi
        const R dw = a11 * J11 - a10 * J01;
        PointGeo pg;
        if (need_x) {
          pg.X[0] = g[6] + g[0] * xi + g[4] * eta + g[2] * xi * eta;
          pg.X[1] = g[7] + g[1] * xi + g[5] * eta + g[3] * xi * eta;
        }
        if constexpr (NGR > 0) {
          pg.J[0] = a11; pg.J[1] = J01; pg.J[2] = a10; pg.J[3] = J11;
        }
        if constexpr (MappedOf<Phys>::value) {  // the policy maps its own integrand
          const R A[4] = {J11, J01, a10, a11};
#pragma unroll
          for (int o = 0; o < NOUT; ++o) fvo[o] = fxo[o] = feo[o] = R(0);
          sfor<Phys::NG>([&](auto gc) {
            constexpr int G = decltype(gc)::value;
            if constexpr (I::batch_of(G) == B)
              Phys::template point_mapped<G>(prm, v + I::slot_offset(G), pg, A, dw, fvo, fxo, feo);
          });
        } else {
          R val[NOUT], gr[NOUT][2];
#pragma unroll
          for (int o = 0; o < NOUT; ++o) { val[o] = 0.0; gr[o][0] = gr[o][1] = 0.0; }
          sfor<Phys::NG>([&](auto gc) {
            constexpr int G = decltype(gc)::value;
            if constexpr (I::batch_of(G) == B) {
              if constexpr (NfgOf<Phys>::any)
                Phys::template point<G>(prm, v + I::slot_offset(G), deta + I::grad_offset(G), pg, val, gr);
              else
                Phys::template point<G>(prm, v + I::slot_offset(G), pg, val, gr);
            }
          });
#pragma unroll
          for (int o = 0; o < NOUT; ++o) {
            fvo[o] = val[o] * dw;
            fxo[o] = J11 * gr[o][0] - J01 * gr[o][1];
            feo[o] = a11 * gr[o][1] - a10 * gr[o][0];
          }
        }
      };
#pragma unroll 1
      for (int k = 0; k < T::QE; ++k) {
        const bool pair = k < QH;
        asm volatile("" ::: "memory");  // keeps the rows in shared memory: hoisted, they spill
        R v1[NS], v2[NS];
#pragma unroll
        for (int fi = 0; fi < NS; ++fi) {
          const R* row = eo + fi * L::SLS;
          R e = MIDN ? tb.Sm[k] * row[2 * H * RS] : R(0), o = R(0);
#pragma unroll
          for (int i = 0; i < H; ++i) {
            e = fmaR(tb.Se[k][i], row[i * RS], e);
            o = fmaR(tb.So[k][i], row[(H + i) * RS], o);  // (0 at a middle point)
          }
          v1[fi] = e + o;
          v2[fi] = e - o;
        }
        // d/deta of the gradient fields: their S-row slots contracted with D along z
        R d1[NGR > 0 ? NGR : 1], d2[NGR > 0 ? NGR : 1];
        if constexpr (NGR > 0) {
          sfor<Phys::NG>([&](auto gc) {
            constexpr int G = decltype(gc)::value;
            if constexpr (I::batch_of(G) == B) {
              using Gi = GroupInfo<Phys, G>;
#pragma unroll
              for (int kk = 0; kk < Gi::NF_GRAD; ++kk) {
                const R* row = eo + (I::slot_offset(G) + Gi::NF_CELL - Gi::NF_GRAD + kk) * L::SLS;
                R e = 0.0, o = 0.0;
#pragma unroll
                for (int i = 0; i < H; ++i) {
                  e = fmaR(tb.De[k][i], row[i * RS], e);
                  o = fmaR(tb.Do[k][i], row[(H + i) * RS], o);  // at the middle point only o remains
                }
                if (MIDN) e = fmaR(tb.Dm[k], row[2 * H * RS], e);
                d1[I::grad_offset(G) + kk] = e + o;
                d2[I::grad_offset(G) + kk] = o - e;
              }
            }
          });
        }
        R fv1[NOUT], fx1[NOUT], fe1[NOUT], fv2[NOUT], fx2[NOUT], fe2[NOUT];
        integrand(v1, d1, k, fv1, fx1, fe1);
        if (pair) {
          integrand(v2, d2, NQ - 1 - k, fv2, fx2, fe2);
        } else {
#pragma unroll
          for (int o = 0; o < NOUT; ++o) fv2[o] = fx2[o] = fe2[o] = R(0);
        }
        sfor<NOUT>([&](auto oc) {
          constexpr int o = decltype(oc)::value;
          constexpr bool hv = TermsOf<Phys>::val(B, o), hg = TermsOf<Phys>::grad(B, o);
          const R se = hv ? fv1[o] + fv2[o] : R(0), so = hv ? fv1[o] - fv2[o] : R(0);
          const R ge = hg ? fe1[o] - fe2[o] : R(0), go = hg ? fe1[o] + fe2[o] : R(0);
          const R xe = hg ? fx1[o] + fx2[o] : R(0), xo = hg ? fx1[o] - fx2[o] : R(0);
#pragma unroll
          for (int i = 0; i < H; ++i) {
            if (hv) {
              aE[o][i] = fmaR(tb.SeW[k][i], se, aE[o][i]);
              aO[o][i] = fmaR(tb.SoW[k][i], so, aO[o][i]);
            }
            if (hg) {
              aE[o][i] = fmaR(tb.DeW[k][i], ge, aE[o][i]);
              aO[o][i] = fmaR(tb.DoW[k][i], go, aO[o][i]);
              bE[o][i] = fmaR(tb.SeW[k][i], xe, bE[o][i]);
              bO[o][i] = fmaR(tb.SoW[k][i], xo, bO[o][i]);
            }
          }
          if (MIDN) {
            if (hv) aM[o] = fmaR(tb.SmW[k], se, aM[o]);
            if (hg) {
              aM[o] = fmaR(tb.DmW[k], ge, aM[o]);
              bM[o] = fmaR(tb.SmW[k], xe, bM[o]);
            }
          }
        });
      }
    }
  });
  if (abort) {  // a staging wait gave up: wait (bounded) for this CTA's copies before leaving
    if (tid == 0) {
      if (pending) mbar_wait(bar, phase);
      if (epi_bulk) mbar_wait(bar_e, 0);
    }
    return;
  }
  __syncthreads();  // the x-contracted rows are consumed -> accumulators
  {
    const int pt = cl * NQP + m;
    const R wx = tb.w[m];
#pragma unroll
    for (int o = 0; o < NOUT; ++o) {
      R* A = s_acc + (o * P1) * RS + pt;           // [output][row], tested with phi
      R* Bx = s_acc + ((NOUT + o) * P1) * RS + pt;  // [output][row], tested with d/dxi phi
      const bool hg = Phys::has_grad(o);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        A[i * RS] = wx * (aE[o][i] + aO[o][i]);
        A[(P - i) * RS] = wx * (aE[o][i] - aO[o][i]);
        if (hg) {
          Bx[i * RS] = wx * (bE[o][i] + bO[o][i]);
          Bx[(P - i) * RS] = wx * (bE[o][i] - bO[o][i]);
        }
      }
      if (MIDN) {
        A[(P / 2) * RS] = wx * aM[o];
        if (hg) Bx[(P / 2) * RS] = wx * bM[o];
      }
    }
  }
  if constexpr (Phys::FACES) {  // the x-face fluxes contracted along z: line = (face, output)
    for (int e = mt; e < 2 * NOUT; e += NQ) {
      R f[NQ], y[P1];
#pragma unroll
      for (int q = 0; q < NQ; ++q) f[q] = s_fx[e * RS + ct * NQP + q];
      contract_eo_T<P, R, NQ>(f, y);
#pragma unroll
      for (int i = 0; i < P1; ++i) s_acc[L::O_XF + (e * P1 + i) * CB + ct] = y[i];
    }
  }
  __syncthreads();
  // ---- x-transpose pass: line (output, row iz) -> P1 outputs, plus the x-faces' nodes
  for (int row = mt; row < NOUT * P1; row += NQ) {
    const int o = row / P1, iz = row % P1;
    const R* A = s_acc + row * RS + ct * NQP;
    const R* Bx = A + NOUT * P1 * RS;
    const bool hg = Phys::has_grad(0);  // (the same for every output of a policy)
    R oE[H > 0 ? H : 1], oO[H > 0 ? H : 1], oM = 0.0;
#pragma unroll
    for (int i = 0; i < H; ++i) oE[i] = oO[i] = 0.0;
#pragma unroll
    for (int k = 0; k < QH; ++k) {
      const R a1 = A[k], a2 = A[NQ - 1 - k];
      const R As = a1 + a2, Ad = a1 - a2;
      R Bs = R(0), Bd = R(0);
      if (hg) {
        const R b1 = Bx[k], b2 = Bx[NQ - 1 - k];
        Bs = b1 + b2;
        Bd = b1 - b2;
      }
#pragma unroll
      for (int i = 0; i < H; ++i) {
        oE[i] = fmaR(tb.Se[k][i], As, oE[i]);
        oO[i] = fmaR(tb.So[k][i], Ad, oO[i]);
        if (hg) {
          oE[i] = fmaR(tb.De[k][i], Bd, oE[i]);
          oO[i] = fmaR(tb.Do[k][i], Bs, oO[i]);
        }
      }
      if (MIDN) {
        oM = fmaR(tb.Sm[k], As, oM);
        if (hg) oM = fmaR(tb.Dm[k], Bd, oM);
      }
    }
    if constexpr (T::QMID) {  // the middle point: even part of S, odd part of D
      const R am = A[QH], bm = hg ? Bx[QH] : R(0);
#pragma unroll
      for (int i = 0; i < H; ++i) {
        oE[i] = fmaR(tb.Se[QH][i], am, oE[i]);
        if (hg) oO[i] = fmaR(tb.Do[QH][i], bm, oO[i]);
      }
      if (MIDN) oM = fmaR(tb.Sm[QH], am, oM);
    }
    R out[P1];
#pragma unroll
    for (int i = 0; i < H; ++i) {
      out[i] = oE[i] + oO[i];
      out[P - i] = oE[i] - oO[i];
    }
    if (MIDN) out[P / 2] = oM;
    if constexpr (Phys::FACES) {
      out[0] += s_acc[L::O_XF + row * CB + ct];
      out[P] += s_acc[L::O_XF + (NOUT * P1 + row) * CB + ct];
    }
    const int w = s_to[o];
    R* dst = s_out + (w & 0xfffff) + ct * (w >> 20) + iz * P1;
    if constexpr (L::EPI == 1 || L::EPI == 3) {
      // the epilogue's first change-of-basis pass on the row in registers:
      // u[iz][qx] = sum_ix Vi[ix][qx] out[ix], stored in place of the row
      const CobT<P, R>& cbx = cobr<P, R>();
#pragma unroll
      for (int qx = 0; qx < P1; ++qx) {
        R t = R(0);
#pragma unroll
        for (int ix = 0; ix < P1; ++ix) t = fmaR(cbx.Vi[ix][qx], out[ix], t);
        dst[qx] = t;
      }
    } else {
#pragma unroll
      for (int ix = 0; ix < P1; ++ix) dst[ix] = out[ix];
    }
  }
  if constexpr (L::EPI == 0) {
    // ---- store: the shared-memory image of an output equals its global chunk, so one bulk copy
    //      per array writes it when the chunk starts and ends on 16 bytes
    bool bst = !Phys::ACCUMULATE && ((size_t)ncb * ND * sizeof(R)) % 16 == 0 && (CB * ND * sizeof(R)) % 16 == 0;
#pragma unroll
    for (int a = 0; a < Phys::NOUT_ARR; ++a)
      bst = bst && (reinterpret_cast<size_t>(ptr.out[a] + (size_t)c0 * Phys::out_ncomp(a) * ND) & 15) == 0;
    if (bst) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (bst) {
      if (tid == 0) {
        sfor<Phys::NOUT_ARR>([&](auto oc) {
          constexpr int OA = decltype(oc)::value;
          constexpr int NC = Phys::out_ncomp(OA);
          constexpr int ob = [] { int b = 0; for (int a = 0; a < OA; ++a) b += Phys::out_ncomp(a); return b; }();
          asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(
                           ptr.out[OA] + (size_t)c0 * NC * ND),
                       "r"((unsigned)__cvta_generic_to_shared(s_out + ob * CB * ND)), "r"((unsigned)(ncb * NC * ND * sizeof(R)))
                       : "memory");
        });
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
      }
    } else {
      sfor<Phys::NOUT_ARR>([&](auto oc) {
        constexpr int OA = decltype(oc)::value;
        constexpr int NC = Phys::out_ncomp(OA);
        constexpr int ob = [] { int b = 0; for (int a = 0; a < OA; ++a) b += Phys::out_ncomp(a); return b; }();
        R* dst = ptr.out[OA] + (size_t)c0 * NC * ND;
        for (int e = tid; e < ncb * NC * ND; e += NT) {
          const R v = s_out[ob * CB * ND + e];
          if (Phys::ACCUMULATE) dst[e] += v;
          else dst[e] = v;
        }
      });
    }
  } else {
    __syncthreads();
    // ---- cell-local epilogue: the inverse weights (copied since kernel start)
    if (epi_bulk) {
      const bool ok = mbar_wait(bar_e, 0);
      if (!ok) report_status(mesh.status, kStatusStageTimeout);
      if (__syncthreads_or(!ok)) {
        if (tid == 0) mbar_wait(bar_e, 0);
        return;
      }
    } else {
      cp_async_wait_all();
      __syncthreads();
    }
    // EPI 2: region A is free after the x-transpose pass: s_y = the updated residual rows,
    // s_u = the values between the passes
    constexpr int NC = L::EPI == 1 ? NOUT : 1;
    R* s_y = smem;
    R* s_u = smem + CB * ND;
    const CobT<P, R>& cb = cobr<P, R>();
    if constexpr (L::EPI == 2) {
      R* r = prm.r + (size_t)c0 * ND;
      const R* s_r = s_minv + CB * ND;  // prefetched residual
      for (int e = tid; e < ncb * ND; e += NT) {
        const int cc = e / ND, k = e % ND;
        const R rn = s_r[e] + s_out[cc * L::NDP + k];
        r[e] = rn;
        s_y[cc * ND + k] = rn;
      }
      __syncthreads();
    }
    // the half-transformed values u of component o of cell cc: EPI 1 and 3 formed them in the
    // x-transpose pass (in place of the output rows), EPI 2 forms them here from the updated
    // residual
    auto ubase = [&](int o, int cc) -> R* {
      if constexpr (L::EPI == 2) return s_u + (o * CB + cc) * ND;
      else return s_out + (o * CB + cc) * L::NDP;
    };
    if constexpr (L::EPI == 2) {
      // pass 1 (along x): u[iz][qx] = sum_ix Vi[ix][qx] y[iz][ix]; task (cell, row)
      for (int e = tid; e < ncb * P1; e += NT) {
        const int cc = e / P1, iz = e % P1;
        R yr[P1];
#pragma unroll
        for (int ix = 0; ix < P1; ++ix) yr[ix] = s_y[cc * ND + iz * P1 + ix];
#pragma unroll
        for (int qx = 0; qx < P1; ++qx) {
          R t = R(0);
#pragma unroll
          for (int ix = 0; ix < P1; ++ix) t = fmaR(cb.Vi[ix][qx], yr[ix], t);
          s_u[cc * ND + iz * P1 + qx] = t;
        }
      }
      __syncthreads();
    }
    // pass 2 (along z, per column qx): to the Gauss points, times the weights, and back
    for (int e = tid; e < NC * ncb * P1; e += NT) {
      const int o = e / (ncb * P1), cc = (e / P1) % ncb, qx = e % P1;
      R* col = ubase(o, cc) + qx;
      R u[P1], t[P1];
#pragma unroll
      for (int iz = 0; iz < P1; ++iz) u[iz] = col[iz * P1];
#pragma unroll
      for (int qz = 0; qz < P1; ++qz) {
        R a = R(0);
#pragma unroll
        for (int iz = 0; iz < P1; ++iz) a = fmaR(cb.Vi[iz][qz], u[iz], a);
        t[qz] = a * s_minv[cc * ND + qz * P1 + qx];
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
    // pass 3 (along x): x[iz][ix] = sum_qx Vi[ix][qx] v[iz][qx], in place of the row
    for (int e = tid; e < NC * ncb * P1; e += NT) {
      const int o = e / (ncb * P1), cc = (e / P1) % ncb, iz = e % P1;
      R* row = ubase(o, cc) + iz * P1;
      R v[P1];
#pragma unroll
      for (int qx = 0; qx < P1; ++qx) v[qx] = row[qx];
#pragma unroll
      for (int ix = 0; ix < P1; ++ix) {
        R y = R(0);
#pragma unroll
        for (int qx = 0; qx < P1; ++qx) y = fmaR(cb.Vi[ix][qx], v[qx], y);
        row[ix] = y;
      }
    }
    __syncthreads();
    // the store or the update, one element per thread in global order (coalesced)
    for (int e = tid; e < NC * ncb * ND; e += NT) {
      if constexpr (L::EPI == 1) {
        // one output array, NOUT components, [cell][comp][node]: e is the offset from the CTA's first
        const int cc = e / (NOUT * ND), o = (e / ND) % NOUT, k = e % ND;
        ptr.out[0][(size_t)c0 * NOUT * ND + e] = prm.scale * ubase(o, cc)[k];
      } else if constexpr (L::EPI == 3) {  // z, din and x come from the prefetched chunks
        const int cc = e / ND, k = e % ND;
        const size_t g = (size_t)c0 * ND + e;
        const R y = ubase(0, cc)[k];
        const R dl = s_minv[2 * CB * ND + e];
        const R zn = s_minv[CB * ND + e] + prm.g * y - dl;
        const R nd = prm.alpha * dl + prm.s * zn;
        prm.r[g] = zn;
        prm.dout[g] = nd;
        prm.x[g] = prm.first ? nd : s_minv[3 * CB * ND + e] + nd;
      } else {  // din and x come from the prefetched chunks
        const int cc = e / ND, k = e % ND;
        const size_t g = (size_t)c0 * ND + e;
        const R y = ubase(0, cc)[k];
        const R nd = (prm.alpha != R(0) ? prm.alpha * s_minv[2 * CB * ND + e] : R(0)) + prm.s * y;
        prm.dout[g] = nd;
        prm.x[g] = prm.first ? nd : s_minv[3 * CB * ND + e] + nd;
      }
    }
  }
}

// Allows a kernel `bytes` of dynamic shared memory on the current device.  The attribute belongs to the
// function on that device: one bit per device (devices 0..63; beyond that it is set on every launch),
// set by whichever thread gets there first (setting it twice is harmless).
template <class K>
cudaError_t allow_smem(K kernel, size_t bytes, std::atomic<unsigned long long>& configured) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (bit == 0 || (configured.load(std::memory_order_acquire) & bit) == 0) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit, std::memory_order_release);
  }
  return cudaSuccess;
}

template <int P, class Phys, int CB_ = default_cells<P, Phys>(), int MINB = Layout<P, Phys, CB_>::CTAS>
cudaError_t launch_cellop(const MeshDev& mesh,
                          const ArgPtrs<PhysInfo<Phys>::NARR_TOTAL, Phys::NOUT_ARR, RealOf<Phys>>& ptr,
                          const typename Phys::Params& prm, int ncell, cudaStream_t stream) {
  using L = Layout<P, Phys, CB_>;
  static std::atomic<unsigned long long> configured{0};
  const cudaError_t e = allow_smem(k_cellop<P, Phys, CB_, MINB>, L::BYTES, configured);
  if (e != cudaSuccess) return e;
  if (mesh.cell0 < 0) return cudaErrorInvalidValue;
  if (ncell <= mesh.cell0) return cudaSuccess;
  const int nblk = (ncell - mesh.cell0 + L::CB - 1) / L::CB;
  if constexpr (!kPDL) {
    k_cellop<P, Phys, CB_, MINB><<<nblk, L::NT, L::BYTES, stream>>>(mesh, ptr, prm, ncell);
    return cudaGetLastError();
  } else {
    // may overlap the previous kernel of the stream; the kernel waits for it (griddepcontrol)
    // before it touches anything that kernel can write
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nblk);
    cfg.blockDim = dim3((unsigned)L::NT);
    cfg.dynamicSmemBytes = L::BYTES;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_cellop<P, Phys, CB_, MINB>, mesh, ptr, prm, ncell);
  }
}

}  // namespace af
