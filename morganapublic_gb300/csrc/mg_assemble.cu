// Assembly kernels for sm_103a: element matrices of the P1/P2 bilinear forms
// reduced into CSR values, plus the Dirichlet elimination, the adjoint-gradient
// kernel and the load vector.
//
// Every element matrix is computed once, along the plan's Morton element order:
//   P1 (one pass)  k_block_asm: one CTA per block of consecutive elements, their
//                  matrices (two per thread, packed) in shared memory, every
//                  diagonal or upper CSR entry summed there (the plan's block map)
//                  and written to the entry and its mirror; entries whose elements
//                  span blocks get a partial sum per block, added in block order by
//                  k_shared_sum;
//   P2 (two passes) k_elem_mat_pair: two elements per thread, packed, their 55
//                  unique entries to the plan's element-matrix array;
//                  k_slot_gather: one thread per diagonal or upper CSR entry, the
//                  sum of its entries in ascending Morton position (the plan's
//                  slot map).
// No atomics touch values; the per-entry summation order is fixed by the plan,
// so the results are bitwise reproducible.
//
// Element math (reference: src/morganaIntegrator/integratorOEL3d_STD.hpp:106-137,
// src/morganaOperators/opEL3dA.hpp:129-165, opEL3dF.hpp:102-133, opEL3dG.hpp:83-108,
// opEL3dM.hpp:129-158, src/morganaFields/fePr3d.hpp:418-442,643-667 in morganaPublic).
// The tetrahedron map is affine, so J, detJ and J^-1 are the same at every
// quadrature point and the quadrature loop folds into reference tables:
//   stiffness  K_ij = coef det sum_q w_q (J^-T g^_i)(J^-T g^_j)
//                   = (coef / det) sum_{a<=b} (C_a . C_b) T^{ab}_ij ,
//              C_a the columns of the cofactor matrix of J (adj J = C^T),
//              T^{ab} = sum_q w_q g^_ia g^_jb (symmetrised for a != b);
//   P1         the reference gradients are constant, so for i, j >= 1
//              K_ij = coef sum_q w_q / det (C_{i-1} . C_{j-1}), and the row of
//              vertex 0 follows from the zero row sums of a stiffness matrix;
//   mass       K_ij = coef det sum_q w_q phi^_i phi^_j.
// detJ is signed, as in the reference (positive on checked meshes).
//
// Arithmetic modes: kF32 (FP32 values), kDW (FP64-accurate values from
// double-word float arithmetic on the FP32 pipes, written as IEEE doubles), kF64
// (native FP64).  GB300 runs FP64 at ~1/60 of its FP32 rate, so MG_F64 uses kDW;
// MG_F64_NATIVE selects kF64 (the full FP64 exponent range).
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "mg_ff.cuh"
#include "mg_internal.h"
#include "mg_launch.cuh"
#include "mg_pair.cuh"

namespace mg {

enum { kF32 = 0, kDW = 1, kF64 = 2 };

// ---------------------------------------------------------- double-word ops --
__device__ __forceinline__ ff operator+(ff a, ff b) { return ff_add_s(a, b); }
__device__ __forceinline__ ff operator-(ff a, ff b) { return ff_add_s(a, ff_neg(b)); }
__device__ __forceinline__ ff operator-(ff a) { return ff_neg(a); }
__device__ __forceinline__ ff operator*(ff a, ff b) { return ff_mul(a, b); }
__device__ __forceinline__ ff operator/(ff a, ff b) { return ff_div(a, b); }

// An element's scale factor inside the range where the double-word assembly is
// FP64-accurate: zero, or |v| in 2^-96 .. 2^112 (the error terms of products
// stay normal floats and no intermediate overflows).
__device__ __forceinline__ bool dw_scale_ok(float hi)
{
  return hi == 0.0f || (fabsf(hi) >= 0x1p-96f && fabsf(hi) < 0x1p113f);
}
__device__ __forceinline__ bool dw_scale_ok(ff v) { return dw_scale_ok(v.hi); }

template <int MODE> struct Arith;
template <> struct Arith<kF32> {
  using T = float;
  using Out = float;
  // double -> float by integer operations (the conversion instruction runs on
  // the FP64 pipe): hi + lo of the double-word split, rounded once
  __device__ static T from(double x)
  {
    const ff t = ff_from_double_bits(x);
    return __fadd_rn(t.hi, t.lo);
  }
  __device__ static T zero() { return 0.0f; }
};
template <> struct Arith<kDW> {
  using T = ff;
  using Out = double;
  __device__ static T from(double x) { return ff_from_double_bits(x); }
  __device__ static T zero() { return ff{0.0f, 0.0f}; }
};
template <> struct Arith<kF64> {
  using T = double;
  using Out = double;
  __device__ static T from(double x) { return x; }
  __device__ static T zero() { return 0.0; }
};

// ---------------------------------------------------------------- geometry --
template <typename T>
struct Cof {
  T c[3][3];  // cofactor matrix C[r][k] of J; column a of C = det * (J^-T e_a)
  T det;
};

template <typename T>
__device__ __forceinline__ void cofactors(const T J[3][3], Cof<T>& f)
{
  f.c[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  f.c[0][1] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  f.c[0][2] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  f.c[1][0] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
  f.c[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
  f.c[1][2] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
  f.c[2][0] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
  f.c[2][1] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
  f.c[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
  f.det = J[0][0] * f.c[0][0] + J[0][1] * f.c[0][1] + J[0][2] * f.c[0][2];
}

struct GeoPtrs {
  const double4_32a* xyz;  // (x, y, z, 0)
  const float4* rec;       // 2 per node: (hx, hy, hz, mx), (my, mz, lx, ly)
  const float* loz;        // lz
};

template <int MODE> struct Fetch;
template <> struct Fetch<kF64> {
  double4_32a x[4];
};

// components of a three-float record: hi, mid, lo
__device__ __forceinline__ float rec_hi(const float4& a, int r) { return r == 0 ? a.x : (r == 1 ? a.y : a.z); }
__device__ __forceinline__ float rec_mid(const float4& a, const float4& b, int r) { return r == 0 ? a.w : (r == 1 ? b.x : b.y); }
__device__ __forceinline__ float rec_lo(const float4& b, float lz, int r) { return r == 0 ? b.z : (r == 1 ? b.w : lz); }
__device__ __forceinline__ double comp(const double4_32a& v, int r) { return r == 0 ? v.x : (r == 1 ? v.y : v.z); }

__device__ __forceinline__ void geometry(const Fetch<kF64>& F, Cof<double>& f)
{
  double J[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) J[r][k] = comp(F.x[k + 1], r) - comp(F.x[0], r);
  cofactors<double>(J, f);
}

// Near-degenerate elements.  The determinant is a cofactor expansion; when its
// terms cancel (sum_k |J0k C0k| > kCancelTol |det|) the relative error of det,
// and of every entry scaled by 1/det, is that many times the arithmetic's own
// (measured on GB300: double-word 2.3e-12 and FP32 7e-6 against the FP64 oracle
// at a cancellation of ~230).  Such elements recompute J, the cofactors and det
// in FP64 from the exact coordinates -- out of line, so that the rare FP64
// path does not occupy the FP64 pipe of every other element.
constexpr float kCancelTol = 16.0f;

// P1 stiffness needs the gradient of every vertex: the columns C_0..C_3 of the
// cofactor matrix (gradients times det).  C_1..C_3 come from the edge vectors at
// vertex 0.  C_0:
//  - FP32: formed for every element from the face opposite vertex 0,
//    (x3 - x1) x (x2 - x1), accurate to its own magnitude -- cheap in FP32, and
//    the zero-row-sum form C_0 = -(C_1 + C_2 + C_3) would cost eps |C_max| / |C_0|
//    relative on the entries of vertex 0, too much at FP32's eps;
//  - double-word and FP64: the zero-row-sum form (eps 2^-47).
// Elements whose gradients differ by more than 8x (|C_max| > 8 |C_min| over all
// four, or a cancelling determinant) take the rare path abs_rare_stiffness: a
// cofactor is a 2x2 minor whose terms then cancel by about that ratio, and so does
// the zero-row sum; the rare path computes the geometry in FP64 from the exact
// coordinates, as the reference does.  On a Kuhn cube jittered by 0.25 h (12.6 M
// tets, ratios up to 21) ~0.01 % of the elements are rare.
__device__ __forceinline__ bool p1_class(const Cof<double>& f)
{
  float n[4];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float na = 0.0f;
#pragma unroll
    for (int r = 0; r < 3; ++r) na = fmaf((float)f.c[r][a], (float)f.c[r][a], na);
    n[a + 1] = na;
  }
  n[0] = 0.0f;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const float s = (float)f.c[r][0] + (float)f.c[r][1] + (float)f.c[r][2];
    n[0] = fmaf(s, s, n[0]);
  }
  const float nmax = fmaxf(fmaxf(n[0], n[1]), fmaxf(n[2], n[3]));
  const float nmin = fminf(fminf(n[0], n[1]), fminf(n[2], n[3]));
  return nmax > 64.0f * nmin;
}

__device__ __forceinline__ void store_geometry(const Cof<double>& d, Cof<float>& f)
{
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) f.c[r][k] = (float)d.c[r][k];
  f.det = (float)d.det;
}
__device__ __forceinline__ void store_geometry(const Cof<double>& d, Cof<ff>& f)
{
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) f.c[r][k] = ff_from_double_bits(d.c[r][k]);
  f.det = ff_from_double_bits(d.det);
}
__device__ __forceinline__ void store_geometry(const Cof<double>& d, Cof<double>& f) { f = d; }

template <typename T> __device__ __forceinline__ T from_double(double x);
template <> __device__ __forceinline__ float from_double<float>(double x) { return (float)x; }
template <> __device__ __forceinline__ ff from_double<ff>(double x) { return ff_from_double_bits(x); }
template <> __device__ __forceinline__ double from_double<double>(double x) { return x; }

// Double-word difference of two three-float numbers x = hi + mid + lo:
// x_b - x_a = (hi_b - hi_a) + (mid_b - mid_a) + (lo_b - lo_a) with the two
// leading differences error-free -- relative error ~2^-47 of the difference.
__device__ __forceinline__ ff dw_diff3(float hb, float ha, float mb, float ma, float lb, float la)
{
  const ff s1 = two_sum(hb, -ha);
  const ff s2 = two_sum(mb, -ma);
  const ff s = two_sum(s1.hi, s2.hi);
  const float t = __fadd_rn(__fadd_rn(__fadd_rn(s.lo, s1.lo), s2.lo), __fsub_rn(lb, la));
  return two_sum(s.hi, t);
}
// ------------------------------------------------------- element matrices --
// P1 stiffness, unique entries in sym_index order:
// (0,0) (0,1) (0,2) (0,3) (1,1) (1,2) (1,3) (2,2) (2,3) (3,3)
__device__ __forceinline__ void p1_stiff_unique(const Cof<double>& f, double s, double K[10])
{
  double d[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      d[a][b] = s * (f.c[0][a] * f.c[0][b] + f.c[1][a] * f.c[1][b] + f.c[2][a] * f.c[2][b]);
      d[b][a] = d[a][b];
    }
  K[4] = d[0][0];
  K[5] = d[0][1];
  K[6] = d[0][2];
  K[7] = d[1][1];
  K[8] = d[1][2];
  K[9] = d[2][2];
  K[1] = -(d[0][0] + d[1][0] + d[2][0]);  // rows sum to zero
  K[2] = -(d[0][1] + d[1][1] + d[2][1]);
  K[3] = -(d[0][2] + d[1][2] + d[2][2]);
  K[0] = -(K[1] + K[2] + K[3]);
}

// P1 stiffness with every vertex gradient explicit: C_0 given, the entries of
// vertex 0 as s (C_0 . C_j); the others as in p1_stiff_unique.
template <typename T>
__device__ __forceinline__ void p1_stiff_direct(const Cof<T>& f, const T C0[3], T s, T K[10])
{
  T d[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      d[a][b] = s * (f.c[0][a] * f.c[0][b] + f.c[1][a] * f.c[1][b] + f.c[2][a] * f.c[2][b]);
      d[b][a] = d[a][b];
    }
  K[0] = s * (C0[0] * C0[0] + C0[1] * C0[1] + C0[2] * C0[2]);
#pragma unroll
  for (int b = 0; b < 3; ++b) K[1 + b] = s * (C0[0] * f.c[0][b] + C0[1] * f.c[1][b] + C0[2] * f.c[2][b]);
  K[4] = d[0][0];
  K[5] = d[0][1];
  K[6] = d[0][2];
  K[7] = d[1][1];
  K[8] = d[1][2];
  K[9] = d[2][2];
}
template <>
__device__ __forceinline__ void p1_stiff_direct<ff>(const Cof<ff>& f, const ff C0[3], ff s, ff K[10])
{
  ff col[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int r = 0; r < 3; ++r) col[a][r] = f.c[r][a];
  K[0] = ff_mul(s, ff_dot3(C0, C0));
#pragma unroll
  for (int b = 0; b < 3; ++b) K[1 + b] = ff_mul(s, ff_dot3(C0, col[b]));
  K[4] = ff_mul(s, ff_dot3(col[0], col[0]));
  K[5] = ff_mul(s, ff_dot3(col[0], col[1]));
  K[6] = ff_mul(s, ff_dot3(col[0], col[2]));
  K[7] = ff_mul(s, ff_dot3(col[1], col[1]));
  K[8] = ff_mul(s, ff_dot3(col[1], col[2]));
  K[9] = ff_mul(s, ff_dot3(col[2], col[2]));
}

// A P1 element matrix returned by value (the out-of-line rare paths: no register
// of the caller is passed by address, so the common path keeps its registers).
template <typename T>
struct RareK {
  T K[10];
};

// The six scaled metric coefficients s (C_a . C_b), ab = 00,11,22,01,02,12.
template <typename T>
__device__ __forceinline__ void metric(const Cof<T>& f, T s, T g[6])
{
  const int pa[6] = {0, 1, 2, 0, 0, 1}, pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int p = 0; p < 6; ++p)
    g[p] = s * (f.c[0][pa[p]] * f.c[0][pb[p]] + f.c[1][pa[p]] * f.c[1][pb[p]] + f.c[2][pa[p]] * f.c[2][pb[p]]);
}

// sum_{p<6} g[p] tab[p * NU + u] (the P2 metric contraction)
__device__ __forceinline__ double metric_dot(const double g[6], const double* tab, int NU, int u)
{
  double v = g[0] * tab[u];
#pragma unroll
  for (int k = 1; k < 6; ++k) v = v + g[k] * tab[k * NU + u];
  return v;
}

// ------------------------------------------------------------ assembly --
// P1: the one-pass block assembly (k_block_asm, k_shared_sum, below).
// P2, two passes, each element computed once:
//   k_elem_mat_pair  two elements per thread, along the plan's Morton order p: the
//                  unique entries u of its (symmetric) element matrix into the
//                  plan's element-matrix array em;
//   k_slot_gather  one thread per diagonal or upper CSR entry: the sum of the em
//                  entries of every element holding both of its dofs, in
//                  ascending p (the slot map, build_slot_map), written to the
//                  entry and to its mirror -- a fixed order, so the values are
//                  bitwise reproducible, with no atomics.

// Geometry of an element from the mesh's FP64 coordinates.
__device__ __forceinline__ void geometry_f64(const GeoPtrs& g, int4 n, Cof<double>& f)
{
  Fetch<kF64> D;
  D.x[0] = g.xyz[n.x];
  D.x[1] = g.xyz[n.y];
  D.x[2] = g.xyz[n.z];
  D.x[3] = g.xyz[n.w];
  geometry(D, f);
}

// Near-degenerate elements: the FP64 geometry from the mesh's FP64 coordinates,
// out of line and returned by value.
template <typename T>
static __device__ __noinline__ Cof<T> abs_geometry_fp64(const double4_32a* xyz, int4 n)
{
  Fetch<kF64> D;
  D.x[0] = xyz[n.x];
  D.x[1] = xyz[n.y];
  D.x[2] = xyz[n.z];
  D.x[3] = xyz[n.w];
  Cof<double> g;
  geometry(D, g);
  Cof<T> f;
  store_geometry(g, f);
  return f;
}

// The rare P1 stiffness elements (p1_class, or a cancelling determinant): the
// geometry in FP64 from the mesh's FP64 coordinates and C_0 from the face
// opposite vertex 0, returned by value (out of line).
template <int MODE>
static __device__ __noinline__ RareK<typename Arith<MODE>::T> abs_rare_stiffness(const double4_32a* xyz, int4 n,
                                                                                 double coef, double wsum,
                                                                                 uint32_t* flags)
{
  using T = typename Arith<MODE>::T;
  Fetch<kF64> D;
  D.x[0] = xyz[n.x];
  D.x[1] = xyz[n.y];
  D.x[2] = xyz[n.z];
  D.x[3] = xyz[n.w];
  Cof<double> d;
  geometry(D, d);
  double f2[3], f3[3], c0[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    f2[r] = comp(D.x[2], r) - comp(D.x[1], r);
    f3[r] = comp(D.x[3], r) - comp(D.x[1], r);
  }
  c0[0] = f3[1] * f2[2] - f3[2] * f2[1];
  c0[1] = f3[2] * f2[0] - f3[0] * f2[2];
  c0[2] = f3[0] * f2[1] - f3[1] * f2[0];
  Cof<T> f;
  store_geometry(d, f);
  T C0[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) C0[k] = from_double<T>(c0[k]);
  const T s = Arith<MODE>::from(coef) * Arith<MODE>::from(wsum) / f.det;
  RareK<T> r;
  p1_stiff_direct<T>(f, C0, s, r.K);
  if constexpr (MODE == kDW)
    if (!dw_scale_ok(s) || !dw_scale_ok(r.K[4])) atomicOr(flags, 2u);
  return r;
}

__device__ __forceinline__ void em_put(void* em, int64_t i, float v) { static_cast<float*>(em)[i] = v; }
__device__ __forceinline__ void em_put(void* em, int64_t i, ff v)
{
  static_cast<float2*>(em)[i] = make_float2(v.hi, v.lo);
}
__device__ __forceinline__ void em_put(void* em, int64_t i, double v) { static_cast<double*>(em)[i] = v; }
template <typename T> __device__ __forceinline__ T em_get(const void* em, uint32_t i);
template <> __device__ __forceinline__ float em_get<float>(const void* em, uint32_t i)
{
  return __ldg(static_cast<const float*>(em) + i);
}
template <> __device__ __forceinline__ ff em_get<ff>(const void* em, uint32_t i)
{
  const float2 v = __ldg(static_cast<const float2*>(em) + i);
  return ff{v.x, v.y};
}
template <> __device__ __forceinline__ double em_get<double>(const void* em, uint32_t i)
{
  return __ldg(static_cast<const double*>(em) + i);
}

struct ElemArgs {
  int64_t n_elem;
  const int32_t* elem_order;  // Morton position -> element (the caller's numbering)
  const int32_t* dofs_m;      // dofs in Morton order (nb each; the first four are the vertices)
  GeoPtrs geo;
  const double* coeff;        // per element in the caller's order, or null
  double cconst;              // used when coeff is null
  const double* tables;       // unique-entry tables: stiff[6][nu], mass[nu], P2: bary[kBaryTerms]
  double wsum;                // times 2^g, see len_scale
  float w_hi, w_lo;           // wsum as a double-word
  // the element kernels see the mesh times 2^-g (mg_mesh::geo_exp): a stiffness is 2^g of
  // theirs, in wsum (P1) and len_scale (P2), a mass 2^(3g), in two factors
  float len_scale, vol_scale1, vol_scale2;
  float sc_min, sc_max;       // the double-word range of coefficient times determinant
  int stiff;
  void* em;                   // out: nu x n_elem entries
  uint32_t* flags;            // bit 0: NaN / Inf coefficient; bit 1: outside the double-word range
};

// NaN or Inf: recorded for mg_plan_status
__device__ __forceinline__ bool coef_not_finite(double c)
{
  return ((__double_as_longlong(c) >> 52) & 0x7ff) == 0x7ff;
}

// The coefficient and the vertex dofs of Morton element p.
__device__ __forceinline__ double elem_coef(const ElemArgs& a, int64_t p)
{
  return a.coeff ? a.coeff[a.elem_order[p]] : a.cconst;
}
__device__ __forceinline__ int4 elem_nodes(const ElemArgs& a, int64_t p)
{
  return __ldg(reinterpret_cast<const int4*>(a.dofs_m) + p);
}

// The P1 element matrix in native FP64 from the element's vertex dofs n and
// coefficient coef.
__device__ __forceinline__ void p1_element_f64(const ElemArgs& a, const double* mass, int4 n, double coef, double K[10])
{
  Cof<double> f;
  geometry_f64(a.geo, n, f);
  if (coef_not_finite(coef)) atomicOr(a.flags, 1u);
  if (a.stiff) {
    // the rare elements (p1_class) go out of line, entered only when a lane of
    // the warp has one
    const bool rare = p1_class(f);
    if (__any_sync(__activemask(), rare)) {
      if (rare) {
        const RareK<double> rk = abs_rare_stiffness<kF64>(a.geo.xyz, n, coef, a.wsum, a.flags);
#pragma unroll
        for (int u = 0; u < 10; ++u) K[u] = rk.K[u];
      }
    }
    if (!rare) p1_stiff_unique(f, coef * a.wsum / f.det, K);
  } else {
    const double sc = coef * f.det;
#pragma unroll
    for (int u = 0; u < 10; ++u) K[u] = sc * mass[u];
  }
}

// ------------------------------------------------- P1 elements, two per thread --
// The same element math on packed pairs (mg_pair.cuh).  The rare elements are
// found from the finished matrix: gradients that differ by more than 8x show as
// diagonal entries that differ by more than 64x (K_aa = s |C_a|^2); a cancelling
// determinant as before; and determinants outside 2^-100 .. 2^100, where the
// reciprocal estimate would leave the normal floats.

// |det| outside the range of the pair division
__device__ __forceinline__ bool det_extreme(float det)
{
  return !(fabsf(det) >= 0x1p-100f && fabsf(det) <= 0x1p100f);
}
// one lane of |J_00 C_00| + |J_01 C_01| + |J_02 C_02| > kCancelTol |det|
__device__ __forceinline__ bool cancels(float t0, float t1, float t2, float det)
{
  return fabsf(t0) + fabsf(t1) + fabsf(t2) > kCancelTol * fabsf(det);
}
__device__ __forceinline__ bool diag_spread(float k0, float k1, float k2, float k3)
{
  k0 = fabsf(k0), k1 = fabsf(k1), k2 = fabsf(k2), k3 = fabsf(k3);
  // true where all are NaN, of a scale factor above the floats
  return !(fmaxf(fmaxf(k0, k1), fmaxf(k2, k3)) <= 64.0f * fminf(fminf(k0, k1), fminf(k2, k3)));
}

// The node records of a block: its unique nodes staged in shared memory, indexed by
// the element's local vertex numbers, or the mesh's in global memory.
struct StagedNodes {
  const float4 *a, *b;  // (hi.xyz, mid.x), (mid.yz, lo.xy)
  const float* z;       // lo.z
  __device__ __forceinline__ float4 first(int i) const { return a[i]; }
  __device__ __forceinline__ float4 second(int i) const { return b[i]; }
  __device__ __forceinline__ float last(int i) const { return z[i]; }
};
struct GlobalNodes {
  GeoPtrs g;
  __device__ __forceinline__ float4 first(int i) const { return __ldg(g.rec + 2 * (int64_t)i); }
  __device__ __forceinline__ float4 second(int i) const { return __ldg(g.rec + 2 * (int64_t)i + 1); }
  __device__ __forceinline__ float last(int i) const { return __ldg(g.loz + i); }
};

// Edge vectors x_k - x_0 of one element as double-words, component r of edge k at
// 3 r + k.  SPLIT: the node records are split on per-axis grids (mg_mesh::grid_split),
// so the differences of the high and of the middle parts are exact and ordered
// (|d hi| >= |d mid| unless d hi = 0): 7 operations per component against 28.
template <bool SPLIT, typename N>
__device__ __forceinline__ void edges_dw(const N& g, int4 n, float (&hi)[9], float (&lo)[9])
{
  const float4 a0 = g.first(n.x), b0 = g.second(n.x);
  const float z0 = g.last(n.x);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int id = k == 0 ? n.y : (k == 1 ? n.z : n.w);
    const float4 ak = g.first(id), bk = g.second(id);
    const float zk = g.last(id);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      ff d;
      if constexpr (SPLIT) {
        d = fast_two_sum(__fsub_rn(rec_hi(ak, r), rec_hi(a0, r)), __fsub_rn(rec_mid(ak, bk, r), rec_mid(a0, b0, r)));
        d.lo = __fadd_rn(d.lo, __fsub_rn(rec_lo(bk, zk, r), rec_lo(b0, z0, r)));
      } else {
        d = dw_diff3(rec_hi(ak, r), rec_hi(a0, r), rec_mid(ak, bk, r), rec_mid(a0, b0, r), rec_lo(bk, zk, r),
                     rec_lo(b0, z0, r));
      }
      hi[3 * r + k] = d.hi;
      lo[3 * r + k] = d.lo;
    }
  }
}
// ... and as floats: (hi_k - hi_0) + (mid_k - mid_0), to a float ulp of the edge
template <typename N>
__device__ __forceinline__ void edges_f32(const N& g, int4 n, float (&x)[9])
{
  const float4 a0 = g.first(n.x), b0 = g.second(n.x);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int id = k == 0 ? n.y : (k == 1 ? n.z : n.w);
    const float4 ak = g.first(id), bk = g.second(id);
#pragma unroll
    for (int r = 0; r < 3; ++r)
      x[3 * r + k] = (rec_hi(ak, r) - rec_hi(a0, r)) + (rec_mid(ak, bk, r) - rec_mid(a0, b0, r));
  }
}
template <int MODE> struct Pair;
template <> struct Pair<kDW> { using T = ff2; };
template <> struct Pair<kF32> { using T = f2; };
// both elements' edges as packed pairs
template <bool SPLIT, typename N>
__device__ __forceinline__ void pair_edges(const N& g, int4 n0, int4 n1, ff2 (&J)[3][3])
{
  float h0[9], l0[9], h1[9], l1[9];
  edges_dw<SPLIT>(g, n0, h0, l0);
  edges_dw<SPLIT>(g, n1, h1, l1);
#pragma unroll
  for (int i = 0; i < 9; ++i) J[i / 3][i % 3] = ff2{f2_make(h0[i], h1[i]), f2_make(l0[i], l1[i])};
}
template <bool, typename N>
__device__ __forceinline__ void pair_edges(const N& g, int4 n0, int4 n1, f2 (&J)[3][3])
{
  float x0[9], x1[9];
  edges_f32(g, n0, x0);
  edges_f32(g, n1, x1);
#pragma unroll
  for (int i = 0; i < 9; ++i) J[i / 3][i % 3] = f2_make(x0[i], x1[i]);
}

// Two element matrices into the block's shared array: entry u of the block's
// element l at em[u kElemBlock + l], the pair at l = lp and lp + 32 (a warp's lanes
// take consecutive elements: their vertices share cache lines, and the stores are
// conflict-free).  Double-word low parts in a second array.
__device__ __forceinline__ void em_pair(float* em, int u, int lp, f2 v)
{
  const float2 x = f2_get(v);
  em[u * kElemBlock + lp] = x.x;
  em[u * kElemBlock + lp + 32] = x.y;
}

// Cofactor columns C[k][r] = cofactor (r, k) of J and the determinant of a pair; per lane
// whether the determinant cancels.
struct PairGeo {
  ff2 C[3][3];
  ff2 det;
  bool degen0, degen1;
};
__device__ __forceinline__ void pair_cofactors(const ff2 (&J)[3][3], PairGeo& f)
{
  f2 nJ[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) nJ[r][k] = -J[r][k].hi;
#define MG_COF(r, k, r1, k1, r2, k2) \
  f.C[k][r] = ff2_cross(J[r1][k1], J[r2][k2], J[r1][k2], J[r2][k1], nJ[r1][k1], nJ[r1][k2], nJ[r2][k1])
  MG_COF(0, 0, 1, 1, 2, 2);
  MG_COF(0, 1, 1, 2, 2, 0);
  MG_COF(0, 2, 1, 0, 2, 1);
  MG_COF(1, 0, 2, 1, 0, 2);
  MG_COF(1, 1, 2, 2, 0, 0);
  MG_COF(1, 2, 2, 0, 0, 1);
  MG_COF(2, 0, 0, 1, 1, 2);
  MG_COF(2, 1, 0, 2, 1, 0);
  MG_COF(2, 2, 0, 0, 1, 1);
#undef MG_COF
  const ff2 c0[3] = {f.C[0][0], f.C[1][0], f.C[2][0]};
  const ff2 d = ff2_dot3(J[0], c0, nJ[0]);
  f.det = f2_fast_two_sum(d.hi, d.lo);
  const float2 dh = f2_get(f.det.hi), t0 = f2_get(J[0][0].hi * c0[0].hi), t1 = f2_get(J[0][1].hi * c0[1].hi),
               t2 = f2_get(J[0][2].hi * c0[2].hi);
  f.degen0 = cancels(t0.x, t1.x, t2.x, dh.x);
  f.degen1 = cancels(t0.y, t1.y, t2.y, dh.y);
}
// n / det: quotient digits q1 + q2 + q3, the remainder of each by FMAs; |det| in 2^-100 .. 2^100
__device__ __forceinline__ ff2 pair_quotient(f2 nh, f2 nl, ff2 det)
{
  const f2 rb = f2_rcp(det.hi), nd = -det.hi;
  const f2 q1 = nh * rb;
  const f2 r1 = fma2(nd, q1, nh) + fma2(-det.lo, q1, nl);
  const f2 q2 = r1 * rb;
  const f2 q3 = fma2(nd, q2, r1) * rb;
  return f2_fast_two_sum(q1, q2 + q3);
}

// Coefficient times determinant of a pair, from the kernels' scale to the mesh's;
// double-words outside their range are recorded.
__device__ __forceinline__ f2 true_volume(const ElemArgs& a, f2 v)
{
  return v * f2_make(a.vol_scale1, a.vol_scale1) * f2_make(a.vol_scale2, a.vol_scale2);
}
__device__ __forceinline__ ff2 true_volume(const ElemArgs& a, ff2 v)
{
  const float2 h = f2_get(v.hi);
  const auto ok = [&](float x) { return x == 0.0f || (fabsf(x) >= a.sc_min && fabsf(x) < a.sc_max); };
  if (!ok(h.x) || !ok(h.y)) atomicOr(a.flags, 2u);
  return ff2{true_volume(a, v.hi), true_volume(a, v.lo)};
}

// From the pair's edges J and coefficients; node(e): the global vertex ids of
// element e of the pair (for the rare paths).
template <typename Node>
__device__ __forceinline__ void p1_pair_dw(const ElemArgs& a, const ff* mass, const ff2 (&J)[3][3], Node node, double coef0,
                                           double coef1, int lp, float* em_hi, float* em_lo)
{
  PairGeo f;
  pair_cofactors(J, f);
  const ff2 (&C)[3][3] = f.C;
  ff2& det = f.det;
  bool &degen0 = f.degen0, &degen1 = f.degen1;
  if (a.stiff) {
    const float2 dh = f2_get(det.hi);
    degen0 |= det_extreme(dh.x);
    degen1 |= det_extreme(dh.y);
  }
  if (coef_not_finite(coef0) || coef_not_finite(coef1)) atomicOr(a.flags, 1u);
  const ff2 coef = ff2_make(ff_from_double_bits(coef0), ff_from_double_bits(coef1));
  if (a.stiff) {
    // s = coef w / det
    const f2 wh = f2_make(a.w_hi, a.w_hi), wl = f2_make(a.w_lo, a.w_lo);
    const f2 nh = coef.hi * wh;
    const f2 nl = fma2(coef.lo, wh, coef.hi * wl) - fma2(-coef.hi, wh, nh);
    const ff2 s = pair_quotient(nh, nl, det);
    ff2 K[10];
    {
      const f2 ns = -s.hi;
      f2 nC[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int r = 0; r < 3; ++r) nC[k][r] = -C[k][r].hi;
      const int ui[6] = {4, 5, 6, 7, 8, 9}, ua[6] = {0, 0, 0, 1, 1, 2}, ub[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
      for (int t = 0; t < 6; ++t) {
        ff2 d = ff2_dot3(C[ua[t]], C[ub[t]], nC[ua[t]]);
        d = f2_fast_two_sum(d.hi, d.lo);
        const f2 p = s.hi * d.hi;
        const f2 lo = fma2(s.hi, d.lo, s.lo * d.hi) - fma2(ns, d.hi, p);
        K[ui[t]] = f2_fast_two_sum(p, lo);
      }
      // vertex 0 from the zero row sums, the sums of the high parts error-free
      const ff2* R[3][3] = {{&K[4], &K[5], &K[6]}, {&K[5], &K[7], &K[8]}, {&K[6], &K[8], &K[9]}};
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const ff2 x = f2_two_sum(R[t][0]->hi, R[t][1]->hi), y = f2_two_sum(x.hi, R[t][2]->hi);
        K[1 + t] = f2_fast_two_sum(y.hi, (R[t][0]->lo + R[t][1]->lo) + (R[t][2]->lo + (x.lo + y.lo)));
      }
      const ff2 x = f2_two_sum(K[1].hi, K[2].hi), y = f2_two_sum(x.hi, K[3].hi);
      K[0] = f2_fast_two_sum(y.hi, (K[1].lo + K[2].lo) + (K[3].lo + (x.lo + y.lo)));
    }
#pragma unroll
    for (int u = 0; u < 10; ++u) {
      const bool neg = u >= 1 && u <= 3;
      em_pair(em_hi, u, lp, neg ? -K[u].hi : K[u].hi);
      em_pair(em_lo, u, lp, neg ? -K[u].lo : K[u].lo);
    }
    const float2 k0 = f2_get(K[0].hi), k1 = f2_get(K[4].hi), k2 = f2_get(K[7].hi), k3 = f2_get(K[9].hi),
                 sh = f2_get(s.hi);
    const bool rare0 = degen0 || diag_spread(k0.x, k1.x, k2.x, k3.x);
    const bool rare1 = degen1 || diag_spread(k0.y, k1.y, k2.y, k3.y);
    if ((!rare0 && !(dw_scale_ok(sh.x) && dw_scale_ok(k1.x))) || (!rare1 && !(dw_scale_ok(sh.y) && dw_scale_ok(k1.y))))
      atomicOr(a.flags, 2u);
    // the rare elements (~0.01 %) again, out of line in FP64 geometry
    if (rare0 || rare1) {
#pragma unroll 1
      for (int e = rare0 ? 0 : 1; e < (rare1 ? 2 : 1); ++e) {
        const RareK<ff> rk = abs_rare_stiffness<kDW>(a.geo.xyz, node(e), e ? coef1 : coef0, a.wsum, a.flags);
#pragma unroll
        for (int u = 0; u < 10; ++u) {
          em_hi[u * kElemBlock + lp + 32 * e] = rk.K[u].hi;
          em_lo[u * kElemBlock + lp + 32 * e] = rk.K[u].lo;
        }
      }
    }
  } else {
    if (degen0 || degen1) {
      const ff x = degen0 ? abs_geometry_fp64<ff>(a.geo.xyz, node(0)).det
                          : ff{f2_get(det.hi).x, f2_get(det.lo).x};
      const ff y = degen1 ? abs_geometry_fp64<ff>(a.geo.xyz, node(1)).det
                          : ff{f2_get(det.hi).y, f2_get(det.lo).y};
      det = ff2_make(x, y);
    }
    const f2 nc = -coef.hi, p = coef.hi * det.hi;
    const f2 lo = fma2(coef.hi, det.lo, coef.lo * det.hi);
    const ff2 sc = true_volume(a, f2_fast_two_sum(p, lo - fma2(nc, det.hi, p)));
    const f2 ns = -sc.hi;
#pragma unroll
    for (int u = 0; u < 10; ++u) {
      const f2 th = f2_make(mass[u].hi, mass[u].hi), tl = f2_make(mass[u].lo, mass[u].lo);
      const f2 q = sc.hi * th;
      const ff2 k = f2_fast_two_sum(q, fma2(sc.hi, tl, sc.lo * th) - fma2(ns, th, q));
      em_pair(em_hi, u, lp, k.hi);
      em_pair(em_lo, u, lp, k.lo);
    }
  }
}

// FP32: C[0] from the face opposite vertex 0, (x3 - x1) x (x2 - x1), then the cofactor
// columns of J; the determinant; per lane whether it cancels.
__device__ __forceinline__ void pair_gradients(const f2 (&J)[3][3], f2 (&C)[4][3], f2& det, bool& degen0, bool& degen1)
{
  f2 nJ[3][3];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) nJ[r][k] = -J[r][k];
#define MG_COF(r, k, r1, k1, r2, k2) C[k + 1][r] = f2_cross(J[r1][k1], J[r2][k2], J[r1][k2], J[r2][k1], nJ[r1][k2])
  MG_COF(0, 0, 1, 1, 2, 2);
  MG_COF(0, 1, 1, 2, 2, 0);
  MG_COF(0, 2, 1, 0, 2, 1);
  MG_COF(1, 0, 2, 1, 0, 2);
  MG_COF(1, 1, 2, 2, 0, 0);
  MG_COF(1, 2, 2, 0, 0, 1);
  MG_COF(2, 0, 0, 1, 1, 2);
  MG_COF(2, 1, 0, 2, 1, 0);
  MG_COF(2, 2, 0, 0, 1, 1);
#undef MG_COF
  f2 e2[3], e3[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    e2[r] = J[r][1] - J[r][0];
    e3[r] = J[r][2] - J[r][0];
  }
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    const int r1 = (r + 1) % 3, r2 = (r + 2) % 3;
    C[0][r] = f2_cross(e3[r1], e2[r2], e3[r2], e2[r1], -e3[r2]);
  }
  det = fma2(J[0][2], C[3][0], fma2(J[0][1], C[2][0], J[0][0] * C[1][0]));
  const float2 dh = f2_get(det), t0 = f2_get(J[0][0] * C[1][0]), t1 = f2_get(J[0][1] * C[2][0]),
               t2 = f2_get(J[0][2] * C[3][0]);
  degen0 = cancels(t0.x, t1.x, t2.x, dh.x);
  degen1 = cancels(t0.y, t1.y, t2.y, dh.y);
}

template <typename Node>
__device__ __forceinline__ void p1_pair_f32(const ElemArgs& a, const float* mass, const f2 (&J)[3][3], Node node,
                                            double coef0, double coef1, int lp, float* em)
{
  f2 C[4][3];
  f2 det;
  bool degen0, degen1;
  pair_gradients(J, C, det, degen0, degen1);
  if (a.stiff) {
    const float2 dh = f2_get(det);
    degen0 |= det_extreme(dh.x);
    degen1 |= det_extreme(dh.y);
  }
  if (coef_not_finite(coef0) || coef_not_finite(coef1)) atomicOr(a.flags, 1u);
  const f2 coef = f2_make(Arith<kF32>::from(coef0), Arith<kF32>::from(coef1));
  if (a.stiff) {
    // s = coef w / det, one correction of the quotient estimate
    const f2 nu = coef * f2_make(a.w_hi, a.w_hi), rb = f2_rcp(det), q = nu * rb;
    const f2 s = fma2(fma2(-det, q, nu), rb, q);
    f2 diag[4];
    int u = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = i; j < 4; ++j, ++u) {
        const f2 k = s * fma2(C[i][2], C[j][2], fma2(C[i][1], C[j][1], C[i][0] * C[j][0]));
        if (j == i) diag[i] = k;
        em_pair(em, u, lp, k);
      }
    const float2 k0 = f2_get(diag[0]), k1 = f2_get(diag[1]), k2 = f2_get(diag[2]), k3 = f2_get(diag[3]);
    const bool rare0 = degen0 || diag_spread(k0.x, k1.x, k2.x, k3.x);
    const bool rare1 = degen1 || diag_spread(k0.y, k1.y, k2.y, k3.y);
    if (rare0 || rare1) {
#pragma unroll 1
      for (int e = rare0 ? 0 : 1; e < (rare1 ? 2 : 1); ++e) {
        const RareK<float> rk = abs_rare_stiffness<kF32>(a.geo.xyz, node(e), e ? coef1 : coef0, a.wsum, a.flags);
#pragma unroll
        for (int v = 0; v < 10; ++v) em[v * kElemBlock + lp + 32 * e] = rk.K[v];
      }
    }
  } else {
    if (degen0 || degen1) {
      const float2 d = f2_get(det);
      det = f2_make(degen0 ? abs_geometry_fp64<float>(a.geo.xyz, node(0)).det : d.x,
                    degen1 ? abs_geometry_fp64<float>(a.geo.xyz, node(1)).det : d.y);
    }
    const f2 sc = true_volume(a, coef * det);
#pragma unroll
    for (int u = 0; u < 10; ++u) em_pair(em, u, lp, sc * f2_make(mass[u], mass[u]));
  }
}

// ------------------------------------------------- P2 elements, two per thread --
// The stiffness in barycentric form: with G_ab = s C_a . C_b (C_0 = -(C_1 + C_2 + C_3),
// C_a / det the gradient of lambda_a) and the P2 gradients (4 lambda_i - 1) grad
// lambda_i and 4 (lambda_a grad lambda_b + lambda_b grad lambda_a), entry
//   (vertex i, vertex j)              one term   G_ij
//   (vertex i, edge (a, b))           two terms  G_ib, G_ia
//   (edge (a, b), edge (c, d))        four terms G_bd, G_bc, G_ad, G_ac
//   (edge (a, b) with itself)         three      G_bb, G_ab, G_aa
// with coefficients summed over the card (RefTables::bary, in this order): 136 products
// per element, where the contraction of the six metric coefficients C_a . C_b with
// tables T^{ab} takes 330.
constexpr int kBaryTerms = 10 + 24 * 2 + 15 * 4 + 6 * 3;
// vertex s of local edge e: (0,1) (1,2) (2,0) (0,3) (1,3) (2,3)
__host__ __device__ constexpr int p2_edge(int e, int s) { return (int)((0x323130022110ull >> (8 * e + 4 * s)) & 0xf); }
// place of G_ab among the ten
__host__ __device__ constexpr int g_index(int a, int b)
{
  return a <= b ? a * 4 - a * (a - 1) / 2 + (b - a) : b * 4 - b * (b - 1) / 2 + (a - b);
}

// sum_k g[i_k] t[k], N terms (i0 .. i3 the indices): packed; double-word: error-free
// products of the high words chained with two_sum, the low-order terms in one float,
// one renormalisation; table entries as (hi, hi, lo, lo)
template <int N>
__device__ __forceinline__ ff2 bary_sum(const ff2 (&g)[10], const f2 (&ng)[10], const float4* t, int i0, int i1, int i2, int i3)
{
  const int id[4] = {i0, i1, i2, i3};
  f2 hi, lo;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const float4 tk = t[k];
    const f2 th = f2_make(tk.x, tk.y), tl = f2_make(tk.z, tk.w);
    const ff2 gk = g[id[k]];
    const f2 q = gk.hi * th, qe = fma2(ng[id[k]], th, q);
    if (k == 0) {
      hi = q;
      lo = fma2(gk.hi, tl, gk.lo * th) - qe;
    } else {
      const ff2 s = f2_two_sum(hi, q);
      hi = s.hi;
      lo = lo + fma2(gk.hi, tl, fma2(gk.lo, th, s.lo - qe));
    }
  }
  return f2_fast_two_sum(hi, lo);
}
template <int N>
__device__ __forceinline__ f2 bary_sum(const f2 (&g)[10], const f2 (&)[10], const float2* t, int i0, int i1, int i2, int i3)
{
  const int id[4] = {i0, i1, i2, i3};
  f2 v = g[i0] * f2_make(t[0].x, t[0].y);
#pragma unroll
  for (int k = 1; k < N; ++k) v = fma2(g[id[k]], f2_make(t[k].x, t[k].y), v);
  return v;
}
// entry u of elements p0 and p1 into the element-matrix array
__device__ __forceinline__ void em_pair_put(void* em, int64_t E, int u, int64_t p0, int64_t p1, ff2 v)
{
  const float2 h = f2_get(v.hi), l = f2_get(v.lo);
  em_put(em, u * E + p0, ff{h.x, l.x});
  em_put(em, u * E + p1, ff{h.y, l.y});
}
__device__ __forceinline__ void em_pair_put(void* em, int64_t E, int u, int64_t p0, int64_t p1, f2 v)
{
  const float2 x = f2_get(v);
  em_put(em, u * E + p0, x.x);
  em_put(em, u * E + p1, x.y);
}
template <typename T2, typename Tab>
__device__ __forceinline__ void p2_stiffness(const T2 (&g)[10], const f2 (&ng)[10], const Tab* t, void* em, int64_t E,
                                             int64_t p0, int64_t p1)
{
  int u = 0;
#pragma unroll
  for (int i = 0; i < 10; ++i)
#pragma unroll
    for (int j = i; j < 10; ++j, ++u) {
      T2 v;
      if (j < 4) {
        v = bary_sum<1>(g, ng, t, g_index(i, j), 0, 0, 0);
        t += 1;
      } else if (i < 4) {
        const int a = p2_edge(j - 4, 0), b = p2_edge(j - 4, 1);
        v = bary_sum<2>(g, ng, t, g_index(i, b), g_index(i, a), 0, 0);
        t += 2;
      } else if (i != j) {
        const int a = p2_edge(i - 4, 0), b = p2_edge(i - 4, 1), c = p2_edge(j - 4, 0), d = p2_edge(j - 4, 1);
        v = bary_sum<4>(g, ng, t, g_index(b, d), g_index(b, c), g_index(a, d), g_index(a, c));
        t += 4;
      } else {
        const int a = p2_edge(i - 4, 0), b = p2_edge(i - 4, 1);
        v = bary_sum<3>(g, ng, t, g_index(b, b), g_index(a, b), g_index(a, a), 0);
        t += 3;
      }
      em_pair_put(em, E, u, p0, p1, v);
    }
}

__device__ __forceinline__ ff2 ff2_mul(ff2 a, ff2 b)
{
  const f2 p = a.hi * b.hi;
  const f2 lo = fma2(a.hi, b.lo, a.lo * b.hi) - fma2(-a.hi, b.hi, p);
  return f2_fast_two_sum(p, lo);
}
// -(a + b + c), the high parts summed error-free
__device__ __forceinline__ ff2 ff2_neg_sum(ff2 a, ff2 b, ff2 c)
{
  const ff2 x = f2_two_sum(a.hi, b.hi), y = f2_two_sum(x.hi, c.hi);
  return -f2_fast_two_sum(y.hi, (a.lo + b.lo) + (c.lo + (x.lo + y.lo)));
}

// The element pass of the two-pass P2 assembly: two elements per thread (Morton
// positions 32 apart: a warp covers 64) as packed pairs, the 55 entries of each to
// em[u * E + p] (entry-major: the stores of one u coalesce across the warp).
// Bound by the element-matrix stores and instruction issue; GB300, P2 48^3, FP64: scalar
// double-words with the six-coefficient contraction 125 us, this form 69 us.
template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(128, 4) k_elem_mat_pair(ElemArgs a)
{
  using A = Arith<MODE>;
  using Tab = typename std::conditional<MODE == kDW, float4, float2>::type;
  constexpr int NU = 55;
  __shared__ Tab tab[kBaryTerms > NU ? kBaryTerms : NU];
  {
    const double* t = a.stiff ? a.tables + 7 * NU : a.tables + 6 * NU;
    for (int i = threadIdx.x; i < (a.stiff ? kBaryTerms : NU); i += blockDim.x) {
      if constexpr (MODE == kDW) {
        const ff v = ff_from_double_bits(t[i]);
        tab[i] = make_float4(v.hi, v.hi, v.lo, v.lo);
      } else {
        const float v = A::from(t[i]);
        tab[i] = make_float2(v, v);
      }
    }
  }
  __syncthreads();
  const int64_t E = a.n_elem;
  const int lane = threadIdx.x & 31;
  const int64_t first = (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 64;
  if (first >= E) return;
  // past the last element the pair repeats it (the same values stored again)
  const int64_t p0 = min(first + lane, E - 1), p1 = min(first + 32 + lane, E - 1);
  const double c0 = a.coeff ? a.coeff[a.elem_order[p0]] : a.cconst;
  const double c1 = a.coeff ? a.coeff[a.elem_order[p1]] : a.cconst;
  const auto vertices = [&](int64_t p) {
    const int2* d = reinterpret_cast<const int2*>(a.dofs_m + p * 10);
    const int2 x = __ldg(d), y = __ldg(d + 1);
    return make_int4(x.x, x.y, y.x, y.y);
  };
  const int4 n0 = vertices(p0), n1 = vertices(p1);
  typename Pair<MODE>::T J[3][3];
  pair_edges<SPLIT>(GlobalNodes{a.geo}, n0, n1, J);
  if (coef_not_finite(c0) || coef_not_finite(c1)) atomicOr(a.flags, 1u);
  if constexpr (MODE == kDW) {
    PairGeo f;
    pair_cofactors(J, f);
    if (f.degen0 || f.degen1) {  // rare: the FP64 geometry of that lane
      const Cof<ff> x = abs_geometry_fp64<ff>(a.geo.xyz, f.degen0 ? n0 : n1), y = abs_geometry_fp64<ff>(a.geo.xyz, f.degen1 ? n1 : n0);
      const auto pick = [&](ff2 v, ff vx, ff vy) {
        const float2 h = f2_get(v.hi), l = f2_get(v.lo);
        return ff2_make(f.degen0 ? vx : ff{h.x, l.x}, f.degen1 ? vy : ff{h.y, l.y});
      };
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int r = 0; r < 3; ++r) f.C[k][r] = pick(f.C[k][r], x.c[r][k], y.c[r][k]);
      f.det = pick(f.det, x.det, y.det);
    }
    const ff2 coef = ff2_make(ff_from_double_bits(c0), ff_from_double_bits(c1));
    if (a.stiff) {
      ff2 s = pair_quotient(coef.hi, coef.lo, f.det);
      const float2 dh = f2_get(f.det.hi);
      if (det_extreme(dh.x) || det_extreme(dh.y)) {  // outside the estimate's range
        const float2 dl = f2_get(f.det.lo), ch = f2_get(coef.hi), cl = f2_get(coef.lo);
        s = ff2_make(ff_div(ff{ch.x, cl.x}, ff{dh.x, dl.x}), ff_div(ff{ch.y, cl.y}, ff{dh.y, dl.y}));
      }
      const f2 ls = f2_make(a.len_scale, a.len_scale);
      s = ff2{s.hi * ls, s.lo * ls};
      ff2 g[10];
      f2 nC[3][3];
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int r = 0; r < 3; ++r) nC[k][r] = -f.C[k][r].hi;
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = k; l < 3; ++l) {
          const ff2 d = ff2_dot3(f.C[k], f.C[l], nC[k]);
          g[g_index(k + 1, l + 1)] = ff2_mul(s, f2_fast_two_sum(d.hi, d.lo));
        }
      // G_0b from the zero sum of the gradients
#pragma unroll
      for (int b = 1; b < 4; ++b) g[g_index(0, b)] = ff2_neg_sum(g[g_index(1, b)], g[g_index(2, b)], g[g_index(3, b)]);
      g[0] = ff2_neg_sum(g[1], g[2], g[3]);
      const float2 sh = f2_get(s.hi), gh = f2_get(g[g_index(1, 1)].hi);
      if (!dw_scale_ok(sh.x) || !dw_scale_ok(gh.x) || !dw_scale_ok(sh.y) || !dw_scale_ok(gh.y)) atomicOr(a.flags, 2u);
      f2 ng[10];
#pragma unroll
      for (int i = 0; i < 10; ++i) ng[i] = -g[i].hi;
      p2_stiffness(g, ng, tab, a.em, E, p0, p1);
    } else {
      const ff2 sc = true_volume(a, ff2_mul(coef, f.det));
      const f2 ns = -sc.hi;
#pragma unroll 5
      for (int u = 0; u < NU; ++u) {
        const float4 t = tab[u];
        const f2 th = f2_make(t.x, t.y), tl = f2_make(t.z, t.w), q = sc.hi * th;
        em_pair_put(a.em, E, u, p0, p1, f2_fast_two_sum(q, fma2(sc.hi, tl, sc.lo * th) - fma2(ns, th, q)));
      }
    }
  } else {
    f2 C[4][3];  // C_0 from the face opposite vertex 0, then the cofactor columns
    f2 det;
    bool degen0, degen1;
    pair_gradients(J, C, det, degen0, degen1);
    if (degen0 || degen1) {
      const Cof<float> x = abs_geometry_fp64<float>(a.geo.xyz, degen0 ? n0 : n1), y = abs_geometry_fp64<float>(a.geo.xyz, degen1 ? n1 : n0);
      const auto pick = [&](f2 v, float vx, float vy) {
        const float2 h = f2_get(v);
        return f2_make(degen0 ? vx : h.x, degen1 ? vy : h.y);
      };
#pragma unroll
      for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int r = 0; r < 3; ++r) C[k + 1][r] = pick(C[k + 1][r], x.c[r][k], y.c[r][k]);
      det = pick(det, x.det, y.det);
    }
    const f2 coef = f2_make(A::from(c0), A::from(c1));
    if (a.stiff) {
      const float2 dh = f2_get(det), ch = f2_get(coef);
      const f2 s = f2_make(ch.x / dh.x, ch.y / dh.y) * f2_make(a.len_scale, a.len_scale);
      f2 g[10];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int l = k; l < 4; ++l)
          g[g_index(k, l)] = s * fma2(C[k][2], C[l][2], fma2(C[k][1], C[l][1], C[k][0] * C[l][0]));
      p2_stiffness(g, g, tab, a.em, E, p0, p1);
    } else {
      const f2 sc = true_volume(a, coef * det);
#pragma unroll 5
      for (int u = 0; u < NU; ++u) em_pair_put(a.em, E, u, p0, p1, sc * f2_make(tab[u].x, tab[u].y));
    }
  }
}

// The P2 element pass in native FP64: one thread per element, the six metric
// coefficients contracted with the tables T^{ab} in shared memory.
__global__ void __launch_bounds__(256, 1) k_elem_mat_f64(ElemArgs a)
{
  constexpr int NU = 55;
  __shared__ double tab[7 * NU];
  for (int i = threadIdx.x; i < 7 * NU; i += blockDim.x) tab[i] = a.tables[i];
  __syncthreads();
  const int64_t E = a.n_elem;
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= E) return;
  const double coef = a.coeff ? a.coeff[a.elem_order[p]] : a.cconst;
  const int32_t* dp = a.dofs_m + p * 10;
  Cof<double> f;
  geometry_f64(a.geo, make_int4(dp[0], dp[1], dp[2], dp[3]), f);
  if (coef_not_finite(coef)) atomicOr(a.flags, 1u);
  if (a.stiff) {
    double g[6];
    metric<double>(f, coef / f.det, g);
#pragma unroll 5
    for (int u = 0; u < NU; ++u) em_put(a.em, u * E + p, metric_dot(g, tab, NU, u));
  } else {
    const double sc = coef * f.det;
#pragma unroll 5
    for (int u = 0; u < NU; ++u) em_put(a.em, u * E + p, sc * tab[6 * NU + u]);
  }
}

// The sum of an entry's sources, two at a time: double-words in two packed accumulators
// (the high parts error-free, the low parts and errors collected) and written as
// one FP64 sum of the two parts; floats packed; FP64 in order.
template <int MODE> struct SourceSum;
template <> struct SourceSum<kDW> {
  ff2 s{f2_make(0.0f, 0.0f), f2_make(0.0f, 0.0f)};
  __device__ __forceinline__ void add(ff a, ff b)
  {
    const ff2 t = f2_two_sum(s.hi, f2_make(a.hi, b.hi));
    s.hi = t.hi;
    s.lo = s.lo + (t.lo + f2_make(a.lo, b.lo));
  }
  __device__ __forceinline__ double result() const
  {
    const float2 h = f2_get(s.hi), l = f2_get(s.lo);
    const ff t = two_sum(h.x, h.y);
    return (double)t.hi + (double)__fadd_rn(t.lo, __fadd_rn(l.x, l.y));
  }
};
template <> struct SourceSum<kF32> {
  f2 s = f2_make(0.0f, 0.0f);
  __device__ __forceinline__ void add(float a, float b) { s = s + f2_make(a, b); }
  __device__ __forceinline__ float result() const
  {
    const float2 h = f2_get(s);
    return h.x + h.y;
  }
};
template <> struct SourceSum<kF64> {
  double s = 0.0;
  __device__ __forceinline__ void add(double a, double b) { s = (s + a) + b; }
  __device__ __forceinline__ double result() const { return s; }
};

// One warp per group of 32 diagonal or upper CSR entries (the slot map's
// layout): lane l sums the sources src[o + 32 j + l] of its entry, j < L, in the
// slot map's order, K at a time, and writes the sum to the entry and to its
// mirror (the operators are symmetric).  Software-pipelined: the indices of the
// next K sources (one coalesced line per j) and the output positions load while
// the current element-matrix values are in flight.  Padding sources
// (kPadSource) read the zero entry `zero` past the element matrices.
// Bound by L2: every source is a sector of its own (59 M sectors read at P2 48^3, 7.4
// TB/s); element-major element matrices and a grid pipelined over groups measured no
// better (256 and 448 us against 248).
template <int MODE, int K>
__global__ void __launch_bounds__(256) k_slot_gather(int64_t n_groups, int64_t n_upper, const int32_t* __restrict__ goff,
                                                     const int32_t* __restrict__ uslot,
                                                     const int32_t* __restrict__ umirror,
                                                     const uint32_t* __restrict__ src, const void* __restrict__ em,
                                                     uint32_t zero, typename Arith<MODE>::Out* __restrict__ values)
{
  using A = Arith<MODE>;
  using T = typename A::T;
  const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (g >= n_groups) return;
  const int lane = threadIdx.x & 31;
  const int64_t t = 32 * g + lane;
  const bool live = t < n_upper;
  const int32_t out_a = live ? __ldg(uslot + t) : 0, out_m = live ? __ldg(umirror + t) : 0;
  const int32_t o = goff[g], L = (goff[g + 1] - o) >> 5;
  const uint32_t* s = src + o + lane;
  uint32_t nxt[K];
#pragma unroll
  for (int i = 0; i < K; ++i) nxt[i] = i < L ? __ldg(s + 32 * i) : kPadSource;
  SourceSum<MODE> sum;
  for (int32_t j = 0; j < L; j += K) {
    uint32_t idx[K];
#pragma unroll
    for (int i = 0; i < K; ++i) idx[i] = min(nxt[i], zero);
#pragma unroll
    for (int i = 0; i < K; ++i) nxt[i] = j + K + i < L ? __ldg(s + 32 * (j + K + i)) : kPadSource;
    T x[K];
#pragma unroll
    for (int i = 0; i < K; ++i) x[i] = j + i < L ? em_get<T>(em, idx[i]) : A::zero();
#pragma unroll
    for (int i = 0; i < K; i += 2) sum.add(x[i], x[i + 1]);
  }
  if (live) {
    const typename A::Out r = sum.result();
    values[out_a] = r;
    if (out_m != out_a) values[out_m] = r;
  }
}

// ---------------------------------------------------- one-pass assembly (P1) --
// k_block_asm: one CTA per block of kElemBlock consecutive Morton positions.
//   1. the records of the block's unique nodes, its coefficients and its part of
//      the block map come into shared memory by cp.async; each thread computes the
//      matrices of two elements as packed pairs into shared memory (10 unique
//      entries each);
//   2. each warp takes groups of 32 of the block's local entries (the block map):
//      lane l sums its entry's local sources, and writes the sum to the CSR entry and
//      its mirror when every source of the entry lies in this block, else to the
//      entry's partial-sum slot.
// k_shared_sum: one warp per group of 32 shared entries: the partial sums in
//   ascending block (coalesced [j][lane]), written to the entry and its mirror.
// Each entry's summation order is fixed by the plan, so the values are bitwise
// reproducible; no atomics, no element matrix leaves the SM.  Both kernels are
// launched with programmatic dependent launch: what they read of the plan overlaps
// the tail of the kernel before.
//
// What bounds it on GB300 (P1 128^3, FP64, one assembly 949 -> 711 us; FP32 at 64^3
// 74 -> 56 us, both with k_shared_sum).  One element per thread and scalar
// double-words took 46 warp instructions per element at 57 % issue.  The packed
// pairs with grid-split coordinates take 30, and left latency as the bound:
//   - random vertex and coefficient loads need an L1 line each while in flight,
//     and the blocks' shared memory leaves few lines: nodes staged by cp.async 833 ->
//     743 us, coefficients by cp.async 782 -> 745 us;
//   - occupancy: three CTAs of 256 threads at 80 registers 789 us, two at 128
//     registers 889 us, four at 64 registers (spills) 880 us;
//   - the map rows' outputs staged beside the sources, uniform loop bounds in the
//     sums: 750 -> 727 us.
// About half of the issue slots are used; the rest is the latency of the block's phases,
// the scattered 8-byte writes of the sums (~30 us) and k_shared_sum (~130 us).
struct BlockArgs {
  const int32_t* bgrp;
  const int32_t* bsrc0;
  const int32_t* bgoff;
  const uint16_t* bsrc;
  const int2* bout;
  void* partial;  // 8-byte slots: a double, or a float in the low half
  const int32_t* bnode;        // kStageNodes per block: its unique nodes, the last repeated
  const int32_t* bnode_n;      // their number, or -1 (more than kStageNodes)
  const uchar4* elem_local;    // per Morton position, the vertices' places among them
};

// Block-map staging in shared memory: the block's local sources (kStageSrc) and its
// groups' outputs and offsets (kStageGroups), copied with cp.async while the element
// matrices are computed.  A block of 512 elements of a volume mesh has about 5,500
// sources in 33 groups; one with more than the stage holds copies the first of them
// and reads its map from global memory.
constexpr int kStageSrc = 6144;
constexpr int kStageGroups = 40;
// The block's element matrices in shared memory: entry u of local element l at
// u kElemBlock + l -- consecutive elements in consecutive words, so a warp's stores
// are conflict-free -- then the zero of the padding sources.  Double-words keep
// their low parts in a second array of kEmStride floats.
constexpr int kEmStride = 10 * kElemBlock + 4;
template <int MODE>
constexpr size_t kEmBytes = (MODE == kF32 ? sizeof(float) : sizeof(double)) * kEmStride;
// dynamic shared memory of a block: its element matrices, the staged sources, node
// records and ids, and group offsets
constexpr size_t kNodeStageBytes = kStageNodes * (2 * sizeof(float4) + sizeof(float) + sizeof(int32_t));
template <int MODE>
__host__ __device__ constexpr size_t block_smem_bytes()
{
  return kEmBytes<MODE> + 2 * kStageSrc + 256 * kStageGroups + (MODE == kF64 ? 0 : kNodeStageBytes) +
         4 * (kStageGroups + 1);
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem));
}
// The double c[e] of an array of n, copied asynchronously into the 16-byte slot
// `smem` as the aligned 16 bytes that hold it (read back with coef_slot).  The bypassing copy
// takes no L1 line: random 8-byte loads would each hold one while in flight, and the
// blocks' shared memory leaves few.  Where those 16 bytes reach past the array
// (an end of an array that is odd in length or off the 16-byte grid) the value is stored.
__device__ __forceinline__ void coef_fetch(double* smem, const double* c, int64_t e, int64_t n)
{
  const int odd = (int)((reinterpret_cast<uintptr_t>(c + e) >> 3) & 1);
  const int64_t e0 = e - odd;
  if (e0 >= 0 && e0 + 1 < n) cp_async16(smem, c + e0);
  else smem[odd] = c[e];
}
__device__ __forceinline__ double coef_slot(const double* smem, const double* c, int64_t e)
{
  return smem[(reinterpret_cast<uintptr_t>(c + e) >> 3) & 1];
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem));
}

// The block's map rows into shared memory with cp.async (waited for by the
// caller's cp.async.wait_all): whole 16-byte chunks of its local sources (group
// offsets are multiples of 32 sources, so the range is 64-byte aligned) and its
// group offsets, each up to the stage's size.
template <int THREADS>
__device__ __forceinline__ void stage_block_map(const BlockArgs& bm, int32_t g0, int32_t g1, int32_t src0,
                                                int32_t src1, uint16_t* s_src, int2* s_out, int32_t* s_goff)
{
  const int32_t n_src = min(src1 - src0, kStageSrc), n_goff = min(g1 - g0, kStageGroups) + 1;
  const int32_t n_out = 32 * min(g1 - g0, kStageGroups);
  for (int i = threadIdx.x; i < n_src / 8; i += THREADS) cp_async16(s_src + 8 * i, bm.bsrc + src0 + 8 * i);
  for (int i = threadIdx.x; i < n_out / 2; i += THREADS) cp_async16(s_out + 2 * i, bm.bout + 32 * (int64_t)g0 + 2 * i);
  for (int i = threadIdx.x; i < n_goff; i += THREADS) cp_async4(s_goff + i, bm.bgoff + g0 + i);
  asm volatile("cp.async.commit_group;\n" ::);
}

// One run's sum by one lane, four sources per step, from the byte offsets `src`
// (row j at src[32 j]) of the block's entries; rows past L read the zero entry.
__device__ __forceinline__ uint32_t src_row(const uint16_t* src, int32_t j, int32_t L)
{
  return j < L ? src[32 * j] : 4u * 10u * kElemBlock;
}
__device__ __forceinline__ float em_at(const unsigned char* em, uint32_t off)
{
  return *reinterpret_cast<const float*>(em + off);
}
template <int MODE>
__device__ __forceinline__ typename Arith<MODE>::T em_value(const unsigned char* em, uint32_t off)
{
  if constexpr (MODE == kDW) return ff{em_at(em, off), em_at(em + 4 * kEmStride, off)};
  else if constexpr (MODE == kF32) return em_at(em, off);
  else return *reinterpret_cast<const double*>(em + 2 * off);
}
template <int MODE>
__device__ __forceinline__ typename Arith<MODE>::Out run_sum(const unsigned char* em, const uint16_t* src, int32_t L)
{
  if constexpr (MODE == kF64) {
    // no rows past L: an addition, of zero too, holds the FP64 pipe that bounds this mode
    // (P1 128^3: 2.40 ms with them, 2.36 without)
    double v = 0.0;
    int32_t j = 0;
    for (; j + 4 <= L; j += 4) {
      const double x0 = em_value<MODE>(em, src[32 * j]), x1 = em_value<MODE>(em, src[32 * j + 32]),
                   x2 = em_value<MODE>(em, src[32 * j + 64]), x3 = em_value<MODE>(em, src[32 * j + 96]);
      v = (((v + x0) + x1) + x2) + x3;
    }
    for (; j < L; ++j) v += em_value<MODE>(em, src[32 * j]);
    return v;
  }
  SourceSum<MODE> sum;
  for (int32_t j = 0; j < L; j += 4) {
    const uint32_t i0 = src_row(src, j, L), i1 = src_row(src, j + 1, L), i2 = src_row(src, j + 2, L),
                   i3 = src_row(src, j + 3, L);
    sum.add(em_value<MODE>(em, i0), em_value<MODE>(em, i1));
    sum.add(em_value<MODE>(em, i2), em_value<MODE>(em, i3));
  }
  return sum.result();
}

// Phase 2 of the block assembly: each warp takes groups of 32 of the block's
// runs; lane l sums its run's sources from the element matrices em in shared
// memory and writes a complete entry to its CSR position and mirror, a shared
// entry's partial to its slot.  A block whose map exceeds the stage (rare) reads it
// from global memory.  Loop bounds go through shuffles, which makes them uniform
// for the compiler: no divergence handling around the loops.
template <int MODE, int THREADS>
__device__ __forceinline__ void block_sums_from(const BlockArgs& bm, int32_t g0, int32_t g1, int32_t src0,
                                                const uint16_t* src, const int2* out_of, const int32_t* goff,
                                                const unsigned char* em, typename Arith<MODE>::Out* __restrict__ values)
{
  using Out = typename Arith<MODE>::Out;
  const int lane = threadIdx.x & 31;
  const int n = g1 - g0;
  for (int gi = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); gi < n; gi += THREADS / 32) {
    const int2 out = out_of[32 * gi + lane];
    const int32_t o = goff[gi];
    const int32_t L = __shfl_sync(0xffffffffu, (goff[gi + 1] - o) >> 5, 0);
    const Out r = run_sum<MODE>(em, src + (o - src0) + lane, L);
    // a partial takes an 8-byte slot in every precision
    Out* at = out.x >= 0 ? values + out.x
                         : reinterpret_cast<Out*>(static_cast<double*>(bm.partial) + (-1 - (int64_t)out.x));
    if (out.x != kNoOutput) *at = r;
    if (out.x >= 0 && out.y != out.x) values[out.y] = r;
  }
}
template <int MODE, int THREADS>
__device__ __forceinline__ void block_sums(const BlockArgs& bm, int32_t g0, int32_t g1, int32_t src0, int32_t src1,
                                           const uint16_t* s_src, const int2* s_out, const int32_t* s_goff,
                                           const unsigned char* em, typename Arith<MODE>::Out* __restrict__ values)
{
  if (src1 - src0 <= kStageSrc && g1 - g0 <= kStageGroups)
    block_sums_from<MODE, THREADS>(bm, g0, g1, src0, s_src, s_out, s_goff, em, values);
  else
    block_sums_from<MODE, THREADS>(bm, g0, g1, 0, bm.bsrc, bm.bout + 32 * (int64_t)g0, bm.bgoff + g0, em, values);
}

// P1: one CTA per block of kElemBlock elements.  Double-word and FP32: 256 threads,
// two elements each as packed pairs; native FP64: 512 threads, one element each.
// SPLIT: the node records are split on grids (edges_dw; FP32 reads either form).
template <int MODE> constexpr int kBlockThreads = MODE == kF64 ? 512 : 256;
template <int MODE, bool SPLIT>
__global__ void __launch_bounds__(kBlockThreads<MODE>, MODE == kF32 ? 4 : (MODE == kDW ? 3 : 2))
    k_block_asm(ElemArgs a, BlockArgs bm, typename Arith<MODE>::Out* __restrict__ values)
{
  using A = Arith<MODE>;
  using T = typename A::T;
  constexpr int NU = 10, THREADS = kBlockThreads<MODE>;
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* s_src = reinterpret_cast<uint16_t*>(smem + kEmBytes<MODE>);
  int2* s_out = reinterpret_cast<int2*>(s_src + kStageSrc);
  float4* s_a = reinterpret_cast<float4*>(s_out + 32 * kStageGroups);
  float4* s_b = s_a + kStageNodes;
  float* s_z = reinterpret_cast<float*>(s_b + kStageNodes);
  int32_t* s_id = reinterpret_cast<int32_t*>(s_z + kStageNodes);
  int32_t* s_goff = MODE == kF64 ? reinterpret_cast<int32_t*>(s_a) : s_id + kStageNodes;
  __shared__ T mass[NU];
  pdl_trigger();
  const int64_t p0 = (int64_t)blockIdx.x * kElemBlock;
  const int64_t E = a.n_elem;
  if constexpr (MODE == kF64) {
    const int32_t g0 = bm.bgrp[blockIdx.x], g1 = bm.bgrp[blockIdx.x + 1];
    const int32_t src0 = bm.bsrc0[blockIdx.x], src1 = bm.bsrc0[blockIdx.x + 1];
    stage_block_map<THREADS>(bm, g0, g1, src0, src1, s_src, s_out, s_goff);
    pdl_wait();
    double* em = reinterpret_cast<double*>(smem);
    if (threadIdx.x < NU) mass[threadIdx.x] = a.tables[6 * NU + threadIdx.x];
    if (threadIdx.x == 0) em[NU * kElemBlock] = 0.0;
    __syncthreads();
    const int lp = threadIdx.x;
    if (p0 + lp < E) {
      double K[NU];
      p1_element_f64(a, mass, elem_nodes(a, p0 + lp), elem_coef(a, p0 + lp), K);
#pragma unroll
      for (int u = 0; u < NU; ++u) em[u * kElemBlock + lp] = K[u];
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    block_sums<MODE, THREADS>(bm, g0, g1, src0, src1, s_src, s_out, s_goff, smem, values);
  } else {
    // asynchronous copies in the order of need: the records of the block's unique
    // nodes, the pair's coefficients, the block map.  A warp's coefficient slots lie in
    // the shared rows that only its own elements' entries overwrite.
    float* em = reinterpret_cast<float*>(smem);
    const int lane = threadIdx.x & 31, lp = threadIdx.x + (threadIdx.x & ~31);
    // past the last element the pair repeats it (no source refers to the copies)
    const int64_t p1 = min(p0 + lp, E - 1), p2 = min(p0 + lp + 32, E - 1);
    const int32_t id = bm.bnode[(int64_t)blockIdx.x * kStageNodes + threadIdx.x];
    const int64_t e1 = a.elem_order[p1], e2 = a.elem_order[p2];
    const bool staged = bm.bnode_n[blockIdx.x] >= 0;
    const int32_t g0 = bm.bgrp[blockIdx.x], g1 = bm.bgrp[blockIdx.x + 1];
    const int32_t src0 = bm.bsrc0[blockIdx.x], src1 = bm.bsrc0[blockIdx.x + 1];
    cp_async16(s_a + threadIdx.x, a.geo.rec + 2 * (int64_t)id);
    cp_async16(s_b + threadIdx.x, a.geo.rec + 2 * (int64_t)id + 1);
    if (MODE == kDW) cp_async4(s_z + threadIdx.x, a.geo.loz + id);
    s_id[threadIdx.x] = id;
    asm volatile("cp.async.commit_group;\n" ::);
    // up to here only the plan was read; the coefficients, the partial sums and the
    // values belong to the kernels before this one until they are complete
    pdl_wait();
    double* slot1 = reinterpret_cast<double*>(em + (lane >> 4) * kElemBlock + (lp - lane) + 4 * (lane & 15));
    double* slot2 = slot1 + kElemBlock;  // two rows on
    if (a.coeff) {
      coef_fetch(slot1, a.coeff, e1, E);
      coef_fetch(slot2, a.coeff, e2, E);
    }
    asm volatile("cp.async.commit_group;\n" ::);
    stage_block_map<THREADS>(bm, g0, g1, src0, src1, s_src, s_out, s_goff);
    if (threadIdx.x < (MODE == kDW ? 2 : 1)) em[threadIdx.x * kEmStride + NU * kElemBlock] = 0.0f;
    if (!a.stiff && threadIdx.x < NU) mass[threadIdx.x] = A::from(a.tables[6 * NU + threadIdx.x]);
    typename Pair<MODE>::T J[3][3];
    int4 n0, n1;
    if (staged) {
      const uchar4 l0 = __ldg(bm.elem_local + p1), l1 = __ldg(bm.elem_local + p2);
      n0 = make_int4(l0.x, l0.y, l0.z, l0.w);
      n1 = make_int4(l1.x, l1.y, l1.z, l1.w);
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      __syncthreads();
      pair_edges<SPLIT>(StagedNodes{s_a, s_b, s_z}, n0, n1, J);
    } else {
      n0 = elem_nodes(a, p1);
      n1 = elem_nodes(a, p2);
      __syncthreads();  // mass
      pair_edges<SPLIT>(GlobalNodes{a.geo}, n0, n1, J);
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    const double c0 = a.coeff ? coef_slot(slot1, a.coeff, e1) : a.cconst;
    const double c1 = a.coeff ? coef_slot(slot2, a.coeff, e2) : a.cconst;
    __syncwarp();  // before the entries overwrite the slots
    const auto node = [&](int e) {
      const int4 n = e ? n1 : n0;
      return staged ? make_int4(s_id[n.x], s_id[n.y], s_id[n.z], s_id[n.w]) : n;
    };
    if constexpr (MODE == kDW) p1_pair_dw(a, mass, J, node, c0, c1, lp, em, em + kEmStride);
    else p1_pair_f32(a, mass, J, node, c0, c1, lp, em);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    block_sums<MODE, THREADS>(bm, g0, g1, src0, src1, s_src, s_out, s_goff, smem, values);
  }
}

template <typename V>
__global__ void __launch_bounds__(256) k_shared_sum(int64_t n_groups, const int32_t* __restrict__ sgoff,
                                                    const int2* __restrict__ sout, const double* partial, V* values)
{
  pdl_trigger();
  const int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const bool live = g < n_groups;
  const int lane = threadIdx.x & 31;
  const int2 out = live ? sout[32 * g + lane] : make_int2(kNoOutput, 0);
  const int32_t o = live ? sgoff[g] : 0, L = live ? (sgoff[g + 1] - o) >> 5 : 0;
  pdl_wait();  // every CTA waits, so that this kernel's end implies the one before's
  V v = V(0);
  // 8 partials in flight, summed in ascending j
  for (int32_t j = 0; j < L; j += 8) {
    V x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      x[i] = j + i < L ? *reinterpret_cast<const V*>(partial + o + 32 * (j + i) + lane) : V(0);
#pragma unroll
    for (int i = 0; i < 8; ++i) v += x[i];
  }
  if (out.x >= 0) {
    values[out.x] = v;
    if (out.y != out.x) values[out.y] = v;
  }
}

template <int MODE, bool SPLIT>
static mg_status launch_block_t(mg_plan* p, const ElemArgs& a, void* d_values, cudaStream_t st)
{
  using Out = typename Arith<MODE>::Out;
  const BlockArgs bm{p->d_bgrp,    p->d_bsrc0, p->d_bgoff,   p->d_bsrc,      p->d_bout,
                     p->d_partial, p->d_bnode, p->d_bnode_n, p->d_elem_local};
  static std::once_flag once[64];
  if (a.n_elem > 0) {
    constexpr size_t smem = block_smem_bytes<MODE>();
    MG_TRY(allow_smem(k_block_asm<MODE, SPLIT>, smem, once));
    MG_CUDA(launch_smem(true, k_block_asm<MODE, SPLIT>, (int)p->n_blocks, kBlockThreads<MODE>, smem, st, a, bm,
                        static_cast<Out*>(d_values)));
  }
  if (p->n_sgroups > 0)
    MG_CUDA(launch_pdl(k_shared_sum<Out>, (int)((p->n_sgroups + 7) / 8), 256, st, p->n_sgroups,
                       (const int32_t*)p->d_sgoff, (const int2*)p->d_sout, (const double*)p->d_partial,
                       static_cast<Out*>(d_values)));
  return MG_OK;
}

// The element-matrix array of a plan (allocated by its first assembly).
static mg_status plan_gather(mg_plan* p)
{
  std::lock_guard<std::mutex> lock(p->upload_mu);
  if (!p->d_em) {
    // nunique x n_elem entries of up to 8 bytes, then one zero entry (8 bytes:
    // the FP32 gather reads its first float) for the padding sources
    const int64_t n = (int64_t)nunique(p->mesh->order) * p->mesh->n_elem;
    MG_CUDA(cudaMalloc(&p->d_em, sizeof(double) * (size_t)(n + 1)));
    MG_CUDA(cudaMemset(static_cast<double*>(p->d_em) + n, 0, sizeof(double)));
    MG_TRY(legacy_done());
  }
  return MG_OK;
}

template <int MODE>
static mg_status launch_gather_t(mg_plan* p, const ElemArgs& a, void* d_values, cudaStream_t st)
{
  constexpr int ORDER = 2;
  const int64_t E = a.n_elem;
  if (E > 0) {
    if constexpr (MODE == kF64) k_elem_mat_f64<<<(unsigned)((E + 255) / 256), 256, 0, st>>>(a);
    else if (MODE == kDW && p->mesh->grid_split) k_elem_mat_pair<MODE, true><<<(unsigned)((E + 255) / 256), 128, 0, st>>>(a);
    else k_elem_mat_pair<MODE, false><<<(unsigned)((E + 255) / 256), 128, 0, st>>>(a);
  }
  MG_CUDA(cudaGetLastError());
  using Out = typename Arith<MODE>::Out;
  const unsigned blocks = (unsigned)((p->n_groups + 7) / 8);  // 8 warps (groups) per CTA
  // the zero entry: index nunique * n_elem of the 8-byte entries, 2 * that of floats
  const uint32_t zero = (uint32_t)((MODE == kF32 ? 2 : 1) * (int64_t)nunique(ORDER) * E);
  // 8 sources in flight per thread (measured on GB300 at P1 128^3 and P2 48^3
  // against 4 and 16)
  if (p->n_groups > 0)
    k_slot_gather<MODE, 8><<<blocks, 256, 0, st>>>(p->n_groups, p->n_upper, p->d_goff, p->d_uslot, p->d_umirror,
                                                   p->d_src, p->d_em, zero, static_cast<Out*>(d_values));
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

static mg_status launch_assemble_gather(mg_plan* p, int op, const double* d_coeff, double c, const RefTables* t,
                                        const double* d_tab, int prec, void* d_values, cudaStream_t st)
{
  mg_mesh* m = p->mesh;
  if (!uses_block_map(m->order)) MG_TRY(plan_gather(p));
  const bool needs_coeff = (op == MG_OP_STIFF_KAPPA || op == MG_OP_MASS_COEFF);
  ElemArgs a;
  a.n_elem = m->n_elem;
  a.elem_order = p->d_elem_order;
  a.dofs_m = p->d_dofs_morton;
  const int ge = prec == MG_F64_NATIVE ? 0 : m->geo_exp;  // native FP64 reads the coordinates as they are
  a.geo = GeoPtrs{ge ? m->d_xyz_rec : m->d_xyz, m->d_node_rec, m->d_lo_z};
  a.coeff = needs_coeff ? d_coeff : nullptr;
  a.cconst = op == MG_OP_STIFF_CONST ? c : 1.0;
  a.tables = d_tab;
  a.wsum = std::ldexp(t->wsum, ge);
  a.w_hi = (float)a.wsum;
  a.w_lo = (float)(a.wsum - (double)a.w_hi);
  a.len_scale = std::ldexp(1.0f, ge);
  a.vol_scale1 = std::ldexp(1.0f, 3 * ge / 2);
  a.vol_scale2 = std::ldexp(1.0f, 3 * ge - 3 * ge / 2);
  a.sc_min = std::ldexp(1.0f, -96 - 3 * ge);
  a.sc_max = std::ldexp(1.0f, 113 - 3 * ge);
  a.stiff = (op == MG_OP_STIFF_KAPPA || op == MG_OP_STIFF_CONST);
  a.em = p->d_em;
  a.flags = p->d_counters + 4;
  if (uses_block_map(m->order)) {
    if (prec == MG_F32) return launch_block_t<kF32, false>(p, a, d_values, st);
    if (prec == MG_F64_NATIVE) return launch_block_t<kF64, false>(p, a, d_values, st);
    return m->grid_split ? launch_block_t<kDW, true>(p, a, d_values, st) : launch_block_t<kDW, false>(p, a, d_values, st);
  }
  if (prec == MG_F32) return launch_gather_t<kF32>(p, a, d_values, st);
  return prec == MG_F64_NATIVE ? launch_gather_t<kF64>(p, a, d_values, st) : launch_gather_t<kDW>(p, a, d_values, st);
}

mg_status launch_assemble(mg_plan* p, int op, const double* d_coeff, double c, int quad, int prec,
                          void* d_values, cudaStream_t st)
{
  if (op < MG_OP_STIFF_KAPPA || op > MG_OP_MASS_COEFF)
    return set_error(MG_ERR_INVALID_ARG, "unknown operator " + std::to_string(op));
  if (!prec_valid(prec)) return set_error(MG_ERR_INVALID_ARG, "prec must be MG_F64, MG_F32 or MG_F64_NATIVE");
  const bool needs_coeff = (op == MG_OP_STIFF_KAPPA || op == MG_OP_MASS_COEFF);
  if (needs_coeff && !d_coeff && p->mesh->n_elem > 0)
    return set_error(MG_ERR_INVALID_ARG, "this operator needs the per-element coefficient array");
  const RefTables* t = nullptr;
  const double* d_tab = nullptr;
  MG_TRY(plan_tables(p, quad, &t, &d_tab));  // validates quad
  if (p->nnz == 0) return MG_OK;  // empty mesh: nothing to write
  if (!d_values) return set_error(MG_ERR_INVALID_ARG, "mg_assemble: null values");
  MG_TRY(plan_device(p));
  return launch_assemble_gather(p, op, d_coeff, c, t, d_tab, prec, d_values, st);
}

// --------------------------------------------------------------- Dirichlet --
template <typename V>
__global__ void k_dirichlet(int64_t ndof, const int32_t* rowptr, const int32_t* colind, const uint8_t* mask,
                            V* values, double* b)
{
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r >= ndof) return;
  const bool mr = mask[r] != 0;
  for (int s = rowptr[r]; s < rowptr[r + 1]; ++s) {
    const int c = colind[s];
    if (mr) values[s] = (c == r) ? V(1) : V(0);
    else if (mask[c]) values[s] = V(0);
  }
  if (b && mr) b[r] = 0.0;
}

// ----------------------------------------------------------------- adjoint --
// grad_e = -sum_{i,j} lambda[dof_j] Khat_ij u[dof_i], Khat the kappa = 1
// stiffness of element e (symmetric, rows summing to zero).  Because of the
// zero row sums the form only sees differences to the element's first vertex:
// grad_e = -sum_{i,j >= 1} (lambda_j - lambda_0) Khat_ij (u_i - u_0), which removes
// the cancellation of a smooth field against the stiffness.  The differences
// are FP64 (exact for nearby values); each group (u or lambda) is rescaled by
// the power of two of its largest difference, so the double-word arithmetic on
// the FP32 pipes sees values near 1 whatever the scale of u and lambda, and the
// result is scaled back in FP64.

// biased FP64 exponent
__device__ __forceinline__ int dexp(double v) { return (int)((__double_as_longlong(v) >> 52) & 0x7ff); }

// v * 2^(1023 - emax) as a double-word value, by exponent arithmetic (emax = the
// largest biased exponent of the group, a normal number).  Parts more than 2^-74
// below the largest are dropped (a relative 2^-74 of the group).
template <bool RENORM>
__device__ __forceinline__ ff ff_rescaled(double v, int emax)
{
  const long long b = __double_as_longlong(v);
  if (dexp(v) + 74 < emax) return ff{0.0f, 0.0f};
  return ff_from_double_bits<RENORM>(__longlong_as_double(b - ((long long)(emax - 1023) << 52)));
}

// v * 2^k for |k| <= 2044 (two exact power-of-two products unless the result
// leaves the FP64 range); out of line, like the other rare FP64 paths
__device__ __noinline__ double scale_pow2(double v, int k)
{
  const int k1 = k / 2, k2 = k - k1;
  return v * __longlong_as_double((long long)(k1 + 1023) << 52) * __longlong_as_double((long long)(k2 + 1023) << 52);
}

// a * 2^k as a double: scaled on the floats when the result stays well inside
// the normal-float range (then one FP64 addition), else in FP64
__device__ __forceinline__ double ff_to_double_pow2(ff a, int k)
{
  if (a.hi == 0.0f) return 0.0;
  const int ex = (int)((__float_as_uint(a.hi) >> 23) & 0xffu) - 127 + k;
  if (k >= -100 && k <= 100 && ex >= -90 && ex <= 100) {
    const float fs = __uint_as_float((uint32_t)(k + 127) << 23);
    return ff_to_double_bits(ff{a.hi * fs, a.lo * fs});
  }
  return scale_pow2(ff_to_double_bits(a), k);
}

// Element geometry cache: the double-word Jacobian determinant and cofactors of every
// element, written once per plan in the Morton order p, structure of arrays
// (coalesced for the kernels that read them: load vector, adjoint).  Two elements per
// thread (64 per warp) as packed pairs from the node records; cancelling determinants
// in FP64.
template <int NB, bool SPLIT>
__global__ void __launch_bounds__(128) k_elem_geometry(int64_t n_elem, const int32_t* dofs_m, GeoPtrs geo, float2* det,
                                                       float2* cof)
{
  const int lane = threadIdx.x & 31;
  const int64_t first = (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 64;
  if (first >= n_elem) return;
  const int64_t p0 = min(first + lane, n_elem - 1), p1 = min(first + 32 + lane, n_elem - 1);
  const auto vertices = [&](int64_t p) {
    if constexpr (NB == 4) return __ldg(reinterpret_cast<const int4*>(dofs_m) + p);
    const int2* d = reinterpret_cast<const int2*>(dofs_m + p * NB);
    const int2 x = __ldg(d), y = __ldg(d + 1);
    return make_int4(x.x, x.y, y.x, y.y);
  };
  const int4 n0 = vertices(p0), n1 = vertices(p1);
  ff2 J[3][3];
  pair_edges<SPLIT>(GlobalNodes{geo}, n0, n1, J);
  PairGeo f;
  pair_cofactors(J, f);
  const auto put = [&](int64_t p, float2 h, float2 l, float2* out, bool second) {
    out[p] = second ? make_float2(h.y, l.y) : make_float2(h.x, l.x);
  };
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int64_t p = e ? p1 : p0;
    if (e ? f.degen1 : f.degen0) {
      const Cof<ff> x = abs_geometry_fp64<ff>(geo.xyz, e ? n1 : n0);
      det[p] = make_float2(x.det.hi, x.det.lo);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) cof[(3 * r + c) * n_elem + p] = make_float2(x.c[r][c].hi, x.c[r][c].lo);
    } else {
      put(p, f2_get(f.det.hi), f2_get(f.det.lo), det, e);
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) put(p, f2_get(f.C[c][r].hi), f2_get(f.C[c][r].lo), cof + (3 * r + c) * n_elem, e);
    }
  }
}

__device__ __forceinline__ void cached_geometry(const float2* det, const float2* cof, int64_t n_elem, int64_t p,
                                                Cof<ff>& f)
{
  const float2 d = det[p];
  f.det = ff{d.x, d.y};
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float2 v = cof[(3 * r + c) * n_elem + p];
      f.c[r][c] = ff{v.x, v.y};
    }
}

// Elements are visited along a Morton curve of their centroids (elem_order,
// dofs_m = their dofs in that order), so neighbouring threads gather
// neighbouring dof values.  factor: 2^g of the geometry cache's scale (mg_mesh::geo_exp),
// for P1 times the card's weights.
// P1 is bound by instruction issue: dot products with one renormalisation each (instead of
// one per operation) and five CTAs per SM took it from 52 to 45 us at P1 64^3 on GB300 (4:
// 49, 6: 47.5), no table staged and the plan read before the wait to 41.4.  Two elements per thread as packed pairs measured 59 to 68 us, and the
// geometry formed from nodes staged per block 70 us: fewer warps for the same gathers.
template <int ORDER>
__global__ void __launch_bounds__(256, ORDER == 1 ? 5 : 1) k_adjoint(int64_t n_elem, const int32_t* elem_order, const int32_t* dofs_m,
                                                 const float2* gdet, const float2* gcof, const double* tables,
                                                 double factor, const double* u, const double* lam, double* grad)
{
  constexpr int NB = ORDER == 1 ? 4 : 10, NU = ORDER == 1 ? 10 : 55;
  __shared__ ff tab[ORDER == 1 ? 1 : 6 * NU];  // P1 takes the zero row sums, no table
  // P1 is launched with programmatic dependence; P2, whose CTAs fill the SM's registers,
  // takes 17 us without and 27 with it at 13 k elements
  if constexpr (ORDER == 1) {
    pdl_trigger();
  } else {
    for (int i = threadIdx.x; i < 6 * NU; i += blockDim.x) tab[i] = ff_from_double(tables[i]);
    __syncthreads();
  }
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n_elem) {
    if constexpr (ORDER == 1) pdl_wait();
    return;
  }
  const int64_t e = elem_order[i];
  const int32_t* dofs = dofs_m + i * NB;  // this element's dofs; the first four are its vertices
  const int4 n = ORDER == 1 ? reinterpret_cast<const int4*>(dofs_m)[i] : make_int4(dofs[0], dofs[1], dofs[2], dofs[3]);
  if constexpr (ORDER == 1) pdl_wait();  // u, lambda and grad belong to the kernels before this one
  // FP64 differences to the first dof and the largest exponent of each group
  double du[NB - 1], dl[NB - 1];
  int eu = 0, el = 0;
  {
    const double u0 = u[n.x], l0 = lam[n.x];
#pragma unroll
    for (int k = 1; k < NB; ++k) {
      const int dof = ORDER == 1 ? (k == 1 ? n.y : k == 2 ? n.z : n.w) : dofs[k];
      du[k - 1] = u[dof] - u0;
      dl[k - 1] = lam[dof] - l0;
      eu = max(eu, dexp(du[k - 1]));
      el = max(el, dexp(dl[k - 1]));
    }
  }
  if (eu == 0x7ff || el == 0x7ff) {  // Inf or NaN among u, lambda
    grad[e] = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  if (eu == 0 || el == 0) {  // constant (or denormal-scale) u or lambda on the element
    grad[e] = -0.0;
    return;
  }
  Cof<ff> f;
  cached_geometry(gdet, gcof, n_elem, i, f);
  ff s = ff_make(0.0f);
  if (ORDER == 1) {
    // lambda^T K u = (factor / det) (sum_b dl_b C_b) . (sum_b du_b C_b), C_b the cofactor columns
    // (one renormalisation per dot product instead of one per operation)
    ff gu[3], gl[3], a[3], c[3];
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      a[b] = ff_rescaled<true>(du[b], eu);
      c[b] = ff_rescaled<true>(dl[b], el);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      gu[r] = ff_dot3(a, f.c[r]);
      gl[r] = ff_dot3(c, f.c[r]);
    }
    s = ff_dot3(gl, gu) * (ff_from_double_bits(factor) / f.det);
  } else {
    ff ue[NB - 1], le[NB - 1];
#pragma unroll
    for (int k = 0; k < NB - 1; ++k) {
      ue[k] = ff_rescaled<false>(du[k], eu);
      le[k] = ff_rescaled<false>(dl[k], el);
    }
    ff g[6];
    metric<ff>(f, ff_make((float)factor) / f.det, g);
#pragma unroll
    for (int a = 1; a < NB; ++a) {
      ff row = ff_make(0.0f);
#pragma unroll
      for (int b = 1; b < NB; ++b) {
        const int uidx = sym_index(a, b, NB);
        ff v = g[0] * tab[uidx];
#pragma unroll
        for (int p = 1; p < 6; ++p) v = v + g[p] * tab[p * NU + uidx];
        row = row + le[b - 1] * v;
      }
      s = s + row * ue[a - 1];
    }
  }
  grad[e] = -ff_to_double_pow2(s, (eu - 1023) + (el - 1023));
}

// v 2^(1023 - emax) as a double-word value, emax the block's largest biased exponent and
// v zero or a normal number within 2^70 of it
__device__ __forceinline__ ff ff_scaled(double v, int emax)
{
  if (dexp(v) == 0) return ff{0.0f, 0.0f};
  return ff_from_double_bits(__longlong_as_double(__double_as_longlong(v) - ((long long)(emax - 1023) << 52)));
}

// ------------------------------------------------------------- load vector --
// P1 meshes whose blocks fit the stage take the one-pass form below (k_rhs_block); P2 and
// the others these two passes.
// b_i = sum_e s_e int_e f_h phi_i with f_h = sum_k f_k phi_k (f = 1 without a
// field): the reference's vector builder (fnEL3dA / fnEL3dB under
// traitsVectorBuilder) as two deterministic passes.
// Pass 1, one thread per element along the Morton order (position p): the
// element vector y[p nb + l] = s_e det_e sum_k Mhat_lk f_k, Mhat the reference
// mass table of the quadrature card.  Double-word arithmetic; s_e and the f_k
// are rescaled by powers of two (their largest exponents), so the result keeps
// FP64 accuracy at any scale, and is written as an IEEE double.
// SCALED: the geometry cache is on another scale than the mesh (volume = 2^(3 geo_exp)); the
// test in one kernel for both took P2 32^3 from 43.2 to 45.1 us.
template <int ORDER, bool SCALED>
__global__ void __launch_bounds__(256) k_rhs_elem(int64_t n_elem, const int32_t* elem_order, const int32_t* dofs_m,
                                                  const float2* gdet, const double* mass, const double* field,
                                                  const double* scale, double* y, int two_valued, double volume)
{
  constexpr int NB = ORDER == 1 ? 4 : 10, NU = ORDER == 1 ? 10 : 55;
  __shared__ ff tab[NU];
  __shared__ ff rsum[NB];
  for (int i = threadIdx.x; i < NU; i += blockDim.x) tab[i] = ff_from_double(mass[i]);
  if (threadIdx.x < NB) {
    double r = 0.0;
    for (int j = 0; j < NB; ++j) r += mass[sym_index((int)threadIdx.x, j, NB)];
    rsum[threadIdx.x] = ff_from_double(r);
  }
  __syncthreads();
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= n_elem) return;
  const int32_t* dofs = dofs_m + p * NB;
  const double sd = scale ? scale[elem_order[p]] : 1.0;
  const int es = dexp(sd);
  double f[NB];
  int ef = 1023;  // exponent of 1 without a field
  if (field) {
    ef = 0;
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      f[k] = field[dofs[k]];
      ef = max(ef, dexp(f[k]));
    }
  }
  double2* out = reinterpret_cast<double2*>(y + p * NB);
  if (es == 0x7ff || ef == 0x7ff || es == 0 || ef == 0) {
    // Inf / NaN in s or f: NaN; zero (or denormal-scale) s or f: zero
    const double v = (es == 0x7ff || ef == 0x7ff) ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
#pragma unroll
    for (int l = 0; l < NB / 2; ++l) out[l] = make_double2(v, v);
    return;
  }
  const float2 dt = gdet[p];
  const ff sdet = ff_rescaled<false>(sd, es) * ff{dt.x, dt.y};
  ff v[NB];
  if (field) {
    ff fr[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) fr[k] = ff_rescaled<false>(f[k], ef);
    if (ORDER == 1 && two_valued) {
      // M^_lk = o + (d - o) [l = k]: (M^ f)_l = o sum_k f_k + (d - o) f_l, with
      // d = tab(0,0) and o = tab(0,1) from the table
      const ff o = tab[1], dmo = tab[0] - tab[1];
      ff sf = fr[0];
#pragma unroll
      for (int k = 1; k < NB; ++k) sf = sf + fr[k];
      const ff base = o * sf;
#pragma unroll
      for (int l = 0; l < NB; ++l) v[l] = (base + dmo * fr[l]) * sdet;
    } else {
#pragma unroll
      for (int l = 0; l < NB; ++l) {
        ff a = tab[sym_index(l, 0, NB)] * fr[0];
#pragma unroll
        for (int k = 1; k < NB; ++k) a = a + tab[sym_index(l, k, NB)] * fr[k];
        v[l] = a * sdet;
      }
    }
  } else {
#pragma unroll
    for (int l = 0; l < NB; ++l) v[l] = rsum[l] * sdet;
  }
  // back to the true scale 2^k2
  const int k2 = (es - 1023) + (ef - 1023);
#pragma unroll
  for (int l = 0; l < NB / 2; ++l) {
    double2 w = make_double2(ff_to_double_pow2(v[2 * l], k2), ff_to_double_pow2(v[2 * l + 1], k2));
    if constexpr (SCALED) w = make_double2(w.x * volume, w.y * volume);
    out[l] = w;
  }
}

// Pass 2, G lanes per dof: b_i = the FP64 sum of its element-vector entries,
// each lane over every G-th entry in ascending slot order, the lanes combined
// by xor shuffles in a fixed tree (bitwise reproducible, no atomics).
template <int G, int U>
__global__ void __launch_bounds__(256) k_rhs_gather(int64_t ndof, const int32_t* __restrict__ ptr,
                                                    const int32_t* __restrict__ slot, const double* __restrict__ y,
                                                    double* __restrict__ b)
{
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int lane = threadIdx.x & (G - 1);
  if (i >= ndof) return;  // whole groups: G divides the block
  const int s0 = __ldg(ptr + i), s1 = __ldg(ptr + i + 1);
  double acc = 0.0;
  for (int base = s0 + lane; base < s1; base += G * U) {
    int q[U];
#pragma unroll
    for (int u = 0; u < U; ++u) q[u] = base + u * G < s1 ? __ldg(slot + base + u * G) : -1;
    double t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = q[u] >= 0 ? __ldg(y + q[u]) : 0.0;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (q[u] >= 0) acc += t[u];
  }
  if constexpr (G > 1) {
    const unsigned mask = ((1u << G) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(G - 1));
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(mask, acc, off, G);
  }
  if (lane == 0) b[i] = acc;
}

// P1, one pass: a CTA per block of kElemBlock elements computes its element vectors into
// shared memory, two elements per thread as packed pairs, and sums them per node of
// the block (build_rhs_map): a node whose elements all lie in the block gets its sum
// written, another one a partial, added in block order by k_rhs_shared.
//   y_l = s det (M^ f)_l
// f (converted once per node), s and det are scaled by the powers of two of their largest
// values in the block; where their spreads together exceed 2^70, a value is Inf, NaN or
// subnormal, or a determinant is 2^127 or more (its inverse power would be
// subnormal), every element takes its own (rhs_block_wide).
// The two passes wrote and gathered 32 bytes per element through memory and issued 21
// warp instructions per element, a third of them conversions: GB300, P1 96^3, 217 ->
// 141 us (block kernel 126, shared nodes 14; bound by issue and the L1 data path, 61 %
// each), 134 with programmatic launches, the table staged only where it is used and
// no FP64 comparisons, 123 with the powers of two in the factor's exponent and the spread
// blocks out of line; the map is built on the GPU (first call on a plan 76 -> 1.6 ms).
struct RhsArgs {
  int64_t n_elem;
  const int32_t *elem_order, *bnode, *bnode_n;
  const uchar4* elem_local;
  const float2* gdet;
  const double *mass, *field, *scale;
  const uint16_t* bpos;    // per block 4 kElemBlock byte offsets 4 (l kElemBlock + element), by node
  const uint16_t* bstart;  // per block kStageNodes + 1 starts
  const int32_t* bout;     // per block kStageNodes outputs: node, or -1 - partial slot
  double *partial, *b;
  const int32_t* all_partial;  // rhs_ptr where b may overlap an input, else null (rhs_put)
  int form;     // of M^ f
  int det_exp;  // gdet holds 2^-det_exp of the determinants (3 mg_mesh::geo_exp)
  double unit;  // factor of the sums (1 with the full table), a normal number
};
// M^ f: u (sum_k f_k + f_l) where the table is u (1 + [l = k]) (the symmetric cards of two
// and more degrees), u sum_k f_k where it is constant (the one-point card), else the
// full table.  u multiplies the node's sum in FP64.
enum { kRhsTable = 0, kRhsSumPlus = 1, kRhsSum = 2 };

// Where b overlaps the field or the scale, which other blocks may still read, every sum
// goes to its partial slot (a node with one has it at rhs_ptr[node]).
__device__ __forceinline__ void rhs_put(const RhsArgs& a, int32_t out, double v)
{
  if (out < 0) a.partial[-1 - (int64_t)out] = v;
  else if (a.all_partial) a.partial[a.all_partial[out]] = v;
  else a.b[out] = v;
}

// (M^ f)_l s det of a pair, without the unit, in the form's arithmetic
__device__ __forceinline__ void rhs_pair(int form, const ff* tab, const ff2 (&F)[4], ff2 sd, ff2 (&v)[4])
{
  const auto add = [](ff2 x, ff2 z) {
    const ff2 t = f2_two_sum(x.hi, z.hi);
    return f2_fast_two_sum(t.hi, t.lo + (x.lo + z.lo));
  };
  const auto dup = [](ff t) { return ff2_make(t, t); };
  if (form != kRhsTable) {
    const ff2 x = f2_two_sum(F[0].hi, F[1].hi), z = f2_two_sum(F[2].hi, F[3].hi), w = f2_two_sum(x.hi, z.hi);
    const f2 slo = ((F[0].lo + F[1].lo) + (F[2].lo + F[3].lo)) + ((x.lo + z.lo) + w.lo);
    const ff2 one = ff2_mul(f2_fast_two_sum(w.hi, slo), sd);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      const ff2 t = f2_two_sum(w.hi, F[l].hi);
      v[l] = form == kRhsSum ? one : ff2_mul(f2_fast_two_sum(t.hi, slo + (t.lo + F[l].lo)), sd);
    }
  } else {
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      ff2 t = ff2_mul(dup(tab[sym_index(l, 0, 4)]), F[0]);
#pragma unroll
      for (int k = 1; k < 4; ++k) t = add(t, ff2_mul(dup(tab[sym_index(l, k, 4)]), F[k]));
      v[l] = ff2_mul(t, sd);
    }
  }
}

// One element's share of rhs_block_wide: s, f and det near one, the powers of two that were
// taken out (the determinant's apart), and whether the vector is NaN (s or an f
// Inf or NaN) or zero (s, or all f, zero or subnormal), the rules of k_rhs_elem.
struct RhsElement {
  ff F[4], s, det;
  int k, kdet;
  bool nan, zero;
};
__device__ __forceinline__ RhsElement rhs_element(const double* f, uchar4 q, double s, float2 d)
{
  RhsElement e;
  const double v[4] = {f[q.x], f[q.y], f[q.z], f[q.w]};
  const int es = dexp(s), ef = max(max(dexp(v[0]), dexp(v[1])), max(dexp(v[2]), dexp(v[3])));
  e.nan = es == 0x7ff || ef == 0x7ff;
  e.zero = es == 0 || ef == 0;
  e.k = (es - 1023) + (ef - 1023);
  // (products of a determinant as it is may overflow, or lose their errors below the floats)
  e.kdet = min(max((int)((__float_as_uint(d.x) >> 23) & 0xffu) - 127, -126), 126);
  const float dscale = __uint_as_float((uint32_t)(127 - e.kdet) << 23);
  e.det = ff{d.x * dscale, d.y * dscale};
  if (e.nan || e.zero) {
#pragma unroll
    for (int k = 0; k < 4; ++k) e.F[k] = ff{0.0f, 0.0f};
    e.s = ff{0.0f, 0.0f};
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      // (subnormal, and not 2^-74 of the largest: its exponent is no power of two to take out)
      e.F[k] = dexp(v[k]) == 0 && ef <= 74 ? ff_from_double(scale_pow2(v[k], 1023 - ef)) : ff_rescaled<true>(v[k], ef);
    e.s = ff_rescaled<true>(s, es);
  }
  return e;
}
__device__ __forceinline__ double rhs_value(const RhsElement& e, int det_exp, ff v)
{
  if (e.nan) return __longlong_as_double(0x7ff8000000000000ll);
  const double x = ff_to_double_bits(v);
  // in the normal range the powers go into the exponent, off the FP64 pipe
  const int ex = dexp(x), kdet = e.kdet + det_exp, k = e.k + kdet;
  if (ex == 0 || ex == 0x7ff) return x;
  if (ex + k >= 1 && ex + k <= 2046) return __longlong_as_double(__double_as_longlong(x) + ((long long)k << 52));
  return scale_pow2(x * __longlong_as_double((long long)(kdet + 1023) << 52), e.k);
}

// Shared memory of a block
struct RhsShared {
  __align__(16) float y[8 * kElemBlock];       // element vectors: high parts, low parts (or doubles)
  __align__(16) float f[2 * kStageNodes];      // the nodes' f: high parts, low parts (or doubles)
  __align__(16) uint16_t pos[4 * kElemBlock];
  uint16_t start[kStageNodes + 1];
  ff tab[10];
  int red[6][8];
};

// A block whose values spread too far for one scale: s and f of every element by their own
// powers of two, as k_rhs_elem takes them, and the element vectors as doubles.  GB300,
// P1 96^3, every block of this kind: 213 us, 727 with the block in native FP64 (the
// two-pass form: 216; two FP64 products per entry for its power of two: 228).
static __device__ __noinline__ void rhs_block_wide(const RhsArgs& a, RhsShared& sh, int n_nodes, int32_t out)
{
  double *y = reinterpret_cast<double*>(sh.y), *s_f = reinterpret_cast<double*>(sh.f);
  // everything is read again, so that the common path holds nothing for this one
  const int64_t p0 = (int64_t)blockIdx.x * kElemBlock;
  const int lp = threadIdx.x + (threadIdx.x & ~31);
  const int64_t p1 = min(p0 + lp, a.n_elem - 1), p2 = min(p0 + lp + 32, a.n_elem - 1);
  s_f[threadIdx.x] = a.field ? a.field[a.bnode[(int64_t)blockIdx.x * kStageNodes + threadIdx.x]] : 1.0;
  __syncthreads();
  const RhsElement e1 = rhs_element(s_f, a.elem_local[p1], a.scale ? a.scale[a.elem_order[p1]] : 1.0, a.gdet[p1]);
  const RhsElement e2 = rhs_element(s_f, a.elem_local[p2], a.scale ? a.scale[a.elem_order[p2]] : 1.0, a.gdet[p2]);
  ff2 F[4], v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) F[k] = ff2_make(e1.F[k], e2.F[k]);
  rhs_pair(a.form, sh.tab, F, ff2_mul(ff2_make(e1.s, e2.s), ff2_make(e1.det, e2.det)), v);
  const ff u = ff_from_double_bits(a.unit);
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const ff2 w = ff2_mul(v[l], ff2_make(u, u));
    const float2 h = f2_get(w.hi), lo = f2_get(w.lo);
    y[l * kElemBlock + lp] = rhs_value(e1, a.det_exp, ff{h.x, lo.x});
    y[l * kElemBlock + lp + 32] = rhs_value(e2, a.det_exp, ff{h.y, lo.y});
  }
  __syncthreads();
  if ((int)threadIdx.x < n_nodes) {
    double sum = 0.0;
    for (int j = sh.start[threadIdx.x]; j < sh.start[threadIdx.x + 1]; ++j) sum += y[sh.pos[j] / 4];
    rhs_put(a, out, sum);
  }
}

// The sum of a node's element-vector entries, two at a time in two packed accumulators:
// the high parts error-free, and the low parts and their errors error-free into a
// second and plain into a third part, so the sum adds no error of its own beside the
// entries' (a plain sum of the low parts measured 3.0e-15 against 2.1e-15 at 96^3).
struct NodeSum {
  f2 hi = f2_make(0.0f, 0.0f), lo = f2_make(0.0f, 0.0f), er = f2_make(0.0f, 0.0f);
  __device__ __forceinline__ void add(ff a, ff b)
  {
    const ff2 t = f2_two_sum(hi, f2_make(a.hi, b.hi));
    const ff2 x = f2_two_sum(lo, f2_make(a.lo, b.lo)), y = f2_two_sum(x.hi, t.lo);
    hi = t.hi;
    lo = y.hi;
    er = er + (x.lo + y.lo);
  }
  __device__ __forceinline__ double result() const
  {
    const float2 h = f2_get(hi), l = f2_get(lo), e = f2_get(er);
    const ff t = two_sum(h.x, h.y), v = two_sum(l.x, l.y);
    return (double)t.hi + (((double)t.lo + (double)v.hi) + (double)__fadd_rn(v.lo, __fadd_rn(e.x, e.y)));
  }
};

__global__ void __launch_bounds__(256, 5) k_rhs_block(RhsArgs a)
{
  constexpr int Y = 4 * kElemBlock;
  __shared__ RhsShared sh;
  float *const y = sh.y, *const s_fh = sh.f, *const s_fl = sh.f + kStageNodes;
  uint16_t *const s_pos = sh.pos, *const s_start = sh.start;
  ff* const tab = sh.tab;
  int(&red)[6][8] = sh.red;
  const int tid = threadIdx.x, lane = tid & 31, lp = tid + (tid & ~31);
  const int64_t blk = blockIdx.x, p0 = blk * kElemBlock, E = a.n_elem;
  const int64_t p1 = min(p0 + lp, E - 1), p2 = min(p0 + lp + 32, E - 1);  // past the end: the last element again
  pdl_trigger();
  const int n_nodes = a.bnode_n[blk];
  const int32_t id = a.bnode[blk * kStageNodes + tid];
  // a warp's coefficient slots lie in the rows that only its own elements overwrite
  double* slot1 = reinterpret_cast<double*>(y + (lane >> 4) * kElemBlock + (lp - lane) + 4 * (lane & 15));
  double* slot2 = slot1 + kElemBlock;
  int64_t e1 = 0, e2 = 0;
  if (a.scale) e1 = a.elem_order[p1], e2 = a.elem_order[p2];
  cp_async16(s_pos + 8 * tid, a.bpos + blk * Y + 8 * tid);
  const float2 d1 = a.gdet[p1], d2 = a.gdet[p2];
  const uchar4 q1 = __ldg(a.elem_local + p1), q2 = __ldg(a.elem_local + p2);
  const int32_t out = a.bout[blk * kStageNodes + tid];
  for (int i = tid; i <= kStageNodes; i += 256) s_start[i] = a.bstart[blk * (kStageNodes + 1) + i];
  if (a.form == kRhsTable && tid < 10) tab[tid] = ff_from_double(a.mass[tid]);
  // up to here only the plan was read
  pdl_wait();
  if (a.scale) {
    coef_fetch(slot1, a.scale, e1, E);
    coef_fetch(slot2, a.scale, e2, E);
  }
  asm volatile("cp.async.commit_group;\n" ::);
  const double f = a.field ? a.field[id] : 1.0;
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  const double s1 = a.scale ? coef_slot(slot1, a.scale, e1) : 1.0, s2 = a.scale ? coef_slot(slot2, a.scale, e2) : 1.0;
  // largest and smallest biased exponents of f, s and det over the block; zeros do not
  // count for the smallest, subnormals count as exponent zero
  {
    const auto low = [](double v) { return (__double_as_longlong(v) << 1) == 0 ? 0x7ff : dexp(v); };
    const auto fexp = [](float v) { return (int)((__float_as_uint(v) >> 23) & 0xffu); };
    int m[6] = {dexp(f), 0x7ff - low(f), max(dexp(s1), dexp(s2)), 0x7ff - min(low(s1), low(s2)),
                max(fexp(d1.x), fexp(d2.x)), 0x7ff - min(fexp(d1.x), fexp(d2.x))};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      m[k] = __reduce_max_sync(0xffffffffu, m[k]);
      if (lane == 0) red[k][tid >> 5] = m[k];
    }
  }
  __syncthreads();
  int m[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) m[k] = __reduce_max_sync(0xffffffffu, red[k][lane & 7]);
  const int ef = m[0], es = m[2], ed = m[4];
  const int lf = 0x7ff - m[1], ls = 0x7ff - m[3], ld = 0x7ff - m[5];
  // (all zero: the largest is 0 and the smallest 0x7ff)
  const int spread = (ef > 0 ? ef - lf : 0) + (es > 0 ? es - ls : 0) + (ed - ld);
  if (ef == 0x7ff || es == 0x7ff || lf == 0 || ls == 0 || ed >= 0xfe || ld == 0 || spread > 70) {
    rhs_block_wide(a, sh, n_nodes, out);
    return;
  }
  {
    const ff v = ff_scaled(f, ef);
    s_fh[tid] = v.hi;
    s_fl[tid] = v.lo;
  }
  __syncthreads();
  {
    // det 2^(127 - ed): near one
    const float dscale = __uint_as_float((uint32_t)(254 - ed) << 23);
    const ff2 det = ff2_make(ff{d1.x * dscale, d1.y * dscale}, ff{d2.x * dscale, d2.y * dscale});
    const ff2 sd = ff2_mul(ff2_make(ff_scaled(s1, es), ff_scaled(s2, es)), det);
    const int i1[4] = {q1.x, q1.y, q1.z, q1.w}, i2[4] = {q2.x, q2.y, q2.z, q2.w};
    ff2 F[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      F[k] = ff2{f2_make(s_fh[i1[k]], s_fh[i2[k]]), f2_make(s_fl[i1[k]], s_fl[i2[k]])};
    ff2 v[4];
    rhs_pair(a.form, tab, F, sd, v);
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      em_pair(y, l, lp, v[l].hi);
      em_pair(y + Y, l, lp, v[l].lo);
    }
  }
  __syncthreads();
  if (tid < n_nodes) {
    const unsigned char *yh = reinterpret_cast<const unsigned char*>(y), *yl = yh + 4 * Y;
    NodeSum sum;
    const int j1 = s_start[tid + 1];
    for (int j = s_start[tid]; j < j1; j += 2) {
      const uint32_t o0 = s_pos[j], o1 = j + 1 < j1 ? s_pos[j + 1] : o0;
      const bool two = j + 1 < j1;
      sum.add(ff{em_at(yh, o0), em_at(yl, o0)}, two ? ff{em_at(yh, o1), em_at(yl, o1)} : ff{0.0f, 0.0f});
    }
    // det's power goes into the factor (2^-27 .. 1): with the others it would leave
    // scale_pow2's range
    const double unit = __longlong_as_double(__double_as_longlong(a.unit) + ((long long)(ed - 127 + a.det_exp) << 52));
    rhs_put(a, out, scale_pow2(unit * sum.result(), (ef > 0 ? ef - 1023 : 0) + (es > 0 ? es - 1023 : 0)));
  }
}

// One thread per node: the partials of a node with elements in several blocks (or of
// every node, where all are partial) in ascending block; nodes outside every element get
// zero.
__global__ void __launch_bounds__(256) k_rhs_shared(int64_t n, const int32_t* __restrict__ ptr,
                                                    const double* partial, int all_partial, double* __restrict__ b)
{
  pdl_trigger();
  const int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int q0 = d < n ? __ldg(ptr + d) : 0, q1 = d < n ? __ldg(ptr + d + 1) : 0;
  pdl_wait();  // every thread, so that this kernel's end implies the one before's
  if (d >= n || (q1 - q0 == 1 && !all_partial)) return;
  double v = 0.0;
  for (int q = q0; q < q1; ++q) v += partial[q];
  b[d] = v;
}

}  // namespace mg

using namespace mg;

extern "C" {

mg_status mg_assemble(mg_plan* plan, int32_t op, const double* d_coeff, double c, int32_t quad, int32_t prec,
                      void* d_values, void* stream)
{
  NvtxRange nvtx_range("mg_assemble");
  if (!plan) return set_error(MG_ERR_INVALID_ARG, "mg_assemble: null plan");
  return launch_assemble(plan, op, d_coeff, c, quad, prec, d_values, (cudaStream_t)stream);
}

mg_status mg_plan_status(mg_plan* p)
{
  if (!p) return set_error(MG_ERR_INVALID_ARG, "mg_plan_status: null plan");
  if (!p->on_device) return MG_OK;
  MG_CUDA(cudaDeviceSynchronize());
  uint32_t flags = 0;
  MG_CUDA(cudaMemcpy(&flags, p->d_counters + 4, sizeof(flags), cudaMemcpyDeviceToHost));
  if (flags) {
    const uint32_t zero = 0u;
    MG_TRY(copy_to_device(p->d_counters + 4, &zero, sizeof(zero)));
  }
  if (flags & 1u)
    return set_error(MG_ERR_INVALID_ARG, "assembly: the coefficient array holds NaN or Inf (the values are not usable)");
  if (flags & 2u)
    return set_error(MG_ERR_UNSUPPORTED,
                     "assembly: element-matrix scales outside 2^-96 .. 2^112, where the double-word MG_F64 "
                     "assembly keeps 1e-12 accuracy; use MG_F64_NATIVE or rescale the coefficient by a power of two");
  return MG_OK;
}

mg_status mg_assemble_host(mg_plan* p, int32_t op, const double* h_coeff, double c, int32_t quad, int32_t prec,
                           void* h_values, void* stream)
{
  NvtxRange nvtx_range("mg_assemble_host");
  if (!p || (!h_values && p->nnz > 0)) return set_error(MG_ERR_INVALID_ARG, "mg_assemble_host: null argument");
  MG_TRY(plan_device(p));
  cudaStream_t st = (cudaStream_t)stream;
  const size_t vbytes = (size_t)p->nnz * (prec_is_f64(prec) ? 8 : 4);
  if (p->tmp_values_bytes < vbytes) {
    cudaFree(p->d_tmp_values);
    p->d_tmp_values = nullptr;
    p->tmp_values_bytes = 0;
    MG_CUDA(cudaMalloc(&p->d_tmp_values, vbytes));
    p->tmp_values_bytes = vbytes;
  }
  const double* d_coeff = nullptr;
  if (h_coeff) {
    const size_t cbytes = sizeof(double) * (size_t)p->mesh->n_elem;
    if (p->tmp_coeff_bytes < cbytes) {
      cudaFree(p->d_tmp_coeff);
      p->d_tmp_coeff = nullptr;
      p->tmp_coeff_bytes = 0;
      MG_CUDA(cudaMalloc(&p->d_tmp_coeff, cbytes));
      p->tmp_coeff_bytes = cbytes;
    }
    MG_CUDA(cudaMemcpyAsync(p->d_tmp_coeff, h_coeff, cbytes, cudaMemcpyHostToDevice, st));
    d_coeff = p->d_tmp_coeff;
  }
  MG_TRY(launch_assemble(p, op, d_coeff, c, quad, prec, p->d_tmp_values, st));
  if (vbytes) MG_CUDA(cudaMemcpyAsync(h_values, p->d_tmp_values, vbytes, cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaStreamSynchronize(st));
  return mg_plan_status(p);
}

mg_status mg_apply_dirichlet(mg_plan* p, const uint8_t* d_mask, int32_t prec, void* d_values, double* d_b,
                             void* stream)
{
  NvtxRange nvtx_range("mg_apply_dirichlet");
  if (!p || !d_mask || !d_values) return set_error(MG_ERR_INVALID_ARG, "mg_apply_dirichlet: null argument");
  if (!prec_valid(prec)) return set_error(MG_ERR_INVALID_ARG, "bad precision");
  MG_TRY(plan_device(p));
  const int threads = 256;
  const int blocks = (int)((p->ndof + threads - 1) / threads);
  cudaStream_t st = (cudaStream_t)stream;
  if (blocks > 0) {
    if (prec_is_f64(prec))
      k_dirichlet<double><<<blocks, threads, 0, st>>>(p->ndof, p->d_rowptr, p->d_colind, d_mask, (double*)d_values,
                                                      d_b);
    else
      k_dirichlet<float><<<blocks, threads, 0, st>>>(p->ndof, p->d_rowptr, p->d_colind, d_mask, (float*)d_values,
                                                     d_b);
  }
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

// The element geometry cache (once per plan; the mesh is immutable).  Built on
// the caller's stream and waited for, so later calls on any stream see it.
static mg_status plan_geometry(mg_plan* p, cudaStream_t st)
{
  if (p->d_geo_det) return MG_OK;
  mg_mesh* m = p->mesh;
  const int64_t E = m->n_elem;
  if (E == 0) return MG_OK;
  float2 *det = nullptr, *cof = nullptr;
  MG_CUDA(cudaMalloc(&det, sizeof(float2) * E));
  if (cudaMalloc(&cof, sizeof(float2) * 9 * E) != cudaSuccess) {
    cudaFree(det);
    return set_error(MG_ERR_ALLOC, "element geometry cache: out of device memory");
  }
  const GeoPtrs geo{m->geo_exp ? m->d_xyz_rec : m->d_xyz, m->d_node_rec, m->d_lo_z};
  const unsigned blocks = (unsigned)((E + 255) / 256);
  const auto kernel = m->order == 1 ? (m->grid_split ? k_elem_geometry<4, true> : k_elem_geometry<4, false>)
                                    : (m->grid_split ? k_elem_geometry<10, true> : k_elem_geometry<10, false>);
  kernel<<<blocks, 128, 0, st>>>(E, p->d_dofs_morton, geo, det, cof);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(det);
    cudaFree(cof);
    return cuda_error(e, "element geometry cache");
  }
  p->d_geo_det = det;
  p->d_geo_cof = cof;
  return MG_OK;
}

mg_status mg_adjoint_grad(mg_plan* p, const double* d_u, const double* d_lambda, int32_t quad, double* d_grad,
                          void* stream)
{
  NvtxRange nvtx_range("mg_adjoint_grad");
  if (!p || !d_u || !d_lambda || (!d_grad && p->mesh->n_elem > 0))
    return set_error(MG_ERR_INVALID_ARG, "mg_adjoint_grad: null argument");
  const RefTables* t = nullptr;
  const double* d_tab = nullptr;
  MG_TRY(plan_tables(p, quad, &t, &d_tab));
  MG_TRY(plan_device(p));
  mg_mesh* m = p->mesh;
  const int threads = 256;
  const int blocks = (int)((m->n_elem + threads - 1) / threads);
  cudaStream_t st = (cudaStream_t)stream;
  MG_TRY(plan_geometry(p, st));
  if (blocks > 0) {
    if (m->order == 1)
      MG_CUDA(launch_pdl(k_adjoint<1>, blocks, threads, st, m->n_elem, p->d_elem_order, p->d_dofs_morton, p->d_geo_det,
                         p->d_geo_cof, d_tab, std::ldexp(t->wsum, m->geo_exp), d_u, d_lambda, d_grad));
    else
      MG_CUDA(launch_k(false, k_adjoint<2>, blocks, threads, st, m->n_elem, p->d_elem_order, p->d_dofs_morton, p->d_geo_det,
                         p->d_geo_cof, d_tab, std::ldexp(1.0, m->geo_exp), d_u, d_lambda, d_grad));
  }
  return MG_OK;
}

mg_status mg_assemble_rhs(mg_plan* p, const double* d_field, const double* d_elem_scale, int32_t quad, double* d_b,
                          void* stream)
{
  NvtxRange nvtx_range("mg_assemble_rhs");
  if (!p || (!d_b && p->ndof > 0)) return set_error(MG_ERR_INVALID_ARG, "mg_assemble_rhs: null argument");
  const RefTables* t = nullptr;
  const double* d_tab = nullptr;
  MG_TRY(plan_tables(p, quad, &t, &d_tab));  // validates quad
  if (p->ndof == 0) return MG_OK;
  MG_TRY(plan_device(p));
  mg_mesh* m = p->mesh;
  cudaStream_t st = (cudaStream_t)stream;
  const int threads = 256;
  const int nu = m->nb * (m->nb + 1) / 2;
  MG_TRY(plan_geometry(p, st));
  const int eblocks = (int)((m->n_elem + threads - 1) / threads);
  // A P1 mass table with one diagonal and one off-diagonal value (to a few ulps:
  // every symmetric card gives (1 + [i = j]) |T^| / 20) takes the two-value form
  // of the mat-vec in the element pass.
  int two_valued = 0;
  if (m->order == 1) {
    const double d = t->mass[0], o = t->mass[1];
    double mx = 0.0, dev = 0.0;
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < 4; ++j) {
        mx = std::max(mx, std::fabs(t->mass[4 * i + j]));
        dev = std::max(dev, std::fabs(t->mass[4 * i + j] - (i == j ? d : o)));
      }
    two_valued = dev <= 8.0 * DBL_EPSILON * mx ? 1 : 0;
  }
  if (m->order == 1 && p->nodes_staged && m->n_elem > 0) {
    // every block's nodes fit the stage: one pass
    MG_TRY(build_rhs_map(p, st));
    const double diag = t->mass[0] - t->mass[1], off = t->mass[1], ulps = 8.0 * DBL_EPSILON * std::fabs(t->mass[0]);
    const int form = !two_valued || std::fabs(off) < 0x1p-27 ? kRhsTable
                     : std::fabs(diag - off) <= ulps         ? kRhsSumPlus
                     : std::fabs(diag) <= ulps               ? kRhsSum
                                                             : kRhsTable;
    const auto overlaps = [&](const double* q, int64_t n) {
      const uintptr_t b0 = reinterpret_cast<uintptr_t>(d_b), q0 = reinterpret_cast<uintptr_t>(q);
      return q && q0 < b0 + sizeof(double) * (size_t)p->ndof && b0 < q0 + sizeof(double) * (size_t)n;
    };
    const bool in_place = overlaps(d_field, p->ndof) || overlaps(d_elem_scale, m->n_elem);
    const RhsArgs a{m->n_elem,       p->d_elem_order, p->d_bnode,       p->d_bnode_n, p->d_elem_local,
                    p->d_geo_det,    d_tab + 6 * nu,  d_field,          d_elem_scale, p->d_rhs_bpos,
                    p->d_rhs_bstart, p->d_rhs_bout,   p->d_rhs_partial, d_b,          in_place ? p->d_rhs_ptr : nullptr,
                    form,            3 * m->geo_exp,  form == kRhsTable ? 1.0 : off};
    MG_CUDA(launch_pdl(k_rhs_block, (int)p->n_blocks, 256, st, a));
    MG_CUDA(launch_pdl(k_rhs_shared, (int)((p->ndof + 255) / 256), 256, st, p->ndof, (const int32_t*)p->d_rhs_ptr,
                       (const double*)p->d_rhs_partial, in_place ? 1 : 0, d_b));
    return MG_OK;
  }
  MG_TRY(plan_rhs_map(p));
  if (eblocks > 0) {
    const double volume = std::ldexp(1.0, 3 * m->geo_exp);
    const auto elements = [&](auto kernel) {
      kernel<<<eblocks, threads, 0, st>>>(m->n_elem, p->d_elem_order, p->d_dofs_morton, p->d_geo_det, d_tab + 6 * nu,
                                          d_field, d_elem_scale, p->d_rhs_y, m->order == 1 ? two_valued : 0, volume);
    };
    if (m->order == 1) elements(m->geo_exp == 0 ? k_rhs_elem<1, false> : k_rhs_elem<1, true>);
    else elements(m->geo_exp == 0 ? k_rhs_elem<2, false> : k_rhs_elem<2, true>);
    MG_CUDA(cudaGetLastError());
  }
  // two lanes per dof when dofs sum more than 16 entries on average (P1: ~24),
  // else one (P2: ~7); measured on GB300 at P1 64^3 / 128^3 and P2 48^3
  if (m->n_elem * m->nb > 16 * p->ndof)
    k_rhs_gather<2, 8><<<(int)((p->ndof * 2 + threads - 1) / threads), threads, 0, st>>>(
        p->ndof, p->d_rhs_ptr, p->d_rhs_slot, p->d_rhs_y, d_b);
  else
    k_rhs_gather<1, 8><<<(int)((p->ndof + threads - 1) / threads), threads, 0, st>>>(
        p->ndof, p->d_rhs_ptr, p->d_rhs_slot, p->d_rhs_y, d_b);
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

}  // extern "C"
