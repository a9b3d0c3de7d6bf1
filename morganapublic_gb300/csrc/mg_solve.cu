// CSR SpMV and conjugate-gradient solvers for sm_103a.
//
// SpMV: FP64 one thread per row (the FP64 pipe, not HBM, is the narrow
// resource on GB300); FP32 a group of G lanes per row (G from the mean row
// length), values and column indices read coalesced, x gathered through the
// read-only path, the row sum reduced with xor shuffles in a fixed tree --
// deterministic.
//
// CG: the reference hands the assembled Epetra operator to Belos BlockCG
// (src/morganaTrilinos/belosBlockCG.hpp:46-82 in morganaPublic); here every
// iteration is three kernels whose scalars (alpha, beta, r.z, r.r, a done flag)
// live in device memory:
//   K1  q = A p and per-CTA partials of p.q; the last CTA to finish (integer
//       ticket) sums the partials in a fixed order and sets alpha = rz / pq;
//   K2  x += alpha p, r -= alpha q, z = D^-1 r, partials of r.z and r.r; the last
//       CTA forms beta, rz, rr and raises `done` when ||r|| <= tol ||b||;
//   K3  p = z + beta p.
// Once `done` is set the remaining kernels return at entry, so a CUDA graph of
// several iterations can be replayed without a host round trip per iteration.
// Kernels are launched with programmatic dependent launch: a kernel's launch and
// prologue overlap the tail of the one before, and it waits (griddepcontrol)
// before touching memory that kernel wrote.
// Dot products accumulate in FP64 in both precisions; the order of every
// floating-point sum is fixed, so a solve is bitwise reproducible.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>
#include <utility>
#include <vector>

#include "mg_ff.cuh"
#include "mg_internal.h"
#include "mg_launch.cuh"

namespace mg {

constexpr int kSolveThreads = 256;
constexpr int kMaxSolveBlocks = 2048;  // bound of the per-CTA partial arrays

struct CgScalars {
  double rz, alpha, beta, rr, bb, tol2, pq, rz_prev;
  double rr_anchor, delta2, pad[2];  // reliable updates: r.r at the last anchor, trigger ratio^2 (0 = off)
  int32_t done, iter, maxit, pad2;
  uint32_t ticket[4];
};
// done: 0 running, 1 converged (recursive residual), 2 breakdown (p.Ap <= 0),
// 3 maxit, 5 pause for a reliable update

// ------------------------------------------------------------ launch shape --
// GB300 issues FP64 at ~1/60 of its FP32 rate, below the rate at which HBM
// delivers doubles, so FP64 kernels are shaped to issue as few FP64 operations
// per entry as possible: one thread per CSR row (one FMA per entry, no
// shuffle-adds) with 16 entries loaded per pass and two accumulators, and
// several vector entries per thread (the block reduction tree is paid once per
// thread).  FP32 kernels use groups of 2+ lanes x 8 entries per row and more threads.
// SMs of the current device (cached per device; racing first calls store the
// same value)
static int sm_count()
{
  static std::atomic<int> cached[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  int sms = cached[dev].load(std::memory_order_relaxed);
  if (sms <= 0) {
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    cached[dev].store(sms, std::memory_order_relaxed);
  }
  return sms;
}

template <typename V> constexpr int kEntriesPerLane = sizeof(V) == 8 ? 16 : 8;

// FP64 row shape.  GB300 issues 2 FP64 FMA lanes per SM per clock, about as many
// products as HBM delivers matrix entries, and a warp instruction occupies the
// FP64 pipe whatever its active lanes: every lane of a warp issues the FMAs of
// the passes its longest row needs.  The FP64 kernels therefore prefer one
// thread per row (no shuffle-adds) with 15 entries per pass: interior P1 rows
// have 15 entries, one pass; P2 rows (19, 27 and 65 entries) take 2, 2 and 5.
// The standalone SpMV keeps two lanes per row for rows above 16 entries on
// average: there single-lane loads cost more L1 throughput than the FMAs they
// save (measured on GB300 at P2 48^3: 101 us against 99 us with two lanes of
// 16).  Two lanes of 14 (28 entries per pass: P2 rows of 19 and 27 in one pass,
// 65 in three; ~1.38 FMA slots per entry against ~1.56 with 16) measured 90.8
// against 99.0 us there.
constexpr int kF64Entries = 15;
constexpr int kF64PairEntries = 14;

// Lanes per row of the standalone SpMV: FP64 one up to 16 entries on average
// (P1), two above (P2); FP32 the smallest group of at least 2 lanes whose pass
// covers the mean row length (measured on GB300 at P1 128^3 and P2 48^3).
template <typename V>
static int row_group(int64_t rows, int64_t nnz)
{
  const double mean = rows > 0 ? (double)nnz / (double)rows : 1.0;
  if (sizeof(V) == 8) return mean > 16.0 ? 2 : 1;
  const int U = kEntriesPerLane<V>;
  for (int g = 2; g < 32; g *= 2)
    if (mean <= g * U) return g;
  return 32;
}
template <typename V>
static int row_group(const mg_plan* p)
{
  return row_group<V>(p->ndof, p->nnz);
}

// FP32 rows are streamed where the columns are 32-bit (16-bit offsets need each entry's
// row) and rows are long.
static bool stream_rows(const mg_plan* p)
{
  return !p->d_coloff && p->nnz > 16 * p->ndof && p->nnz < INT32_MAX - 1024;  // window ends in 32 bits
}

// CTAs covering every row once (G lanes per row), for the standalone SpMV.
static int spmv_full_grid(int64_t rows, int G)
{
  return (int)std::max<int64_t>(1, std::min<int64_t>((rows * G + kSolveThreads - 1) / kSolveThreads, INT32_MAX));
}

// CTAs of a row kernel with G lanes per row, at most `per_sm` per SM.
static int row_blocks(int64_t rows, int G, int per_sm)
{
  const int64_t need = (rows * G + kSolveThreads - 1) / kSolveThreads;
  const int cap = per_sm * sm_count();
  return (int)std::max<int64_t>(1, std::min<int64_t>({need, (int64_t)cap, (int64_t)kMaxSolveBlocks}));
}
static int row_blocks(const mg_plan* p, int G, int per_sm)
{
  return row_blocks(p->ndof, G, per_sm);
}
template <typename V>
static int row_blocks(const mg_plan* p, int G)
{
  return row_blocks(p, G, 8);
}

// Shape of the CG kernels: FP64 one thread per row, 15 entries per pass (the
// FP64 row shape above; measured on GB300 against two or four lanes of 8: 151
// against 159 us per iteration at P1 128^3, 136 against 142 us at P2 48^3);
// FP32 rows by 2 lanes x 8 entries (more lanes for longer rows).  FP64 at most
// 4 CTAs per SM (fewer partials for the last CTA to sum) and launched without
// programmatic dependent launch (it slowed the FP64 iteration); FP32 up to 8
// CTAs per SM, with programmatic dependent launch.
template <typename V> struct CgShape {
  static constexpr int U = sizeof(V) == 8 ? kF64Entries : 8;
  static constexpr bool pdl = sizeof(V) == 4;
  static int group(const mg_plan* p)
  {
    if (sizeof(V) == 8) return 1;
    const double mean = p->ndof > 0 ? (double)p->nnz / (double)p->ndof : 1.0;
    for (int g = 2; g < 32; g *= 2)
      if (mean <= g * U) return g;
    return 32;
  }
  static int blocks(const mg_plan* p, int G) { return row_blocks(p, G, sizeof(V) == 8 ? 4 : 8); }
};

template <typename V>
static int vec_blocks(int64_t n)
{
  const int64_t need = (n + kSolveThreads - 1) / kSolveThreads;
  const int cap = (sizeof(V) == 8 ? 2 : 4) * sm_count();
  return (int)std::max<int64_t>(1, std::min<int64_t>({need, (int64_t)cap, (int64_t)kMaxSolveBlocks}));
}

template <int G>
__device__ __forceinline__ unsigned group_mask()
{
  if constexpr (G == 32) {
    return 0xffffffffu;
  } else {
    const unsigned lane = threadIdx.x & 31u;
    return ((1u << G) - 1u) << (lane & ~(unsigned)(G - 1));
  }
}

// Dot product of one CSR row with x by a group of G lanes.  Each pass issues
// U independent loads of (column, value) per lane before any gather of x, so
// every lane keeps U requests in flight; the G partial sums are combined by xor
// shuffles in a fixed order.
// Entries u of a pass alternate between two accumulators (halving the chain of
// dependent FMAs), added at the end.
// Column of entry s of `row`: int32 columns, or 16-bit offsets col - row (the
// plan's compressed index stream).
template <typename I>
__device__ __forceinline__ int column(const I* __restrict__ ci, int s, int64_t row)
{
  if constexpr (sizeof(I) == 2) return (int)row + (int)__ldg(ci + s);
  else return __ldg(ci + s);
}

template <typename V, int G, int U = kEntriesPerLane<V>, typename I = int32_t>
__device__ __forceinline__ V row_dot(int64_t row, const int32_t* __restrict__ rp, const I* __restrict__ ci,
                                     const V* __restrict__ val, const V* __restrict__ x)
{
  const int lane = threadIdx.x & (G - 1);
  const int s0 = __ldg(rp + row), s1 = __ldg(rp + row + 1);
  V sa = V(0), sb = V(0);
  for (int base = s0 + lane; base < s1; base += G * U) {
    int c[U];
    V v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = base + u * G;
      c[u] = s < s1 ? column<I>(ci, s, row) : -1;
      v[u] = s < s1 ? __ldg(val + s) : V(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const V xv = c[u] >= 0 ? __ldg(x + c[u]) : V(0);
      if (u & 1) sb = fma(v[u], xv, sb);
      else sa = fma(v[u], xv, sa);
    }
  }
  V sum = sa + sb;
#pragma unroll
  for (int off = G / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(group_mask<G>(), sum, off, G);
  return sum;
}

// 16 rows by one warp, their entries streamed: each lane loads every 32nd entry of the
// rows (coalesced, kStreamBatch in flight before the gathers of x) and writes the
// products to the warp's window of shared memory, then two lanes sum each row's
// products from there with compensation (error-free sums of the rounded products: as
// accurate as a chain of FMAs in several accumulators, and as fast as plain sums here).
// Returns row (row0 + lane / 2)'s sum, in both of its lanes.
// Bound by the gathers of x and the L1 data path (76 % of its wavefronts; with a few
// lanes per row every load touches several rows' lines).  GB300, P2 37 x 51 x 43 in
// FP32: 39.0 -> 35.9 us at 8 CTAs per SM (42.7 at 6).  Whole warps per row (32 lanes,
// eight rows reduced together) measured 63 us.
constexpr int kStreamRows = 16, kStreamWindow = 512, kStreamBatch = 8;
__device__ __forceinline__ float rows_dot_stream(int64_t row0, int64_t n, const int32_t* __restrict__ rp,
                                                 const int32_t* __restrict__ ci, const float* __restrict__ val,
                                                 const float* __restrict__ x, float* window)
{
  const int lane = threadIdx.x & 31;
  const int64_t row = row0 + (lane >> 1);
  const int lo = __ldg(rp + min(row, n)), hi = __ldg(rp + min(row + 1, n));
  const int s0 = __shfl_sync(0xffffffffu, lo, 0), s1 = __shfl_sync(0xffffffffu, hi, 31);
  ff sum{0.0f, 0.0f};
  for (int w0 = s0; w0 < s1; w0 += kStreamWindow) {
    const int w1 = min(w0 + kStreamWindow, s1);
    for (int e0 = w0; e0 < w1; e0 += 32 * kStreamBatch) {
      int c[kStreamBatch];
      float v[kStreamBatch];
#pragma unroll
      for (int u = 0; u < kStreamBatch; ++u) {
        const int e = e0 + 32 * u + lane;
        c[u] = e < w1 ? __ldg(ci + e) : -1;
        v[u] = e < w1 ? __ldg(val + e) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < kStreamBatch; ++u)
        if (c[u] >= 0) window[e0 - w0 + 32 * u + lane] = __fmul_rn(v[u], __ldg(x + c[u]));
    }
    __syncwarp();
    const int i1 = min(hi, w1) - w0;
    for (int i = max(lo, w0) - w0 + (lane & 1); i < i1; i += 8) {
      float q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) q[u] = i + 2 * u < i1 ? window[i + 2 * u] : 0.0f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const ff t = two_sum(sum.hi, q[u]);
        sum.hi = t.hi;
        sum.lo = __fadd_rn(sum.lo, t.lo);
      }
    }
    __syncwarp();
  }
  const ff t = two_sum(sum.hi, __shfl_xor_sync(0xffffffffu, sum.hi, 1));
  const float low = __fadd_rn(t.lo, __fadd_rn(sum.lo, __shfl_xor_sync(0xffffffffu, sum.lo, 1)));
  // an Inf or NaN sum is the row's value: its errors are NaN
  return isfinite(t.hi) ? __fadd_rn(t.hi, low) : t.hi;
}

// Dot-product accumulation: FP64 for FP64 vectors; for FP32 vectors a
// double-word (float pair) sum of exact float products on the FP32 pipes, as
// accurate as FP64 here and free of FP64 operations.
template <typename V> struct Dot;
template <> struct Dot<double> {
  using A = double;
  __device__ static A zero() { return 0.0; }
  __device__ static void mac(A& s, double a, double b) { s = __fma_rn(a, b, s); }
  __device__ static A add(A a, A b) { return a + b; }
  __device__ static A shfl(A v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
  __device__ static double to_double(A v) { return v; }
};
template <> struct Dot<float> {
  using A = ff;
  __device__ static A zero() { return ff{0.0f, 0.0f}; }
  __device__ static void mac(A& s, float a, float b) { s = ff_add_s(s, two_prod(a, b)); }
  __device__ static A add(A a, A b) { return ff_add_s(a, b); }
  __device__ static A shfl(A v, int off)
  {
    return ff{__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off)};
  }
  __device__ static double to_double(A v) { return (double)v.hi + (double)v.lo; }
};

// Block-wide sum in a fixed tree; the result (as double) is valid in thread 0.
template <typename V>
__device__ __forceinline__ double block_sum(typename Dot<V>::A v, typename Dot<V>::A* sh)
{
  using D = Dot<V>;
  const int tid = threadIdx.x;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = D::add(v, D::shfl(v, off));
  if ((tid & 31) == 0) sh[tid >> 5] = v;
  __syncthreads();
  double out = 0.0;
  if (tid < 32) {
    v = tid < (kSolveThreads / 32) ? sh[tid] : D::zero();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v = D::add(v, D::shfl(v, off));
    if (tid == 0) out = D::to_double(v);
  }
  __syncthreads();
  return out;
}

// NV block-wide sums at once (each value the same fixed tree as block_sum, so
// the results are those of NV separate calls, with two barriers instead of 2 NV);
// sh holds NV * 32 values.  Valid in thread 0.
template <typename V, int NV>
__device__ __forceinline__ void block_sum_n(typename Dot<V>::A (&v)[NV], typename Dot<V>::A* sh, double (&out)[NV])
{
  using D = Dot<V>;
  const int tid = threadIdx.x;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = D::add(v[k], D::shfl(v[k], off));
  if ((tid & 31) == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[k * 32 + (tid >> 5)] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) out[k] = 0.0;
  if (tid < 32) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = tid < (kSolveThreads / 32) ? sh[k * 32 + tid] : D::zero();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = D::add(v[k], D::shfl(v[k], off));
    if (tid == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) out[k] = D::to_double(v[k]);
  }
  __syncthreads();
}

// Sum of partials[0..n) in a fixed order by one CTA (valid in thread 0).
__device__ __forceinline__ double reduce_partials(const double* partials, int n, double* sh)
{
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += kSolveThreads) v += partials[i];
  return block_sum<double>(v, sh);
}

// NV arrays of partials (partials[k * n + i]) reduced together, each in the
// order of reduce_partials; sh holds NV * 32 doubles.
template <int NV>
__device__ __forceinline__ void reduce_partials_n(const double* partials, int n, double* sh, double (&out)[NV])
{
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int i = threadIdx.x; i < n; i += kSolveThreads)
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += partials[k * n + i];
  block_sum_n<double, NV>(v, sh, out);
}

// Last-CTA detection: returns true in the single CTA that finishes last.
__device__ __forceinline__ bool last_block(uint32_t* ticket)
{
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const uint32_t t = atomicAdd(ticket, 1u);
    last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

template <typename V, int G, int U, typename I>
__global__ void __launch_bounds__(kSolveThreads) k_spmv(int64_t n, const int32_t* __restrict__ rp,
                                                        const I* __restrict__ ci, const V* __restrict__ val,
                                                        const V* __restrict__ x, V* __restrict__ y)
{
  pdl_wait();
  pdl_trigger();
  const int64_t groups = (int64_t)gridDim.x * (kSolveThreads / G);
  for (int64_t row = (blockIdx.x * (int64_t)kSolveThreads + threadIdx.x) / G; row < n; row += groups) {
    const V s = row_dot<V, G, U, I>(row, rp, ci, val, x);
    if ((threadIdx.x & (G - 1)) == 0) y[row] = s;
  }
}

// y = A x by streamed rows (rows_dot_stream), one warp per 16 rows
__global__ void __launch_bounds__(kSolveThreads, 8)
    k_spmv_stream(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                  const float* __restrict__ val, const float* __restrict__ x, float* __restrict__ y)
{
  __shared__ float window[kSolveThreads / 32][kStreamWindow];
  pdl_wait();
  pdl_trigger();
  const int64_t row0 = (blockIdx.x * (int64_t)(kSolveThreads / 32) + (threadIdx.x >> 5)) * kStreamRows;
  if (row0 >= n) return;
  const float s = rows_dot_stream(row0, n, rp, ci, val, x, window[threadIdx.x >> 5]);
  const int lane = threadIdx.x & 31;
  const int64_t row = row0 + (lane >> 1);
  if ((lane & 1) == 0 && row < n) y[row] = s;
}

// K1: q = A p, alpha = rz / (p . q)
template <typename V, int G, typename I>
__global__ void __launch_bounds__(kSolveThreads) k_cg_spmv(int64_t n, const int32_t* __restrict__ rp,
                                                           const I* __restrict__ ci, const V* __restrict__ val,
                                                           const V* __restrict__ p, V* __restrict__ q,
                                                           double* partials, CgScalars* s)
{
  using D = Dot<V>;
  __shared__ typename D::A sh[32];
  __shared__ double shd[32];
  pdl_wait();
  pdl_trigger();
  if (s->done) return;
  const int64_t groups = (int64_t)gridDim.x * (kSolveThreads / G);
  typename D::A acc = D::zero();
  for (int64_t row = (blockIdx.x * (int64_t)kSolveThreads + threadIdx.x) / G; row < n; row += groups) {
    const V v = row_dot<V, G, CgShape<V>::U, I>(row, rp, ci, val, p);
    if ((threadIdx.x & (G - 1)) == 0) {
      q[row] = v;
      D::mac(acc, p[row], v);
    }
  }
  const double b = block_sum<V>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block(&s->ticket[0])) {
    const double pq = reduce_partials(partials, gridDim.x, shd);
    if (threadIdx.x == 0) {
      s->pq = pq;
      s->alpha = s->rz / pq;
      if (!(pq > 0.0) || !isfinite(s->alpha)) s->done = 2;  // breakdown: A not SPD on the Krylov space
      s->ticket[0] = 0;
    }
  }
}

// K1 by streamed rows (rows_dot_stream), FP32 (P2 48^3, mixed solve: 49.6 -> 47.5 ms)
constexpr int kCgStreamCtas = 6;  // per SM: 40 registers; 8 spill (60.8 ms a solve), 5: 48.9 ms
__global__ void __launch_bounds__(kSolveThreads, kCgStreamCtas)
    k_cg_spmv_stream(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                     const float* __restrict__ val, const float* __restrict__ p, float* __restrict__ q, double* partials,
                     CgScalars* s)
{
  using D = Dot<float>;
  __shared__ float window[kSolveThreads / 32][kStreamWindow];
  __shared__ D::A sh[32];
  __shared__ double shd[32];
  pdl_wait();
  pdl_trigger();
  if (s->done) return;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * (kSolveThreads / 32) * kStreamRows;
  D::A acc = D::zero();
  for (int64_t row0 = (blockIdx.x * (int64_t)(kSolveThreads / 32) + (threadIdx.x >> 5)) * kStreamRows; row0 < n;
       row0 += step) {
    const float v = rows_dot_stream(row0, n, rp, ci, val, p, window[threadIdx.x >> 5]);
    const int64_t row = row0 + (lane >> 1);
    if ((lane & 1) == 0 && row < n) {
      q[row] = v;
      D::mac(acc, p[row], v);
    }
  }
  const double b = block_sum<float>(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = b;
  if (last_block(&s->ticket[0])) {
    const double pq = reduce_partials(partials, gridDim.x, shd);
    if (threadIdx.x == 0) {
      s->pq = pq;
      s->alpha = s->rz / pq;
      if (!(pq > 0.0) || !isfinite(s->alpha)) s->done = 2;
      s->ticket[0] = 0;
    }
  }
}

// K2: x += alpha p; r -= alpha q; z = D^-1 r; rz, rr, beta, convergence
template <typename V>
__global__ void __launch_bounds__(kSolveThreads) k_cg_update(int64_t n, V* __restrict__ x, V* __restrict__ r,
                                                             V* __restrict__ z, const V* __restrict__ p,
                                                             const V* __restrict__ q, const V* __restrict__ dinv,
                                                             double* partials, CgScalars* s)
{
  using D = Dot<V>;
  __shared__ typename D::A sh[2 * 32];
  __shared__ double shd[2 * 32];
  pdl_wait();
  pdl_trigger();
  if (s->done) return;
  const V alpha = (V)s->alpha;
  typename D::A prz = D::zero(), prr = D::zero();
  int64_t i0 = 0;
  if constexpr (sizeof(V) == 4) {
    // FP32: the vectors are the solver's own (16-byte aligned), four entries per step
    // (P2 48^3: update 15.3 -> 12.6 us, direction 6.5 -> 4.9 us)
    const int64_t n4 = n / 4;
    i0 = 4 * n4;
    for (int64_t i = blockIdx.x * (int64_t)kSolveThreads + threadIdx.x; i < n4;
         i += (int64_t)gridDim.x * kSolveThreads) {
      const float4 pv = reinterpret_cast<const float4*>(p)[i], qv = reinterpret_cast<const float4*>(q)[i];
      const float4 dv = reinterpret_cast<const float4*>(dinv)[i];
      float4 xv = reinterpret_cast<float4*>(x)[i], rv = reinterpret_cast<float4*>(r)[i], zv;
      float *xp = &xv.x, *rp = &rv.x, *zp = &zv.x;
      const float *pp = &pv.x, *qp = &qv.x, *dp = &dv.x;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        xp[k] += alpha * pp[k];
        rp[k] -= alpha * qp[k];
        zp[k] = dp[k] * rp[k];
        D::mac(prz, rp[k], zp[k]);
        D::mac(prr, rp[k], rp[k]);
      }
      reinterpret_cast<float4*>(x)[i] = xv;
      reinterpret_cast<float4*>(r)[i] = rv;
      reinterpret_cast<float4*>(z)[i] = zv;
    }
  }
#pragma unroll 4
  for (int64_t i = i0 + blockIdx.x * (int64_t)kSolveThreads + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kSolveThreads) {
    x[i] += alpha * p[i];
    const V ri = r[i] - alpha * q[i];
    r[i] = ri;
    const V zi = dinv[i] * ri;
    z[i] = zi;
    D::mac(prz, ri, zi);
    D::mac(prr, ri, ri);
  }
  typename D::A acc2[2] = {prz, prr};
  double bl[2];
  block_sum_n<V, 2>(acc2, sh, bl);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = bl[0];
    partials[gridDim.x + blockIdx.x] = bl[1];
  }
  if (last_block(&s->ticket[1])) {
    double tot[2];
    reduce_partials_n<2>(partials, gridDim.x, shd, tot);
    const double rz = tot[0], rr = tot[1];
    if (threadIdx.x == 0) {
      s->rz_prev = s->rz;
      s->beta = rz / s->rz;
      s->rz = rz;
      s->rr = rr;
      s->iter += 1;
      if (rr <= s->tol2 * s->bb) s->done = 1;
      else if (s->iter >= s->maxit) s->done = 3;
      else if (rr <= s->delta2 * s->rr_anchor) s->done = 5;  // K3 is skipped: the host re-anchors first
      s->ticket[1] = 0;
    }
  }
}

// K3: p = z + beta p
template <typename V>
__global__ void __launch_bounds__(kSolveThreads) k_cg_dir(int64_t n, const V* __restrict__ z, V* __restrict__ p,
                                                          const CgScalars* s)
{
  pdl_wait();
  pdl_trigger();
  if (s->done) return;
  const V beta = (V)s->beta;
  int64_t i0 = 0;
  if constexpr (sizeof(V) == 4) {
    const int64_t n4 = n / 4;
    i0 = 4 * n4;
    for (int64_t i = blockIdx.x * (int64_t)kSolveThreads + threadIdx.x; i < n4;
         i += (int64_t)gridDim.x * kSolveThreads) {
      const float4 zv = reinterpret_cast<const float4*>(z)[i];
      float4 pv = reinterpret_cast<float4*>(p)[i];
      pv = make_float4(zv.x + beta * pv.x, zv.y + beta * pv.y, zv.z + beta * pv.z, zv.w + beta * pv.w);
      reinterpret_cast<float4*>(p)[i] = pv;
    }
  }
#pragma unroll 4
  for (int64_t i = i0 + blockIdx.x * (int64_t)kSolveThreads + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kSolveThreads)
    p[i] = z[i] + beta * p[i];
}

// ------------------------------------------------------- resident CG --
// The same iteration as K1..K3 in one cooperative kernel: each CTA (one per SM) owns a
// range of rows and, where they are few enough, keeps their x, r, p, q and D^-1 in shared
// memory, so an iteration streams the matrix and exchanges p.  The dot products go
// through CTA 0: it adds the CTAs' partial sums in a fixed order and publishes the
// total, so all take the same alpha, beta and stopping decision, and a solve is
// bitwise reproducible.
//
// A value is published as two 64-bit words, each half of the double with the sum's
// epoch: a word is current when its epoch is, with no fence and no reset.  Two
// sets alternate: a CTA writes its words of the sum after next only when it has the
// next one's total, which CTA 0 publishes after reading all partials of both.
// Every wait is bounded (spin_limit polls): a CTA that gives up records done = 9 and
// returns, the others follow; the caller starts again from the x they leave with the
// three kernels.
//
// What bounds it (GB300, P1 64^3, FP64): the FP64 pipe, 22 operations a row or 10 us of
// an iteration, then the exchanges (~2 us each; every CTA polling every
// other's partials or flags took 3 and 4 us: the polls queue at a few L2 lines).
// K1..K3 took 39.6 us an iteration there and 24 us at any small size.
template <typename V> constexpr int kResidentThreads = sizeof(V) == 8 ? 512 : 768;
constexpr int kResidentIters = 512;  // iterations per launch (the host looks in between)
constexpr int kSpinLimit = 1 << 21;  // polls: a second or so
constexpr int kGaveUp = 9;           // CgScalars::done of a wait that ran out
constexpr int kMaxResidentCtas = 1024;

// Exchange buffer: 2 sets of 4 words (2 values) per CTA, 2 sets of totals on a line of
// their own, and the barrier's counter.
struct GatherBuf {
  unsigned long long* words;   // [set][cta][4]
  unsigned long long* totals;  // [set][16]
  unsigned int* count;
};
constexpr size_t kGatherBytes = sizeof(unsigned long long) * (8 * kMaxResidentCtas + 32) + 128;

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_relaxed2(const unsigned long long* p)
{
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void publish(unsigned long long* w, double v, unsigned int epoch)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
  st_relaxed(w, e | (b >> 32));
  st_relaxed(w + 1, e | (b & 0xffffffffull));
}
// Waits for NV values published at w; false when the wait ran out.
template <int NV>
__device__ __forceinline__ bool receive(const unsigned long long* w, unsigned int epoch, int spin_limit, double (&v)[NV])
{
  for (int spin = 0; spin < spin_limit; ++spin) {
    ulonglong2 x[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) x[k] = ld_relaxed2(w + 2 * k);
    bool current = true;
#pragma unroll
    for (int k = 0; k < NV; ++k)
      current = current && (unsigned int)(x[k].x >> 32) == epoch && (unsigned int)(x[k].y >> 32) == epoch;
    if (current) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        v[k] = __longlong_as_double((long long)((x[k].x << 32) | (x[k].y & 0xffffffffull)));
      return true;
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  return false;
}

// Sum over all threads of all CTAs of NV values, the same in every thread (false
// after a wait that ran out).  red: NV * blockDim.x + 8 values of shared memory; gat:
// NV * gridDim.x + NV + 1 doubles; at least 128 threads.  Per CTA: the threads' values by
// 128 threads in ascending stride, a shuffle tree, four warps' results in order; CTA 0's
// thread c waits for CTA c's partials, its warp k adds the k-th ones in a fixed order.
template <typename V, int NV>
__device__ __forceinline__ bool grid_sum(const typename Dot<V>::A (&v)[NV], typename Dot<V>::A* red, double* gat,
                                         const GatherBuf& gb, unsigned int epoch, int spin_limit, double (&total)[NV])
{
  using D = Dot<V>;
  const int tid = threadIdx.x, T = blockDim.x, lane = tid & 31, C = gridDim.x;
#pragma unroll
  for (int k = 0; k < NV; ++k) red[k * T + tid] = v[k];
  __syncthreads();
  if (tid < 128) {
    typename D::A a[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      a[k] = red[k * T + tid];
      for (int i = tid + 128; i < T; i += 128) a[k] = D::add(a[k], red[k * T + i]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
      for (int k = 0; k < NV; ++k) a[k] = D::add(a[k], D::shfl(a[k], off));
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NV; ++k) red[NV * T + 4 * k + (tid >> 5)] = a[k];
  }
  __syncthreads();
  unsigned long long* set = gb.words + (size_t)(epoch & 1u) * 4 * kMaxResidentCtas;
  unsigned long long* result = gb.totals + (epoch & 1u) * 16;
  if (tid < NV) {  // thread k publishes value k
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 4; ++w) s += D::to_double(red[NV * T + 4 * tid + w]);
    publish(set + 4 * blockIdx.x + 2 * tid, s, epoch);
  }
  bool ok = true;
  if (blockIdx.x == 0) {
    for (int c = tid; c < C; c += T) {
      double p[NV];
      ok = receive<NV>(set + 4 * c, epoch, spin_limit, p) && ok;
#pragma unroll
      for (int k = 0; k < NV; ++k) gat[k * C + c] = p[k];
    }
    ok = __syncthreads_and(ok) != 0;
    if (tid < 32 * NV) {
      const int k = tid >> 5;
      double a = 0.0;
      for (int c = lane; c < C; c += 32) a += gat[k * C + c];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) a += __shfl_xor_sync(0xffffffffu, a, off);
      if (lane == 0) {
        gat[NV * C + k] = a;
        if (ok) publish(result + 2 * k, a, epoch);
      }
    }
  } else if (tid == 0) {
    double p[NV];
    ok = receive<NV>(result, epoch, spin_limit, p);
#pragma unroll
    for (int k = 0; k < NV; ++k) gat[NV * C + k] = p[k];
  }
  ok = __syncthreads_and(ok) != 0;
#pragma unroll
  for (int k = 0; k < NV; ++k) total[k] = gat[NV * C + k];
  return ok;
}

// All CTAs' global writes before the barrier are seen by all CTAs' plain loads after it:
// one thread's fence releases the CTA's writes, and after the wait drops its stale L1
// lines.  `target`: the arrivals of all CTAs so far and at this barrier.
__device__ __forceinline__ bool grid_barrier(const GatherBuf& gb, unsigned int target, int spin_limit)
{
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(gb.count) : "memory");
    int spin = 0;
    for (; spin < spin_limit; ++spin) {
      unsigned int f;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(f) : "l"(gb.count) : "memory");
      if ((int)(f - target) >= 0) break;
    }
    ok = spin < spin_limit;
    __threadfence();
  }
  return __syncthreads_and(ok) != 0;
}

// U entries of one lane of a group of G, and their products with p
template <typename V, int G, int U, typename I>
__device__ __forceinline__ void load_entries(const I* __restrict__ ci, const V* __restrict__ val, int row, int b0, int s1,
                                             int (&c)[U], V (&v)[U])
{
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int k = b0 + u * G;
    c[u] = k < s1 ? column<I>(ci, k, row) : -1;
    v[u] = k < s1 ? __ldg(val + k) : V(0);
  }
}
template <typename V, int U>
__device__ __forceinline__ void gather_entries(const V* p, const int (&c)[U], const V (&v)[U], V& sa, V& sb)
{
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const V xv = c[u] >= 0 ? p[c[u]] : V(0);
    // one chain in FP64: its pipe is busy with the other warps meanwhile, and a second
    // accumulator costs an addition per row
    if (sizeof(V) == 4 && (u & 1)) sb = fma(v[u], xv, sb);
    else sa = fma(v[u], xv, sa);
  }
}

// Up to `iters` iterations from the state of k_cg_start (or of an earlier launch).
// p is read by plain loads (its values change within the kernel).
template <typename V, int G, int U, typename I>
__global__ void __launch_bounds__(kResidentThreads<V>, 1)
    k_cg_resident(const int32_t* __restrict__ part, int max_rows, const int32_t* __restrict__ rp,
                  const I* __restrict__ ci, const V* __restrict__ val, V* dinv, V* x, V* r, V* z, V* p, V* q_out,
                  int in_smem, GatherBuf gb, unsigned int epoch, int iters, CgScalars* s, int spin_limit)
{
  using D = Dot<V>;
  extern __shared__ __align__(16) unsigned char smem[];
  double* gat = reinterpret_cast<double*>(smem);
  typename D::A* red = reinterpret_cast<typename D::A*>(gat + 2 * gridDim.x + 2);
  int32_t* srp = reinterpret_cast<int32_t*>(red + 2 * blockDim.x + 8);  // the rows' starts
  const int tid = threadIdx.x, T = blockDim.x;
  // one reading for the CTA: another one that gave up may set it meanwhile
  if (__syncthreads_or(tid == 0 && s->done != 0)) return;
  const int r0 = part[blockIdx.x], rows = part[blockIdx.x + 1] - r0;
  // the rows' vectors: in shared memory, or where they are
  V *sx = x + r0, *sr = r + r0, *sd = dinv + r0, *sp = p + r0, *sq = q_out + r0;
  if (in_smem) {
    V* v = reinterpret_cast<V*>(srp + (max_rows + 2) / 2 * 2);
    sx = v, sr = v + max_rows, sd = v + 2 * max_rows, sp = v + 3 * max_rows, sq = v + 4 * max_rows;
    for (int i = tid; i < rows; i += T) {
      sx[i] = x[r0 + i];
      sr[i] = r[r0 + i];
      sp[i] = p[r0 + i];
      sd[i] = dinv[r0 + i];
    }
  }
  for (int i = tid; i <= rows; i += T) srp[i] = rp[r0 + i];
  double rz = s->rz, rz_prev = s->rz_prev, rr = s->rr, beta = s->beta, alpha = s->alpha, pq = s->pq;
  const double target = s->tol2 * s->bb, anchor = s->delta2 * s->rr_anchor;
  const int maxit = s->maxit;
  int iter = s->iter, done = 0;
  unsigned int arrivals = 0;  // at the barriers so far (the counter starts at zero)
  __syncthreads();
  for (int it = 0; it < iters; ++it) {
    // q = A p, p . q: the next row's first entries load while this row's gathers are
    // in flight
    typename D::A acc[1] = {D::zero()};
    {
      const int lane = tid & (G - 1), step = T / G;
      int c[U];
      V v[U];
      int base = tid / G, s0 = 0, s1 = 0;
      if (base < rows) {
        s0 = srp[base] + lane, s1 = srp[base + 1];
        load_entries<V, G, U, I>(ci, val, r0 + base, s0, s1, c, v);
      }
      while (base < rows) {
        const int next = base + step;
        int n0 = 0, n1 = 0;
        int cn[U];
        V vn[U];
        if (next < rows) n0 = srp[next] + lane, n1 = srp[next + 1];
        load_entries<V, G, U, I>(ci, val, r0 + next, n0, n1, cn, vn);
        V sa = V(0), sb = V(0);
        gather_entries<V, U>(p, c, v, sa, sb);
        for (int b0 = s0 + G * U; b0 < s1; b0 += G * U) {
          load_entries<V, G, U, I>(ci, val, r0 + base, b0, s1, c, v);
          gather_entries<V, U>(p, c, v, sa, sb);
        }
        V q = sizeof(V) == 4 ? sa + sb : sa;
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) q += __shfl_xor_sync(group_mask<G>(), q, off, G);
        if (lane == 0) {
          sq[base] = q;
          D::mac(acc[0], sp[base], q);
        }
        base = next, s0 = n0, s1 = n1;
#pragma unroll
        for (int u = 0; u < U; ++u) c[u] = cn[u], v[u] = vn[u];
      }
    }
    double tot[1];
    if (!grid_sum<V, 1>(acc, red, gat, gb, ++epoch, spin_limit, tot)) { done = kGaveUp; break; }
    pq = tot[0];
    alpha = rz / pq;
    if (!(pq > 0.0) || !isfinite(alpha)) { done = 2; break; }  // A not SPD on the Krylov space
    // x += alpha p, r -= alpha q, z = D^-1 r, r . z, r . r
    const V al = (V)alpha;
    typename D::A acc2[2] = {D::zero(), D::zero()};
    for (int i = tid; i < rows; i += T) {
      sx[i] += al * sp[i];
      const V ri = sr[i] - al * sq[i];
      sr[i] = ri;
      const V zi = sd[i] * ri;
      sq[i] = zi;
      D::mac(acc2[0], ri, zi);
      D::mac(acc2[1], ri, ri);
    }
    double tot2[2];
    if (!grid_sum<V, 2>(acc2, red, gat, gb, ++epoch, spin_limit, tot2)) { done = kGaveUp; break; }
    rz_prev = rz;
    beta = tot2[0] / rz;
    rz = tot2[0];
    rr = tot2[1];
    ++iter;
    if (rr <= target) done = 1;
    else if (iter >= maxit) done = 3;
    else if (rr <= anchor) done = 5;  // the host re-anchors, then forms the direction
    if (done) break;
    // p = z + beta p
    const V be = (V)beta;
    for (int i = tid; i < rows; i += T) {
      const V pi = sq[i] + be * sp[i];
      sp[i] = pi;
      p[r0 + i] = pi;
    }
    if (!grid_barrier(gb, arrivals += gridDim.x, spin_limit)) { done = kGaveUp; break; }
  }
  for (int i = tid; i < rows; i += T) {
    if (in_smem) {
      x[r0 + i] = sx[i];
      r[r0 + i] = sr[i];
    }
    z[r0 + i] = sd[i] * sr[i];
  }
  if (tid == 0 && (blockIdx.x == 0 || done == kGaveUp)) {
    if (blockIdx.x == 0) {
      s->rz = rz;
      s->rz_prev = rz_prev;
      s->rr = rr;
      s->beta = beta;
      s->alpha = alpha;
      s->pq = pq;
      s->iter = iter;
    }
    s->done = done;
  }
}

// Start of a solve: r = b - A x (or r = b when x is zero), z = D^-1 r, p = z,
// D^-1 from the diagonal, partials of r.z, r.r, b.b.
template <typename V, int G>
__global__ void __launch_bounds__(kSolveThreads) k_cg_start(int64_t n, const int32_t* __restrict__ rp,
                                                            const int32_t* __restrict__ ci, const V* __restrict__ val,
                                                            const int32_t* __restrict__ diag, const V* __restrict__ b,
                                                            const V* __restrict__ x, int zero_x, int jacobi,
                                                            V* __restrict__ r, V* __restrict__ z, V* __restrict__ p,
                                                            V* __restrict__ dinv, double* partials, CgScalars* s)
{
  using D = Dot<V>;
  __shared__ typename D::A sh[3 * 32];
  __shared__ double shd[3 * 32];
  const int64_t groups = (int64_t)gridDim.x * (kSolveThreads / G);
  typename D::A prz = D::zero(), prr = D::zero(), pbb = D::zero();
  for (int64_t row = (blockIdx.x * (int64_t)kSolveThreads + threadIdx.x) / G; row < n; row += groups) {
    V ax = V(0);
    if (!zero_x) ax = row_dot<V, G, CgShape<V>::U>(row, rp, ci, val, x);
    if ((threadIdx.x & (G - 1)) == 0) {
      const V dv = val[diag[row]];
      const V di = (jacobi && dv != V(0)) ? V(1) / dv : V(1);
      const V ri = b[row] - ax;
      const V zi = di * ri;
      dinv[row] = di;
      r[row] = ri;
      z[row] = zi;
      p[row] = zi;
      D::mac(prz, ri, zi);
      D::mac(prr, ri, ri);
      D::mac(pbb, b[row], b[row]);
    }
  }
  typename D::A acc3[3] = {prz, prr, pbb};
  double bl[3];
  block_sum_n<V, 3>(acc3, sh, bl);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = bl[0];
    partials[gridDim.x + blockIdx.x] = bl[1];
    partials[2 * gridDim.x + blockIdx.x] = bl[2];
  }
  if (last_block(&s->ticket[2])) {
    double tot[3];
    reduce_partials_n<3>(partials, gridDim.x, shd, tot);
    const double rz = tot[0], rr = tot[1], bb = tot[2];
    if (threadIdx.x == 0) {
      s->rz = rz;
      s->rr = rr;
      s->bb = bb > 0.0 ? bb : 1.0;
      s->iter = 0;
      s->done = (rr <= s->tol2 * s->bb) ? 1 : 0;
      s->ticket[2] = 0;
    }
  }
}

// Refinement residual: r64 = b - A64 x, rr = r64 . r64 (last CTA); the scaled
// FP32 right-hand side r32 = r64 / ||r64|| is then written by k_scale_cast.
template <int G>
__global__ void __launch_bounds__(kSolveThreads) k_residual64(int64_t n, const int32_t* __restrict__ rp,
                                                              const int32_t* __restrict__ ci,
                                                              const double* __restrict__ val,
                                                              const double* __restrict__ b,
                                                              const double* __restrict__ x, double* __restrict__ r,
                                                              double* partials, CgScalars* s)
{
  __shared__ double sh[2 * 32];
  const int64_t groups = (int64_t)gridDim.x * (kSolveThreads / G);
  double prr = 0.0, pbb = 0.0;
  for (int64_t row = (blockIdx.x * (int64_t)kSolveThreads + threadIdx.x) / G; row < n; row += groups) {
    const double ax = row_dot<double, G, CgShape<double>::U>(row, rp, ci, val, x);
    if ((threadIdx.x & (G - 1)) == 0) {
      const double ri = b[row] - ax;
      r[row] = ri;
      prr = __fma_rn(ri, ri, prr);
      pbb = __fma_rn(b[row], b[row], pbb);
    }
  }
  double acc2[2] = {prr, pbb}, bl[2];
  block_sum_n<double, 2>(acc2, sh, bl);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = bl[0];
    partials[gridDim.x + blockIdx.x] = bl[1];
  }
  if (last_block(&s->ticket[3])) {
    double tot[2];
    reduce_partials_n<2>(partials, gridDim.x, sh, tot);
    const double rr = tot[0], bb = tot[1];
    if (threadIdx.x == 0) {
      s->rr = rr;
      s->bb = bb > 0.0 ? bb : 1.0;
      s->ticket[3] = 0;
    }
  }
}

__global__ void k_scale_cast(int64_t n, const double* r, double scale, float* r32, float* d32)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    r32[i] = (float)(r[i] * scale);
    d32[i] = 0.0f;
  }
}

// Reliable update, part 1: x64 += x32, x32 = 0.
__global__ void k_anchor_x(int64_t n, double* __restrict__ x, float* __restrict__ x32)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    x[i] += (double)x32[i];
    x32[i] = 0.0f;
  }
}

// Reliable update, part 2 (after r64 = b - A64 x): r32 = r64, z32 = D^-1 r32,
// r.z and r.r of the replaced residual; the last CTA forms beta with the r.z
// of the iteration that paused, re-anchors and resumes (K3 then runs).
__global__ void __launch_bounds__(kSolveThreads) k_anchor_r(int64_t n, const double* __restrict__ r64,
                                                            float* __restrict__ r, float* __restrict__ z,
                                                            const float* __restrict__ dinv, double* partials,
                                                            CgScalars* s)
{
  using D = Dot<float>;
  __shared__ D::A sh[2 * 32];
  __shared__ double shd[2 * 32];
  D::A prz = D::zero(), prr = D::zero();
  for (int64_t i = blockIdx.x * (int64_t)kSolveThreads + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kSolveThreads) {
    const float ri = (float)r64[i];
    const float zi = dinv[i] * ri;
    r[i] = ri;
    z[i] = zi;
    D::mac(prz, ri, zi);
    D::mac(prr, ri, ri);
  }
  D::A acc2[2] = {prz, prr};
  double bl[2];
  block_sum_n<float, 2>(acc2, sh, bl);
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = bl[0];
    partials[gridDim.x + blockIdx.x] = bl[1];
  }
  if (last_block(&s->ticket[1])) {
    double tot[2];
    reduce_partials_n<2>(partials, gridDim.x, shd, tot);
    const double rz = tot[0], rr = tot[1];
    if (threadIdx.x == 0) {
      s->beta = rz / s->rz_prev;
      s->rz = rz;
      s->rr = rr;
      s->rr_anchor = rr;
      s->done = 0;
      s->ticket[1] = 0;
    }
  }
}

#define MG_DISPATCH_G(G, ...)                                \
  switch (G) {                                               \
    case 32: { constexpr int g = 32; __VA_ARGS__; } break;   \
    case 16: { constexpr int g = 16; __VA_ARGS__; } break;   \
    case 8: { constexpr int g = 8; __VA_ARGS__; } break;     \
    case 4: { constexpr int g = 4; __VA_ARGS__; } break;     \
    case 2: { constexpr int g = 2; __VA_ARGS__; } break;     \
    default: { constexpr int g = 1; __VA_ARGS__; } break;    \
  }

mg_status launch_spmv(mg_plan* p, int prec, const void* vals, const void* x, void* y, cudaStream_t st)
{
  if (!prec_valid(prec)) return set_error(MG_ERR_INVALID_ARG, "bad precision");
  if (p->ndof == 0) return MG_OK;
  if (!vals || !x || !y) return set_error(MG_ERR_INVALID_ARG, "mg_spmv: null argument");
  MG_TRY(plan_device(p));
  if (prec_is_f64(prec)) {
    // FP64: one thread per row, a CTA for every 256 rows, no grid-stride loop
    // (measured on GB300 at P1 128^3: 84.7 us against 88.7 us with 8 CTAs per SM
    // and a grid-stride loop)
    const int G = row_group<double>(p), nb = spmv_full_grid(p->ndof, G);
    const double *v = (const double*)vals, *xx = (const double*)x;
    double* yy = (double*)y;
    const int32_t* rp = p->d_rowptr;
    const int64_t n = p->ndof;
    if (p->d_coloff) {
      const int16_t* c = p->d_coloff;
      if (G == 1) launch_pdl(k_spmv<double, 1, kF64Entries, int16_t>, nb, kSolveThreads, st, n, rp, c, v, xx, yy);
      else launch_pdl(k_spmv<double, 2, kF64PairEntries, int16_t>, nb, kSolveThreads, st, n, rp, c, v, xx, yy);
    } else {
      const int32_t* c = p->d_colind;
      if (G == 1) launch_pdl(k_spmv<double, 1, kF64Entries, int32_t>, nb, kSolveThreads, st, n, rp, c, v, xx, yy);
      else launch_pdl(k_spmv<double, 2, kF64PairEntries, int32_t>, nb, kSolveThreads, st, n, rp, c, v, xx, yy);
    }
  } else if (stream_rows(p)) {
    const int64_t warps = (p->ndof + kStreamRows - 1) / kStreamRows, per = kSolveThreads / 32;
    launch_pdl(k_spmv_stream, (int)((warps + per - 1) / per), kSolveThreads, st, p->ndof, (const int32_t*)p->d_rowptr,
               (const int32_t*)p->d_colind, (const float*)vals, (const float*)x, (float*)y);
  } else {
    const int G = row_group<float>(p), nb = row_blocks<float>(p, G);
    if (p->d_coloff) {
      MG_DISPATCH_G(G, (launch_pdl(k_spmv<float, g, kEntriesPerLane<float>, int16_t>, nb, kSolveThreads, st, p->ndof,
                                   (const int32_t*)p->d_rowptr, (const int16_t*)p->d_coloff, (const float*)vals,
                                   (const float*)x, (float*)y)));
    } else {
      MG_DISPATCH_G(G, (launch_pdl(k_spmv<float, g, kEntriesPerLane<float>, int32_t>, nb, kSolveThreads, st, p->ndof,
                                   (const int32_t*)p->d_rowptr, (const int32_t*)p->d_colind, (const float*)vals,
                                   (const float*)x, (float*)y)));
    }
  }
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

// y = A x for a CSR matrix of any shape: the standalone SpMV kernel with the
// lane group of the FP64 path, int32 columns.
mg_status launch_spmv_csr(int64_t rows, int64_t nnz, const int32_t* rowptr, const int32_t* colind,
                          const double* vals, const double* x, double* y, cudaStream_t st)
{
  if (rows == 0) return MG_OK;
  const int G = row_group<double>(rows, nnz), nb = row_blocks(rows, G, 8);
  if (G == 1)
    launch_pdl(k_spmv<double, 1, kF64Entries, int32_t>, nb, kSolveThreads, st, rows, rowptr, colind, vals, x, y);
  else
    launch_pdl(k_spmv<double, 2, kF64PairEntries, int32_t>, nb, kSolveThreads, st, rows, rowptr, colind, vals, x,
               y);
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}


// Workspace of one CG run over vectors of type V.
template <typename V>
struct CgWork {
  V *r, *z, *p, *q, *dinv;
  double* partials;  // 3 * kMaxSolveBlocks
  CgScalars* s;
  GatherBuf gather;
};

template <typename V>
static size_t cg_work_bytes(int64_t n)
{
  const size_t vec = ((size_t)n * sizeof(V) + 255) / 256 * 256;
  return 5 * vec + 3 * kMaxSolveBlocks * sizeof(double) + kGatherBytes + 256;
}

template <typename V>
static CgWork<V> cg_work_carve(void* base, int64_t n)
{
  char* c = (char*)base;
  const size_t vec = ((size_t)n * sizeof(V) + 255) / 256 * 256;
  CgWork<V> w;
  w.s = (CgScalars*)c;
  c += 256;
  w.partials = (double*)c;
  c += 3 * kMaxSolveBlocks * sizeof(double);
  w.gather.words = (unsigned long long*)c;
  w.gather.totals = w.gather.words + 8 * kMaxResidentCtas;
  w.gather.count = (unsigned int*)(w.gather.totals + 32);
  c += kGatherBytes;
  w.r = (V*)c; c += vec;
  w.z = (V*)c; c += vec;
  w.p = (V*)c; c += vec;
  w.q = (V*)c; c += vec;
  w.dinv = (V*)c;
  return w;
}

// Smallest reliable-update trigger ratio of the mixed-precision CG.
constexpr double kMinAnchorRatio = 1e-3;

// Iterations per replay of the captured CG graph between two host checks.
constexpr int kGraphIters = 16;

// Shape of the resident CG.  The vectors go to shared memory only while that leaves most
// of the SM's 256 KB to L1, which the matrix stream and the gathers of p need (measured:
// 213 KB of vectors at P2 48^3 left 15 KB of lines, 95 ms a solve).
constexpr size_t kResidentVectors = 112 * 1024;
// ... and only for systems that stay in L2: streaming from HBM one CTA per SM has too few
// loads in flight (P2 48^3 in FP32, 222 MB: 103 us an iteration against 81 us with the
// three kernels; P2 36^3, 94 MB: 44.2 against 45.3; P1 64^3 in FP64, 53 MB: 23.6 against 39.6).
constexpr int64_t kResidentBytes = 100ll << 20;
template <typename V>
static size_t resident_smem(int ctas, int threads, int max_rows, bool vectors)
{
  return (2 * ctas + 2) * sizeof(double) + sizeof(typename Dot<V>::A) * (2 * threads + 8) +
         sizeof(int32_t) * (size_t)((max_rows + 2) / 2 * 2) + (vectors ? 5 * sizeof(V) * (size_t)max_rows : 0);
}
// Threads per CTA: the passes over the rows evenly filled.
template <typename V>
static int resident_threads(int max_rows, int G)
{
  const int64_t units = (int64_t)max_rows * G, most = kResidentThreads<V>;
  const int64_t passes = std::max<int64_t>(1, (units + most - 1) / most);
  const int64_t t = ((units + passes - 1) / passes + 31) / 32 * 32;
  return (int)std::min(most, std::max<int64_t>(t, 128));
}
// The plan's row partition for vectors of type V: as many CTAs as SMs, at least 256 rows
// each on average, with equal shares of the rows' cost: FP64 the FMA slots of the row's
// passes (U entries each) and 8 of the vector updates; FP32 its entries and 12.
template <typename V>
static mg_status resident_partition(mg_plan* p, const RowPartition** out)
{
  std::lock_guard<std::mutex> lock(p->upload_mu);
  RowPartition& rp = p->cg_part[sizeof(V) == 8 ? 0 : 1];
  *out = &rp;
  if (rp.ctas != 0) return MG_OK;
  const int64_t n = p->ndof;
  const int ctas = (int)std::max<int64_t>(1, std::min<int64_t>({(int64_t)sm_count(), (n + 255) / 256, (int64_t)kMaxResidentCtas}));
  const auto cost = [&](int64_t r) -> int64_t {
    const int64_t len = p->rowptr[r + 1] - p->rowptr[r];
    constexpr int U = CgShape<V>::U;
    return sizeof(V) == 8 ? U * std::max<int64_t>(1, (len + U - 1) / U) + 8 : len + 12;
  };
  int64_t total = 0;
  for (int64_t r = 0; r < n; ++r) total += cost(r);
  std::vector<int32_t> part(ctas + 1, (int32_t)n);
  part[0] = 0;
  int64_t sum = 0;
  int c = 1;
  for (int64_t r = 0; r < n && c < ctas; ++r) {
    sum += cost(r);
    while (c < ctas && sum * ctas >= total * c) part[c++] = (int32_t)(r + 1);
  }
  int max_rows = 0;
  for (int k = 0; k < ctas; ++k) max_rows = std::max(max_rows, part[k + 1] - part[k]);
  int32_t* d = nullptr;
  MG_CUDA(cudaMalloc(&d, sizeof(int32_t) * part.size()));
  const mg_status copied = copy_to_device(d, part.data(), sizeof(int32_t) * part.size());
  if (copied != MG_OK) {
    cudaFree(d);
    return copied;
  }
  rp.d_rows = d;
  rp.max_rows = max_rows;
  rp.ctas = ctas;
  return MG_OK;
}

template <typename V, int G, int U, typename I>
static cudaError_t resident_launch(mg_plan* p, const RowPartition* part, const V* vals, V* x, CgWork<V>& w, int threads, size_t smem,
                                 bool in_smem, unsigned int epoch, cudaStream_t st)
{
  const auto kernel = k_cg_resident<V, G, U, I>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)part->ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const I* ci;
  if constexpr (sizeof(I) == 2) ci = p->d_coloff;
  else ci = p->d_colind;
  return cudaLaunchKernelEx(&cfg, kernel, (const int32_t*)part->d_rows, part->max_rows, (const int32_t*)p->d_rowptr, ci,
                            vals, w.dinv, x, w.r, w.z, w.p, w.q, in_smem ? 1 : 0, w.gather, epoch, kResidentIters, w.s, kSpinLimit);
}
// Whether all CTAs of the kernel can be resident at once on the whole device.
template <typename V, int G, int U, typename I>
static mg_status resident_fits(int ctas, int threads, size_t smem, bool* fits)
{
  const auto kernel = k_cg_resident<V, G, U, I>;
  static std::once_flag once[64];
  MG_TRY(allow_smem(kernel, kResidentVectors, once));  // smem <= kResidentVectors (cg_iterate)
  int per_sm = 0;
  MG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  *fits = (int64_t)per_sm * sm_count() >= ctas;
  return MG_OK;
}

// Runs CG on A (vals) from the state set up by k_cg_start until `done`: by the resident
// kernel, or by the three kernels where the system is too large for it or its launch is
// refused (a process or stream that has a part of the SMs), from the state it is in.
// *try_resident: whether the kernel may be tried; false after a wait of it ran out, done is
// kGaveUp then and x holds every row's value of one of the iterations.
template <typename V>
static mg_status cg_iterate(mg_plan* p, const V* vals, V* x, CgWork<V>& w, int G, int nb, int maxit,
                            cudaStream_t st, CgScalars* h_s, unsigned int* epoch, bool* try_resident)
{
  const int64_t n = p->ndof;
  const int vb = vec_blocks<V>(n);
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool use_graph = true;
  cudaStreamCaptureStatus cs;
  MG_CUDA(cudaStreamIsCapturing(st, &cs));
  constexpr int U = CgShape<V>::U;
  const int64_t bytes = p->nnz * (int64_t)(sizeof(V) + (p->d_coloff ? 2 : 4)) + 6 * n * (int64_t)sizeof(V);
  bool resident = *try_resident && bytes <= kResidentBytes && cs == cudaStreamCaptureStatusNone;
  const RowPartition* part = nullptr;
  int threads = 0;
  bool in_smem = false;
  size_t smem = 0;
  if (resident) {
    MG_TRY(resident_partition<V>(p, &part));
    threads = resident_threads<V>(part->max_rows, G);
    in_smem = resident_smem<V>(part->ctas, threads, part->max_rows, true) <= kResidentVectors;
    smem = resident_smem<V>(part->ctas, threads, part->max_rows, in_smem);
    resident = smem <= kResidentVectors;
  }
  const auto on_kernel = [&](auto&& f) -> mg_status {  // f(lanes per row, index type) of this system
    if constexpr (sizeof(V) == 8) {
      return p->d_coloff ? f(std::integral_constant<int, 1>(), int16_t()) : f(std::integral_constant<int, 1>(), int32_t());
    } else {
      MG_DISPATCH_G(G, return p->d_coloff ? f(std::integral_constant<int, g>(), int16_t())
                                          : f(std::integral_constant<int, g>(), int32_t()))
    }
    return MG_OK;
  };
  if (resident)
    MG_TRY(on_kernel([&](auto g, auto i) {
      return resident_fits<V, decltype(g)::value, U, decltype(i)>(part->ctas, threads, smem, &resident);
    }));
  if (resident) {
    for (;;) {
      MG_CUDA(cudaMemsetAsync(w.gather.count, 0, sizeof(unsigned int), st));
      cudaError_t refused = cudaSuccess;
      MG_TRY(on_kernel([&](auto g, auto i) {
        refused = resident_launch<V, decltype(g)::value, U, decltype(i)>(p, part, vals, x, w, threads, smem, in_smem, *epoch, st);
        return MG_OK;
      }));
      if (refused != cudaSuccess) {
        cudaGetLastError();  // an error of the context comes up again below
        break;
      }
      *epoch += 2 * kResidentIters;
      MG_CUDA(cudaMemcpyAsync(h_s, w.s, sizeof(CgScalars), cudaMemcpyDeviceToHost, st));
      MG_CUDA(cudaStreamSynchronize(st));
      if (h_s->done == kGaveUp) *try_resident = false;
      if (h_s->done) return MG_OK;
    }
  }
  if (cs != cudaStreamCaptureStatusNone || st == nullptr) use_graph = false;  // no nested capture; legacy stream cannot capture
  constexpr bool pdl = CgShape<V>::pdl;
  auto body = [&]() {
    if constexpr (sizeof(V) == 4) {
      if (stream_rows(p))
        launch_k(pdl, k_cg_spmv_stream, row_blocks((n + kStreamRows - 1) / kStreamRows, 32, kCgStreamCtas), kSolveThreads, st, n,
                 (const int32_t*)p->d_rowptr, (const int32_t*)p->d_colind, vals, (const float*)w.p, w.q, w.partials,
                 w.s);
    }
    if (sizeof(V) == 4 && stream_rows(p)) {
      // launched above
    } else if (p->d_coloff) {
      MG_DISPATCH_G(G, (launch_k(pdl, k_cg_spmv<V, g, int16_t>, nb, kSolveThreads, st, n,
                                 (const int32_t*)p->d_rowptr, (const int16_t*)p->d_coloff, vals, (const V*)w.p, w.q,
                                 w.partials, w.s)));
    } else {
      MG_DISPATCH_G(G, (launch_k(pdl, k_cg_spmv<V, g, int32_t>, nb, kSolveThreads, st, n,
                                 (const int32_t*)p->d_rowptr, (const int32_t*)p->d_colind, vals, (const V*)w.p, w.q,
                                 w.partials, w.s)));
    }
    launch_k(pdl, k_cg_update<V>, vb, kSolveThreads, st, n, x, w.r, w.z, (const V*)w.p, (const V*)w.q,
             (const V*)w.dinv, w.partials, w.s);
    launch_k(pdl, k_cg_dir<V>, vb, kSolveThreads, st, n, (const V*)w.z, w.p, (const CgScalars*)w.s);
  };
  if (use_graph) {
    MG_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    for (int k = 0; k < kGraphIters; ++k) body();
    MG_CUDA(cudaStreamEndCapture(st, &graph));
    MG_CUDA(cudaGraphInstantiate(&exec, graph, 0));
  }
  mg_status status = MG_OK;
  for (int launched = 0;; launched += kGraphIters) {
    if (use_graph) {
      cudaError_t e = cudaGraphLaunch(exec, st);
      if (e != cudaSuccess) { status = cuda_error(e, "cudaGraphLaunch"); break; }
    } else {
      for (int k = 0; k < kGraphIters; ++k) body();
      cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) { status = cuda_error(e, "cg kernels"); break; }
    }
    cudaError_t e = cudaMemcpyAsync(h_s, w.s, sizeof(CgScalars), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) { status = cuda_error(e, "cg scalars"); break; }
    if (h_s->done) break;
    if (launched + kGraphIters > maxit + kGraphIters) break;
  }
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  return status;
}

template <typename V>
static mg_status cg_start(mg_plan* p, const V* vals, const V* b, const V* x, int zero_x, int jacobi,
                          double tol, int maxit, CgWork<V>& w, int G, int nb, cudaStream_t st)
{
  CgScalars init{};
  init.tol2 = tol * tol;
  init.maxit = maxit;
  MG_CUDA(cudaMemcpyAsync(w.s, &init, sizeof(CgScalars), cudaMemcpyHostToDevice, st));
  MG_CUDA(cudaMemsetAsync(w.gather.words, 0, kGatherBytes, st));  // no epoch is current
  const int64_t n = p->ndof;
  MG_DISPATCH_G(G, (k_cg_start<V, g><<<nb, kSolveThreads, 0, st>>>(n, p->d_rowptr, p->d_colind, vals, p->d_diag, b,
                                                                     x, zero_x, jacobi, w.r, w.z, w.p, w.dinv,
                                                                     w.partials, w.s)));
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

// ||r|| / ||b|| from the squared norms; with b = 0 the absolute residual ||r||
// (0 when r = 0 as well), never NaN
static double rel_residual(double rr, double bb)
{
  if (rr == 0.0) return 0.0;
  return bb > 0.0 ? std::sqrt(rr / bb) : std::sqrt(rr);
}

// ------------------------------------------------- CG without allocation --
// Work space of mg_cg_solve_noalloc: a file-scope device array (16 MiB, 256-byte
// aligned), enough for the CG vectors of MG_CG_NOALLOC_MAX_NDOF dofs.  Host code
// must not use the symbol itself as a pointer: its device address is looked up
// once per device with cudaGetSymbolAddress.
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
static_assert(MG_CG_NOALLOC_MAX_NDOF > 0, "limit");

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mutex;
static void* g_noalloc_ptr[kNoAllocMaxDevices] = {};

static mg_status noalloc_scratch(void** out)
{
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return set_error(MG_ERR_UNSUPPORTED, "device index above 63");
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev]) {
    void* ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    g_noalloc_ptr[dev] = ptr;
  }
  *out = g_noalloc_ptr[dev];
  return MG_OK;
}

}  // namespace mg

using namespace mg;

extern "C" {

mg_status mg_cg_solve_noalloc(mg_plan* p, const double* d_values, const double* d_b, double* d_x, double rtol,
                              int32_t maxit, int32_t precond, mg_cg_info* info, void* stream)
{
  NvtxRange nvtx_range("mg_cg_solve_noalloc");
  if (!p || !d_values || !d_b || !d_x) return set_error(MG_ERR_INVALID_ARG, "mg_cg_solve_noalloc: null argument");
  if (!(rtol > 0.0) || maxit < 0)
    return set_error(MG_ERR_INVALID_ARG, "mg_cg_solve_noalloc: rtol must be > 0, maxit >= 0");
  if (p->ndof > MG_CG_NOALLOC_MAX_NDOF)
    return set_error(MG_ERR_SIZE, "mg_cg_solve_noalloc: ndof " + std::to_string(p->ndof) +
                                      " exceeds MG_CG_NOALLOC_MAX_NDOF (" +
                                      std::to_string(MG_CG_NOALLOC_MAX_NDOF) + ") of the fixed work array");
  if (!p->on_device)
    return set_error(MG_ERR_INVALID_ARG,
                     "mg_cg_solve_noalloc: the plan is not resident on the device yet (make one regular GPU call "
                     "on it first, e.g. mg_assemble)");
  if (cg_work_bytes<double>(p->ndof) > kNoAllocScratchBytes)
    return set_error(MG_ERR_SIZE, "mg_cg_solve_noalloc: work space above the fixed array");
  // the scratch address below is the current device's; the plan's arrays must be there too
  MG_TRY(check_device(p->mesh->device, "mg_cg_solve_noalloc: the plan"));
  void* base = nullptr;
  MG_TRY(noalloc_scratch(&base));
  cudaStream_t st = (cudaStream_t)stream;
  CgWork<double> w = cg_work_carve<double>(base, p->ndof);
  const int G = CgShape<double>::group(p), nb = CgShape<double>::blocks(p, G);
  const int64_t n = p->ndof;
  const int vb = vec_blocks<double>(n);
  const auto t0 = std::chrono::steady_clock::now();
  // cg_start writes the scalars from the host (tickets and flags start at zero)
  MG_TRY(cg_start<double>(p, d_values, d_b, d_x, 0, precond == MG_PREC_JACOBI, rtol, maxit, w, G, nb, st));
  CgScalars hs{};
  for (int launched = 0;; launched += kGraphIters) {
    for (int k = 0; k < kGraphIters; ++k) {
      constexpr bool pdl = CgShape<double>::pdl;
      if (p->d_coloff) {
        MG_DISPATCH_G(G, (launch_k(pdl, k_cg_spmv<double, g, int16_t>, nb, kSolveThreads, st, n,
                                   (const int32_t*)p->d_rowptr, (const int16_t*)p->d_coloff, d_values,
                                   (const double*)w.p, w.q, w.partials, w.s)));
      } else {
        MG_DISPATCH_G(G, (launch_k(pdl, k_cg_spmv<double, g, int32_t>, nb, kSolveThreads, st, n,
                                   (const int32_t*)p->d_rowptr, (const int32_t*)p->d_colind, d_values,
                                   (const double*)w.p, w.q, w.partials, w.s)));
      }
      launch_k(pdl, k_cg_update<double>, vb, kSolveThreads, st, n, d_x, w.r, w.z, (const double*)w.p,
               (const double*)w.q, (const double*)w.dinv, w.partials, w.s);
      launch_k(pdl, k_cg_dir<double>, vb, kSolveThreads, st, n, (const double*)w.z, w.p, (const CgScalars*)w.s);
    }
    MG_CUDA(cudaGetLastError());
    MG_CUDA(cudaMemcpyAsync(&hs, w.s, sizeof(CgScalars), cudaMemcpyDeviceToHost, st));
    MG_CUDA(cudaStreamSynchronize(st));
    if (hs.done) break;
    if (launched + kGraphIters > maxit + kGraphIters) break;
  }
  const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  if (info) {
    info->iterations = hs.iter;
    info->outer_iterations = 0;
    info->converged = hs.done == 1;
    info->rel_residual = rel_residual(hs.rr, hs.bb);
    info->seconds = secs;
  }
  if (hs.done == 2) return set_error(MG_ERR_NOT_CONVERGED, "CG breakdown: p.Ap <= 0");
  if (hs.done != 1) return set_error(MG_ERR_NOT_CONVERGED, "CG reached maxit");
  return MG_OK;
}

mg_status mg_spmv(mg_plan* plan, int32_t prec, const void* d_values, const void* d_x, void* d_y, void* stream)
{
  NvtxRange nvtx_range("mg_spmv");
  if (!plan) return set_error(MG_ERR_INVALID_ARG, "mg_spmv: null plan");
  return launch_spmv(plan, prec, d_values, d_x, d_y, (cudaStream_t)stream);
}

mg_status mg_cg_solve(mg_plan* p, const double* d_values, const double* d_b, double* d_x, double rtol,
                      int32_t maxit, int32_t precond, mg_cg_info* info, void* stream)
{
  NvtxRange nvtx_range("mg_cg_solve");
  if (!p || !d_values || !d_b || !d_x) return set_error(MG_ERR_INVALID_ARG, "mg_cg_solve: null argument");
  if (!(rtol > 0.0) || maxit < 0) return set_error(MG_ERR_INVALID_ARG, "mg_cg_solve: rtol must be > 0, maxit >= 0");
  MG_TRY(plan_device(p));
  cudaStream_t st = (cudaStream_t)stream;
  void* base = nullptr;
  MG_TRY(plan_work(p, cg_work_bytes<double>(p->ndof), &base));
  CgWork<double> w = cg_work_carve<double>(base, p->ndof);
  const int G = CgShape<double>::group(p), nb = CgShape<double>::blocks(p, G);
  cudaEvent_t e0, e1;
  MG_CUDA(cudaEventCreate(&e0));
  MG_CUDA(cudaEventCreate(&e1));
  MG_CUDA(cudaEventRecord(e0, st));
  CgScalars* hs = reinterpret_cast<CgScalars*>(p->h_pinned);
  mg_status s = MG_OK;
  int before = 0;  // iterations of a resident kernel that gave up
  bool try_resident = true;
  for (;;) {
    s = cg_start<double>(p, d_values, d_b, d_x, 0, precond == MG_PREC_JACOBI, rtol, maxit - before, w, G, nb, st);
    unsigned int epoch = 0;
    if (s == MG_OK) s = cg_iterate<double>(p, d_values, d_x, w, G, nb, maxit - before, st, hs, &epoch, &try_resident);
    if (s != MG_OK || hs->done != kGaveUp) break;
    before += hs->iter;
  }
  MG_CUDA(cudaEventRecord(e1, st));
  MG_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (s != MG_OK) return s;
  MG_CUDA(cudaMemcpy(hs, w.s, sizeof(CgScalars), cudaMemcpyDeviceToHost));
  if (info) {
    info->iterations = before + hs->iter;
    info->outer_iterations = 0;
    info->converged = hs->done == 1;
    info->rel_residual = rel_residual(hs->rr, hs->bb);
    info->seconds = ms * 1e-3;
  }
  if (hs->done == 2) return set_error(MG_ERR_NOT_CONVERGED, "CG breakdown: p.Ap <= 0");
  if (hs->done != 1) return set_error(MG_ERR_NOT_CONVERGED, "CG reached maxit");
  return MG_OK;
}

mg_status mg_cg_refined(mg_plan* p, const double* d_values64, const float* d_values32, const double* d_b,
                        double* d_x, double rtol, int32_t max_outer, int32_t max_inner, double inner_rtol,
                        int32_t precond, mg_cg_info* info, void* stream)
{
  NvtxRange nvtx_range("mg_cg_refined");
  if (!p || !d_values64 || !d_values32 || !d_b || !d_x)
    return set_error(MG_ERR_INVALID_ARG, "mg_cg_refined: null argument");
  if (!(rtol > 0.0) || !(inner_rtol > 0.0) || !(inner_rtol < 1.0) || max_outer < 1 || max_inner < 1)
    return set_error(MG_ERR_INVALID_ARG, "mg_cg_refined: bad tolerance or iteration limits");
  MG_TRY(plan_device(p));
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = p->ndof;
  // layout: [CgWork<float>][r64][x32][scalars of the FP64 residual]
  const size_t wbytes = cg_work_bytes<float>(n);
  const size_t v64 = ((size_t)n * 8 + 255) / 256 * 256, v32 = ((size_t)n * 4 + 255) / 256 * 256;
  void* base = nullptr;
  MG_TRY(plan_work(p, wbytes + v64 + v32 + 256, &base));
  CgWork<float> w = cg_work_carve<float>(base, n);
  double* r64 = (double*)((char*)base + wbytes);
  float* x32 = (float*)((char*)r64 + v64);
  CgScalars* s64 = (CgScalars*)((char*)x32 + v32);
  const int G64 = CgShape<double>::group(p), nb64 = CgShape<double>::blocks(p, G64);
  const int G = CgShape<float>::group(p), nb = CgShape<float>::blocks(p, G);
  const int eb = vec_blocks<float>(n);
  CgScalars* hs = reinterpret_cast<CgScalars*>(p->h_pinned);
  cudaEvent_t e0, e1;
  MG_CUDA(cudaEventCreate(&e0));
  MG_CUDA(cudaEventCreate(&e1));
  MG_CUDA(cudaEventRecord(e0, st));
  int anchors = 0, inner = 0;
  unsigned int epoch = 0;
  bool converged = false, try_resident = true;
  double relres = INFINITY, bb64 = 1.0;
  mg_status s = MG_OK;
  // FP64 residual of the current x (into r64, s64->rr, s64->bb)
  auto residual64 = [&]() -> mg_status {
    MG_CUDA(cudaMemsetAsync(s64, 0, sizeof(CgScalars), st));
    MG_DISPATCH_G(G64, (k_residual64<g><<<nb64, kSolveThreads, 0, st>>>(n, p->d_rowptr, p->d_colind, d_values64,
                                                                          d_b, d_x, r64, w.partials, s64)));
    MG_CUDA(cudaGetLastError());
    MG_CUDA(cudaMemcpyAsync(hs, s64, sizeof(CgScalars), cudaMemcpyDeviceToHost, st));
    MG_CUDA(cudaStreamSynchronize(st));
    bb64 = hs->bb;
    relres = rel_residual(hs->rr, hs->bb);
    return MG_OK;
  };
  s = residual64();
  if (s == MG_OK && relres <= rtol) converged = true;
  if (s == MG_OK && !converged) {
    // first anchor: a plain FP32 CG start on r32 = r64 (x32 = 0), then the
    // target and the reliable-update trigger in its scalars
    k_scale_cast<<<eb, 256, 0, st>>>(n, r64, 1.0, w.r, x32);
    s = cg_start<float>(p, d_values32, w.r, x32, 1, precond == MG_PREC_JACOBI, 1.0, max_inner, w, G, nb, st);
    if (s == MG_OK) {
      MG_CUDA(cudaMemcpyAsync(hs, w.s, sizeof(CgScalars), cudaMemcpyDeviceToHost, st));
      MG_CUDA(cudaStreamSynchronize(st));
      hs->bb = 1.0;
      hs->tol2 = rtol * rtol * bb64;  // recursive-residual target: ||r|| <= rtol ||b||
      hs->rr_anchor = hs->rr;
      // the FP32 recursion drifts from the true residual beyond ~3 decades
      // between anchors (measured: 1e-4 took 33x the iterations on P2 48^3)
      const double delta = std::max(inner_rtol, kMinAnchorRatio);
      hs->delta2 = delta * delta;
      hs->done = 0;
      MG_CUDA(cudaMemcpyAsync(w.s, hs, sizeof(CgScalars), cudaMemcpyHostToDevice, st));
    }
    while (s == MG_OK) {
      s = cg_iterate<float>(p, d_values32, x32, w, G, nb, max_inner, st, hs, &epoch, &try_resident);
      if (s != MG_OK) break;
      inner = hs->iter;
      const int why = hs->done;
      if (why == 2) { s = set_error(MG_ERR_NOT_CONVERGED, "refined CG breakdown: p.Ap <= 0"); break; }
      // anchor: x += x32, r64 = b - A64 x
      k_anchor_x<<<eb, 256, 0, st>>>(n, d_x, x32);
      if (why != kGaveUp) ++anchors;
      s = residual64();
      if (s != MG_OK) break;
      if (relres <= rtol) { converged = true; break; }
      if (why == 3 || anchors >= max_outer) break;
      // replace the FP32 residual, keep the direction, resume; after a wait that ran out the
      // direction is of no one iteration, and z takes its place
      k_anchor_r<<<eb, kSolveThreads, 0, st>>>(n, r64, w.r, w.z, w.dinv, w.partials, w.s);
      if (why == kGaveUp) MG_CUDA(cudaMemcpyAsync(w.p, w.z, sizeof(float) * (size_t)n, cudaMemcpyDeviceToDevice, st));
      else launch_k(false, k_cg_dir<float>, eb, kSolveThreads, st, n, (const float*)w.z, w.p, (const CgScalars*)w.s);
      MG_CUDA(cudaGetLastError());
    }
  }
  MG_CUDA(cudaEventRecord(e1, st));
  MG_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (s != MG_OK) return s;
  if (info) {
    info->iterations = inner;
    info->outer_iterations = anchors;
    info->converged = converged;
    info->rel_residual = relres;
    info->seconds = ms * 1e-3;
  }
  if (!converged) return set_error(MG_ERR_NOT_CONVERGED, "refined CG: no convergence within max_outer / max_inner");
  return MG_OK;
}

}  // extern "C"
