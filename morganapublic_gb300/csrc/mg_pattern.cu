// Mesh preprocessing on the GPU: edge enumeration / numbering and the CSR
// pattern, each giving the host build's arrays bit for bit.
//
// Edges (connect3d.hpp:417-491 with pMapItem / pMapItemShare numbering in
// morganaPublic): the 6 E element-edge incidences as keys min << 32 | max,
// radix-sorted with the incidence index as value (a stable sort, so the first
// incidence of an edge heads its run); run heads give the lexicographic edge
// ids (the LEX rule), and a second sort of the edges by first incidence gives
// the FIRST rule's ids.
//
// CSR pattern on the GPU: the same rows and columns as the host build (the
// union of every element's (test dof, field dof) couplings, columns sorted,
// explicit zeros kept -- traitsMatrixBuilder.hpp:443-544 and the insert /
// GlobalAssemble of buildEpetraCrs, :363-441, in morganaPublic), computed as
//   1. one 64-bit key (row, col) per element coupling with row < col,
//   2. a radix sort of the keys and removal of duplicates (CUB): the upper entries;
//      the same with row and column swapped, sorted again: the lower ones,
//   3. row starts by binary search over both, and each entry to its place.
// The pattern is copied to the host (the export calls and the boundary-multiplier
// build read it there) and, for the device plan build, kept on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include <cub/cub.cuh>

#include "mg_internal.h"
#include "mg_scratch.h"

namespace mg {

// ------------------------------------------------------------ node records --
// The device coordinates and the three-float node records x = hi + mid + lo.
// Where the mesh allows, the parts are split on per-axis grids: with |x| <= 2^e on
// the axis, hi is a multiple of 2^(e-23) and mid of 2^(e-47), so that the
// differences of two nodes' hi and mid parts are exact floats, and lo carries the
// rest to 2^(e-72).  An edge vector then keeps an absolute error of 2^(e-70), a
// relative 2^-50 of every gradient as long as no element is thinner than 2^-20 of
// the largest coordinate; thinner elements, and coordinates whose lower parts
// would leave the normal floats, take the general split (each part the remainder
// rounded to a float, exact), whose differences cost error-free sums.

// The records of a mesh that lies within 2^kSmallMesh of the origin are of its coordinates
// times a power of two that brings the largest near one: the element kernels' products
// of cofactors, the fourth power of an edge, would leave the normal floats (a mesh of
// 1e-9 edges: FP64 stiffness to 5e-9, of 1e-12 edges: zero).  The power, which only
// shifts exponents, is taken back with the entries' weights.  The least keeps 2^geo_exp
// and its products with the weights normal floats.
constexpr int kSmallMesh = -8, kLeastGeoExp = -90;

// stats: per axis the largest |x| (bits of a double), then the smallest altitude
// over 2^emax (bits of a float)
__global__ void __launch_bounds__(256) k_node_xyz(int64_t N, const double* __restrict__ raw, double4_32a* __restrict__ xyz,
                                                  unsigned long long* __restrict__ stats)
{
  __shared__ unsigned long long mx[3];
  if (threadIdx.x < 3) mx[threadIdx.x] = 0ull;
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < N) {
    const double x = raw[3 * i], y = raw[3 * i + 1], z = raw[3 * i + 2];
    xyz[i] = make_double4_32a(x, y, z, 0.0);
    atomicMax(&mx[0], (unsigned long long)__double_as_longlong(fabs(x)));
    atomicMax(&mx[1], (unsigned long long)__double_as_longlong(fabs(y)));
    atomicMax(&mx[2], (unsigned long long)__double_as_longlong(fabs(z)));
  }
  __syncthreads();
  if (threadIdx.x < 3) atomicMax(&stats[threadIdx.x], mx[threadIdx.x]);
}

// e with 2^(e-1) <= |x| < 2^e from the bits of a normal double (-1074 for smaller)
__host__ __device__ __forceinline__ int grid_exponent(unsigned long long bits)
{
  const int ex = (int)((bits >> 52) & 0x7ff);
  return ex == 0 ? -1074 : ex - 1022;
}

// 2^k as a double, |k| <= 1022
__host__ __device__ __forceinline__ double pow2(int k)
{
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)(k + 1023) << 52);
#else
  return std::ldexp(1.0, k);
#endif
}

// The smallest altitude det / |C_a| of the elements, in units of 2^emax: edge
// differences in FP64, the rest in FP32 (only its size against 2^-20 matters).
__global__ void __launch_bounds__(256) k_min_altitude(int64_t E, const int4* __restrict__ conn,
                                                      const double4_32a* __restrict__ xyz, double scale,
                                                      uint32_t* __restrict__ min_alt)
{
  __shared__ uint32_t mn;
  if (threadIdx.x == 0) mn = 0x7f800000u;
  __syncthreads();
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e < E) {
    const int4 n = conn[e];
    const double4_32a p = xyz[n.x], q[3] = {xyz[n.y], xyz[n.z], xyz[n.w]};
    float d[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      d[k][0] = (float)((q[k].x - p.x) * scale);
      d[k][1] = (float)((q[k].y - p.y) * scale);
      d[k][2] = (float)((q[k].z - p.z) * scale);
    }
    float c[4][3], big = 0.0f;
#pragma unroll
    for (int r = 0; r < 3; ++r) c[3][r] = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float *a = d[(k + 1) % 3], *b = d[(k + 2) % 3];
      c[k][0] = a[1] * b[2] - a[2] * b[1];
      c[k][1] = a[2] * b[0] - a[0] * b[2];
      c[k][2] = a[0] * b[1] - a[1] * b[0];
#pragma unroll
      for (int r = 0; r < 3; ++r) c[3][r] -= c[k][r];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) big = fmaxf(big, c[k][0] * c[k][0] + c[k][1] * c[k][1] + c[k][2] * c[k][2]);
    const float det = d[0][0] * c[0][0] + d[0][1] * c[0][1] + d[0][2] * c[0][2];
    // squares below the floats (elements under 2^-37 or so) leave Inf or NaN: zero, as
    // faces of that size rule out an altitude of 2^-20
    const float alt = fabsf(det) * rsqrtf(big);
    atomicMin(&mn, alt > 0.0f && alt < INFINITY ? __float_as_uint(alt) : 0u);
  }
  __syncthreads();
  if (threadIdx.x == 0) atomicMin(min_alt, mn);
}

struct SplitGrid {
  int on;
  int e[3];      // per axis, of scale * x
  double scale;  // a power of two
};

__device__ __forceinline__ void split3(double x, const SplitGrid& g, int k, float& h, float& m, float& l)
{
  if (g.on) {
    const double hd = rint(x * pow2(23 - g.e[k])) * pow2(g.e[k] - 23);
    const double r1 = x - hd;
    const double md = rint(r1 * pow2(47 - g.e[k])) * pow2(g.e[k] - 47);
    h = (float)hd;
    m = (float)md;
    l = (float)(r1 - md);
  } else {  // each remainder is exact in double
    h = (float)x;
    const double r1 = x - (double)h;
    m = (float)r1;
    l = (float)(r1 - (double)m);
  }
}

__global__ void __launch_bounds__(256) k_node_split(int64_t N, const double4_32a* __restrict__ xyz, SplitGrid g,
                                                    double4_32a* __restrict__ scaled, float4* __restrict__ rec,
                                                    float* __restrict__ loz)
{
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= N) return;
  double4_32a p = xyz[i];
  p.x *= g.scale, p.y *= g.scale, p.z *= g.scale;
  if (scaled) scaled[i] = p;
  float h[3], m[3], l[3];
  split3(p.x, g, 0, h[0], m[0], l[0]);
  split3(p.y, g, 1, h[1], m[1], l[1]);
  split3(p.z, g, 2, h[2], m[2], l[2]);
  rec[2 * i] = make_float4(h[0], h[1], h[2], m[0]);
  rec[2 * i + 1] = make_float4(m[1], m[2], l[0], l[1]);
  loz[i] = l[2];
}

mg_status build_node_records(mg_mesh* m)
{
  const int64_t N = m->n_nodes, E = m->n_elem;
  m->grid_split = false;
  m->geo_exp = 0;
  if (N == 0) return MG_OK;
  // the coordinates as they are on the host (24 bytes a node) and the statistics wait in
  // the records' own memory (32) and in lo's (kStatsFloats at least)
  double* raw = reinterpret_cast<double*>(m->d_node_rec);
  unsigned long long* stats = reinterpret_cast<unsigned long long*>(m->d_lo_z);
  uint32_t* min_alt = reinterpret_cast<uint32_t*>(stats + 3);
  const cudaStream_t st = cudaStreamLegacy;
  const uint32_t inf = 0x7f800000u;
  unsigned long long h[3] = {0, 0, 0};
  uint32_t halt = 0;
  SplitGrid g{};
  const unsigned nb = (unsigned)((N + 255) / 256), eb = (unsigned)((E + 255) / 256);
  cudaError_t e = cudaMemcpyAsync(raw, m->xyz.data(), sizeof(double) * 3 * N, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(stats, 0, 4 * sizeof(double), st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(min_alt, &inf, sizeof(inf), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    k_node_xyz<<<nb, 256, 0, st>>>(N, raw, m->d_xyz, stats);
    e = cudaMemcpyAsync(h, stats, sizeof(h), cudaMemcpyDeviceToHost, st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) {
    int emax = -1074;
    bool fits = true;
    for (int k = 0; k < 3; ++k) {
      g.e[k] = grid_exponent(h[k]);
      emax = std::max(emax, g.e[k]);
    }
    m->geo_exp = emax < kSmallMesh ? std::max(emax, kLeastGeoExp) : 0;
    g.scale = pow2(-m->geo_exp);
    for (int k = 0; k < 3; ++k) {
      g.e[k] -= m->geo_exp;
      if (g.e[k] < -50 || g.e[k] > 100) fits = false;
    }
    if (fits && eb > 0) {
      k_min_altitude<<<eb, 256, 0, st>>>(E, m->d_conn, m->d_xyz, pow2(-emax), min_alt);
      e = cudaMemcpyAsync(&halt, min_alt, sizeof(halt), cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
      float alt;
      std::memcpy(&alt, &halt, sizeof(alt));
      g.on = alt >= 0x1p-20f;
    }
  }
  if (e == cudaSuccess) {
    if (m->geo_exp != 0) e = cudaMalloc(&m->d_xyz_rec, sizeof(double4_32a) * N);
  }
  if (e == cudaSuccess) {
    k_node_split<<<nb, 256, 0, st>>>(N, m->d_xyz, g, m->d_xyz_rec, m->d_node_rec, m->d_lo_z);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  if (e != cudaSuccess) return cuda_error(e, "node records");
  m->grid_split = g.on != 0;
  return MG_OK;
}

static int key_bits(int64_t n)  // bits that hold every value < n
{
  int b = 0;
  while (b < 62 && (1ll << b) < n) ++b;
  return b;
}

// ---------------------------------------------------------------- pattern --
// The pattern is symmetric with a diagonal entry for every dof of an element, so only
// the couplings row < column are sorted: nb (nb - 1) / 2 keys per element, P1 6 of 16,
// P2 45 of 100, of 2 bits(ndof) bits; the lower entries are the unique ones with the
// words swapped, sorted again (a sixth of the keys).  Measured at 64^3 P1 (25 M
// couplings): all of them sorted 1.4 ms, the upper ones 0.7 and the lower ones 0.25,
// from a third of the memory (its allocation and free: 0.6 -> 0.4 ms).

// one thread per (element, test basis j): its couplings with the later basis functions
__global__ void __launch_bounds__(256) k_pattern_keys(int64_t n_elem, int nb, int col_bits, const int32_t* __restrict__ dofs,
                                                      unsigned long long* __restrict__ keys, int32_t* __restrict__ used)
{
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n_elem * nb) return;
  const int64_t e = t / nb;
  const int j = (int)(t - e * nb);
  const uint32_t a = (uint32_t)dofs[t];
  used[a] = 1;
  unsigned long long* out = keys + e * (nb * (nb - 1) / 2) + j * (2 * nb - 1 - j) / 2;
  for (int i = j + 1; i < nb; ++i) {
    const uint32_t b = (uint32_t)dofs[e * nb + i];
    out[i - j - 1] = ((unsigned long long)min(a, b) << col_bits) | max(a, b);
  }
}

__global__ void __launch_bounds__(256) k_pattern_swap(int64_t n, int col_bits, const unsigned long long* __restrict__ keys,
                                                      unsigned long long* __restrict__ out)
{
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) out[k] = ((keys[k] & ((1ull << col_bits) - 1ull)) << col_bits) | (keys[k] >> col_bits);
}

// first of the n sorted keys with a row >= r
__device__ __forceinline__ int64_t row_start(int64_t r, int64_t n, int col_bits, const unsigned long long* keys)
{
  const unsigned long long target = (unsigned long long)r << col_bits;
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (keys[mid] < target) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Starts of row r among the lower and the upper entries, the row pointer (diag: the
// diagonal entries before row r), and the diagonal entry's column.
__global__ void __launch_bounds__(256) k_pattern_rows(int64_t nd, int64_t n, int col_bits,
                                                      const unsigned long long* __restrict__ lower,
                                                      const unsigned long long* __restrict__ upper,
                                                      const int32_t* __restrict__ diag, int32_t* __restrict__ lo_start,
                                                      int32_t* __restrict__ up_start, int32_t* __restrict__ rowptr)
{
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r > nd) return;
  const int64_t lo = row_start(r, n, col_bits, lower), up = row_start(r, n, col_bits, upper);
  lo_start[r] = (int32_t)lo;
  up_start[r] = (int32_t)up;
  rowptr[r] = (int32_t)(lo + up + diag[r]);
}

// A row holds its lower entries, its diagonal one and its upper ones: entry k of a list
// goes to k plus the other two lists' entries before it.  Thread k < n: lower and
// upper entry k; thread n + r: row r's diagonal.
__global__ void __launch_bounds__(256) k_pattern_cols(int64_t nd, int64_t n, int col_bits,
                                                      const unsigned long long* __restrict__ lower,
                                                      const unsigned long long* __restrict__ upper,
                                                      const int32_t* __restrict__ diag,
                                                      const int32_t* __restrict__ lo_start,
                                                      const int32_t* __restrict__ up_start, int32_t* __restrict__ colind)
{
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const unsigned long long mask = (1ull << col_bits) - 1ull;
  if (k < n) {
    const int64_t rl = (int64_t)(lower[k] >> col_bits), ru = (int64_t)(upper[k] >> col_bits);
    colind[k + up_start[rl] + diag[rl]] = (int32_t)(lower[k] & mask);
    colind[k + lo_start[ru + 1] + diag[ru + 1]] = (int32_t)(upper[k] & mask);
  } else if (k < n + nd) {
    const int64_t r = k - n;
    if (diag[r + 1] > diag[r]) colind[lo_start[r + 1] + up_start[r] + diag[r]] = (int32_t)r;
  }
}

// local edge j of a tet joins its vertices kEdge[j][0] and kEdge[j][1]
__constant__ int kEdgeDev[6][2] = {{0, 1}, {1, 2}, {2, 0}, {0, 3}, {1, 3}, {2, 3}};

__global__ void __launch_bounds__(256) k_edge_keys(int64_t M, const int32_t* __restrict__ conn,
                                                   unsigned long long* __restrict__ keys, int32_t* __restrict__ vals)
{
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= M) return;
  const int64_t e = t / 6;
  const int j = (int)(t % 6);
  const uint32_t a = (uint32_t)conn[4 * e + kEdgeDev[j][0]], b = (uint32_t)conn[4 * e + kEdgeDev[j][1]];
  keys[t] = ((unsigned long long)min(a, b) << 32) | max(a, b);
  vals[t] = (int32_t)t;
}

__global__ void __launch_bounds__(256) k_edge_heads(int64_t M, const unsigned long long* __restrict__ keys,
                                                    int32_t* __restrict__ head)
{
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < M) head[k] = (k == 0 || keys[k] != keys[k - 1]) ? 1 : 0;
}

// first incidence of each edge (lexicographic id g = lex[k] - 1 at its run head)
__global__ void __launch_bounds__(256) k_edge_first(int64_t M, const int32_t* __restrict__ head,
                                                    const int32_t* __restrict__ lex, const int32_t* __restrict__ inc,
                                                    int32_t* __restrict__ first, int32_t* __restrict__ ids)
{
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < M && head[k]) {
    first[lex[k] - 1] = inc[k];
    ids[lex[k] - 1] = lex[k] - 1;
  }
}

// gid_of_lex from the edges sorted by first incidence (FIRST rule)
__global__ void __launch_bounds__(256) k_edge_rank(int64_t nE, const int32_t* __restrict__ sorted_g,
                                                   int32_t* __restrict__ gid_of_lex)
{
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (r < nE) gid_of_lex[sorted_g[r]] = (int32_t)r;
}

__global__ void __launch_bounds__(256) k_edge_scatter(int64_t M, const int32_t* __restrict__ lex,
                                                      const int32_t* __restrict__ inc,
                                                      const int32_t* __restrict__ gid_of_lex,
                                                      int32_t* __restrict__ elem_edge)
{
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < M) elem_edge[inc[k]] = gid_of_lex ? gid_of_lex[lex[k] - 1] : lex[k] - 1;
}

// end points of each edge, oriented as in its first incidence
__global__ void __launch_bounds__(256) k_edge_nodes(int64_t nE, const int32_t* __restrict__ first,
                                                    const int32_t* __restrict__ gid_of_lex,
                                                    const int32_t* __restrict__ conn, int32_t* __restrict__ nodes)
{
  const int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (g >= nE) return;
  const int64_t t = first[g], e = t / 6;
  const int j = (int)(t % 6);
  const int64_t gid = gid_of_lex ? gid_of_lex[g] : g;
  nodes[2 * gid] = conn[4 * e + kEdgeDev[j][0]];
  nodes[2 * gid + 1] = conn[4 * e + kEdgeDev[j][1]];
}

struct EdgeBuffers {
  int32_t *conn = nullptr, *vals = nullptr, *vals_s = nullptr, *head = nullptr, *lex = nullptr, *first = nullptr,
          *ids = nullptr, *ids_s = nullptr, *first_s = nullptr, *gid = nullptr, *elem_edge = nullptr,
          *nodes = nullptr;
  unsigned long long *keys = nullptr, *keys_s = nullptr;
  unsigned char* tmp = nullptr;
};

mg_status build_edges_device(mg_mesh* m, cudaStream_t st)
{
  if (m->n_edges >= 0) return MG_OK;
  const int64_t N = m->n_nodes, E = m->n_elem, M = 6 * E;
  if (M >= INT32_MAX) return set_error(MG_ERR_SIZE, "device edge build: more than 2^31 edge incidences");
  if (M == 0) {
    m->elem_edge.clear();
    m->edge_nodes.clear();
    m->n_edges = 0;
    return MG_OK;
  }
  EdgeBuffers d;
  DeviceScratch scratch;
  const size_t i4 = sizeof(int32_t) * M;
  MG_TRY(scratch.reserve(64 * (size_t)M + 4096));  // 12 four-byte arrays and two of keys
  MG_TRY(scratch.take(&d.conn, 4 * E));
  for (int32_t** q : {&d.vals, &d.vals_s, &d.head, &d.lex, &d.first, &d.ids, &d.ids_s, &d.first_s, &d.gid,
                      &d.elem_edge})
    MG_TRY(scratch.take(q, M));
  MG_TRY(scratch.take(&d.keys, M));
  MG_TRY(scratch.take(&d.keys_s, M));
  size_t b1 = 0, b2 = 0, b3 = 0;
  const int kb = 32 + key_bits(N), fb = key_bits(M);
  MG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b1, d.keys, d.keys_s, d.vals, d.vals_s, (int)M, 0, kb, st));
  MG_CUDA(cub::DeviceScan::InclusiveSum(nullptr, b2, d.head, d.lex, (int)M, st));
  MG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b3, d.first, d.first_s, d.ids, d.ids_s, (int)M, 0, fb, st));
  MG_TRY(scratch.take(&d.tmp, (int64_t)std::max({b1, b2, b3})));
  MG_CUDA(cudaMemcpyAsync(d.conn, m->conn.data(), sizeof(int32_t) * 4 * E, cudaMemcpyHostToDevice, st));
  const int T = 256;
  const int gm = (int)((M + T - 1) / T);
  k_edge_keys<<<gm, T, 0, st>>>(M, d.conn, d.keys, d.vals);
  MG_CUDA(cub::DeviceRadixSort::SortPairs(d.tmp, b1, d.keys, d.keys_s, d.vals, d.vals_s, (int)M, 0, kb, st));
  k_edge_heads<<<gm, T, 0, st>>>(M, d.keys_s, d.head);
  MG_CUDA(cub::DeviceScan::InclusiveSum(d.tmp, b2, d.head, d.lex, (int)M, st));
  int32_t nE = 0;
  MG_CUDA(cudaMemcpyAsync(&nE, d.lex + (M - 1), sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  k_edge_first<<<gm, T, 0, st>>>(M, d.head, d.lex, d.vals_s, d.first, d.ids);
  MG_CUDA(cudaGetLastError());
  MG_CUDA(cudaStreamSynchronize(st));
  const int ge = (int)((nE + T - 1) / T);
  const int32_t* gid = nullptr;
  if (m->edge_rule == MG_EDGES_FIRST) {
    // edges ordered by their first incidence (distinct values)
    MG_CUDA(cub::DeviceRadixSort::SortPairs(d.tmp, b3, d.first, d.first_s, d.ids, d.ids_s, (int)nE, 0, fb, st));
    k_edge_rank<<<ge, T, 0, st>>>(nE, d.ids_s, d.gid);
    gid = d.gid;
  }
  k_edge_scatter<<<gm, T, 0, st>>>(M, d.lex, d.vals_s, gid, d.elem_edge);
  MG_TRY(scratch.take(&d.nodes, 2 * (int64_t)nE));
  k_edge_nodes<<<ge, T, 0, st>>>(nE, d.first, gid, d.conn, d.nodes);
  MG_CUDA(cudaGetLastError());
  m->elem_edge.resize(M);
  m->edge_nodes.resize(2 * (int64_t)nE);
  MG_CUDA(cudaMemcpyAsync(m->elem_edge.data(), d.elem_edge, i4, cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaMemcpyAsync(m->edge_nodes.data(), d.nodes, sizeof(int32_t) * 2 * nE, cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaStreamSynchronize(st));
  m->n_edges = nE;
  return MG_OK;
}

mg_status build_pattern_device(mg_plan* p, DeviceScratch& scratch, cudaStream_t st, bool keep_device)
{
  mg_mesh* m = p->mesh;
  const int nb = m->nb;
  const int64_t E = m->n_elem, nd = m->ndof, n = E * nb * nb;
  if (n >= INT32_MAX) return set_error(MG_ERR_SIZE, "device pattern build: more than 2^31 element couplings");
  if (nd >= INT32_MAX) return set_error(MG_ERR_SIZE, "device pattern build: ndof above 2^31");
  MG_TRY(mesh_device(m));
  p->ndof = nd;
  p->rowptr.assign(nd + 1, 0);
  p->colind.clear();
  p->nnz = 0;
  if (n == 0) {  // no elements: every row empty
    if (keep_device) {
      MG_CUDA(cudaMalloc(&p->d_rowptr, sizeof(int32_t) * (nd + 1)));
      MG_CUDA(cudaMalloc(&p->d_colind, sizeof(int32_t)));
      MG_CUDA(cudaMemsetAsync(p->d_rowptr, 0, sizeof(int32_t) * (nd + 1), st));
      MG_CUDA(cudaStreamSynchronize(st));
    }
    return MG_OK;
  }
  BuildBuffers B(scratch);
  unsigned long long *a, *upper, *lower;
  int64_t* count;
  unsigned char* tmp;
  int32_t *used, *diag, *lo_start, *up_start, *d_rowptr, *d_colind;
  const int64_t m_keys = E * (nb * (nb - 1) / 2);
  const int col_bits = std::max(1, key_bits(nd)), end_bit = 2 * col_bits;
  size_t sort_bytes = 0, uniq_bytes = 0, scan_bytes = 0;
  MG_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                         (int)m_keys, 0, end_bit, st));
  MG_CUDA(cub::DeviceSelect::Unique(nullptr, uniq_bytes, (unsigned long long*)nullptr, (unsigned long long*)nullptr,
                                    (int64_t*)nullptr, (int)m_keys, st));
  MG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (int32_t*)nullptr, (int32_t*)nullptr, (int)(nd + 1), st));
  const size_t tmp_bytes = std::max({sort_bytes, uniq_bytes, scan_bytes});
  MG_TRY(scratch.reserve(2 * sizeof(unsigned long long) * (size_t)m_keys + 4 * sizeof(int32_t) * (size_t)(nd + 1) +
                         tmp_bytes + 4096));
  MG_TRY(B.temp(&a, m_keys));
  MG_TRY(B.temp(&upper, m_keys));
  MG_TRY(B.temp(&used, nd + 1));
  MG_TRY(B.temp(&diag, nd + 1));
  MG_TRY(B.temp(&lo_start, nd + 1));
  MG_TRY(B.temp(&up_start, nd + 1));
  MG_TRY(B.temp(&count, 1));
  MG_TRY(B.temp(&tmp, (int64_t)tmp_bytes));
  const int threads = 256;
  MG_CUDA(cudaMemsetAsync(used, 0, sizeof(int32_t) * (nd + 1), st));
  k_pattern_keys<<<(int)((E * nb + threads - 1) / threads), threads, 0, st>>>(E, nb, col_bits, m->d_dofs, a, used);
  MG_CUDA(cudaGetLastError());
  size_t tb = tmp_bytes;
  MG_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, used, diag, (int)(nd + 1), st));
  tb = tmp_bytes;
  MG_CUDA(cub::DeviceRadixSort::SortKeys(tmp, tb, a, upper, (int)m_keys, 0, end_bit, st));
  tb = tmp_bytes;
  MG_CUDA(cub::DeviceSelect::Unique(tmp, tb, upper, a, count, (int)m_keys, st));
  std::swap(a, upper);  // the unique keys; a is free again
  int64_t n_up = 0;
  int32_t n_diag = 0;
  MG_CUDA(cudaMemcpyAsync(&n_up, count, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaMemcpyAsync(&n_diag, diag + nd, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaStreamSynchronize(st));
  const int64_t nnz = 2 * n_up + n_diag;
  if (nnz >= INT32_MAX) return set_error(MG_ERR_SIZE, "nnz above 2^31-1");
  unsigned long long* swapped;
  MG_TRY(B.temp(&swapped, n_up));
  lower = a;
  k_pattern_swap<<<(int)((n_up + threads - 1) / threads), threads, 0, st>>>(n_up, col_bits, upper, swapped);
  tb = tmp_bytes;
  MG_CUDA(cub::DeviceRadixSort::SortKeys(tmp, tb, swapped, lower, (int)n_up, 0, end_bit, st));
  MG_TRY(B.alloc(&d_rowptr, nd + 1));
  MG_TRY(B.alloc(&d_colind, nnz));
  k_pattern_rows<<<(int)((nd + 1 + threads - 1) / threads), threads, 0, st>>>(nd, n_up, col_bits, lower, upper, diag,
                                                                              lo_start, up_start, d_rowptr);
  k_pattern_cols<<<(int)((n_up + nd + threads - 1) / threads), threads, 0, st>>>(nd, n_up, col_bits, lower, upper, diag,
                                                                                 lo_start, up_start, d_colind);
  MG_CUDA(cudaGetLastError());
  p->colind.resize(nnz);
  MG_CUDA(cudaMemcpyAsync(p->rowptr.data(), d_rowptr, sizeof(int32_t) * (nd + 1), cudaMemcpyDeviceToHost, st));
  if (nnz > 0)
    MG_CUDA(cudaMemcpyAsync(p->colind.data(), d_colind, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost, st));
  MG_CUDA(cudaStreamSynchronize(st));
  p->nnz = nnz;
  if (keep_device) {  // the device copies become the plan's (the plan's device state is built from them)
    p->d_rowptr = d_rowptr;
    p->d_colind = d_colind;
    B.keep(d_rowptr);
    B.keep(d_colind);
  }
  return MG_OK;
}

}  // namespace mg
