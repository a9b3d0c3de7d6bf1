// Boundary multipliers on the GPU: values of B = opLA3dA, of the saddle matrix
// [K B^T; B 0], and the products with them.
//
// B is assembled in two deterministic passes.  A face's local matrix is its area2 =
// |Vx ^ Vy| times a matrix of its local face and the card alone (mg_lagrange.cuh), so
//   k_face_area    one thread per boundary face: area2, in native FP64;
//   k_gather_sum   one thread per entry of B: the sum of area2 times the table's entry
//                  over the faces that the entry sums, in the reference's insertion
//                  order (element, local face, face vertex, basis), from the
//                  host-built list of the entry.
// No atomics, so every run gives the same bits.  (Summing each face's local matrix at
// its quadrature points instead cost 130 to 2000 FP64 instructions per face, on a pipe
// that starts one per warp every 16 cycles, and 8 nt nb bytes of staging per face:
// 41 x 47 x 35, P1, B and the saddle values: 27 us against 9.)
// The saddle values are a gather from K's and B's values through a per-entry
// source map (plus, for setMTM / setMMT, one thread per entry of B^T B or
// B B^T summing its products); the products with the matrices use the CSR SpMV
// kernel of mg_solve.cu.
// The three kernels are launched with programmatic dependence: each reads the
// plan's lists before it waits for the kernel before it.
#include <algorithm>
#include <climits>

#include "mg_internal.h"
#include "mg_lagrange.cuh"
#include "mg_launch.cuh"

namespace mg {

namespace {

constexpr int kFaceThreads = 256, kAreaThreads = 128, kFillItems = 4;

int grid_for(int64_t n, int per_cta = kFaceThreads)
{
  const int64_t b = (n + per_cta - 1) / per_cta;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 65535));
}

// Bound by latency: the face's node ids, its nodes and an FP64 chain; 128 threads per
// CTA spread a small surface's faces over more SMs.
__global__ void __launch_bounds__(kAreaThreads) k_face_area(int64_t n_faces, const int4* __restrict__ faces,
                                                            const double4_32a* __restrict__ xyz,
                                                            double2* __restrict__ area)
{
  pdl_trigger();
  bool waited = false;
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < n_faces; f += (int64_t)gridDim.x * blockDim.x) {
    const int4 c = faces[f];
    const int v[3] = {c.x, c.y, c.z};
    double P[3][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double4_32a p = xyz[v[a]];
      P[a][0] = p.x;
      P[a][1] = p.y;
      P[a][2] = p.z;
    }
    const double s = face_area2(P);
    if (!waited) pdl_wait();  // an earlier gather may still read the areas
    waited = true;
    area[f] = make_double2(s, __hiloint2double(0, c.w));
  }
  if (!waited) pdl_wait();
}

// vals[k] = sum over j in [ptr[k], ptr[k+1]), in list order, of area2 of face src[j] / nt
// nb times the entry src[j] % (nt nb) of its local face's table.  Bound by the latency
// of its loads: the list's are taken two at a time, the first ones before the wait.
template <int NTB>
__global__ void __launch_bounds__(kFaceThreads) k_gather_sum(int64_t n, const int32_t* __restrict__ ptr,
                                                             const int32_t* __restrict__ src,
                                                             const double2* area, const double* __restrict__ tab,
                                                             double* __restrict__ vals)
{
  pdl_trigger();
  bool waited = false;
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    const int32_t j1 = ptr[k + 1];
    for (int32_t j = ptr[k]; j < j1; j += 2) {
      int32_t q[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) q[i] = src[min(j + i, j1 - 1)];
      if (!waited) pdl_wait();
      waited = true;
      double2 a[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = area[q[i] / NTB];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (j + i < j1) s += a[i].x * tab[__double2loint(a[i].y) * NTB + q[i] % NTB];
    }
    if (!waited) pdl_wait();  // an earlier kernel may still read vals
    waited = true;
    vals[k] = s;
  }
  if (!waited) pdl_wait();
}

// Saddle entry k: K's entry src (>= 0), B's entry -(src + 1), eye_lam
// (kSrcLamDiag) or zero (kSrcZero, a B^T B entry outside K).  Bound by the latency of
// two dependent loads: four entries per thread, and their sources read before the wait
// (1.26 M entries: 3.2 us, with two or eight per thread 3.8 and 3.6).
__global__ void __launch_bounds__(kFaceThreads) k_saddle_fill(int64_t n, const int32_t* __restrict__ src,
                                                          const double* kv, const double* bv, double eye_lam,
                                                          double* __restrict__ out)
{
  pdl_trigger();
  const int64_t step = (int64_t)gridDim.x * (kFillItems * kFaceThreads);
  bool waited = false;
  for (int64_t k0 = blockIdx.x * (int64_t)(kFillItems * kFaceThreads) + threadIdx.x; k0 < n; k0 += step) {
    int32_t s[kFillItems];
    double v[kFillItems];
#pragma unroll
    for (int i = 0; i < kFillItems; ++i) s[i] = k0 + i * kFaceThreads < n ? src[k0 + i * kFaceThreads] : kSrcZero;
    if (!waited) pdl_wait();
    waited = true;
#pragma unroll
    for (int i = 0; i < kFillItems; ++i)
      v[i] = s[i] >= 0 ? kv[s[i]] : (s[i] == kSrcLamDiag ? eye_lam : (s[i] == kSrcZero ? 0.0 : bv[-(s[i] + 1)]));
#pragma unroll
    for (int i = 0; i < kFillItems; ++i)
      if (k0 + i * kFaceThreads < n) out[k0 + i * kFaceThreads] = v[i];
  }
  if (!waited) pdl_wait();
}

// Product entry m (B^T B or B B^T): scale * sum of bv[k1] bv[k2] over its
// pairs (in their fixed order), added to its saddle entry (one entry per m: no
// atomics)
__global__ void __launch_bounds__(kFaceThreads) k_saddle_products(int64_t n, const int32_t* __restrict__ pair_ptr,
                                                         const int2* __restrict__ pairs,
                                                         const int32_t* __restrict__ slot,
                                                         const double* __restrict__ bv, double scale,
                                                         double* __restrict__ out)
{
  for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < n; m += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    const int32_t j1 = pair_ptr[m + 1];
    for (int32_t j = pair_ptr[m]; j < j1; ++j) {
      const int2 pr = pairs[j];
      s += bv[pr.x] * bv[pr.y];
    }
    out[slot[m]] += scale * s;
  }
}

// Adds eye to the diagonal of the field block, at each row's diagonal entry
// (s_diag[r]; rows without one, dofs outside every element, are left alone).
__global__ void __launch_bounds__(kFaceThreads) k_saddle_eye(int64_t nd, const int32_t* __restrict__ s_diag,
                                                         double eye, double* __restrict__ out)
{
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nd; r += (int64_t)gridDim.x * blockDim.x) {
    const int32_t d = s_diag[r];
    if (d >= 0) out[d] += eye;
  }
}

}  // namespace

}  // namespace mg

using namespace mg;

extern "C" {

mg_status mg_lagrange_assemble(mg_lagrange* lg, int32_t quad, double* d_b_values, void* stream)
{
  NvtxRange nvtx_range("mg_lagrange_assemble");
  if (!lg) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble: null handle");
  FaceRule rule{};
  if (!face_rule(quad, &rule)) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble: face card must be 1, 3, 4 or 6");
  if (lg->nnz_b == 0) return MG_OK;
  if (!d_b_values) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble: null values");
  MG_TRY(lagrange_device(lg));
  cudaStream_t st = (cudaStream_t)stream;
  const mg_mesh* m = lg->plan->mesh;
  const int ntb = lg->nt * lg->nb;
  const double* tab = lg->d_face_tab;
  for (const int card : kFaceCards) {
    if (card == quad) break;
    tab += 4 * ntb;
  }
  MG_CUDA(launch_pdl(k_face_area, grid_for(lg->n_faces, kAreaThreads), kAreaThreads, st, lg->n_faces, lg->d_faces,
                     m->d_xyz, lg->d_face_area));
  const auto gather = [&](auto kernel) {
    return launch_pdl(kernel, grid_for(lg->nnz_b), kFaceThreads, st, lg->nnz_b, lg->d_b_src_ptr, lg->d_b_src,
                      lg->d_face_area, tab, d_b_values);
  };
  switch (ntb) {
    case 4: MG_CUDA(gather(k_gather_sum<4>)); break;
    case 10: MG_CUDA(gather(k_gather_sum<10>)); break;
    case 12: MG_CUDA(gather(k_gather_sum<12>)); break;
    case 24: MG_CUDA(gather(k_gather_sum<24>)); break;
    case 30: MG_CUDA(gather(k_gather_sum<30>)); break;
    default: MG_CUDA(gather(k_gather_sum<60>)); break;
  }
  return MG_OK;
}

mg_status mg_lagrange_assemble_host(mg_lagrange* lg, int32_t quad, double* h_b_values)
{
  NvtxRange nvtx_range("mg_lagrange_assemble_host");
  if (!lg) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble_host: null handle");
  FaceRule rule{};
  if (!face_rule(quad, &rule))
    return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble_host: face card must be 1, 3, 4 or 6");
  if (lg->nnz_b == 0) return MG_OK;
  if (!h_b_values) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_assemble_host: null values");
  double* d = nullptr;
  MG_CUDA(cudaMalloc(&d, sizeof(double) * lg->nnz_b));
  mg_status s = mg_lagrange_assemble(lg, quad, d, nullptr);
  if (s == MG_OK) {
    const cudaError_t e = cudaMemcpy(h_b_values, d, sizeof(double) * lg->nnz_b, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) s = cuda_error(e, "cudaMemcpy(B values)");
  }
  cudaFree(d);
  return s;
}

mg_status mg_saddle_assemble(mg_lagrange* lg, const double* d_k_values, const double* d_b_values,
                             const mg_saddle_scales* scales, double* d_values, void* stream)
{
  NvtxRange nvtx_range("mg_saddle_assemble");
  if (!lg) return set_error(MG_ERR_INVALID_ARG, "mg_saddle_assemble: null handle");
  const mg_saddle_scales sc = scales ? *scales : mg_saddle_scales{0.0, 0.0, 0.0, 0.0};
  const double eye_field = sc.eye_field, eye_lam = sc.eye_lam, mtm_scale = sc.mtm, mmt_scale = sc.mmt;
  if (eye_lam != 0.0 && !lg->lam_diag)
    return set_error(MG_ERR_INVALID_ARG, "mg_saddle_assemble: eye_lam needs a pattern built with MG_SADDLE_LAM_DIAG");
  if (mtm_scale != 0.0 && !lg->mtm)
    return set_error(MG_ERR_INVALID_ARG, "mg_saddle_assemble: mtm needs a pattern built with MG_SADDLE_MTM");
  if (mmt_scale != 0.0 && !lg->mmt)
    return set_error(MG_ERR_INVALID_ARG, "mg_saddle_assemble: mmt needs a pattern built with MG_SADDLE_MMT");
  if (lg->nnz_s == 0) return MG_OK;
  if (!d_values || (lg->plan->nnz && !d_k_values) || (lg->nnz_b && !d_b_values))
    return set_error(MG_ERR_INVALID_ARG, "mg_saddle_assemble: null argument");
  MG_TRY(lagrange_device(lg));
  cudaStream_t st = (cudaStream_t)stream;
  MG_CUDA(launch_pdl(k_saddle_fill, grid_for(lg->nnz_s, kFillItems * kFaceThreads), kFaceThreads, st, lg->nnz_s,
                     lg->d_s_src, d_k_values, d_b_values, eye_lam, d_values));
  if (eye_field != 0.0 && lg->ndof > 0) {
    k_saddle_eye<<<grid_for(lg->ndof), kFaceThreads, 0, st>>>(lg->ndof, lg->d_s_diag, eye_field, d_values);
    MG_CUDA(cudaGetLastError());
  }
  if (mtm_scale != 0.0 && lg->nnz_m > 0) {
    k_saddle_products<<<grid_for(lg->nnz_m), kFaceThreads, 0, st>>>(lg->nnz_m, lg->d_m_pair_ptr, lg->d_m_pairs,
                                                                    lg->d_m_slot, d_b_values, mtm_scale, d_values);
    MG_CUDA(cudaGetLastError());
  }
  if (mmt_scale != 0.0 && lg->nnz_p > 0) {
    k_saddle_products<<<grid_for(lg->nnz_p), kFaceThreads, 0, st>>>(lg->nnz_p, lg->d_p_pair_ptr, lg->d_p_pairs,
                                                                    lg->d_p_slot, d_b_values, mmt_scale, d_values);
    MG_CUDA(cudaGetLastError());
  }
  return MG_OK;
}

mg_status mg_saddle_spmv(mg_lagrange* lg, const double* d_values, const double* d_x, double* d_y, void* stream)
{
  NvtxRange nvtx_range("mg_saddle_spmv");
  if (!lg) return set_error(MG_ERR_INVALID_ARG, "mg_saddle_spmv: null handle");
  const int64_t rows = lg->ndof + lg->nl;
  if (rows == 0) return MG_OK;
  if (!d_values || !d_x || !d_y) return set_error(MG_ERR_INVALID_ARG, "mg_saddle_spmv: null argument");
  MG_TRY(lagrange_device(lg));
  return launch_spmv_csr(rows, lg->nnz_s, lg->d_s_rowptr, lg->d_s_colind, d_values, d_x, d_y, (cudaStream_t)stream);
}

mg_status mg_lagrange_apply(mg_lagrange* lg, const double* d_b_values, const double* d_u, double* d_g, void* stream)
{
  NvtxRange nvtx_range("mg_lagrange_apply");
  if (!lg) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_apply: null handle");
  if (lg->nl == 0) return MG_OK;
  if (!d_b_values || !d_u || !d_g) return set_error(MG_ERR_INVALID_ARG, "mg_lagrange_apply: null argument");
  MG_TRY(lagrange_device(lg));
  return launch_spmv_csr(lg->nl, lg->nnz_b, lg->d_b_rowptr, lg->d_b_colind, d_b_values, d_u, d_g,
                         (cudaStream_t)stream);
}

}  // extern "C"
