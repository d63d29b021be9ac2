// demap.cu -- NUC max-log soft demapper with the BICM bit de-interleaver
// fused into its epilogue (sm_100a).
//
// Reference semantics: lab/m44_ldm.py:2431-2494 (`_point_metric`,
// `demap_batch_qam`), the float32 form of lab/m6_bicm.py:213-225
// (`demap_llr`) and lab/m16_demap_fast.py:80-119 (`demap_llr_fast`):
//
//   q_k   = ((zr*pr_k + zi*pi_k) * -2) + |p_k|^2      every op rounded to f32
//   a_i   = min over labels with bit i = 1 of q_k       (y0 = MSB)
//   b_i   = min over labels with bit i = 0 of q_k
//   llr_i = (a_i - b_i) / sigma2                        IEEE f32 division
//   lam[lam_of_q[MOD*s + i]] = llr_i                    (lab/m9_fast.py:1120)
//
// The |z|^2 term common to every point cancels in a_i - b_i
// (lab/m16_demap_fast.py:27-58), so it is only used by the sigma2 estimator.
//
// Work split: one thread per cell; the alphabet (Re, Im,
// |p|^2, 3*M values) is staged in shared memory; cells and per-cell sigma2 are
// read coalesced.  The point distance is work of K=2: no tensor-core shape.

#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/atsc3_fec.h"
#include "common.cuh"
#include "demap_core.cuh"

namespace atsc3 {

constexpr int DEMAP_T = 256;    // threads per CTA, a cell each
// CTAs per SM the compiler has to leave room for: the fully unrolled 64- and
// 256-point kernels run best with just the registers of four (75 x 64800-bit
// Blocks: 64 points 31.2 us without the bound, 23.0 with it; 256 points 37.4
// and 31.6; the grids lose by it).  16 points are bound by memory latency and the
// scattered stores, so by the warps in flight (codeword order, one sigma2 / one per
// cell: 16.9 / 18.4 us without the bound, which takes 62 registers, 15.5 / 16.8 with
// five CTAs, 14.5 / 15.6 with six, 13.8 / 14.7 with eight, which do not spill; 13.0 /
// 14.0 with one 32-bit division a cell instead of a 64-bit one and a 32-bit one).
template <int NB, typename T>
constexpr int demap_ctas() {
  return sizeof(T) != 4 ? 1 : NB == 4 ? 8 : NB == 6 || NB == 8 ? 4 : 1;
}

// Writes one cell's LLRs: through lam_of_q (nullable) or in transmission
// order, the table and the contiguous LLRs in the widest aligned pieces.
template <int NB, typename T>
__device__ __forceinline__ void store_llrs(const T (&d)[NB], int s,
                                           const int32_t *__restrict__ lam_of_q,
                                           T *__restrict__ o) {
  const int q0 = s * NB;
  if (lam_of_q) {
    int32_t at[NB];
    if (NB % 4 == 0 && (reinterpret_cast<uintptr_t>(lam_of_q) & 15) == 0) {
#pragma unroll
      for (int i = 0; i + 4 <= NB; i += 4) {
        const int4 v = __ldg(reinterpret_cast<const int4 *>(lam_of_q + q0 + i));
        at[i] = v.x;
        at[i + 1] = v.y;
        at[i + 2] = v.z;
        at[i + 3] = v.w;
      }
    } else if ((reinterpret_cast<uintptr_t>(lam_of_q) & 7) == 0) {
#pragma unroll
      for (int i = 0; i < NB; i += 2) {
        const int2 v = __ldg(reinterpret_cast<const int2 *>(lam_of_q + q0 + i));
        at[i] = v.x;
        at[i + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < NB; ++i) at[i] = __ldg(lam_of_q + q0 + i);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) o[at[i]] = d[i];
    return;
  }
  T *r = o + q0;
  if (sizeof(T) == 4 && (reinterpret_cast<uintptr_t>(r) & 7) == 0) {
#pragma unroll
    for (int i = 0; i < NB; i += 2)
      *reinterpret_cast<float2 *>(r + i) = make_float2((float)d[i], (float)d[i + 1]);
  } else if (sizeof(T) == 8 && (reinterpret_cast<uintptr_t>(r) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < NB; i += 2)
      *reinterpret_cast<double2 *>(r + i) = make_double2(d[i], d[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < NB; ++i) r[i] = d[i];
  }
}

template <typename T> struct Cell2;
template <> struct Cell2<float> { using type = float2; };
template <> struct Cell2<double> { using type = double2; };

// T = float: the decode path; T = double: the drop-in for the reference's
// default float64 demap_llr_fast (lab/m16_demap_fast.py:80-119).
template <int NB, typename T>
__global__ void __launch_bounds__(DEMAP_T, (demap_ctas<NB, T>())) demap_kernel(
    const typename Cell2<T>::type *__restrict__ cells, int64_t ld_cells, int nblk,
    int ncell, const T *__restrict__ pts, int sigma_mode,
    const T *__restrict__ sigma2, int64_t ld_sigma, T s2scalar,
    const int32_t *__restrict__ lam_of_q, T *__restrict__ out,
    int64_t ld_out) {
  using A = DemapArith<T>;
  extern __shared__ __align__(16) unsigned char demap_smem[];
  T *sp = reinterpret_cast<T *>(demap_smem);
  const int form = stage_points<NB, T>(sp, pts);
  const int64_t total = (int64_t)nblk * ncell;
  for (int64_t g0 = (int64_t)blockIdx.x * DEMAP_T; g0 < total;
       g0 += (int64_t)gridDim.x * DEMAP_T) {
    // row and cell: one 32-bit division where the batch allows it, else the CTA's
    // first cell and a 32-bit step from it
    int64_t b;
    uint32_t x = threadIdx.x;
    if (total <= 0xFFFFFFFFll - DEMAP_T) {
      x += (uint32_t)g0;
      b = 0;
    } else {
      b = g0 / ncell;
      x += (uint32_t)(g0 - b * ncell);
    }
    const uint32_t step = x / (uint32_t)ncell;
    b += step;
    const int s = (int)(x - step * (uint32_t)ncell);
    if (b >= nblk) break;
    const typename Cell2<T>::type z = cells[(size_t)b * ld_cells + s];
    T mn[NB][2];
    cell_minima<NB, T>(z.x, z.y, sp, form, mn);
    T s2 = s2scalar;
    if (sigma_mode == 1) s2 = sigma2[(size_t)b * ld_sigma + s];
    else if (sigma_mode == 2) s2 = sigma2[b];
    T d[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      d[i] = A::sub(mn[i][1], mn[i][0]);
      if (sigma_mode != 3) d[i] = A::div(d[i], s2);
    }
    store_llrs<NB, T>(d, s, lam_of_q, out + (size_t)b * ld_out);
  }
}

// sigma2[b] = max(mean_s(|z|^2 + min_k q_k), 1e-9); float64 accumulation.
template <int NB>
__global__ void __launch_bounds__(256) row_sigma_kernel(
    const float2 *__restrict__ cells, int64_t ld_cells, int ncell,
    const float *__restrict__ pts, float *__restrict__ sigma2) {
  extern __shared__ __align__(16) unsigned char demap_smem[];
  __shared__ double red[32];
  float *sp = reinterpret_cast<float *>(demap_smem);
  const int form = stage_points<NB, float>(sp, pts);
  const int b = blockIdx.x;
  double acc = 0.0;
  for (int s = threadIdx.x; s < ncell; s += blockDim.x) {
    const float2 z = cells[(size_t)b * ld_cells + s];
    float mn[NB][2];
    cell_minima<NB, float>(z.x, z.y, sp, form, mn);
    const float qmin = fminf(mn[0][0], mn[0][1]);
    const float z2 = __fadd_rn(__fmul_rn(z.x, z.x), __fmul_rn(z.y, z.y));
    acc += (double)__fadd_rn(z2, qmin);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    const float m = (float)(t / (double)ncell);
    sigma2[b] = fmaxf(m, 1e-9f);
  }
}

// sigma2[b] = max(mean_s(|z|^2 + min_k q_k), 1e-9) in float64 (the estimate
// of lab/m16_demap_fast.py:104-106).
template <int NB>
__global__ void __launch_bounds__(256) row_sigma_f64_kernel(
    const double2 *__restrict__ cells, int64_t ld_cells, int ncell,
    const double *__restrict__ pts, double *__restrict__ sigma2) {
  using A = DemapArith<double>;
  extern __shared__ __align__(16) unsigned char demap_smem[];
  __shared__ double red[32];
  double *sp = reinterpret_cast<double *>(demap_smem);
  const int form = stage_points<NB, double>(sp, pts);
  const int b = blockIdx.x;
  double acc = 0.0;
  for (int s = threadIdx.x; s < ncell; s += blockDim.x) {
    const double2 z = cells[(size_t)b * ld_cells + s];
    double mn[NB][2];
    cell_minima<NB, double>(z.x, z.y, sp, form, mn);
    const double qmin = A::min(mn[0][0], mn[0][1]);
    const double z2 = A::add(A::mul(z.x, z.x), A::mul(z.y, z.y));
    acc += A::add(z2, qmin);
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    sigma2[b] = fmax(t / (double)ncell, 1e-9);
  }
}

// ---- sigma2 estimated from the cells ----------------------------------------
// A row's estimate needs the same minima as its LLRs, so one pass writes the
// undivided LLRs and per-CTA sums of |z|^2 + min_k q_k (float64), and a second
// adds a row's sums in a fixed order and divides.  Rows are cut into `chunks`
// pieces: one CTA a row, as a separate estimate had it, left a single long row
// (the reference's call) on one SM: 113401 cells of 256 points in float64 took
// 2774 us for the estimate and 52 for the LLRs; the two passes now take 29.
template <int NB, typename T>
__global__ void __launch_bounds__(DEMAP_T, (demap_ctas<NB, T>())) demap_sum_kernel(
    const typename Cell2<T>::type *__restrict__ cells, int64_t ld_cells, int ncell,
    int chunks, const T *__restrict__ pts, const int32_t *__restrict__ lam_of_q,
    T *__restrict__ out, int64_t ld_out, double *__restrict__ sums) {
  using A = DemapArith<T>;
  extern __shared__ __align__(16) unsigned char demap_smem[];
  __shared__ double red[DEMAP_T / 32];
  T *sp = reinterpret_cast<T *>(demap_smem);
  const int form = stage_points<NB, T>(sp, pts);
  const int b = blockIdx.x / chunks, chunk = blockIdx.x - b * chunks;
  const typename Cell2<T>::type *row = cells + (size_t)b * ld_cells;
  T *o = out + (size_t)b * ld_out;
  double acc = 0.0;
  for (int64_t s = (int64_t)chunk * DEMAP_T + threadIdx.x; s < ncell;
       s += (int64_t)chunks * DEMAP_T) {
    const typename Cell2<T>::type z = row[s];
    T mn[NB][2];
    cell_minima<NB, T>(z.x, z.y, sp, form, mn);
    const T z2 = A::add(A::mul(z.x, z.x), A::mul(z.y, z.y));
    acc += (double)A::add(z2, A::min(mn[0][0], mn[0][1]));
    T d[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) d[i] = A::sub(mn[i][1], mn[i][0]);
    store_llrs<NB, T>(d, (int)s, lam_of_q, o);
  }
  for (int w = 16; w > 0; w >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, w);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < DEMAP_T / 32; ++w) t += red[w];
    sums[blockIdx.x] = t;
  }
}

__device__ __forceinline__ float row_sigma2(double mean, float) {
  return fmaxf((float)mean, 1e-9f);
}
__device__ __forceinline__ double row_sigma2(double mean, double) { return fmax(mean, 1e-9); }

template <typename T>
__global__ void __launch_bounds__(DEMAP_T) demap_scale_kernel(
    const double *__restrict__ sums, int sum_chunks, int ncell, int chunks, int width,
    T *__restrict__ out, int64_t ld_out) {
  using A = DemapArith<T>;
  using T2 = typename Cell2<T>::type;
  __shared__ double red[DEMAP_T / 32];
  const int b = blockIdx.x / chunks, chunk = blockIdx.x - b * chunks;
  double acc = 0.0;
  for (int k = threadIdx.x; k < sum_chunks; k += DEMAP_T) acc += sums[(size_t)b * sum_chunks + k];
  for (int w = 16; w > 0; w >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, w);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < DEMAP_T / 32; ++w) t += red[w];
  const T s2 = row_sigma2(t / (double)ncell, T(0));
  T *o = out + (size_t)b * ld_out;
  const int64_t at = (int64_t)chunk * DEMAP_T + threadIdx.x, step = (int64_t)chunks * DEMAP_T;
  if (width % 2 == 0 && (reinterpret_cast<uintptr_t>(o) & (sizeof(T2) - 1)) == 0) {
    T2 *v = reinterpret_cast<T2 *>(o);
    for (int64_t i = at; i < width / 2; i += step) {
      T2 d = v[i];
      d.x = A::div(d.x, s2);
      d.y = A::div(d.y, s2);
      v[i] = d;
    }
  } else {
    for (int64_t i = at; i < width; i += step) o[i] = A::div(o[i], s2);
  }
}

typedef void (*DemapF64Fn)(const double2 *, int64_t, int, int, const double *,
                           int, const double *, int64_t, double,
                           const int32_t *, double *, int64_t);
typedef void (*SigmaF64Fn)(const double2 *, int64_t, int, const double *,
                           double *);

static DemapF64Fn demap_f64_fn(int nb) {
  switch (nb) {
    case 2: return demap_kernel<2, double>;
    case 4: return demap_kernel<4, double>;
    case 6: return demap_kernel<6, double>;
    case 8: return demap_kernel<8, double>;
    case 10: return demap_kernel<10, double>;
    case 12: return demap_kernel<12, double>;
  }
  return nullptr;
}

static SigmaF64Fn sigma_f64_fn(int nb) {
  switch (nb) {
    case 2: return row_sigma_f64_kernel<2>;
    case 4: return row_sigma_f64_kernel<4>;
    case 6: return row_sigma_f64_kernel<6>;
    case 8: return row_sigma_f64_kernel<8>;
    case 10: return row_sigma_f64_kernel<10>;
    case 12: return row_sigma_f64_kernel<12>;
  }
  return nullptr;
}

typedef void (*DemapFn)(const float2 *, int64_t, int, int, const float *, int,
                        const float *, int64_t, float, const int32_t *,
                        float *, int64_t);
typedef void (*SigmaFn)(const float2 *, int64_t, int, const float *, float *);

static DemapFn demap_fn(int nb) {
  switch (nb) {
    case 2: return demap_kernel<2, float>;
    case 4: return demap_kernel<4, float>;
    case 6: return demap_kernel<6, float>;
    case 8: return demap_kernel<8, float>;
    case 10: return demap_kernel<10, float>;
    case 12: return demap_kernel<12, float>;
  }
  return nullptr;
}

static SigmaFn sigma_fn(int nb) {
  switch (nb) {
    case 2: return row_sigma_kernel<2>;
    case 4: return row_sigma_kernel<4>;
    case 6: return row_sigma_kernel<6>;
    case 8: return row_sigma_kernel<8>;
    case 10: return row_sigma_kernel<10>;
    case 12: return row_sigma_kernel<12>;
  }
  return nullptr;
}

// CTAs per SM at most: enough for the hardware to even out the last wave; where
// staging the alphabet costs as much as demapping a CTA's cells (12 or 48 KB of
// grid points, a few labels formed per cell), no more than are resident at once.
static int demap_waves(int nbits) { return nbits >= 10 ? 3 : 32; }

static int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

int32_t demap_launch(const float *cells, int64_t ld_cells, int nblk, int ncell,
                     const float *pts, int nbits, int sigma_mode,
                     const float *sigma2, int64_t ld_sigma, float s2scalar,
                     const int32_t *lam_of_q, float *out, int64_t ld_out,
                     cudaStream_t st) {
  ATSC3_ARG(nblk >= 0 && ncell >= 0, "negative size");
  ATSC3_ARG(sigma_mode >= 0 && sigma_mode <= 3, "sigma_mode must be 0..3");
  DemapFn fn = demap_fn(nbits);
  ATSC3_ARG(fn != nullptr, "nbits must be 2, 4, 6, 8, 10 or 12");
  if (nblk == 0 || ncell == 0) return 0;
  ATSC3_ARG(cells && pts && out, "null pointer");
  ATSC3_ARG(ld_cells >= ncell, "ld_cells < ncell");
  ATSC3_ARG(ld_out >= (int64_t)ncell * nbits, "ld_out < ncell*nbits");
  ATSC3_ARG(((uintptr_t)cells & 7) == 0, "cells must be 8-byte aligned");
  ATSC3_ARG(!(sigma_mode == 1 || sigma_mode == 2) || sigma2 != nullptr,
            "sigma2 array required");
  ATSC3_ARG(sigma_mode != 1 || ld_sigma >= ncell, "ld_sigma < ncell");
  const int smem = demap_smem_bytes(nbits, 4);
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)fn,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    smem));
  const int64_t total = (int64_t)nblk * ncell;
  int64_t grid = (total + DEMAP_T - 1) / DEMAP_T;
  const int64_t cap = (int64_t)num_sms() * demap_waves(nbits);
  if (grid > cap) grid = cap;
  fn<<<(unsigned)grid, DEMAP_T, smem, st>>>((const float2 *)cells, ld_cells, nblk,
                                       ncell, pts, sigma_mode, sigma2,
                                       ld_sigma, s2scalar, lam_of_q, out,
                                       ld_out);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

int32_t demap_f64_launch(const double *cells, int64_t ld_cells, int nblk,
                         int ncell, const double *pts, int nbits,
                         int sigma_mode, const double *sigma2,
                         int64_t ld_sigma, double s2scalar,
                         const int32_t *lam_of_q, double *out, int64_t ld_out,
                         cudaStream_t st) {
  ATSC3_ARG(nblk >= 0 && ncell >= 0, "negative size");
  ATSC3_ARG(sigma_mode >= 0 && sigma_mode <= 2, "sigma_mode must be 0..2");
  DemapF64Fn fn = demap_f64_fn(nbits);
  ATSC3_ARG(fn != nullptr, "nbits must be 2, 4, 6, 8, 10 or 12");
  if (nblk == 0 || ncell == 0) return 0;
  ATSC3_ARG(cells && pts && out, "null pointer");
  ATSC3_ARG(ld_cells >= ncell, "ld_cells < ncell");
  ATSC3_ARG(ld_out >= (int64_t)ncell * nbits, "ld_out < ncell*nbits");
  ATSC3_ARG(((uintptr_t)cells & 15) == 0, "cells must be 16-byte aligned");
  ATSC3_ARG(sigma_mode == 0 || sigma2 != nullptr, "sigma2 array required");
  ATSC3_ARG(sigma_mode != 1 || ld_sigma >= ncell, "ld_sigma < ncell");
  const int smem = demap_smem_bytes(nbits, 8);
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)fn,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    smem));
  const int64_t total = (int64_t)nblk * ncell;
  int64_t grid = (total + DEMAP_T - 1) / DEMAP_T;
  const int64_t cap = (int64_t)num_sms() * demap_waves(nbits);
  if (grid > cap) grid = cap;
  fn<<<(unsigned)grid, DEMAP_T, smem, st>>>((const double2 *)cells, ld_cells, nblk,
                                       ncell, pts, sigma_mode, sigma2,
                                       ld_sigma, s2scalar, lam_of_q, out,
                                       ld_out);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

int32_t row_sigma_f64_launch(const double *cells, int64_t ld_cells, int nblk,
                             int ncell, const double *pts, int nbits,
                             double *sigma2, cudaStream_t st) {
  SigmaF64Fn fn = sigma_f64_fn(nbits);
  ATSC3_ARG(fn != nullptr, "nbits must be 2, 4, 6, 8, 10 or 12");
  ATSC3_ARG(nblk >= 0 && ncell > 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(cells && pts && sigma2, "null pointer");
  ATSC3_ARG(ld_cells >= ncell, "ld_cells < ncell");
  ATSC3_ARG(((uintptr_t)cells & 15) == 0, "cells must be 16-byte aligned");
  const int smem = demap_smem_bytes(nbits, 8);
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)fn,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    smem));
  fn<<<nblk, 256, smem, st>>>((const double2 *)cells, ld_cells, ncell, pts,
                              sigma2);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

int32_t row_sigma_launch(const float *cells, int64_t ld_cells, int nblk,
                         int ncell, const float *pts, int nbits, float *sigma2,
                         cudaStream_t st) {
  SigmaFn fn = sigma_fn(nbits);
  ATSC3_ARG(fn != nullptr, "nbits must be 2, 4, 6, 8, 10 or 12");
  ATSC3_ARG(nblk >= 0 && ncell > 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(cells && pts && sigma2, "null pointer");
  ATSC3_ARG(((uintptr_t)cells & 7) == 0, "cells must be 8-byte aligned");
  const int smem = demap_smem_bytes(nbits, 4);
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)fn,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    smem));
  fn<<<nblk, 256, smem, st>>>((const float2 *)cells, ld_cells, ncell, pts,
                              sigma2);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

// CTAs a row of the estimating pass: what fills the chip, at most the row's
// cells and the 4096 sums the workspace holds beyond one per row.
template <int NB, typename T>
static int32_t demap_estimate_nb(const T *cells, int64_t ld_cells, int nblk, int ncell,
                                 const T *pts, const int32_t *lam_of_q, T *out,
                                 int64_t ld_out, double *work, cudaStream_t st) {
  using T2 = typename Cell2<T>::type;
  auto *fn = demap_sum_kernel<NB, T>;
  const int smem = demap_smem_bytes(NB, sizeof(T));
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)fn,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  const int full = std::max(1, std::min(4096, num_sms() * demap_waves(NB)) / nblk);
  const int chunks = std::min((ncell + DEMAP_T - 1) / DEMAP_T, full);
  fn<<<nblk * chunks, DEMAP_T, smem, st>>>((const T2 *)cells, ld_cells, ncell, chunks, pts,
                                           lam_of_q, out, ld_out, work);
  ATSC3_CUDA(cudaGetLastError());
  const int width = ncell * NB;
  const int wide = std::max(1, std::min((width + 4 * DEMAP_T - 1) / (4 * DEMAP_T),
                                        num_sms() * 8 / nblk));
  demap_scale_kernel<T><<<nblk * wide, DEMAP_T, 0, st>>>(work, chunks, ncell, wide, width, out,
                                                        ld_out);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

// Many short rows: one pass over the rows for the estimates and one over all cells
// for the LLRs.  A row's own CTA in both passes leaves most threads idle below 256
// cells, and QPSK's minima cost less than reading its LLRs back (us, one pass that
// is divided after / two passes, float32: 6666 rows of 30 cells, QPSK 23.0 / 10.9,
// 64 points 31.6 / 18.8; 1562 of 128, 9.1 / 6.5 and 13.1 / 11.8; 778 of 257, 256
// points 21.0 / 21.6; QPSK 1481 of 1350 cells 19.5 / 16.6).
static bool demap_short_rows(int nblk, int ncell, int nbits) {
  return nblk >= num_sms() && (ncell <= 256 || (nbits == 2 && ncell <= 4096));
}

static int32_t demap_short(const float *cells, int64_t ld_cells, int nblk, int ncell,
                           const float *pts, int nbits, const int32_t *lam_of_q, float *out,
                           int64_t ld_out, void *work, cudaStream_t st) {
  float *s2 = (float *)work;
  const int32_t rc = row_sigma_launch(cells, ld_cells, nblk, ncell, pts, nbits, s2, st);
  return rc ? rc : demap_launch(cells, ld_cells, nblk, ncell, pts, nbits, 2, s2, 0, 1.f, lam_of_q,
                                out, ld_out, st);
}

static int32_t demap_short(const double *cells, int64_t ld_cells, int nblk, int ncell,
                           const double *pts, int nbits, const int32_t *lam_of_q, double *out,
                           int64_t ld_out, void *work, cudaStream_t st) {
  double *s2 = (double *)work;
  const int32_t rc = row_sigma_f64_launch(cells, ld_cells, nblk, ncell, pts, nbits, s2, st);
  return rc ? rc : demap_f64_launch(cells, ld_cells, nblk, ncell, pts, nbits, 2, s2, 0, 1.0,
                                    lam_of_q, out, ld_out, st);
}

template <typename T>
static int32_t demap_estimate_launch(const T *cells, int64_t ld_cells, int nblk, int ncell,
                                     const T *pts, int nbits, const int32_t *lam_of_q, T *out,
                                     int64_t ld_out, void *work, cudaStream_t st) {
  ATSC3_ARG(nbits >= 2 && nbits <= 12 && nbits % 2 == 0, "nbits must be 2, 4, 6, 8, 10 or 12");
  ATSC3_ARG(nblk >= 0 && ncell > 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(cells && pts && out && work, "null pointer");
  ATSC3_ARG(ld_cells >= ncell, "ld_cells < ncell");
  ATSC3_ARG(ld_out >= (int64_t)ncell * nbits, "ld_out < ncell*nbits");
  ATSC3_ARG((int64_t)ncell * nbits <= INT32_MAX, "a row of more than 2^31 - 1 LLRs");
  ATSC3_ARG(((uintptr_t)cells & (2 * sizeof(T) - 1)) == 0, "cells must be aligned to a cell");
  if (demap_short_rows(nblk, ncell, nbits))
    return demap_short(cells, ld_cells, nblk, ncell, pts, nbits, lam_of_q, out, ld_out, work, st);
  double *w = (double *)work;
  switch (nbits) {
    case 2: return demap_estimate_nb<2, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
    case 4: return demap_estimate_nb<4, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
    case 6: return demap_estimate_nb<6, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
    case 8: return demap_estimate_nb<8, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
    case 10: return demap_estimate_nb<10, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
    default: return demap_estimate_nb<12, T>(cells, ld_cells, nblk, ncell, pts, lam_of_q, out, ld_out, w, st);
  }
}

// ---- uneven batches: every block its own constellation ---------------------
// One CTA per chunk of up to 256 cells of one block (chunk_blk / chunk_start
// built on the host); the CTA stages its block's alphabet (up to 4096
// points) and dispatches on the block's bits per symbol.
struct DemapBatchArgs {
  const float2 *cells;
  const int64_t *cell_off;
  const int32_t *ncell;
  const int32_t *nbits;
  const float *pts;
  const int64_t *pts_off;     // floats, 3*M per alphabet
  const float *sigma2;        // one per block
  const int32_t *lq;
  const int64_t *lq_off;
  float *llr;
  const int64_t *llr_off;
  const int32_t *chunk_blk;
  const int32_t *chunk_start;
};

template <int NB>
__device__ __forceinline__ void demap_cell_batch(const DemapBatchArgs &a, int b,
                                                 int s, float *sp) {
  const int form = stage_points<NB, float>(sp, a.pts + a.pts_off[b]);
  if (s >= a.ncell[b]) return;
  const float2 z = a.cells[a.cell_off[b] + s];
  float mn[NB][2];
  cell_minima<NB, float>(z.x, z.y, sp, form, mn);
  const float s2 = a.sigma2[b];
  float d[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i) d[i] = __fdiv_rn(__fsub_rn(mn[i][1], mn[i][0]), s2);
  store_llrs<NB, float>(d, s, a.lq + a.lq_off[b], a.llr + a.llr_off[b]);
}

__global__ void __launch_bounds__(256) demap_batch_kernel(const DemapBatchArgs a) {
  extern __shared__ __align__(16) unsigned char demap_smem[];
  float *sp = reinterpret_cast<float *>(demap_smem);
  const int b = a.chunk_blk[blockIdx.x];
  const int s = a.chunk_start[blockIdx.x] + threadIdx.x;
  switch (a.nbits[b]) {
    case 2: demap_cell_batch<2>(a, b, s, sp); break;
    case 4: demap_cell_batch<4>(a, b, s, sp); break;
    case 6: demap_cell_batch<6>(a, b, s, sp); break;
    case 8: demap_cell_batch<8>(a, b, s, sp); break;
    case 10: demap_cell_batch<10>(a, b, s, sp); break;
    case 12: demap_cell_batch<12>(a, b, s, sp); break;
  }
}

}  // namespace atsc3

extern "C" {

int32_t atsc3_demap_batch(const float *cells, const int64_t *cell_off,
                          const int32_t *ncell, const int32_t *nbits,
                          const float *pts, const int64_t *pts_off,
                          const float *sigma2, const int32_t *lq,
                          const int64_t *lq_off, float *llr,
                          const int64_t *llr_off, const int32_t *chunk_blk,
                          const int32_t *chunk_start, int32_t nchunks,
                          int32_t max_nbits, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(nchunks >= 0, "negative size");
  if (nchunks == 0) return 0;
  ATSC3_ARG(cells && cell_off && ncell && nbits && pts && pts_off && sigma2 &&
                lq && lq_off && llr && llr_off && chunk_blk && chunk_start,
            "null pointer");
  ATSC3_ARG(max_nbits >= 2 && max_nbits <= 12, "max_nbits must be 2..12");
  const int smem = demap_smem_bytes(max_nbits, 4);
  if (smem > 48 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)demap_batch_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  DemapBatchArgs a{(const float2 *)cells, cell_off, ncell, nbits, pts, pts_off,
                   sigma2, lq, lq_off, llr, llr_off, chunk_blk, chunk_start};
  demap_batch_kernel<<<nchunks, 256, smem, (cudaStream_t)stream>>>(a);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}


int32_t atsc3_demap(const float *cells, int64_t ld_cells, int32_t nblk,
                    int32_t ncell, const float *pts, int32_t nbits,
                    int32_t sigma_mode, const float *sigma2, int64_t ld_sigma,
                    float sigma2_scalar, const int32_t *lam_of_q, float *out,
                    int64_t ld_out, void *stream) {
  return atsc3::demap_launch(cells, ld_cells, nblk, ncell, pts, nbits,
                             sigma_mode, sigma2, ld_sigma, sigma2_scalar,
                             lam_of_q, out, ld_out, (cudaStream_t)stream);
}

int32_t atsc3_demap_f64(const double *cells, int64_t ld_cells, int32_t nblk,
                        int32_t ncell, const double *pts, int32_t nbits,
                        int32_t sigma_mode, const double *sigma2,
                        int64_t ld_sigma, double sigma2_scalar,
                        const int32_t *lam_of_q, double *out, int64_t ld_out,
                        void *stream) {
  return atsc3::demap_f64_launch(cells, ld_cells, nblk, ncell, pts, nbits,
                                 sigma_mode, sigma2, ld_sigma, sigma2_scalar,
                                 lam_of_q, out, ld_out, (cudaStream_t)stream);
}

int32_t atsc3_demap_estimate(const float *cells, int64_t ld_cells, int32_t nblk,
                             int32_t ncell, const float *pts, int32_t nbits,
                             const int32_t *lam_of_q, float *out, int64_t ld_out,
                             void *work, void *stream) {
  return atsc3::demap_estimate_launch<float>(cells, ld_cells, nblk, ncell, pts, nbits, lam_of_q,
                                             out, ld_out, work, (cudaStream_t)stream);
}

int32_t atsc3_demap_estimate_f64(const double *cells, int64_t ld_cells, int32_t nblk,
                                 int32_t ncell, const double *pts, int32_t nbits,
                                 const int32_t *lam_of_q, double *out, int64_t ld_out,
                                 void *work, void *stream) {
  return atsc3::demap_estimate_launch<double>(cells, ld_cells, nblk, ncell, pts, nbits, lam_of_q,
                                              out, ld_out, work, (cudaStream_t)stream);
}

int32_t atsc3_demap_row_sigma2_f64(const double *cells, int64_t ld_cells,
                                   int32_t nblk, int32_t ncell,
                                   const double *pts, int32_t nbits,
                                   double *sigma2, void *stream) {
  return atsc3::row_sigma_f64_launch(cells, ld_cells, nblk, ncell, pts, nbits,
                                     sigma2, (cudaStream_t)stream);
}

int32_t atsc3_demap_row_sigma2(const float *cells, int64_t ld_cells,
                               int32_t nblk, int32_t ncell, const float *pts,
                               int32_t nbits, float *sigma2, void *stream) {
  return atsc3::row_sigma_launch(cells, ld_cells, nblk, ncell, pts, nbits,
                                 sigma2, (cudaStream_t)stream);
}

}  // extern "C"
