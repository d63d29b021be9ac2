// cpe.cu -- common phase error correction of an OFDM cell pool (sm_100a):
// the decision-directed per-symbol complex gain of lab/m6_cells.py:176-209
// (cpe_correct; the same algorithm as lab/m9_gpu.py:283-299 and
// lab/m9_fast.py:619-753), the stage before the demapper.
//
//   z = pool / sqrt(mean |pool|^2)
//   per OFDM symbol, `iters` times:
//     hard = nearest point of the cell's region alphabet (argmin |z - p|,
//            first minimum wins), or the known dummy value (region 2);
//     c = sum conj(hard)*z / max(sum |hard|^2, 1e-12);  z /= c;  gain *= c
//
// Results in float64 throughout.  A cluster of CTAs per symbol (symbols are
// contiguous ranges of the pool); the per-symbol sums are added in a fixed
// order, so results are deterministic.  Agreement with the numpy reference is
// to float64 rounding (its sums are BLAS dot products and numpy pairwise means,
// summed in other orders; z is formed from the pool and the total gain in each
// iteration, not divided again); hard decisions agree.
//
// Work: 3 x cells x points distances.  A float32 screen finds the decision and
// proves it: where the best point leads every other by more than the screen's
// rounding, it is the float64 answer; elsewhere (about 1 cell in 1000) the
// points within the rounding are compared as the reference does, by float64
// hypot in label order.  On quadrant-symmetric alphabets (A/322's) the screen
// looks at the quarter of the points around the cell's own quadrant.
// 61 symbols of 19949 cells, 256 and 16 points, 3 iterations, B200: 6662 us
// (one CTA per symbol, hypot of every point) -> 152 us.

#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/atsc3_fec.h"
#include "common.cuh"

namespace atsc3 {

constexpr int CPE_T = 256;
constexpr int CPE_CL = 8;         // CTAs per symbol at most (portable cluster)
constexpr int CPE_BLK = 8;        // points per block of the screen

struct CpeArgs {
  const double2 *pool;
  int64_t n;
  const int32_t *sym_ptr;
  int nsym;
  const uint8_t *region;
  const double2 *alph0;
  int m0;
  const double2 *alph1;
  int m1;
  const double2 *dummy;
  int iters;
  double *work;          // power partials
  int nparts;
  double2 *out;
  double2 *gains;
};

// Smith's algorithm for a / b (Smith, CACM 5(8), 1962), the form numpy's
// complex128 division uses; b's part of it, formed once for many a
struct SmithDiv {
  double rat, scl;
  bool re;               // |Re b| >= |Im b|
  __device__ explicit SmithDiv(double2 b) {
    re = fabs(b.x) >= fabs(b.y);
    rat = re ? b.y / b.x : b.x / b.y;
    scl = re ? 1.0 / (b.x + b.y * rat) : 1.0 / (b.y + b.x * rat);
  }
  __device__ double2 operator()(double2 a) const {
    return re ? make_double2((a.x + a.y * rat) * scl, (a.y - a.x * rat) * scl)
              : make_double2((a.x * rat + a.y) * scl, (a.y * rat - a.x) * scl);
  }
};

// sum over the CTA in a fixed order (every thread gets it)
template <int K>
__device__ __forceinline__ void cpe_block_sum(double (&v)[K], double (*red)[CPE_T / 32]) {
#pragma unroll
  for (int k = 0; k < K; ++k) {
    for (int w = 16; w > 0; w >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], w);
    if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    v[k] = 0.0;
    for (int w = 0; w < CPE_T / 32; ++w) v[k] += red[k][w];
  }
  __syncthreads();
}

// per-block partial sums of |pool|^2
__global__ void __launch_bounds__(CPE_T) cpe_power_kernel(const CpeArgs a) {
  __shared__ double red[1][CPE_T / 32];
  const int64_t per = (a.n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = per * blockIdx.x;
  const int64_t hi = min(a.n, lo + per);
  double s[1] = {0.0};
  for (int64_t i = lo + threadIdx.x; i < hi; i += CPE_T) {
    const double2 p = a.pool[i];
    s[0] += p.x * p.x + p.y * p.y;
  }
  cpe_block_sum<1>(s, red);
  if (threadIdx.x == 0) a.work[blockIdx.x] = s[0];
}

// One alphabet in shared memory as the float32 screen reads it: Re, Im and
// |p|^2 of every point, padded to whole blocks with points no cell is near.
struct CpeTable {
  const float *re, *im, *p2;
  const double2 *exact;
  int m;                 // points
  int look;              // points the screen looks at: m / 4 with fold, else m
  bool fold;             // label = quadrant * m/4 + j, mirrored as A/322's NUCs
  float big, pow;        // largest |re|, |im|; largest |p|^2 (NaN: no screen)
};

__host__ __device__ inline int cpe_padded(int m) { return (m + CPE_BLK - 1) / CPE_BLK * CPE_BLK; }

// Every thread of the CTA calls it; red: two words of shared memory.
__device__ CpeTable cpe_stage(const double2 *p, int m, float *sm, int *red) {
  const int mp = cpe_padded(m);
  CpeTable t{sm, sm + mp, sm + 2 * mp, p, m, m, false, 0.f, 0.f};
  if (threadIdx.x < 2) red[threadIdx.x] = 0;
  __syncthreads();
  const int j4 = m / 4;
  bool mirrored = m >= 4 && m % 4 == 0, sane = true;
  for (int k = threadIdx.x; k < mp; k += CPE_T) {
    float x = 0.f, y = 0.f, q = 1e30f;
    if (k < m) {
      const double2 v = p[k];
      x = (float)v.x;
      y = (float)v.y;
      q = (float)(v.x * v.x + v.y * v.y);
      sane = sane && q < 1e12f;
      atomicMax(red, __float_as_int(fmaxf(fabsf(x), fabsf(y))));
      atomicMax(red + 1, __float_as_int(q));
      if (mirrored) {
        const int u = k / j4;
        const double2 w = p[k - u * j4];
        mirrored = w.x > 0.0 && w.y > 0.0 && v.x == (u & 1 ? -w.x : w.x) &&
                   v.y == (u & 2 ? -w.y : w.y);
      }
    }
    sm[k] = x;
    sm[mp + k] = y;
    sm[2 * mp + k] = q;
  }
  mirrored = __syncthreads_and(mirrored);
  sane = __syncthreads_and(sane);
  t.big = sane ? __int_as_float(red[0]) : __int_as_float(0x7fffffff);
  t.pow = __int_as_float(red[1]);
  __syncthreads();
  // folded only where a quarter is whole blocks (64 points and more): the
  // screen would otherwise run into the next quadrant's points
  if (mirrored && j4 % CPE_BLK == 0) {
    t.fold = true;
    t.look = j4;
  }
  return t;
}

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 cpe_dup(float v) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}
__device__ __forceinline__ f32x2 cpe_fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// |p|^2 - 2 Re(z conj p) of a block's points
__device__ __forceinline__ void cpe_metric(const CpeTable &t, int k0, f32x2 x, f32x2 y,
                                           float (&q)[CPE_BLK]) {
#pragma unroll
  for (int l = 0; l < CPE_BLK; l += 4) {
    const ulonglong2 r = *reinterpret_cast<const ulonglong2 *>(t.re + k0 + l);
    const ulonglong2 i = *reinterpret_cast<const ulonglong2 *>(t.im + k0 + l);
    const ulonglong2 p = *reinterpret_cast<const ulonglong2 *>(t.p2 + k0 + l);
    const f32x2 a = cpe_fma2(x, r.x, cpe_fma2(y, i.x, p.x));
    const f32x2 b = cpe_fma2(x, r.y, cpe_fma2(y, i.y, p.y));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(q[l]), "=f"(q[l + 1]) : "l"(a));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(q[l + 2]), "=f"(q[l + 3]) : "l"(b));
  }
}

// the reference's decision over every point: first minimum of the float64 hypot
__device__ __noinline__ int cpe_decide_all(const double2 *exact, int m, double2 z) {
  double best = hypot(z.x - exact[0].x, z.y - exact[0].y);
  int bi = 0;
  for (int k = 1; k < m; ++k) {
    const double d = hypot(z.x - exact[k].x, z.y - exact[k].y);
    if (d < best) {
      best = d;
      bi = k;
    }
  }
  return bi;
}

// the same over the points whose screen value (x2, y2: -2 z, folded like the
// screen's) is at most `most`, their mirror images among them
__device__ __noinline__ int cpe_decide_near(CpeTable t, double2 z, float x2, float y2, float most) {
  const f32x2 x = cpe_dup(x2), y = cpe_dup(y2);
  double best = 0.0;
  int bi = -1;
  for (int k0 = 0; k0 < t.look; k0 += CPE_BLK) {
    float q[CPE_BLK];
    cpe_metric(t, k0, x, y, q);
    uint32_t near = 0;
#pragma unroll
    for (int l = 0; l < CPE_BLK; ++l) near |= q[l] <= most ? 1u << l : 0u;
    while (near) {
      const int j = k0 + __ffs(near) - 1;
      near &= near - 1;
      for (int k = j; k < t.m; k += t.fold ? t.look : t.m) {
        const double2 p = t.exact[k];
        const double d = hypot(z.x - p.x, z.y - p.y);
        if (bi < 0 || d < best || (d == best && k < bi)) {
          best = d;
          bi = k;
        }
      }
    }
  }
  return bi;
}

// Nearest point of z.  The screen's q differs from the real |p|^2 - 2 Re(z
// conj p) by at most u (8 B (|Re z| + |Im z|) + 3 P), u = 2^-24, B and P the
// largest coordinate and power: conversions, two products' inputs and two fused
// roundings.  A point that leads all others by twice that is the nearest one.
__device__ __forceinline__ int cpe_decide(const CpeTable &t, double2 z) {
  const float fx = (float)z.x, fy = (float)z.y;
  const float ax = fabsf(fx), ay = fabsf(fy);
  const float margin = 5.9604645e-8f * (17.f * t.big * (ax + ay) + 7.f * t.pow);
  // (far out, or with an alphabet the screen cannot hold: every point)
  if (!(margin < 1e12f && ax + ay <= 1e6f * t.big)) return cpe_decide_all(t.exact, t.m, z);
  const float x2 = -2.f * (t.fold ? ax : fx), y2 = -2.f * (t.fold ? ay : fy);
  const f32x2 x = cpe_dup(x2), y = cpe_dup(y2);
  float best = 3e38f, next = 3e38f;
  int at = 0;
  for (int k0 = 0; k0 < t.look; k0 += CPE_BLK) {
    float q[CPE_BLK];
    cpe_metric(t, k0, x, y, q);
    float m = q[0];
#pragma unroll
    for (int l = 1; l < CPE_BLK; ++l) m = fminf(m, q[l]);
    next = fminf(next, fmaxf(best, m));
    at = m < best ? k0 : at;
    best = fminf(best, m);
  }
  const float most = best + margin;
  float q[CPE_BLK];
  cpe_metric(t, at, x, y, q);
  int n = 0, k = at;
#pragma unroll
  for (int l = 0; l < CPE_BLK; ++l) {
    const bool near = q[l] <= most;
    n += near;
    k = near ? at + l : k;
  }
  bool sure = n == 1 && next > most;
  if (t.fold) {
    // the mirror images of the point found are 4 |Re z| Re p and 4 |Im z| Im p
    // further
    sure = sure && 3.99f * ax * t.re[k] > margin && 3.99f * ay * t.im[k] > margin;
    k += t.look * ((fx < 0.f ? 1 : 0) + (fy < 0.f ? 2 : 0));
  }
  if (sure) return k;
  return cpe_decide_near(t, z, x2, y2, most);
}

__global__ void __launch_bounds__(CPE_T, 4) cpe_symbol_kernel(const CpeArgs a) {
  extern __shared__ __align__(16) float cpe_smem[];
  __shared__ double red[3][CPE_T / 32];
  __shared__ double part[2][3];      // this CTA's sums, alternating iterations
  __shared__ int ired[2];
  const CpeTable t0 = cpe_stage(a.alph0, a.m0, cpe_smem, ired);
  const CpeTable t1 = cpe_stage(a.alph1, a.m1, cpe_smem + 3 * cpe_padded(a.m0), ired);
  const int cl = (int)cluster_nctarank(), rank = (int)cluster_ctarank();
  const int s = blockIdx.x / cl;
  const int64_t s0 = a.sym_ptr[s], s1 = a.sym_ptr[s + 1];
  const int64_t seg = (s1 - s0 + cl - 1) / cl;
  const int64_t lo = s0 + seg * rank, hi = min(s1, lo + seg);
  // unit mean power over the whole pool
  double pw[1] = {0.0};
  for (int k = threadIdx.x; k < a.nparts; k += CPE_T) pw[0] += a.work[k];
  cpe_block_sum<1>(pw, red);
  const double rt = sqrt(pw[0] / (double)a.n);
  const double irt = 1.0 / rt;
  double2 ctot = make_double2(1.0, 0.0);
  for (int it = 0; it < a.iters; ++it) {
    double2 g = SmithDiv(ctot)(make_double2(1.0, 0.0));
    g.x *= irt;
    g.y *= irt;
    double v[3] = {0.0, 0.0, 0.0};
    for (int64_t i = lo + threadIdx.x; i < hi; i += CPE_T) {
      const double2 q = a.pool[i];
      const int r = a.region[i];
      const double2 z = make_double2(q.x * g.x - q.y * g.y, q.x * g.y + q.y * g.x);
      // region 0 / 1: nearest point of that alphabet; 2: the known dummy
      // value; anything else (or a missing table) contributes nothing
      double2 h = make_double2(0.0, 0.0);
      if (r == 2) {
        if (a.dummy) h = a.dummy[i];
      } else if (r < 2) {
        CpeTable t = t0;
        if (r == 1) t = t1;
        if (t.m > 0) h = t.exact[cpe_decide(t, z)];
      }
      v[0] += h.x * z.x + h.y * z.y;      // conj(h) * z
      v[1] += h.x * z.y - h.y * z.x;
      v[2] += h.x * h.x + h.y * h.y;
    }
    cpe_block_sum<3>(v, red);
    double2 c;
    if (cl > 1) {
      if (threadIdx.x == 0) {
        part[it & 1][0] = v[0];
        part[it & 1][1] = v[1];
        part[it & 1][2] = v[2];
      }
      cluster_sync_all();
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        v[k] = 0.0;
        for (int q = 0; q < cl; ++q)
          v[k] += dsmem_ld_f64(dsmem_map(smem_u32(&part[it & 1][k]), (uint32_t)q));
      }
    }
    const double den = fmax(v[2], 1e-12);
    c = make_double2(v[0] / den, v[1] / den);
    ctot = make_double2(ctot.x * c.x - ctot.y * c.y, ctot.x * c.y + ctot.y * c.x);
  }
  const SmithDiv by(ctot);
  for (int64_t i = lo + threadIdx.x; i < hi; i += CPE_T) {
    const double2 q = a.pool[i];
    const double2 z = make_double2(q.x / rt, q.y / rt);
    a.out[i] = a.iters > 0 ? by(z) : z;
  }
  if (rank == 0 && threadIdx.x == 0) a.gains[s] = ctot;
  if (cl > 1) cluster_sync_all();    // no CTA leaves while another reads its sums
}

}  // namespace atsc3

extern "C" {

int32_t atsc3_cpe_workspace(int64_t *work_bytes) {
  ATSC3_ARG(work_bytes != nullptr, "null output");
  *work_bytes = (1 + 1024) * 8;
  return 0;
}

int32_t atsc3_cpe_correct(const double *pool, int64_t ncells,
                          const int32_t *sym_ptr, int32_t nsym,
                          const uint8_t *region, const double *alphabet0,
                          int32_t m0, const double *alphabet1, int32_t m1,
                          const double *dummy, int32_t iters, double *out,
                          double *gains, void *work, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(ncells >= 0 && nsym >= 0 && iters >= 0, "negative size");
  ATSC3_ARG(m0 >= 1 && m1 >= 0 && m0 <= 4096 && m1 <= 4096,
            "alphabets of 1..4096 (and 0..4096) points");
  if (ncells == 0 || nsym == 0) return 0;
  ATSC3_ARG(pool && sym_ptr && region && alphabet0 && out && gains && work,
            "null pointer");
  ATSC3_ARG(m1 == 0 || alphabet1 != nullptr, "alphabet1 required");
  CpeArgs a;
  a.pool = (const double2 *)pool;
  a.n = ncells;
  a.sym_ptr = sym_ptr;
  a.nsym = nsym;
  a.region = region;
  a.alph0 = (const double2 *)alphabet0;
  a.m0 = m0;
  a.alph1 = (const double2 *)(alphabet1 ? alphabet1 : alphabet0);
  a.m1 = m1;
  a.dummy = (const double2 *)dummy;
  a.iters = iters;
  a.work = (double *)work;
  a.out = (double2 *)out;
  a.gains = (double2 *)gains;
  cudaStream_t st = (cudaStream_t)stream;
  const int nparts = (int)std::min<int64_t>(1024, (ncells + CPE_T - 1) / CPE_T);
  a.nparts = nparts;
  cpe_power_kernel<<<nparts, CPE_T, 0, st>>>(a);
  const int smem = 3 * 4 * (cpe_padded(m0) + cpe_padded(m1));
  // 4096 points are 48 KB by themselves, and the kernel's static shared memory
  // counts towards the 48 KB that a launch gets without asking.  Every caller asks
  // for the largest alphabets' size, so none lowers another thread's limit.
  if (smem > 40 * 1024)
    ATSC3_CUDA(cudaFuncSetAttribute((const void *)cpe_symbol_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    3 * 4 * 2 * 4096));
  // CTAs per symbol: what it takes to have four CTAs on every SM (their
  // registers' limit), as long as each keeps a cell for every thread
  // (61 symbols of 19949 cells: 8 CTAs each 151 us, 7 164, 6 at three an SM 148;
  // 10 of 6000: 46, 55, 51)
  int dev = 0, sms = 148;
  ATSC3_CUDA(cudaGetDevice(&dev));
  ATSC3_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int cl = 1;
  while (cl < CPE_CL && (int64_t)nsym * cl * 2 <= 4 * sms && ncells / nsym >= 2 * cl * CPE_T) cl *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(nsym * cl, 1, 1);
  cfg.blockDim = dim3(CPE_T, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ATSC3_CUDA(cudaLaunchKernelEx(&cfg, cpe_symbol_kernel, a));
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

}  // extern "C"
