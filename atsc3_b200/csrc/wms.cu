// wms.cu -- unrolled weighted min-sum with a hand-written backward (sm_100a).
//
// Forward, flooding schedule, iterations t = 1..T (messages m^(0) = 0,
// posterior tot^(0) = llr):
//   x_e   = tot^(t-1)[v(e)] - m^(t-1)_e                       (bit -> check)
//   mu_e  = min over the other edges of |x|  (min1, or min2 at the first
//           minimum; first-minimum rule with strict <)
//   m_e^(t) = sgn_e * relu(alpha[t][d] * mu_e - beta[t][d]),
//           sgn_e = (product of signs of the check's x) * sign(x_e),
//           sign(x) = -1 iff x < 0, d = degree bucket of the check
//   tot^(t)[v] = llr[v] + sum_e m^(t)_e    (ascending edge order)
// Output: tot^(T).  With alpha = a, beta = 0 this is the normalised min-sum
// of lab/ldpc_kernel.c for T fixed iterations (no early stop).
//
// Memory: per iteration one 16-byte record per check {min1, min2, first,
// second, sign bits of x} (checkpoint); the per-edge messages live for one
// iteration only.  The backward walks t = T..1 over the records alone (the
// signs of x^(t) are in them, so no posterior is formed again):
//   G_e   = gtot^(t)[v(e)] - gx^(t+1)_e                       (dL/dm^(t)_e)
//   a_e = alpha*mu_e - beta > 0:  galpha += G sgn mu, gbeta -= G sgn,
//                                 gmu_e = G sgn alpha
//   gx^(t)_first  += sign(x_first)  * sum_{e != first} gmu_e
//   gx^(t)_second += sign(x_second) * gmu_first
//   gtot^(t-1)[v] = sum_e gx^(t)_e
// (signs and the arg-min choice are piecewise constant).  REC selects the
// stored record precision: float (FP32 messages) or bfloat16 minima (BF16
// messages, the low-precision variant).
//
// Layout: every array is [item][block], blocks fastest, and a thread takes VEC
// consecutive blocks of one item (2 or 4, the block count padded up; 1 for
// callers whose buffers have no room for that).  A warp reads consecutive blocks of one
// check, bit or edge, whatever permutation the code applies, and its lanes
// share an index load; the caller's (nblk, n) arrays are transposed on the way in
// and out.  With [block][item] the gathers of one iteration touched a 32-byte
// sector per 4- or 16-byte value.  What bounds it now is moving the messages:
// 4 passes over 4 bytes an edge an iteration forward, 4 backward.
// 64 blocks of 64800 8/15, 12 iterations, forward and backward with the loss:
// 10.5 ms -> 1.9 ms.
//
// Tables are CSR (cptr/cidx check-major; vptr/vedge variable-major edge ids).
// Parameter gradients are reduced per warp (a warp's checks mostly share a
// bucket), then per CTA in shared memory, one atomicAdd per CTA and parameter.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/atsc3_fec.h"
#include "common.cuh"

namespace atsc3 {

struct WmsTables {
  const int32_t *cptr, *cidx, *vptr, *vedge;
  const int8_t *cbucket;     // degree bucket per check
  int n, nc, ne, nbucket;
};

struct WmsRec {              // 16 bytes
  float min1, min2;
  uint16_t first, second;
  uint32_t sx;               // bit j: x_j < 0
};

constexpr int WMS_T = 256;
// Blocks per thread of the check kernels: 2 (64 blocks of 64800 8/15, us a
// launch forward / backward: 63 / 81 with one, 48 / 57 with two, 75 / 66 with
// four, whose registers leave too few threads); the variable kernels take 4 (44 /
// 42 with one, 20 / 18 with four).
constexpr int WMS_CHECK_VEC = 2;

template <bool BF16>
__device__ __forceinline__ float rq(float v) {
  if constexpr (BF16) return __bfloat162float(__float2bfloat16_rn(v));
  return v;
}

// VEC blocks of one value: a thread's share of a load or store
template <int VEC>
struct __align__(4 * VEC) WmsVec {
  float v[VEC];
};

// Where the record of check c and the i-th of this thread's blocks stands in an
// iteration's records: blocks fastest; one block a thread (the entry points
// without padding, whose callers know the records) checks fastest.
template <int VEC>
__device__ __forceinline__ size_t wms_rec_at(int nc, int nv, int c, int b, int i) {
  return VEC == 1 ? (size_t)b * nc + c : ((size_t)c * nv + b) * VEC + i;
}

// item and first block / VEC of this thread (nv = blocks / VEC); false past the end
__device__ __forceinline__ bool wms_item(int items, int nv, int &item, int &b) {
  const int64_t g = (int64_t)blockIdx.x * WMS_T + threadIdx.x;
  if (g >= (int64_t)items * nv) return false;
  if (g <= 0xFFFFFFFFll) {
    const uint32_t i = (uint32_t)g / (uint32_t)nv;
    item = (int)i;
    b = (int)((uint32_t)g - i * (uint32_t)nv);
  } else {
    item = (int)(g / nv);
    b = (int)(g - (int64_t)item * nv);
  }
  return true;
}

// (nblk, n) -> (n, nbp), zeros in the padding; dst2 (nullable): a second copy
__global__ void __launch_bounds__(256) wms_blocks_last(const float *src, int nblk, int n, int nbp,
                                                       float *dst, float *dst2) {
  __shared__ float tile[32][33];
  const int tiles = (n + 31) / 32;
  const int b0 = (int)(blockIdx.x / tiles) * 32, v0 = (int)(blockIdx.x % tiles) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int b = ty; b < 32; b += 8)
    tile[b][tx] = b0 + b < nblk && v0 + tx < n ? src[(size_t)(b0 + b) * n + v0 + tx] : 0.f;
  __syncthreads();
  for (int v = ty; v < 32; v += 8)
    if (v0 + v < n && b0 + tx < nbp) {
      const size_t at = (size_t)(v0 + v) * nbp + b0 + tx;
      dst[at] = tile[tx][v];
      if (dst2) dst2[at] = tile[tx][v];
    }
}

// (n, nbp) -> (nblk, n)
__global__ void __launch_bounds__(256) wms_blocks_first(const float *src, int nblk, int n, int nbp,
                                                        float *dst) {
  __shared__ float tile[32][33];
  const int tiles = (n + 31) / 32;
  const int b0 = (int)(blockIdx.x / tiles) * 32, v0 = (int)(blockIdx.x % tiles) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int v = ty; v < 32; v += 8)
    if (v0 + v < n && b0 + tx < nblk) tile[v][tx] = src[(size_t)(v0 + v) * nbp + b0 + tx];
  __syncthreads();
  for (int b = ty; b < 32; b += 8)
    if (b0 + b < nblk && v0 + tx < n) dst[(size_t)(b0 + b) * n + v0 + tx] = tile[tx][b];
}

// ---- forward: check update of iteration t: record and messages ---------------
// m: messages of iteration t-1 on entry (ignored when FIRST: they are 0), of t
// on return; al/be: scale and offset rows of iteration t
template <int VEC, bool BF16, bool FIRST>
__global__ void __launch_bounds__(WMS_T) wms_check_fwd(WmsTables T, int nv,
                                                       const WmsVec<VEC> *tot, WmsVec<VEC> *m,
                                                       WmsRec *rec, const float *alpha,
                                                       const float *beta) {
  int c, b;
  if (!wms_item(T.nc, nv, c, b)) return;
  const int e0 = T.cptr[c], deg = T.cptr[c + 1] - e0;
  WmsVec<VEC> *mb = m + (size_t)e0 * nv + b;
  float min1[VEC], min2[VEC];
  int first[VEC], second[VEC];
  uint32_t sx[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    min1[i] = min2[i] = __int_as_float(0x7f800000);
    first[i] = second[i] = 0;
    sx[i] = 0;
  }
#pragma unroll 4
  for (int j = 0; j < deg; ++j) {
    const WmsVec<VEC> t = tot[(size_t)T.cidx[e0 + j] * nv + b];
    WmsVec<VEC> mo;
    if (!FIRST) mo = mb[(size_t)j * nv];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const float x = FIRST ? t.v[i] : __fsub_rn(t.v[i], mo.v[i]);
      if (x < 0.f) sx[i] |= 1u << j;
      const float mag = fabsf(x);
      if (mag < min1[i]) {
        min2[i] = min1[i];
        second[i] = first[i];
        min1[i] = mag;
        first[i] = j;
      } else if (mag < min2[i]) {
        min2[i] = mag;
        second[i] = j;
      }
    }
  }
  const int d = T.cbucket[c];
  const float al = alpha[d], be = beta[d];
  float v1[VEC], v2[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    WmsRec r;
    r.min1 = rq<BF16>(min1[i]);
    r.min2 = rq<BF16>(min2[i]);
    r.first = (uint16_t)first[i];
    r.second = (uint16_t)second[i];
    r.sx = sx[i];
    rec[wms_rec_at<VEC>(T.nc, nv, c, b, i)] = r;
    const float a1 = __fsub_rn(__fmul_rn(al, r.min1), be);
    const float a2 = __fsub_rn(__fmul_rn(al, r.min2), be);
    v1[i] = a1 > 0.f ? a1 : 0.f;
    v2[i] = a2 > 0.f ? a2 : 0.f;
    if (__popc(sx[i]) & 1) sx[i] = ~sx[i];      // now the messages' signs
  }
#pragma unroll 4
  for (int j = 0; j < deg; ++j) {
    WmsVec<VEC> o;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const float v = j == first[i] ? v2[i] : v1[i];
      o.v[i] = (sx[i] >> j) & 1u ? -v : v;
    }
    mb[(size_t)j * nv] = o;
  }
}

// ---- forward: variable update: tot^(t) = llr + messages (ascending edges) -----
template <int VEC>
__global__ void __launch_bounds__(WMS_T) wms_var_fwd(WmsTables T, int nv, const WmsVec<VEC> *llr,
                                                     const WmsVec<VEC> *m, WmsVec<VEC> *tot) {
  int v, b;
  if (!wms_item(T.n, nv, v, b)) return;
  WmsVec<VEC> s = llr[(size_t)v * nv + b];
  const int k1 = T.vptr[v + 1];
#pragma unroll 4
  for (int k = T.vptr[v]; k < k1; ++k) {
    const WmsVec<VEC> x = m[(size_t)T.vedge[k] * nv + b];
#pragma unroll
    for (int i = 0; i < VEC; ++i) s.v[i] = __fadd_rn(s.v[i], x.v[i]);
  }
  tot[(size_t)v * nv + b] = s;
}

// ---- backward: check step of iteration t ------------------------------------
// rec: records of t; al/be: its scale and offset rows; gtot: dL/dtot^(t);
// gx_next: dL/dx^(t+1) (null at T); writes gx (dL/dx^(t); null: not wanted) and
// accumulates ga/gb[bucket] of t over the nblk blocks (the padding adds nothing).
template <int VEC, int MAXB>
__global__ void __launch_bounds__(WMS_T) wms_check_bwd(WmsTables T, int nv, int nblk,
                                                       const WmsRec *rec, const float *alpha,
                                                       const float *beta, const WmsVec<VEC> *gtot,
                                                       const WmsVec<VEC> *gx_next, WmsVec<VEC> *gx,
                                                       float *galpha, float *gbeta) {
  __shared__ float sa[MAXB], sb[MAXB];
  for (int i = threadIdx.x; i < MAXB; i += WMS_T) sa[i] = sb[i] = 0.f;
  __syncthreads();
  int c, b, d = -1;
  float sum_a = 0.f, sum_b = 0.f;
  if (wms_item(T.nc, nv, c, b)) {
    const int e0 = T.cptr[c], deg = T.cptr[c + 1] - e0;
    d = T.cbucket[c];
    const float al = alpha[d], be = beta[d];
    const size_t eb = (size_t)e0 * nv + b;
    WmsRec r[VEC];
    float ga[VEC], gb[VEC], gmu_rest[VEC], gmu_first[VEC];
    uint32_t sg[VEC];                            // the messages' signs
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      r[i] = rec[wms_rec_at<VEC>(T.nc, nv, c, b, i)];
      sg[i] = __popc(r[i].sx) & 1 ? ~r[i].sx : r[i].sx;
      ga[i] = gb[i] = gmu_rest[i] = gmu_first[i] = 0.f;
    }
#pragma unroll 4
    for (int j = 0; j < deg; ++j) {
      const WmsVec<VEC> g = gtot[(size_t)T.cidx[e0 + j] * nv + b];
      WmsVec<VEC> gn;
      if (gx_next) gn = gx_next[eb + (size_t)j * nv];
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const float G = g.v[i] - (gx_next ? gn.v[i] : 0.f);
        const float mu = (j == r[i].first) ? r[i].min2 : r[i].min1;
        const float a = al * mu - be;
        if (a > 0.f) {
          const float gaj = (sg[i] >> j) & 1u ? -G : G;
          ga[i] += gaj * mu;
          gb[i] -= gaj;
          const float gmu = gaj * al;
          if (j == r[i].first) gmu_first[i] += gmu; else gmu_rest[i] += gmu;
        }
      }
    }
    if (gx) {
#pragma unroll 4
      for (int j = 0; j < deg; ++j) {
        WmsVec<VEC> o;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          float gxv = 0.f;
          const float sx = (r[i].sx >> j) & 1u ? -1.f : 1.f;
          if (j == r[i].first) gxv += sx * gmu_rest[i];
          if (j == r[i].second && deg > 1) gxv += sx * gmu_first[i];
          o.v[i] = gxv;
        }
        gx[eb + (size_t)j * nv] = o;
      }
    }
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      sum_a += b * VEC + i < nblk ? ga[i] : 0.f;
      sum_b += b * VEC + i < nblk ? gb[i] : 0.f;
    }
  }
  // per bucket: the warp's sum (one turn per bucket present), then the CTA's
  uint32_t left = __ballot_sync(0xffffffffu, d >= 0);
  while (left) {
    const int turn = __shfl_sync(0xffffffffu, d, __ffs(left) - 1);
    const bool mine = d == turn;
    float xa = mine ? sum_a : 0.f, xb = mine ? sum_b : 0.f;
    for (int o = 16; o > 0; o >>= 1) {
      xa += __shfl_xor_sync(0xffffffffu, xa, o);
      xb += __shfl_xor_sync(0xffffffffu, xb, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&sa[turn], xa);
      atomicAdd(&sb[turn], xb);
    }
    left &= ~__ballot_sync(0xffffffffu, mine);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < T.nbucket; i += WMS_T) {
    if (sa[i] != 0.f) atomicAdd(&galpha[i], sa[i]);
    if (sb[i] != 0.f) atomicAdd(&gbeta[i], sb[i]);
  }
}

// ---- backward: gtot^(t-1)[v] = sum of gx^(t) over v's edges --------------------
template <int VEC>
__global__ void __launch_bounds__(WMS_T) wms_var_bwd(WmsTables T, int nv, const WmsVec<VEC> *gx,
                                                     WmsVec<VEC> *gtot_prev) {
  int v, b;
  if (!wms_item(T.n, nv, v, b)) return;
  WmsVec<VEC> s;
#pragma unroll
  for (int i = 0; i < VEC; ++i) s.v[i] = 0.f;
  const int k1 = T.vptr[v + 1];
#pragma unroll 4
  for (int k = T.vptr[v]; k < k1; ++k) {
    const WmsVec<VEC> x = gx[(size_t)T.vedge[k] * nv + b];
#pragma unroll
    for (int i = 0; i < VEC; ++i) s.v[i] += x.v[i];
  }
  gtot_prev[(size_t)v * nv + b] = s;
}

static inline unsigned nblocks(int64_t items, int nv) {
  return (unsigned)((items * nv + WMS_T - 1) / WMS_T);
}

static inline unsigned tiles(int n, int blocks) {
  return (unsigned)((n + 31) / 32) * (unsigned)((blocks + 31) / 32);
}

// nbp: blocks of the records and workspace, nblk rounded up to VEC
template <int VEC>
static int32_t wms_forward(const WmsTables &T, int nblk, int iters, const float *llr,
                           const float *alpha, const float *beta, bool bf16, WmsRec *rec,
                           float *tot_out, float *work, cudaStream_t st) {
  constexpr int CV = VEC > 1 ? WMS_CHECK_VEC : 1;
  using V = WmsVec<VEC>;
  using C = WmsVec<CV>;
  const int nv = (nblk + VEC - 1) / VEC, nbp = nv * VEC;
  float *llr_t = work;                               // [v][b]
  float *tot = llr_t + (size_t)nbp * T.n;            // [v][b]
  float *m = tot + (size_t)nbp * T.n;                // [e][b]
  // tot^(0) = llr
  wms_blocks_last<<<tiles(T.n, nbp), 256, 0, st>>>(llr, nblk, T.n, nbp, llr_t, tot);
  const unsigned gc = nblocks(T.nc, nbp / CV), gv = nblocks(T.n, nv);
  for (int t = 0; t < iters; ++t) {
    WmsRec *r = rec + (size_t)t * nbp * T.nc;
    const float *al = alpha + (size_t)t * T.nbucket, *be = beta + (size_t)t * T.nbucket;
    auto *fn = bf16 ? (t ? wms_check_fwd<CV, true, false> : wms_check_fwd<CV, true, true>)
                    : (t ? wms_check_fwd<CV, false, false> : wms_check_fwd<CV, false, true>);
    fn<<<gc, WMS_T, 0, st>>>(T, nbp / CV, (const C *)tot, (C *)m, r, al, be);
    wms_var_fwd<VEC><<<gv, WMS_T, 0, st>>>(T, nv, (const V *)llr_t, (const V *)m, (V *)tot);
  }
  wms_blocks_first<<<tiles(T.n, nblk), 256, 0, st>>>(tot, nblk, T.n, nbp, tot_out);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

// gtot0 (nullable): dL/dtot^(0), (nblk, n); may be gtot
template <int VEC>
static int32_t wms_backward(const WmsTables &T, int nblk, int iters, const float *alpha,
                            const float *beta, const WmsRec *rec, const float *gtot, float *gtot0,
                            float *galpha, float *gbeta, float *work, cudaStream_t st) {
  constexpr int CV = VEC > 1 ? WMS_CHECK_VEC : 1;
  using V = WmsVec<VEC>;
  using C = WmsVec<CV>;
  const int nv = (nblk + VEC - 1) / VEC, nbp = nv * VEC;
  float *gt = work;                                  // [v][b]
  float *gxa = gt + (size_t)nbp * T.n;               // [e][b]
  float *gxb = gxa + (size_t)nbp * T.ne;
  wms_blocks_last<<<tiles(T.n, nbp), 256, 0, st>>>(gtot, nblk, T.n, nbp, gt, nullptr);
  const unsigned gc = nblocks(T.nc, nbp / CV), gv = nblocks(T.n, nv);
  // per-CTA gradient partials in shared memory, one entry per bucket (check
  // degrees: a handful; block rows: up to 127)
  auto *check = T.nbucket <= 64 ? wms_check_bwd<CV, 64> : wms_check_bwd<CV, 128>;
  float *gx_next = nullptr;
  for (int t = iters - 1; t >= 0; --t) {
    const size_t p = (size_t)t * T.nbucket;
    float *gx = (gx_next == gxa) ? gxb : gxa;
    if (t == 0 && !gtot0) gx = nullptr;
    check<<<gc, WMS_T, 0, st>>>(T, nbp / CV, nblk, rec + (size_t)t * nbp * T.nc, alpha + p,
                                beta + p, (const C *)gt, (const C *)gx_next, (C *)gx, galpha + p,
                                gbeta + p);
    if (gx) wms_var_bwd<VEC><<<gv, WMS_T, 0, st>>>(T, nv, (const V *)gx, (V *)gt);
    gx_next = gx;
  }
  if (gtot0) wms_blocks_first<<<tiles(T.n, nblk), 256, 0, st>>>(gt, nblk, T.n, nbp, gtot0);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace atsc3

extern "C" {

// tables: int32 pointers (device) cptr, cidx, vptr, vedge; int8 cbucket.
// nbp: nblk rounded up to a multiple of 4.  work: nbp * (2n + ne) floats,
// 16-byte aligned; records for nbp blocks.
int32_t atsc3_wms_forward_work(const int32_t *cptr, const int32_t *cidx,
                               const int32_t *vptr, const int32_t *vedge,
                               const int8_t *cbucket, int32_t n, int32_t nc,
                               int32_t ne, int32_t nbucket, int32_t nblk,
                               int32_t iters, const float *llr, const float *alpha,
                               const float *beta, int32_t bf16, void *records,
                               float *tot_out, float *work, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(n > 0 && nc > 0 && ne > 0 && nbucket > 0 && nbucket <= 127, "bad sizes");
  ATSC3_ARG(iters >= 1 && nblk >= 0, "bad sizes");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && cbucket && llr && alpha && beta && records &&
                tot_out && work,
            "null pointer");
  ATSC3_ARG((((uintptr_t)work | (uintptr_t)records) & 15) == 0, "work and records must be 16-byte aligned");
  return wms_forward<4>(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk,
                        iters, llr, alpha, beta, bf16 != 0, (WmsRec *)records, tot_out, work,
                        (cudaStream_t)stream);
}

// Without padding and with the workspace taken from the stream's memory pool for
// the call (vchk and vpos are not read).
int32_t atsc3_wms_forward(const int32_t *cptr, const int32_t *cidx,
                          const int32_t *vptr, const int32_t *vedge,
                          const int32_t *vchk, const int32_t *vpos,
                          const int8_t *cbucket, int32_t n, int32_t nc,
                          int32_t ne, int32_t nbucket, int32_t nblk,
                          int32_t iters, const float *llr, const float *alpha,
                          const float *beta, int32_t bf16, void *records,
                          float *tot_out, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(n > 0 && nc > 0 && ne > 0 && nbucket > 0 && nbucket <= 127, "bad sizes");
  ATSC3_ARG(iters >= 1 && nblk >= 0, "bad sizes");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && vchk && vpos && cbucket && llr &&
                alpha && beta && records && tot_out,
            "null pointer");
  void *work = nullptr;
  ATSC3_CUDA(cudaMallocAsync(&work, (size_t)nblk * (2 * (size_t)n + ne) * 4, (cudaStream_t)stream));
  const int32_t rc = wms_forward<1>(
      WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk, iters, llr, alpha,
      beta, bf16 != 0, (WmsRec *)records, tot_out, (float *)work, (cudaStream_t)stream);
  ATSC3_CUDA(cudaFreeAsync(work, (cudaStream_t)stream));
  return rc;
}

// Parameter gradients only: gtot (nblk, n) dL/dtot^(T) is read; records of
// atsc3_wms_forward_work.  work: nbp * (n + 2 ne) floats, 16-byte aligned.
int32_t atsc3_wms_gradients(const int32_t *cptr, const int32_t *cidx,
                            const int32_t *vptr, const int32_t *vedge,
                            const int8_t *cbucket, int32_t n, int32_t nc,
                            int32_t ne, int32_t nbucket, int32_t nblk,
                            int32_t iters, const float *alpha, const float *beta,
                            const void *records, const float *gtot, float *galpha,
                            float *gbeta, float *work, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(n > 0 && nc > 0 && ne > 0 && nbucket > 0 && nbucket <= 127, "bad sizes");
  ATSC3_ARG(iters >= 1 && nblk >= 0, "bad sizes");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && cbucket && alpha && beta && gtot && galpha && gbeta &&
                work && records,
            "null pointer");
  ATSC3_ARG((((uintptr_t)work | (uintptr_t)records) & 15) == 0, "work and records must be 16-byte aligned");
  return wms_backward<4>(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk,
                         iters, alpha, beta, (const WmsRec *)records, gtot, nullptr, galpha, gbeta,
                         work, (cudaStream_t)stream);
}

// gtot: (nblk, n) dL/dtot^(T) on input, overwritten with dL/dtot^(0) (through the
// messages; llr also enters every later tot^(t) directly).
// work: nblk * (n + 2 ne) floats; records of atsc3_wms_forward (llr, vchk and
// vpos are not read).
int32_t atsc3_wms_backward(const int32_t *cptr, const int32_t *cidx,
                           const int32_t *vptr, const int32_t *vedge,
                           const int32_t *vchk, const int32_t *vpos,
                           const int8_t *cbucket, int32_t n, int32_t nc,
                           int32_t ne, int32_t nbucket, int32_t nblk,
                           int32_t iters, const float *llr, const float *alpha,
                           const float *beta, const void *records, float *gtot,
                           float *galpha, float *gbeta, float *work,
                           void *stream) {
  using namespace atsc3;
  (void)vchk;
  (void)vpos;
  (void)llr;
  ATSC3_ARG(n > 0 && nc > 0 && ne > 0 && nbucket > 0 && nbucket <= 127, "bad sizes");
  ATSC3_ARG(iters >= 1 && nblk >= 0, "bad sizes");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && cbucket && alpha && beta && gtot && galpha && gbeta &&
                work && records,
            "null pointer");
  return wms_backward<1>(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk,
                         iters, alpha, beta, (const WmsRec *)records, gtot, gtot, galpha, gbeta,
                         work, (cudaStream_t)stream);
}

}  // extern "C"
