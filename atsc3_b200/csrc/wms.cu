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
// Layout: every array is [item][block], blocks fastest, and thread g takes item
// g / nblk of block g mod nblk.  A warp reads consecutive blocks of one check,
// bit or edge, whatever permutation the code applies, and its indices are the
// same for all lanes; the caller's (nblk, n) arrays are transposed on the way in
// and out.  With [block][item] the gathers of one iteration touched a 32-byte
// sector per 4- or 16-byte value.  What bounds it now is moving the messages:
// 5 passes over 4 bytes an edge an iteration forward, 5 backward.
// 64 blocks of 64800 8/15, 12 iterations, forward and backward with the loss:
// 10.5 ms -> NOW ms.
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

template <bool BF16>
__device__ __forceinline__ float rq(float v) {
  if constexpr (BF16) return __bfloat162float(__float2bfloat16_rn(v));
  return v;
}

// item and block of this thread; false past the end
__device__ __forceinline__ bool wms_item(int items, int nblk, int &item, int &b) {
  const int64_t g = (int64_t)blockIdx.x * WMS_T + threadIdx.x;
  if (g >= (int64_t)items * nblk) return false;
  if (g <= 0xFFFFFFFFll) {
    const uint32_t i = (uint32_t)g / (uint32_t)nblk;
    item = (int)i;
    b = (int)((uint32_t)g - i * (uint32_t)nblk);
  } else {
    item = (int)(g / nblk);
    b = (int)(g - (int64_t)item * nblk);
  }
  return true;
}

// (rows, cols) -> (cols, rows); dst2 (nullable): a second copy
__global__ void __launch_bounds__(256) wms_transpose(const float *src, int rows, int cols,
                                                     float *dst, float *dst2) {
  __shared__ float tile[32][33];
  const int tiles = (cols + 31) / 32;
  const int r0 = (int)(blockIdx.x / tiles) * 32, c0 = (int)(blockIdx.x % tiles) * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8)
    if (r0 + r < rows && c0 + tx < cols) tile[r][tx] = src[(size_t)(r0 + r) * cols + c0 + tx];
  __syncthreads();
  for (int c = ty; c < 32; c += 8)
    if (c0 + c < cols && r0 + tx < rows) {
      const size_t at = (size_t)(c0 + c) * rows + r0 + tx;
      dst[at] = tile[tx][c];
      if (dst2) dst2[at] = tile[tx][c];
    }
}

// ---- forward: check update of iteration t: record and messages ---------------
// m: messages of iteration t-1 on entry (ignored when FIRST: they are 0), of t
// on return; al/be: scale and offset rows of iteration t
template <bool BF16, bool FIRST>
__global__ void __launch_bounds__(WMS_T) wms_check_fwd(WmsTables T, int nblk, const float *tot,
                                                       float *m, WmsRec *rec, const float *alpha,
                                                       const float *beta) {
  int c, b;
  if (!wms_item(T.nc, nblk, c, b)) return;
  const int e0 = T.cptr[c], deg = T.cptr[c + 1] - e0;
  float *mb = m + (size_t)e0 * nblk + b;
  float min1 = __int_as_float(0x7f800000), min2 = min1;
  int first = 0, second = 0;
  uint32_t sx = 0;
#pragma unroll 4
  for (int j = 0; j < deg; ++j) {
    const float mo = FIRST ? 0.f : mb[(size_t)j * nblk];
    const float x = __fsub_rn(tot[(size_t)T.cidx[e0 + j] * nblk + b], mo);
    if (x < 0.f) sx |= 1u << j;
    const float mag = fabsf(x);
    if (mag < min1) { min2 = min1; second = first; min1 = mag; first = j; }
    else if (mag < min2) { min2 = mag; second = j; }
  }
  WmsRec r;
  r.min1 = rq<BF16>(min1);
  r.min2 = rq<BF16>(min2);
  r.first = (uint16_t)first;
  r.second = (uint16_t)second;
  r.sx = sx;
  rec[(size_t)c * nblk + b] = r;
  const int d = T.cbucket[c];
  const float al = alpha[d], be = beta[d];
  const float a1 = __fsub_rn(__fmul_rn(al, r.min1), be);
  const float a2 = __fsub_rn(__fmul_rn(al, r.min2), be);
  const float v1 = a1 > 0.f ? a1 : 0.f, v2 = a2 > 0.f ? a2 : 0.f;
  const uint32_t par = __popc(sx) & 1u;
#pragma unroll 4
  for (int j = 0; j < deg; ++j) {
    const float v = j == first ? v2 : v1;
    mb[(size_t)j * nblk] = (par ^ (sx >> j)) & 1u ? -v : v;
  }
}

// ---- forward: variable update: tot^(t) = llr + messages (ascending edges) -----
__global__ void __launch_bounds__(WMS_T) wms_var_fwd(WmsTables T, int nblk, const float *llr,
                                                     const float *m, float *tot) {
  int v, b;
  if (!wms_item(T.n, nblk, v, b)) return;
  float s = llr[(size_t)v * nblk + b];
  const int k1 = T.vptr[v + 1];
#pragma unroll 4
  for (int k = T.vptr[v]; k < k1; ++k)
    s = __fadd_rn(s, m[(size_t)T.vedge[k] * nblk + b]);
  tot[(size_t)v * nblk + b] = s;
}

// ---- backward: check step of iteration t ------------------------------------
// rec: records of t; al/be: its scale and offset rows; gtot: dL/dtot^(t);
// gx_next: dL/dx^(t+1) (null at T); writes gx (dL/dx^(t); null: not wanted) and
// accumulates ga/gb[bucket] of t.
template <int MAXB>
__global__ void __launch_bounds__(WMS_T) wms_check_bwd(WmsTables T, int nblk, const WmsRec *rec,
                                                       const float *alpha, const float *beta,
                                                       const float *gtot, const float *gx_next,
                                                       float *gx, float *galpha, float *gbeta) {
  __shared__ float sa[MAXB], sb[MAXB];
  for (int i = threadIdx.x; i < MAXB; i += WMS_T) sa[i] = sb[i] = 0.f;
  __syncthreads();
  int c, b, d = -1;
  float ga = 0.f, gb = 0.f;
  if (wms_item(T.nc, nblk, c, b)) {
    const int e0 = T.cptr[c], deg = T.cptr[c + 1] - e0;
    d = T.cbucket[c];
    const float al = alpha[d], be = beta[d];
    const WmsRec r = rec[(size_t)c * nblk + b];
    const size_t eb = (size_t)e0 * nblk + b;
    const uint32_t par = __popc(r.sx) & 1u;
    float gmu_rest = 0.f, gmu_first = 0.f;
#pragma unroll 4
    for (int j = 0; j < deg; ++j) {
      const float G = gtot[(size_t)T.cidx[e0 + j] * nblk + b] -
                      (gx_next ? gx_next[eb + (size_t)j * nblk] : 0.f);
      const float mu = (j == r.first) ? r.min2 : r.min1;
      const float a = al * mu - be;
      if (a > 0.f) {
        const float sg = (par ^ ((r.sx >> j) & 1u)) ? -1.f : 1.f;
        const float gaj = G * sg;
        ga += gaj * mu;
        gb -= gaj;
        const float gmu = gaj * al;
        if (j == r.first) gmu_first += gmu; else gmu_rest += gmu;
      }
    }
    if (gx) {
#pragma unroll 4
      for (int j = 0; j < deg; ++j) {
        float gxv = 0.f;
        const float sx = (r.sx >> j) & 1u ? -1.f : 1.f;
        if (j == r.first) gxv += sx * gmu_rest;
        if (j == r.second && deg > 1) gxv += sx * gmu_first;
        gx[eb + (size_t)j * nblk] = gxv;
      }
    }
  }
  // per bucket: the warp's sum (one turn per bucket present), then the CTA's
  uint32_t left = __ballot_sync(0xffffffffu, d >= 0);
  while (left) {
    const int turn = __shfl_sync(0xffffffffu, d, __ffs(left) - 1);
    const bool mine = d == turn;
    float xa = mine ? ga : 0.f, xb = mine ? gb : 0.f;
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
__global__ void __launch_bounds__(WMS_T) wms_var_bwd(WmsTables T, int nblk, const float *gx,
                                                     float *gtot_prev) {
  int v, b;
  if (!wms_item(T.n, nblk, v, b)) return;
  float s = 0.f;
  const int k1 = T.vptr[v + 1];
#pragma unroll 4
  for (int k = T.vptr[v]; k < k1; ++k) s += gx[(size_t)T.vedge[k] * nblk + b];
  gtot_prev[(size_t)v * nblk + b] = s;
}

static inline unsigned nblocks(int64_t items, int nblk) {
  return (unsigned)((items * nblk + WMS_T - 1) / WMS_T);
}

static inline unsigned tiles(int rows, int cols) {
  return (unsigned)((rows + 31) / 32) * (unsigned)((cols + 31) / 32);
}

static int32_t wms_forward(const WmsTables &T, int nblk, int iters, const float *llr,
                           const float *alpha, const float *beta, bool bf16, WmsRec *rec,
                           float *tot_out, float *work, cudaStream_t st) {
  float *llr_t = work;                               // [v][b]
  float *tot = llr_t + (size_t)nblk * T.n;           // [v][b]
  float *m = tot + (size_t)nblk * T.n;               // [e][b]
  // tot^(0) = llr
  wms_transpose<<<tiles(nblk, T.n), 256, 0, st>>>(llr, nblk, T.n, llr_t, tot);
  const unsigned gc = nblocks(T.nc, nblk), gv = nblocks(T.n, nblk);
  for (int t = 0; t < iters; ++t) {
    WmsRec *r = rec + (size_t)t * nblk * T.nc;
    const float *al = alpha + (size_t)t * T.nbucket, *be = beta + (size_t)t * T.nbucket;
    auto *fn = bf16 ? (t ? wms_check_fwd<true, false> : wms_check_fwd<true, true>)
                    : (t ? wms_check_fwd<false, false> : wms_check_fwd<false, true>);
    fn<<<gc, WMS_T, 0, st>>>(T, nblk, tot, m, r, al, be);
    wms_var_fwd<<<gv, WMS_T, 0, st>>>(T, nblk, llr_t, m, tot);
  }
  wms_transpose<<<tiles(T.n, nblk), 256, 0, st>>>(tot, T.n, nblk, tot_out, nullptr);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

// gllr (nullable): dL/dllr, (nblk, n); may be gtot
static int32_t wms_backward(const WmsTables &T, int nblk, int iters, const float *alpha,
                            const float *beta, const WmsRec *rec, const float *gtot, float *gllr,
                            float *galpha, float *gbeta, float *work, cudaStream_t st) {
  float *gt = work;                                  // [v][b]
  float *gxa = gt + (size_t)nblk * T.n;              // [e][b]
  float *gxb = gxa + (size_t)nblk * T.ne;
  wms_transpose<<<tiles(nblk, T.n), 256, 0, st>>>(gtot, nblk, T.n, gt, nullptr);
  const unsigned gc = nblocks(T.nc, nblk), gv = nblocks(T.n, nblk);
  // per-CTA gradient partials in shared memory, one entry per bucket (check
  // degrees: a handful; block rows: up to 127)
  auto *check = T.nbucket <= 64 ? wms_check_bwd<64> : wms_check_bwd<128>;
  float *gx_next = nullptr;
  for (int t = iters - 1; t >= 0; --t) {
    const size_t p = (size_t)t * T.nbucket;
    float *gx = (gx_next == gxa) ? gxb : gxa;
    if (t == 0 && !gllr) gx = nullptr;
    check<<<gc, WMS_T, 0, st>>>(T, nblk, rec + (size_t)t * nblk * T.nc, alpha + p, beta + p, gt,
                                gx_next, gx, galpha + p, gbeta + p);
    if (gx) wms_var_bwd<<<gv, WMS_T, 0, st>>>(T, nblk, gx, gt);
    gx_next = gx;
  }
  if (gllr) wms_transpose<<<tiles(T.n, nblk), 256, 0, st>>>(gt, T.n, nblk, gllr, nullptr);
  ATSC3_CUDA(cudaGetLastError());
  return 0;
}

}  // namespace atsc3

extern "C" {

// tables: int32 pointers (device) cptr, cidx, vptr, vedge; int8 cbucket.
// work: nblk * (2n + ne) floats.
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
  return wms_forward(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk, iters,
                     llr, alpha, beta, bf16 != 0, (WmsRec *)records, tot_out, work,
                     (cudaStream_t)stream);
}

// The same with its workspace taken from the stream's memory pool for the call
// (vchk and vpos are not read).
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
  const int32_t rc = atsc3_wms_forward_work(cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket,
                                            nblk, iters, llr, alpha, beta, bf16, records, tot_out,
                                            (float *)work, stream);
  ATSC3_CUDA(cudaFreeAsync(work, (cudaStream_t)stream));
  return rc;
}

// Parameter gradients only: gtot (nblk, n) dL/dtot^(T) is read.
// work: nblk * (n + 2 ne) floats.
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
  return wms_backward(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk, iters,
                      alpha, beta, (const WmsRec *)records, gtot, nullptr, galpha, gbeta, work,
                      (cudaStream_t)stream);
}

// gtot: (nblk, n) dL/dtot^(T) on input, overwritten with dL/dllr on output.
// work: as atsc3_wms_gradients (llr, vchk and vpos are not read).
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
  ATSC3_ARG(gtot && galpha && gbeta && work && records, "null pointer");
  return wms_backward(WmsTables{cptr, cidx, vptr, vedge, cbucket, n, nc, ne, nbucket}, nblk, iters,
                      alpha, beta, (const WmsRec *)records, gtot, gtot, galpha, gbeta, work,
                      (cudaStream_t)stream);
}

}  // extern "C"
