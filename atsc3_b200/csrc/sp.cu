// sp.cu -- exact (log-tanh) sum-product decoding in float64 for the blocks
// min-sum could not close (sm_100a): the near-miss rescue of the reference
// receiver, lab/m16_margin.py:325-390 (sum_product_decode_batch), called from
// lab/m44_ldm.py:2527-2554 on rows whose unsatisfied-check count is small.
//
// Per iteration (it = 0 .. iters), for every block still decoding:
//   syndrome of tot (hard decision tot < 0); zero -> converged at `it`;
//   it == iters -> stop with the current decisions;
//   else per check, per edge e:  v = tot[var(e)] - m[e],
//        t = tanh(clip(v, -38, 38) / 2), parity of (t < 0),
//        lt = log(clip(|t|, 1e-300, 1)), lsum = sum of lt over the check,
//        m[e] = +-2 atanh(clip(exp(clip(lsum - lt, -700, -1e-16)), 0,
//               1 - 1e-16)), negative when parity ^ (t < 0);
//   per variable: tot = llr + sum of its messages in ascending check order.
// tanh, log, exp and atanh are CUDA's float64 functions (not restated); the
// messages agree with the numpy float64 reference to rounding, the decisions
// (bits, convergence, iteration) are what the tests compare.
//
// One cooperative kernel runs all iterations: two phases with a grid barrier
// after each, the blocks still decoding in a list that every CTA forms alike
// from the syndrome counts, and an end as soon as the list is empty.  Four
// launches per iteration, all of them queued for every iteration, spent more
// time on blocks that had ended than on decoding.  State is [item][block]: the
// lanes of a warp read consecutive blocks of one check, edge or bit.  The check
// phase keeps log |t| and the sign of t of each edge in its message slot, so
// tanh and log are taken once per edge; the float64 functions bound it.
// 8 blocks of 64800 6/15 that need about 25 iterations: 3.34 ms -> 1.27 ms.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/atsc3_fec.h"
#include "common.cuh"

namespace atsc3 {

constexpr int SP_T = 256;
constexpr int SP_BLK = 256;        // blocks of one launch

struct SpArgs {
  const int32_t *cptr, *cidx, *vptr, *vedge;
  int n, nc;
  int nblk, ldb;     // blocks of this launch; blocks of the state arrays
  int it0, steps;    // first iteration, iterations of this launch at most
  int iters;         // iteration that ends every block
  const double *llr;
  int64_t ld_llr;
  double *tot;       // [bit][block]
  double *msg;       // [edge][block]
  int32_t *active;   // per block: still decoding (between launches)
  int32_t *count;    // (2, ldb) unsatisfied checks, alternating iterations
  uint8_t *bits;
  int64_t ld_bits;
  uint8_t *conv;
  int32_t *its;
  int32_t *bad;
  int32_t *counts;   // nullable: {blocks still decoding, blocks stopped unconverged}
};

__device__ __forceinline__ double sp_t(double v) {
  const double x = fmin(fmax(v, -38.0), 38.0) * 0.5;
  return tanh(x);
}

__device__ __forceinline__ double sp_lt(double t) {
  return log(fmin(fmax(fabs(t), 1e-300), 1.0));
}

// g = item * k + rest
__device__ __forceinline__ void sp_split(int64_t g, int k, int &item, int &rest) {
  if (g <= 0xFFFFFFFFll) {
    const uint32_t i = (uint32_t)g / (uint32_t)k;
    item = (int)i;
    rest = (int)((uint32_t)g - i * (uint32_t)k);
  } else {
    item = (int)(g / k);
    rest = (int)(g - (int64_t)item * k);
  }
}

// one check of one block: returns its syndrome bit; upd: also its messages
__device__ __forceinline__ int sp_check(const SpArgs &a, int c, int b, bool upd, bool first) {
  const int e0 = __ldg(a.cptr + c), e1 = __ldg(a.cptr + c + 1);
  int syn = 0, par = 0;
  double lsum = 0.0;
  for (int e = e0; e < e1; ++e) {
    const double tv = a.tot[(size_t)__ldg(a.cidx + e) * a.ldb + b];
    syn ^= tv < 0.0 ? 1 : 0;
    if (upd) {
      double *m = a.msg + (size_t)e * a.ldb + b;
      const double t = sp_t(first ? tv : tv - *m);
      const double lt = sp_lt(t);
      par ^= t < 0.0 ? 1 : 0;
      lsum += lt;
      // log |t| is not positive: its sign bit is free for t's
      *m = copysign(lt, t < 0.0 ? -1.0 : 1.0);
    }
  }
  if (!upd) return syn;
  for (int e = e0; e < e1; ++e) {
    double *m = a.msg + (size_t)e * a.ldb + b;
    const double s = *m;
    const int neg = __double2hiint(s) < 0 ? 1 : 0;
    const double le = fmin(fmax(lsum + fabs(s), -700.0), -1e-16);
    const double mag = fmin(fmax(exp(le), 0.0), 1.0 - 1e-16);
    const double mn = 2.0 * atanh(mag);
    *m = (par ^ neg) ? -mn : mn;
  }
  return syn;
}

__global__ void __launch_bounds__(SP_T, 2) sp_kernel(const SpArgs a) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  __shared__ int act[SP_BLK], cnt[SP_BLK];    // blocks decoding; their syndrome counts
  __shared__ int ends[SP_BLK];                // per list entry: ends at this iteration
  __shared__ int nact_s, stop_s;
  const int64_t g0 = (int64_t)blockIdx.x * SP_T + threadIdx.x, gs = (int64_t)gridDim.x * SP_T;
  if (a.it0 == 0) {
    for (int64_t g = g0; g < (int64_t)a.nblk * a.n; g += gs) {
      int v, b;
      sp_split(g, a.nblk, v, b);
      a.tot[(size_t)v * a.ldb + b] = a.llr[(size_t)b * a.ld_llr + v];
    }
    if (blockIdx.x == 0)
      for (int b = threadIdx.x; b < a.nblk; b += SP_T) {
        a.active[b] = 1;
        a.count[b] = a.count[a.ldb + b] = 0;
      }
    grid.sync();
  }
  if (threadIdx.x == 0) {
    int k = 0;
    for (int b = 0; b < a.nblk; ++b)
      if (__ldcg(a.active + b)) act[k++] = b;
    nact_s = k;
  }
  __syncthreads();
  int nact = nact_s;
  for (int it = a.it0; it < a.it0 + a.steps && nact > 0; ++it) {
    const bool upd = it < a.iters;
    int32_t *count = a.count + (it & 1) * a.ldb;
    // ---- checks: syndrome of tot, and the new messages ---------------------
    for (int k = threadIdx.x; k < nact; k += SP_T) cnt[k] = 0;
    __syncthreads();
    for (int64_t g = g0; g < (int64_t)a.nc * nact; g += gs) {
      int c, k;
      sp_split(g, nact, c, k);
      if (sp_check(a, c, act[k], upd, it == 0)) atomicAdd(cnt + k, 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nact; k += SP_T)
      if (cnt[k]) atomicAdd(count + act[k], cnt[k]);
    grid.sync();
    // ---- which blocks end: every CTA reads the same counts -------------------
    for (int k = threadIdx.x; k < nact; k += SP_T) {
      const int b = act[k], bad = __ldcg(count + b);
      ends[k] = bad == 0 || !upd;
      if (blockIdx.x == 0) {
        if (ends[k]) {
          a.conv[b] = bad == 0 ? 1 : 0;
          a.its[b] = it;
          a.bad[b] = bad;
          a.active[b] = 0;
        }
        // the other counter was last read an iteration (two barriers) ago
        a.count[((it + 1) & 1) * a.ldb + b] = 0;
      }
    }
    __syncthreads();
    // ---- bits: decisions of the blocks that ended, tot = llr + messages in
    // ascending check order (vedge) of the others -----------------------------
    for (int64_t g = g0; g < (int64_t)a.n * nact; g += gs) {
      int v, k;
      sp_split(g, nact, v, k);
      const int b = act[k];
      double *tot = a.tot + (size_t)v * a.ldb + b;
      if (ends[k]) {
        a.bits[(size_t)b * a.ld_bits + v] = *tot < 0.0 ? 1 : 0;
        continue;
      }
      double s = a.llr[(size_t)b * a.ld_llr + v];
      const int k1 = __ldg(a.vptr + v + 1);
      for (int e = __ldg(a.vptr + v); e < k1; ++e)
        s += a.msg[(size_t)__ldg(a.vedge + e) * a.ldb + b];
      *tot = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int k = 0, stop = 0;
      for (int q = 0; q < nact; ++q) {
        if (!ends[q]) act[k++] = act[q];
        else if (__ldcg(count + act[q])) ++stop;
      }
      nact_s = k;
      stop_s = stop;
    }
    __syncthreads();
    nact = nact_s;
    if (a.counts && blockIdx.x == 0 && threadIdx.x == 0) {
      a.counts[0] += nact;
      a.counts[1] += stop_s;
    }
    if (nact > 0 && it + 1 < a.it0 + a.steps) grid.sync();
  }
}

static int32_t sp_launch(const int32_t *cptr, const int32_t *cidx, const int32_t *vptr,
                         const int32_t *vedge, int n, int nc, int nedges, const double *llr,
                         int64_t ld_llr, int nblk, int it0, int steps, int iters, uint8_t *bits,
                         int64_t ld_bits, uint8_t *conv, int32_t *its, int32_t *bad, void *work,
                         int32_t *counts, cudaStream_t st) {
  int dev = 0, sms = 148, per = 0;
  ATSC3_CUDA(cudaGetDevice(&dev));
  ATSC3_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ATSC3_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, sp_kernel, SP_T, 0));
  SpArgs a;
  a.cptr = cptr;
  a.cidx = cidx;
  a.vptr = vptr;
  a.vedge = vedge;
  a.n = n;
  a.nc = nc;
  a.it0 = it0;
  a.steps = steps;
  a.iters = iters;
  a.ld_llr = ld_llr;
  a.ld_bits = ld_bits;
  a.counts = counts;
  // up to SP_BLK blocks a launch, each launch with its own share of the state
  if (counts) ATSC3_CUDA(cudaMemsetAsync(counts, 0, 8, st));
  double *dw = (double *)work;
  int32_t *iw = (int32_t *)(dw + (size_t)nblk * ((size_t)n + nedges));
  for (int b0 = 0; b0 < nblk; b0 += SP_BLK) {
    const int nb = std::min(SP_BLK, nblk - b0);
    a.nblk = a.ldb = nb;
    a.llr = llr + (size_t)b0 * ld_llr;
    a.tot = dw + (size_t)b0 * ((size_t)n + nedges);
    a.msg = a.tot + (size_t)nb * n;
    a.active = iw + (size_t)3 * b0;
    a.count = a.active + nb;
    a.bits = bits + (size_t)b0 * ld_bits;
    a.conv = conv + b0;
    a.its = its + b0;
    a.bad = bad + b0;
    const int64_t want = ((int64_t)nb * std::max(n, nc) + SP_T - 1) / SP_T;
    const int grid = (int)std::min<int64_t>((int64_t)sms * std::max(per, 1), want);
    void *args[] = {&a};
    ATSC3_CUDA(cudaLaunchCooperativeKernel((const void *)sp_kernel, dim3(grid), dim3(SP_T), args, 0, st));
  }
  return 0;
}

}  // namespace atsc3

extern "C" {

int32_t atsc3_ldpc_sp_workspace(int32_t n, int32_t nedges, int32_t nblk,
                                int64_t *work_bytes) {
  ATSC3_ARG(work_bytes != nullptr, "null output");
  ATSC3_ARG(n > 0 && nedges > 0 && nblk >= 0, "bad size");
  *work_bytes = (int64_t)nblk * ((int64_t)n + nedges) * 8 + (int64_t)nblk * 12;
  return 0;
}

int32_t atsc3_ldpc_sp_decode(const int32_t *cptr, const int32_t *cidx,
                             const int32_t *vptr, const int32_t *vedge,
                             int32_t n, int32_t nc, int32_t nedges,
                             const double *llr, int64_t ld_llr, int32_t nblk,
                             int32_t iters, uint8_t *bits, int64_t ld_bits,
                             uint8_t *conv, int32_t *its, int32_t *bad,
                             void *work, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(n > 0 && nc > 0 && nedges > 0 && nblk >= 0 && iters >= 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && llr && bits && conv && its && bad && work,
            "null pointer");
  ATSC3_ARG(ld_llr >= n && ld_bits >= n, "leading dimension below n");
  ATSC3_ARG(((uintptr_t)work & 7) == 0 && ((uintptr_t)llr & 7) == 0,
            "llr and work must be 8-byte aligned");
  return sp_launch(cptr, cidx, vptr, vedge, n, nc, nedges, llr, ld_llr, nblk, 0, iters + 1, iters,
                   bits, ld_bits, conv, its, bad, work, nullptr, (cudaStream_t)stream);
}

int32_t atsc3_ldpc_sp_step(const int32_t *cptr, const int32_t *cidx,
                           const int32_t *vptr, const int32_t *vedge,
                           int32_t n, int32_t nc, int32_t nedges,
                           const double *llr, int64_t ld_llr, int32_t nblk,
                           int32_t it, int32_t last, uint8_t *bits,
                           int64_t ld_bits, uint8_t *conv, int32_t *its,
                           int32_t *bad, void *work, int32_t *counts,
                           void *stream) {
  using namespace atsc3;
  ATSC3_ARG(n > 0 && nc > 0 && nedges > 0 && nblk >= 0 && it >= 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(cptr && cidx && vptr && vedge && llr && bits && conv && its && bad &&
                work && counts, "null pointer");
  ATSC3_ARG(ld_llr >= n && ld_bits >= n, "leading dimension below n");
  ATSC3_ARG(((uintptr_t)work & 7) == 0 && ((uintptr_t)llr & 7) == 0,
            "llr and work must be 8-byte aligned");
  // the last step retires every block still decoding (as iteration `iters`
  // of a full decode does); any other step retires only converged blocks
  return sp_launch(cptr, cidx, vptr, vedge, n, nc, nedges, llr, ld_llr, nblk, it, 1,
                   last ? it : it + 1, bits, ld_bits, conv, its, bad, work, counts,
                   (cudaStream_t)stream);
}

}  // extern "C"
