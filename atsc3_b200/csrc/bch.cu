// bch.cu -- BCH zero-syndrome check (A/322 6.1.2.1) and Baseband Packet
// descramble for sm_100a.
//
// The syndrome of the K_ldpc-bit BCH codeword m (MSB first, bit 0 = x^(K-1))
// is m(x) mod g(x), deg g = 192 (Ninner 64800) or 168 (16200).  It is linear
// in the bits, so it is the XOR over the set bits of the precomputed rows
// R[pos] = x^(K-1-pos) mod g(x) -- the same GF(2) matrix product
// lab/m9_accel.py:169-236 evaluates with popcounts.  Zero syndrome = BCH OK.
//
// A cluster of CTAs per codeword.  A warp folds the table rows of one 32-bit word
// of decisions at a time, a row per lane (the word's 32 rows are 768 contiguous
// bytes, those of clear bits predicated off) and eight words in flight; then a
// warp XOR, a shared-memory XOR, and the first CTA adds the others' through
// distributed shared memory.  The table sits in L2; with one CTA a codeword and a
// word a thread, its latency and the 32 lines each load touched were the bound
// (one 16200 11/15 codeword 13.3 us, 7 of 64800 10/15 37.8, 75 of 6/15 26.6; now
// 3.6, 5.8 and 8.3).
// The descrambled payload (lab/m9_fast.py:942-949: hard bits XOR the
// scrambling sequence, packed MSB-first) is written by the same cluster.

#include <cuda_runtime.h>

#include "../../include/atsc3_fec.h"
#include "common.cuh"

namespace atsc3 {

constexpr int BCH_T = 256;
constexpr int BCH_CL = 8;             // CTAs per codeword at most (portable cluster)

__device__ __forceinline__ void fold_row(uint32_t (&acc)[6], const uint32_t *__restrict__ rtab,
                                         int pos) {
  const uint2 *r = reinterpret_cast<const uint2 *>(rtab + (size_t)pos * 6);
  const uint2 a = __ldg(r), b = __ldg(r + 1), c = __ldg(r + 2);
  acc[0] ^= a.x; acc[1] ^= a.y; acc[2] ^= b.x;
  acc[3] ^= b.y; acc[4] ^= c.x; acc[5] ^= c.y;
}

// The cluster's XOR of acc, written by its first CTA.  The kernel has arrived at
// the cluster barrier at its entry; the wait here, behind the fold, shows that the
// first CTA has started before its shared memory is written.
__device__ __forceinline__ void reduce_store(uint32_t (&acc)[6], uint32_t *syn, uint8_t *ok) {
  __shared__ uint32_t red[BCH_T / 32][6];
  __shared__ uint32_t all[BCH_CL][6];           // rank 0: every CTA's words
  const int rank = (int)cluster_ctarank(), cl = (int)cluster_nctarank();
#pragma unroll
  for (int w = 0; w < 6; ++w) acc[w] = __reduce_xor_sync(0xffffffffu, acc[w]);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int w = 0; w < 6; ++w) red[warp][w] = acc[w];
  __syncthreads();
  cluster_wait();
  if (threadIdx.x < 6) {
    uint32_t v = 0;
    for (int q = 0; q < BCH_T / 32; ++q) v ^= red[q][threadIdx.x];
    dsmem_st_u32(dsmem_map(smem_u32(&all[rank][threadIdx.x]), 0u), v);
  }
  cluster_sync_all();
  if (rank == 0 && warp == 0) {
    uint32_t v = 0;
    if (lane < 6) {
      for (int q = 0; q < cl; ++q) v ^= all[q][lane];
      syn[lane] = v;
    }
    const bool any = __any_sync(0xffffffffu, v != 0);
    if (lane == 0 && ok) *ok = any ? 0 : 1;
  }
}

// this warp's words of a packed codeword and this thread's share of the payload
__device__ __forceinline__ void fold_packed(uint32_t (&acc)[6], const uint8_t *h, int kldpc,
                                            const uint32_t *__restrict__ rtab,
                                            const uint8_t *__restrict__ scr, int kpay,
                                            uint8_t *__restrict__ po) {
  const int t0 = (int)cluster_ctarank() * BCH_T + threadIdx.x;
  const int step = (int)cluster_nctarank() * BCH_T;
  const int nword = kldpc >> 5;              // whole 32-bit words
  const uint32_t *hw = reinterpret_cast<const uint32_t *>(h);
  const int lane = threadIdx.x & 31;
  // row 32w + l of word w is decided by bit l of the packed order: byte l>>3,
  // MSB first (byte 4w is the word's low byte)
  const int bit = (lane & ~7) + 7 - (lane & 7);
  const int per = (nword + step / 32 - 1) / (step / 32);
  const int w0 = (t0 >> 5) * per, w1 = min(nword, w0 + per);
  for (int wb = w0; wb < w1; wb += 32) {
    const int cnt = min(32, w1 - wb);
    const uint32_t mine = lane < cnt ? __ldg(hw + wb + lane) : 0u;
    for (int k0 = 0; k0 < cnt; k0 += 8) {
      uint2 x[8][3];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t v = __shfl_sync(0xffffffffu, mine, (k0 + k) & 31);
        const bool on = k0 + k < cnt && ((v >> bit) & 1u);
        const uint2 *r = reinterpret_cast<const uint2 *>(rtab + ((size_t)(wb + k0 + k) * 32 + lane) * 6);
#pragma unroll
        for (int q = 0; q < 3; ++q) x[k][q] = on ? __ldg(r + q) : make_uint2(0u, 0u);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          acc[2 * q] ^= x[k][q].x;
          acc[2 * q + 1] ^= x[k][q].y;
        }
    }
  }
  for (int pos = nword * 32 + t0; pos < kldpc; pos += step)
    if ((h[pos >> 3] >> (7 - (pos & 7))) & 1) fold_row(acc, rtab, pos);
  if (po && scr)
    for (int j = t0; j < (kpay >> 3); j += step) po[j] = h[j] ^ __ldg(scr + j);
}

__global__ void __launch_bounds__(BCH_T) bch_packed_kernel(
    const uint8_t *__restrict__ hard, int64_t ld_hard, int kldpc,
    const uint32_t *__restrict__ rtab, uint32_t *__restrict__ syn,
    uint8_t *__restrict__ ok, const uint8_t *__restrict__ scr, int kpay,
    uint8_t *__restrict__ payload, int64_t ld_payload) {
  cluster_arrive();
  const int b = (int)cluster_id_x();
  uint32_t acc[6] = {0, 0, 0, 0, 0, 0};
  fold_packed(acc, hard + (size_t)b * ld_hard, kldpc, rtab, scr, kpay,
              payload ? payload + (size_t)b * ld_payload : nullptr);
  reduce_store(acc, syn + (size_t)b * 6, ok ? ok + b : nullptr);
}

__global__ void __launch_bounds__(BCH_T) bch_bits_kernel(
    const uint8_t *__restrict__ bits, int64_t ld_bits, int kldpc,
    const uint32_t *__restrict__ rtab, uint32_t *__restrict__ syn) {
  cluster_arrive();
  const int b = (int)cluster_id_x();
  const uint8_t *h = bits + (size_t)b * ld_bits;
  uint32_t acc[6] = {0, 0, 0, 0, 0, 0};
  const int step = (int)cluster_nctarank() * BCH_T;
#pragma unroll 8
  for (int pos = (int)cluster_ctarank() * BCH_T + threadIdx.x; pos < kldpc; pos += step)
    if (h[pos] & 1) fold_row(acc, rtab, pos);
  reduce_store(acc, syn + (size_t)b * 6, nullptr);
}

// CTAs per codeword: as many as leave the whole batch resident at once, which is
// three CTAs an SM by their registers, and two in clusters of eight (us with 1 / 2 /
// 4 / 8 CTAs a codeword: 37 of 64800 6/15 16.9 / 10.4 / 7.1 / 5.9, 74 17.4 / 10.8 /
// 8.3 / 10.1, 148 18.1 / 11.3 / 15.1 / 17.4, 300 20.4 / 23.2 / 22.1 / 30.2; 148 of
// 16200 2/15 5.2 / 4.5 / 7.2 / 11.2).
static int bch_cluster(int64_t nblk, int kldpc) {
  int cl = BCH_CL;
  const auto room = [](int c) { return c == 8 ? 2 * 148 : c == 4 ? 400 : 3 * 148; };
  while (cl > 1 && (nblk * cl > room(cl) || kldpc / 32 < cl * (BCH_T / 32))) cl /= 2;
  return cl;
}

// launches `fn` with a cluster of `cl` CTAs for each of nblk codewords
template <typename... P, typename... A>
static cudaError_t bch_launch(void (*fn)(P...), int nblk, int cl, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)nblk * (unsigned)cl, 1, 1);
  cfg.blockDim = dim3(BCH_T, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

int32_t bch_check_launch(const uint8_t *hard, int64_t ld_hard, int nblk,
                         int kldpc, const uint32_t *rtab, uint32_t *syn,
                         uint8_t *ok, const uint8_t *scr, int kpay,
                         uint8_t *payload, int64_t ld_payload,
                         cudaStream_t st) {
  ATSC3_ARG(nblk >= 0 && kldpc > 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(hard && rtab && syn, "null pointer");
  ATSC3_ARG(ld_hard * 8 >= kldpc, "ld_hard*8 < kldpc");
  ATSC3_ARG(ld_hard % 4 == 0 && ((uintptr_t)hard & 3) == 0,
            "hard must be 4-byte aligned with ld_hard a multiple of 4");
  ATSC3_ARG(((uintptr_t)rtab & 7) == 0, "rtab must be 8-byte aligned");
  if (payload) {
    ATSC3_ARG(scr != nullptr, "payload needs the scrambling bytes");
    ATSC3_ARG(kpay % 8 == 0 && kpay <= kldpc, "kpayload must be a multiple of 8");
    ATSC3_ARG(ld_payload >= kpay / 8, "ld_payload < kpayload/8");
  }
  ATSC3_CUDA(bch_launch(bch_packed_kernel, nblk, bch_cluster(nblk, kldpc), st, hard, ld_hard,
                        kldpc, rtab, syn, ok, scr, kpay, payload, ld_payload));
  return 0;
}

int32_t bch_bits_launch(const uint8_t *bits, int64_t ld_bits, int nblk,
                        int kldpc, const uint32_t *rtab, uint32_t *syn,
                        cudaStream_t st) {
  ATSC3_ARG(nblk >= 0 && kldpc > 0, "bad size");
  if (nblk == 0) return 0;
  ATSC3_ARG(bits && rtab && syn, "null pointer");
  ATSC3_ARG(ld_bits >= kldpc, "ld_bits < kldpc");
  ATSC3_ARG(((uintptr_t)rtab & 7) == 0, "rtab must be 8-byte aligned");
  ATSC3_CUDA(bch_launch(bch_bits_kernel, nblk, bch_cluster(nblk, kldpc), st, bits, ld_bits, kldpc,
                        rtab, syn));
  return 0;
}

// ---- uneven batches: per-block BCH length, tables and payload -------------
struct BchBatchArgs {
  const uint8_t *hard;
  const int64_t *hard_off;
  const int32_t *kldpc;
  const uint32_t *rtab;
  const int64_t *rtab_off;    // uint32 words
  const uint8_t *scr;         // scrambling bytes (longest payload)
  const int32_t *kpay;
  uint8_t *payload;
  const int64_t *pay_off;
  uint32_t *syn;
  uint8_t *ok;
};

__global__ void __launch_bounds__(BCH_T) bch_batch_kernel(const BchBatchArgs a) {
  cluster_arrive();
  const int b = (int)cluster_id_x();
  uint32_t acc[6] = {0, 0, 0, 0, 0, 0};
  fold_packed(acc, a.hard + a.hard_off[b], a.kldpc[b], a.rtab + a.rtab_off[b], a.scr,
              a.payload ? a.kpay[b] : 0, a.payload ? a.payload + a.pay_off[b] : nullptr);
  reduce_store(acc, a.syn + (size_t)b * 6, a.ok + b);
}

}  // namespace atsc3

extern "C" {

int32_t atsc3_bch_batch(const uint8_t *hard, const int64_t *hard_off,
                        const int32_t *kldpc, const uint32_t *rtab,
                        const int64_t *rtab_off, const uint8_t *scr,
                        const int32_t *kpay, uint8_t *payload,
                        const int64_t *pay_off, uint32_t *syn, uint8_t *ok,
                        int32_t nblk, void *stream) {
  using namespace atsc3;
  ATSC3_ARG(nblk >= 0, "negative size");
  if (nblk == 0) return 0;
  ATSC3_ARG(hard && hard_off && kldpc && rtab && rtab_off && syn && ok, "null pointer");
  ATSC3_ARG(!payload || (scr && kpay && pay_off), "payload needs scr, kpay, pay_off");
  BchBatchArgs a{hard, hard_off, kldpc, rtab, rtab_off, scr, kpay, payload,
                 pay_off, syn, ok};
  // the lengths are on the device: the cluster of the longest
  ATSC3_CUDA(bch_launch(bch_batch_kernel, nblk, bch_cluster(nblk, 64800), (cudaStream_t)stream, a));
  return 0;
}


int32_t atsc3_bch_check(const uint8_t *hard, int64_t ld_hard, int32_t nblk,
                        int32_t kldpc, const uint32_t *rtab, uint32_t *syn,
                        uint8_t *ok, const uint8_t *scr, int32_t kpayload,
                        uint8_t *payload, int64_t ld_payload, void *stream) {
  return atsc3::bch_check_launch(hard, ld_hard, nblk, kldpc, rtab, syn, ok,
                                 scr, kpayload, payload, ld_payload,
                                 (cudaStream_t)stream);
}

int32_t atsc3_bch_syndrome_bits(const uint8_t *bits, int64_t ld_bits,
                                int32_t nblk, int32_t kldpc,
                                const uint32_t *rtab, uint32_t *syn,
                                void *stream) {
  return atsc3::bch_bits_launch(bits, ld_bits, nblk, kldpc, rtab, syn,
                                (cudaStream_t)stream);
}

}  // extern "C"
