// reduce.cuh -- block-wide sums of field elements and the grid-size helpers
// shared by the reduction kernels (sumcheck, dot products, WHIR rounds).
//
// Each thread accumulates a grid-stride slice, a CTA adds its threads' sums,
// and one partial per CTA goes to a small scratch array that a single CTA
// sums.  Field addition is exact, so the result does not depend on the
// reduction order.
#pragma once
#include <algorithm>

#include "fr.cuh"
#include "fr_sum.cuh"
#include "pk_common.cuh"

namespace pk {

constexpr int kRedThreads = 256;

// Sums of field elements as integers, limb by limb: 256 limbs of 24 bits fit
// 32 bits, so a warp adds each limb with one redux and a total is reduced
// once.  (Modular additions down a shuffle tree were 5 dependent levels of 8
// shuffles and a 16-step carry chain each.)
constexpr int kSumLimbs = 11;  // 24-bit limbs of an element

// This warp's sum of x, limb by limb, in every lane.
__device__ __forceinline__ void warp_limbs(const Fr& v, uint32_t* sum) {
  constexpr uint32_t M = 0xffffffu;
  const uint32_t* x = v.v;
  const uint32_t d[kSumLimbs] = {x[0] & M,
                                 __funnelshift_r(x[0], x[1], 24) & M,
                                 __funnelshift_r(x[1], x[2], 16) & M,
                                 x[2] >> 8,
                                 x[3] & M,
                                 __funnelshift_r(x[3], x[4], 24) & M,
                                 __funnelshift_r(x[4], x[5], 16) & M,
                                 x[5] >> 8,
                                 x[6] & M,
                                 __funnelshift_r(x[6], x[7], 24) & M,
                                 x[7] >> 16};
#pragma unroll
  for (int i = 0; i < kSumLimbs; i++) sum[i] = __reduce_add_sync(0xffffffffu, d[i]);
}

// sum limbs[i] 2^(24 i) mod p, fully reduced, of at most 256 elements
__device__ __forceinline__ Fr limbs_reduce(const uint32_t* limbs) {
  constexpr uint32_t M = 0xffffffu;
  uint32_t d[kSumLimbs + 1], S[9];
  uint64_t carry = 0;
#pragma unroll
  for (int i = 0; i < kSumLimbs; i++) {
    carry += limbs[i];
    d[i] = (uint32_t)carry & M;
    carry >>= 24;
  }
  d[kSumLimbs] = (uint32_t)carry;
  S[0] = d[0] | (d[1] << 24);
  S[1] = (d[1] >> 8) | (d[2] << 16);
  S[2] = (d[2] >> 16) | (d[3] << 8);
  S[3] = d[4] | (d[5] << 24);
  S[4] = (d[5] >> 8) | (d[6] << 16);
  S[5] = (d[6] >> 16) | (d[7] << 8);
  S[6] = d[8] | (d[9] << 24);
  S[7] = (d[9] >> 8) | (d[10] << 16);
  S[8] = (d[10] >> 16) | (d[11] << 8);
  return fr_reduce_once(tc::quotient_step(S));
}

// This warp's sum of x in every lane.
__device__ __forceinline__ Fr warp_sum(const Fr& x) {
  uint32_t limbs[kSumLimbs];
  warp_limbs(x, limbs);
  return limbs_reduce(limbs);
}

// Block-wide sum of K field elements per thread (at most 256 threads); thread
// 0 gets the result, fully reduced: the warps' limbs are added by one warp.
template <int K>
__device__ __forceinline__ void block_sum(Fr (&v)[K]) {
  __shared__ uint32_t limbs[kRedThreads / 32][K * kSumLimbs];
  __shared__ uint32_t total[K * kSumLimbs];
  __shared__ Fr sums[K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    uint32_t sum[kSumLimbs];
    warp_limbs(v[k], sum);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < kSumLimbs; i++) limbs[warp][k * kSumLimbs + i] = sum[i];
  }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    for (int i = lane; i < K * kSumLimbs; i += 32) {
      uint32_t sum = 0;
      for (int w = 0; w < nw; w++) sum += limbs[w][i];
      total[i] = sum;
    }
    __syncwarp();
    if (lane < K) sums[lane] = limbs_reduce(total + lane * kSumLimbs);
    __syncwarp();
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < K; k++) v[k] = sums[k];
  }
}

// Where a reduction kernel's CTAs leave their sums.  Every CTA takes a ticket after
// storing its partial (K Fr), and the CTA that takes the last one adds all partials,
// writes the K sums to out (mapped host memory) and resets the counter for the next
// launch.
//
// It also announces its completion to the host: after writing the sums, the
// last CTA stores seq (fused_next_seq(), nonzero) into a word of mapped host
// memory whose device address sits in the ticket's block (ticket + 2, see
// fused_slots), so fused_read can poll that word instead of waiting for the
// stream.
struct RedOut {
  uint64_t* part;
  unsigned* ticket;
  uint64_t* out;
  unsigned seq;  // 0: no completion word
};

// 32 bytes through L2 only: partials other CTAs wrote during this launch.
__device__ __forceinline__ Fr fr_load_cg(const uint64_t* base, size_t idx) {
  const uint4* q = reinterpret_cast<const uint4*>(base + 4 * idx);
  const uint4 a = __ldcg(q), b = __ldcg(q + 1);
  Fr r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}

// One thread of the last CTA, after its stores to out: the ticket as it was found, then
// the completion word.
__device__ __forceinline__ void announce(const RedOut& ro) {
  *ro.ticket = 0u;
  if (ro.seq) {
    volatile unsigned* word = *reinterpret_cast<unsigned* const*>(ro.ticket + 2);
    __threadfence_system();  // the sums before the completion word
    *word = ro.seq;
  }
}

// The end of a reduction kernel: block sum, the CTA's partial, and the last CTA's final
// sum.  Every thread of the CTA calls it.
template <int K>
__device__ __forceinline__ void block_finish(Fr (&v)[K], const RedOut& ro) {
  __shared__ bool last;
  block_sum<K>(v);
  if (gridDim.x != 1) {  // else this CTA's sum is the sum
    if (threadIdx.x == 0) {
#pragma unroll
      for (int k = 0; k < K; k++) fr_store(ro.part, (size_t)blockIdx.x * K + k, v[k]);
      __threadfence();
      last = atomicAdd(ro.ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < K; k++) v[k] = fr_zero();
    for (unsigned i = threadIdx.x; i < gridDim.x; i += blockDim.x)
#pragma unroll
      for (int k = 0; k < K; k++) v[k] = fr_add(v[k], fr_load_cg(ro.part, (size_t)i * K + k));
    block_sum<K>(v);
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) fr_store(ro.out, k, v[k]);
    announce(ro);
  }
}

// The end of a kernel with several sums, each over a run of CTAs: thread 0's sum is this
// CTA's partial, and warp w of the last CTA adds the partials first .. end - 1 of sum w
// (count <= the CTA's warps; each thread passes its warp's run).
__device__ __forceinline__ void runs_finish(const Fr& sum, const RedOut& ro, int count,
                                            unsigned first, unsigned end) {
  __shared__ bool last;
  if (threadIdx.x == 0) {
    fr_store(ro.part, blockIdx.x, sum);
    __threadfence();
    last = atomicAdd(ro.ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < count) {
    Fr x = fr_zero();
    for (unsigned k = first + lane; k < end; k += 32) x = fr_add(x, fr_load_cg(ro.part, k));
    x = warp_sum(x);
    if (lane == 0) fr_store(ro.out, warp, x);
  }
  __syncthreads();
  if (threadIdx.x == 0) announce(ro);
}

// CTAs for a reduction over n items (at most 4 per SM).
inline int red_grid(size_t n) {
  size_t b = (n + kRedThreads - 1) / kRedThreads;
  return (int)std::max<size_t>(1, std::min<size_t>(b, (size_t)sm_count() * 4));
}
// CTAs of 256 threads for an element-wise kernel over n items (grid-stride).
inline int ew_grid(size_t n) {
  size_t b = (n + 255) / 256;
  return (int)std::max<size_t>(1, std::min<size_t>(b, (size_t)sm_count() * 32));
}

}  // namespace pk
