// sumcheck_device.cuh -- device-side pieces of the Spartan zk-sumcheck used by
// the batched form: compute_blinding_coefficients_for_round
// (provekit/prover/src/whir_r1cs.rs:427-492) by one warp and the cubic
// evaluation (provekit/common/src/utils/sumcheck.rs:156-158).
#pragma once
#include "fr.cuh"
#include "reduce.cuh"

namespace pk {

__device__ __forceinline__ Fr dev_cubic(const Fr* c, const Fr& x) {
  Fr acc = fr_mul(x, c[3]);
  acc = fr_mul(fr_add(acc, c[2]), x);
  acc = fr_mul(fr_add(acc, c[1]), x);
  return fr_add(acc, c[0]);
}

// (p + 1) / 2 in Montgomery form = 2^-1
__device__ __forceinline__ Fr fr_half_mont() {
  Fr one = fr_one_mont();
  // 2^-1 * R = (R + p) / 2 when R is odd... compute as one * half via shift:
  // R mod p is odd here, so (R mod p + p) / 2 is exact.
  Fr s;
  uint32_t carry = 0;
  // s = one + p (257 bits at most), then >> 1
  asm("add.cc.u32  %0, %9,  %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32    %8, 0, 0;"
      : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]),
        "=r"(s.v[6]), "=r"(s.v[7]), "=r"(carry)
      : "r"(one.v[0]), "r"(one.v[1]), "r"(one.v[2]), "r"(one.v[3]), "r"(one.v[4]), "r"(one.v[5]),
        "r"(one.v[6]), "r"(one.v[7]), "n"(PK_P0), "n"(PK_P1), "n"(PK_P2), "n"(PK_P3), "n"(PK_P4),
        "n"(PK_P5), "n"(PK_P6), "n"(PK_P7));
  Fr h;
#pragma unroll
  for (int i = 0; i < 7; i++) h.v[i] = (s.v[i] >> 1) | (s.v[i + 1] << 31);
  h.v[7] = (s.v[7] >> 1) | (carry << 31);
  return h;
}

// compute_blinding_coefficients_for_round (whir_r1cs.rs:427-492) for
// compute_for < n <= 32 by one warp: lane i takes g_i (n x 4; alphas: at least
// compute_for entries) and the six products by powers of two run in six lanes.
// scratch: six Fr of this warp's.  Every lane gets the result.
__device__ __forceinline__ void warp_blinding_coeffs(const Fr* g, int n, int compute_for,
                                                     const Fr* alphas, int lane, Fr* scratch,
                                                     Fr out[4]) {
  Fr prefix = fr_zero(), suffix = fr_zero();
  if (lane < compute_for) {
    prefix = dev_cubic(g + 4 * lane, alphas[lane]);
  } else if (lane > compute_for && lane < n) {  // at 0 and at 1
    const Fr* c = g + 4 * lane;
    suffix = fr_add(fr_add(fr_add(c[0], c[0]), c[1]), fr_add(c[2], c[3]));
  }
  __syncwarp();
  prefix = warp_sum(prefix);
  suffix = warp_sum(suffix);
  const int e = n - 1 - compute_for;  // 2^e on the current terms and the prefix, 2^(e-1) on the suffix
  Fr pow2 = fr_zero();
  pow2.v[0] = 1u << e;
  const Fr pm = fr_to_mont(pow2);
  if (lane < 6) {
    const Fr x = lane < 4 ? g[4 * compute_for + lane] : (lane == 4 ? prefix : suffix);
    Fr w = pm;
    if (lane == 5) w = fr_mul(pm, fr_half_mont());
    scratch[lane] = fr_mul(x, w);
  }
  __syncwarp();
  out[0] = fr_add(scratch[0], fr_add(scratch[4], scratch[5]));
#pragma unroll
  for (int k = 1; k < 4; k++) out[k] = scratch[k];
  __syncwarp();
}

// The Spartan round code below multiplies 14 times per pair; inlining every
// product made a ~100 KB kernel that runs from cold instruction cache
// (small rounds took ~40 us whatever their size).  One out-of-line product
// keeps the kernel small.
static __device__ __noinline__ Fr fr_mul_call(const Fr a, const Fr b) { return fr_mul(a, b); }

// One pair (t[j], t[j + q]) of a table; with kFold the live size is 4q and
// the top variable is folded first, t[j] += f (t[j+2q] - t[j]) and
// t[j+q] += f (t[j+3q] - t[j+q]), in place.
template <bool kFold>
__device__ __forceinline__ void round_pair(uint64_t* t, size_t j, size_t q, const Fr& fold, Fr& x0,
                                           Fr& x1) {
  x0 = fr_load(t, j);
  x1 = fr_load(t, j + q);
  if (kFold) {
    x0 = fr_add(x0, fr_mul_call(fold, fr_sub(fr_load(t, j + 2 * q), x0)));
    x1 = fr_add(x1, fr_mul_call(fold, fr_sub(fr_load(t, j + 3 * q), x1)));
    fr_store(t, j, x0);
    fr_store(t, j + q, x1);
  }
}

// The Spartan closure (whir_r1cs.rs:552-558) on one pair of each table,
// streaming the tables a, b, c, eq in turn so that only partial products
// stay live:
//   f(0)   = eq0 (a0 b0 - c0)
//   f(-1)  = (2eq0 - eq1) ((2a0 - a1)(2b0 - b1) - (2c0 - c1))
//   f(inf) = (eq1 - eq0)(a1 - a0)(b1 - b0)
template <bool kFold>
__device__ __forceinline__ void spartan_pair(uint64_t* const (&tabs)[4], size_t j, size_t q,
                                             const Fr& fold, Fr (&acc)[3]) {
  Fr x0, x1;
  round_pair<kFold>(tabs[0], j, q, fold, x0, x1);
  const Fr a0 = x0, a2 = fr_sub(fr_add(x0, x0), x1), da = fr_sub(x1, x0);
  round_pair<kFold>(tabs[1], j, q, fold, x0, x1);
  const Fr ab = fr_mul_call(a0, x0);
  const Fr ab2 = fr_mul_call(a2, fr_sub(fr_add(x0, x0), x1));
  const Fr dab = fr_mul_call(da, fr_sub(x1, x0));
  round_pair<kFold>(tabs[2], j, q, fold, x0, x1);
  const Fr t0 = fr_sub(ab, x0), t1 = fr_sub(ab2, fr_sub(fr_add(x0, x0), x1));
  round_pair<kFold>(tabs[3], j, q, fold, x0, x1);
  acc[0] = fr_add(acc[0], fr_mul_call(x0, t0));
  acc[1] = fr_add(acc[1], fr_mul_call(fr_sub(fr_add(x0, x0), x1), t1));
  acc[2] = fr_add(acc[2], fr_mul_call(fr_sub(x1, x0), dab));
}

// Rounds of at most this many pairs take four lanes per pair.  Spartan rounds of
// 2^12, 2^14, 2^15 and 2^16 pairs: 13, 17, 24 and 36 us, against 22, 23, 23 and
// 33 with a thread per pair; WHIR rounds of 2^12, 2^14 and 2^15: 10, 12 and 18
// against 15, 16 and 17.
constexpr size_t kQuadMaxPairs = size_t(1) << 14;

// Sumcheck rounds with four lanes per pair.  A lane folds one table (Spartan) or
// one of the four values (WHIR), the quad exchanges what it has through shared
// memory, and a lane each makes a sum's product: 4 and 2 dependent products
// where one thread has 14 and 7 (small rounds are bound by that chain).
constexpr int kQuadThreads = 256;                // 64 pairs at a time
constexpr int kQuadPairs = kQuadThreads / 4;

struct FrShared {  // a value per thread as two 16-byte halves
  uint4 lo[kQuadThreads], hi[kQuadThreads];
  __device__ __forceinline__ void put(int i, const Fr& x) {
    lo[i] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
    hi[i] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
  }
  __device__ __forceinline__ Fr get(int i) const {
    const uint4 a = lo[i], b = hi[i];
    Fr x;
    x.v[0] = a.x; x.v[1] = a.y; x.v[2] = a.z; x.v[3] = a.w;
    x.v[4] = b.x; x.v[5] = b.y; x.v[6] = b.z; x.v[7] = b.w;
    return x;
  }
};

// The Spartan closure (whir_r1cs.rs:552-558) over pairs (t[j], t[j + q]) of the
// tables a, b, c, eq, j = first, first + step, .., as spartan_pair.  Lane k < 3 of
// a quad returns its share of sum k.  first: the CTA's first pair; all threads
// of the CTA call it together.
template <bool kFold>
__device__ __forceinline__ Fr spartan_quads(uint64_t* const (&tabs)[4], size_t first, size_t step,
                                            size_t q, const Fr& fold, FrShared (&sh)[3]) {
  const int lane = threadIdx.x & 3, quad = threadIdx.x & ~3;
  uint64_t* const t = lane < 2 ? (lane == 0 ? tabs[0] : tabs[1]) : (lane == 2 ? tabs[2] : tabs[3]);
  Fr acc = fr_zero();
  for (size_t base = first; base < q; base += step) {
    const size_t j = base + (threadIdx.x >> 2);
    if (j < q) {
      Fr x0 = fr_load(t, j), x1 = fr_load(t, j + q);
      if (kFold) {
        const Fr d0 = fr_sub(fr_load(t, j + 2 * q), x0), d1 = fr_sub(fr_load(t, j + 3 * q), x1);
        x0 = fr_add(x0, fr_mul(fold, d0));
        x1 = fr_add(x1, fr_mul(fold, d1));
        fr_store(t, j, x0);
        fr_store(t, j + q, x1);
      }
      sh[0].put(threadIdx.x, x0);
      sh[1].put(threadIdx.x, fr_sub(fr_add(x0, x0), x1));
      sh[2].put(threadIdx.x, fr_sub(x1, x0));
    }
    __syncwarp();
    if (j < q && lane < 3) {
      const FrShared& v = sh[lane];
      Fr ab = fr_mul(v.get(quad), v.get(quad + 1));
      if (lane < 2) ab = fr_sub(ab, v.get(quad + 2));
      acc = fr_add(acc, fr_mul(ab, v.get(quad + 3)));
    }
    __syncwarp();
  }
  return acc;
}

// CTAs for a round of q pairs, at most 4 per SM (the partials' room).
inline int round_grid(size_t q) { return red_grid(q <= kQuadMaxPairs ? 4 * q : q); }

// As three sums for block_sum: lane k < 3 of a quad holds a share of sum k.
__device__ __forceinline__ void quad_sums(const Fr& acc, Fr (&v)[3]) {
  const int lane = threadIdx.x & 3;
#pragma unroll
  for (int k = 0; k < 3; k++) v[k] = lane == k ? acc : fr_zero();
}

}  // namespace pk
