// fr_sum.cuh -- sums of field elements and of products as 9-word integers, and
// the step that reduces them once.
#pragma once
#include "fr.cuh"

// Chains of products into X[k], X[k + 1], ...: PK_NEW_PAIR writes a pair that
// nothing wrote before; PK_CHAINn adds n - 1 products to pairs and ends on a
// new one, which takes its carry; PK_CARRYn adds n and returns the carry.
#define PK_NEW_PAIR(X, k, a, b)                    \
  do {                                             \
    const uint64_t w_ = (uint64_t)(a) * (b);       \
    (X)[k] = (uint32_t)w_;                         \
    (X)[(k) + 1] = (uint32_t)(w_ >> 32);           \
  } while (0)
#define PK_CHAIN3(X, k, a0, b0, a1, b1, a2, b2) \
  asm("mad.lo.cc.u32  %0, %6, %7, %0;\n\t" \
      "madc.hi.cc.u32 %1, %6, %7, %1;\n\t" \
      "madc.lo.cc.u32 %2, %8, %9, %2;\n\t" \
      "madc.hi.cc.u32 %3, %8, %9, %3;\n\t" \
      "madc.lo.cc.u32 %4, %10, %11, 0;\n\t" \
      "madc.hi.u32 %5, %10, %11, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "=r"((X)[(k) + 4]), "=r"((X)[(k) + 5]) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2))
#define PK_CHAIN4(X, k, a0, b0, a1, b1, a2, b2, a3, b3) \
  asm("mad.lo.cc.u32  %0, %8, %9, %0;\n\t" \
      "madc.hi.cc.u32 %1, %8, %9, %1;\n\t" \
      "madc.lo.cc.u32 %2, %10, %11, %2;\n\t" \
      "madc.hi.cc.u32 %3, %10, %11, %3;\n\t" \
      "madc.lo.cc.u32 %4, %12, %13, %4;\n\t" \
      "madc.hi.cc.u32 %5, %12, %13, %5;\n\t" \
      "madc.lo.cc.u32 %6, %14, %15, 0;\n\t" \
      "madc.hi.u32 %7, %14, %15, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "=r"((X)[(k) + 6]), "=r"((X)[(k) + 7]) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3))
#define PK_CHAIN5(X, k, a0, b0, a1, b1, a2, b2, a3, b3, a4, b4) \
  asm("mad.lo.cc.u32  %0, %10, %11, %0;\n\t" \
      "madc.hi.cc.u32 %1, %10, %11, %1;\n\t" \
      "madc.lo.cc.u32 %2, %12, %13, %2;\n\t" \
      "madc.hi.cc.u32 %3, %12, %13, %3;\n\t" \
      "madc.lo.cc.u32 %4, %14, %15, %4;\n\t" \
      "madc.hi.cc.u32 %5, %14, %15, %5;\n\t" \
      "madc.lo.cc.u32 %6, %16, %17, %6;\n\t" \
      "madc.hi.cc.u32 %7, %16, %17, %7;\n\t" \
      "madc.lo.cc.u32 %8, %18, %19, 0;\n\t" \
      "madc.hi.u32 %9, %18, %19, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "+r"((X)[(k) + 6]), "+r"((X)[(k) + 7]), "=r"((X)[(k) + 8]), "=r"((X)[(k) + 9]) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3), "r"(a4), "r"(b4))
#define PK_CHAIN6(X, k, a0, b0, a1, b1, a2, b2, a3, b3, a4, b4, a5, b5) \
  asm("mad.lo.cc.u32  %0, %12, %13, %0;\n\t" \
      "madc.hi.cc.u32 %1, %12, %13, %1;\n\t" \
      "madc.lo.cc.u32 %2, %14, %15, %2;\n\t" \
      "madc.hi.cc.u32 %3, %14, %15, %3;\n\t" \
      "madc.lo.cc.u32 %4, %16, %17, %4;\n\t" \
      "madc.hi.cc.u32 %5, %16, %17, %5;\n\t" \
      "madc.lo.cc.u32 %6, %18, %19, %6;\n\t" \
      "madc.hi.cc.u32 %7, %18, %19, %7;\n\t" \
      "madc.lo.cc.u32 %8, %20, %21, %8;\n\t" \
      "madc.hi.cc.u32 %9, %20, %21, %9;\n\t" \
      "madc.lo.cc.u32 %10, %22, %23, 0;\n\t" \
      "madc.hi.u32 %11, %22, %23, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "+r"((X)[(k) + 6]), "+r"((X)[(k) + 7]), "+r"((X)[(k) + 8]), "+r"((X)[(k) + 9]), "=r"((X)[(k) + 10]), "=r"((X)[(k) + 11]) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3), "r"(a4), "r"(b4), "r"(a5), "r"(b5))
#define PK_CARRY1(X, k, a0, b0, c) \
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t" \
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t" \
      "addc.u32 %2, 0, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "=r"(c) \
      : "r"(a0), "r"(b0))
#define PK_CARRY2(X, k, a0, b0, a1, b1, c) \
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t" \
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t" \
      "madc.lo.cc.u32 %2, %7, %8, %2;\n\t" \
      "madc.hi.cc.u32 %3, %7, %8, %3;\n\t" \
      "addc.u32 %4, 0, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "=r"(c) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1))
#define PK_CARRY3(X, k, a0, b0, a1, b1, a2, b2, c) \
  asm("mad.lo.cc.u32  %0, %7, %8, %0;\n\t" \
      "madc.hi.cc.u32 %1, %7, %8, %1;\n\t" \
      "madc.lo.cc.u32 %2, %9, %10, %2;\n\t" \
      "madc.hi.cc.u32 %3, %9, %10, %3;\n\t" \
      "madc.lo.cc.u32 %4, %11, %12, %4;\n\t" \
      "madc.hi.cc.u32 %5, %11, %12, %5;\n\t" \
      "addc.u32 %6, 0, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "=r"(c) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2))
#define PK_CARRY4(X, k, a0, b0, a1, b1, a2, b2, a3, b3, c) \
  asm("mad.lo.cc.u32  %0, %9, %10, %0;\n\t" \
      "madc.hi.cc.u32 %1, %9, %10, %1;\n\t" \
      "madc.lo.cc.u32 %2, %11, %12, %2;\n\t" \
      "madc.hi.cc.u32 %3, %11, %12, %3;\n\t" \
      "madc.lo.cc.u32 %4, %13, %14, %4;\n\t" \
      "madc.hi.cc.u32 %5, %13, %14, %5;\n\t" \
      "madc.lo.cc.u32 %6, %15, %16, %6;\n\t" \
      "madc.hi.cc.u32 %7, %15, %16, %7;\n\t" \
      "addc.u32 %8, 0, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "+r"((X)[(k) + 6]), "+r"((X)[(k) + 7]), "=r"(c) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3))
#define PK_CARRY5(X, k, a0, b0, a1, b1, a2, b2, a3, b3, a4, b4, c) \
  asm("mad.lo.cc.u32  %0, %11, %12, %0;\n\t" \
      "madc.hi.cc.u32 %1, %11, %12, %1;\n\t" \
      "madc.lo.cc.u32 %2, %13, %14, %2;\n\t" \
      "madc.hi.cc.u32 %3, %13, %14, %3;\n\t" \
      "madc.lo.cc.u32 %4, %15, %16, %4;\n\t" \
      "madc.hi.cc.u32 %5, %15, %16, %5;\n\t" \
      "madc.lo.cc.u32 %6, %17, %18, %6;\n\t" \
      "madc.hi.cc.u32 %7, %17, %18, %7;\n\t" \
      "madc.lo.cc.u32 %8, %19, %20, %8;\n\t" \
      "madc.hi.cc.u32 %9, %19, %20, %9;\n\t" \
      "addc.u32 %10, 0, 0;" \
      : "+r"((X)[(k) + 0]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]), "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "+r"((X)[(k) + 6]), "+r"((X)[(k) + 7]), "+r"((X)[(k) + 8]), "+r"((X)[(k) + 9]), "=r"(c) \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3), "r"(a4), "r"(b4))

namespace pk {
namespace tc {

// S (9 words) += v (8 words)
__device__ __forceinline__ void add9(uint32_t* S, const uint32_t* v) {
  asm("add.cc.u32  %0, %0, %9;\n\t"
      "addc.cc.u32 %1, %1, %10;\n\t"
      "addc.cc.u32 %2, %2, %11;\n\t"
      "addc.cc.u32 %3, %3, %12;\n\t"
      "addc.cc.u32 %4, %4, %13;\n\t"
      "addc.cc.u32 %5, %5, %14;\n\t"
      "addc.cc.u32 %6, %6, %15;\n\t"
      "addc.cc.u32 %7, %7, %16;\n\t"
      "addc.u32    %8, %8, 0;"
      : "+r"(S[0]), "+r"(S[1]), "+r"(S[2]), "+r"(S[3]), "+r"(S[4]), "+r"(S[5]), "+r"(S[6]),
        "+r"(S[7]), "+r"(S[8])
      : "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
}

// S mod p in [0, 1.1 p) for S < 2^15 p (9 words).  q = floor(floor(S / 2^240)
// kQ / 2^32) with kQ = floor(2^272 / p): the two truncations lose less than
// 2^15 / 346695 + 2^240 / p < 0.1 of a quotient unit, so q is the quotient or
// one less and S - q p < 1.1 p, taken as S + q (2^256 - p) mod 2^256.
__device__ __forceinline__ Fr quotient_step(const uint32_t* S) {
  constexpr uint32_t kQ = 0x54a47u;
  constexpr uint32_t N[8] = {0x0fffffffu, 0xbc1e0a6cu, 0x86468f6eu, 0xd7cc17b7u,
                             0x7e7ea7a2u, 0x47afba49u, 0x1ece5fd6u, 0xcf9bb18du};  // 2^256 - p
  const uint32_t q = __umulhi(__funnelshift_l(S[7], S[8], 16), kQ);
  uint32_t E[8], O[6];
#pragma unroll
  for (int i = 0; i < 3; i++) PK_NEW_PAIR(O, 2 * i, q, N[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 8; i++) E[i] = S[i];
  fr_chain4(E, q, N[0], N[2], N[4], N[6]);
  E[7] += q * N[7];
  Fr r;
  r.v[0] = E[0];
  asm("add.cc.u32  %0, %7,  %14;\n\t"
      "addc.cc.u32 %1, %8,  %15;\n\t"
      "addc.cc.u32 %2, %9,  %16;\n\t"
      "addc.cc.u32 %3, %10, %17;\n\t"
      "addc.cc.u32 %4, %11, %18;\n\t"
      "addc.cc.u32 %5, %12, %19;\n\t"
      "addc.u32    %6, %13, 0;"
      : "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(O[0]),
        "r"(O[1]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]));
  return r;
}

// a + b + h + top 2^256 mod p in [0, 1.1 p), for a total below 2^15 p (a, b, h: 8
// words; h may be nullptr).  As quotient_step, but the quotient comes from the
// top words alone, before the carries below them are known (they add at most 2
// at word 7, 2^-15 of a unit of S / 2^240), and its multiple of 2^256 - p is
// accumulated onto a and b, so nothing waits for a sum of all three.
__device__ __forceinline__ Fr quotient_sum(const uint32_t* a, const uint32_t* b,
                                           const uint32_t* h, uint32_t top) {
  constexpr uint32_t kQ = 0x54a47u;
  constexpr uint32_t N[8] = {0x0fffffffu, 0xbc1e0a6cu, 0x86468f6eu, 0xd7cc17b7u,
                             0x7e7ea7a2u, 0x47afba49u, 0x1ece5fd6u, 0xcf9bb18du};  // 2^256 - p
  uint32_t lo, hi;
  asm("add.cc.u32 %0, %2, %3;\n\t"
      "addc.u32   %1, %4, 0;"
      : "=r"(lo), "=r"(hi)
      : "r"(a[7]), "r"(b[7]), "r"(top));
  if (h)
    asm("add.cc.u32 %0, %0, %2;\n\t"
        "addc.u32   %1, %1, 0;"
        : "+r"(lo), "+r"(hi)
        : "r"(h[7]));
  const uint32_t q = __umulhi(__funnelshift_l(lo, hi, 16), kQ);
  uint32_t E[8], O[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    E[i] = a[i];
    O[i] = b[i];
  }
  fr_chain4(E, q, N[0], N[2], N[4], N[6]);
  asm("mad.lo.cc.u32  %0, %7, %8,  %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %8,  %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9,  %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9,  %3;\n\t"
      "madc.lo.cc.u32 %4, %7, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %7, %10, %5;\n\t"
      "madc.lo.u32    %6, %7, %11, %6;"
      : "+r"(O[1]), "+r"(O[2]), "+r"(O[3]), "+r"(O[4]), "+r"(O[5]), "+r"(O[6]), "+r"(O[7])
      : "r"(q), "r"(N[1]), "r"(N[3]), "r"(N[5]), "r"(N[7]));
  Fr e;
#pragma unroll
  for (int i = 0; i < 8; i++) e.v[i] = E[i];
  e = fr_add_raw(e, O);
  if (h) e = fr_add_raw(e, h);
  return e;
}

// Any 256-bit value to [0, 1.1 p).
__device__ __forceinline__ Fr reduce_any(const Fr& x) {
  uint32_t S[9];
#pragma unroll
  for (int i = 0; i < 8; i++) S[i] = x.v[i];
  S[8] = 0;
  return quotient_step(S);
}

}  // namespace tc
}  // namespace pk
