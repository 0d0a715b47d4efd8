// fr_lazy.cuh -- exact sums of products of 256-bit values on the integer pipe,
// reduced once per sum.
//
// A sum S = sum_k a_k b_k of products of Montgomery-form values is needed
// reduced only once: its products are added up as integers, and one Montgomery
// reduction follows instead of one per product.
//
// The words a_i b_j of a product are added to two accumulators, those with i + j
// even to one and the rest to the other, so that each product and its addition
// is one 64-bit multiply-add onto an aligned pair.  The products with the same
// i - j lie two words apart, so they form one carry chain; a chain ends above the
// highest word that it wrote, and the carry out of it is counted in a word of its
// own instead of running on to the top.  A term is 64 multiply-adds and 15
// counts, 256 cycles of the multiplier per warp: half of a Montgomery product,
// and half of the 144 binary64 digit products and 24 conversions per term that
// stood here before.  Alone a term takes 310 cycles.
#pragma once
#include "fr_sum.cuh"

namespace pk {
namespace lazy {

constexpr int kMaxTerms = 1024;  // terms per finish(): the sum is below 2^15 p 2^256

// One multiply-add of a chain onto the pair (l, h); the first one starts the carry.
#define PK_FIRST(l, h, a, b) "mad.lo.cc.u32 " l "," a "," b "," l ";\n\tmadc.hi.cc.u32 " h "," a "," b "," h ";\n\t"
#define PK_NEXT(l, h, a, b) "madc.lo.cc.u32 " l "," a "," b "," l ";\n\tmadc.hi.cc.u32 " h "," a "," b "," h ";\n\t"
#define PK_COUNT(c) "addc.u32 " c "," c ",0;\n\t"

struct Acc {
  uint32_t e[16];  // words 0..15
  uint32_t o[14];  // words 1..14
  uint32_t c[8];   // carries into words 9..16

  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 16; i++) e[i] = 0;
#pragma unroll
    for (int i = 0; i < 14; i++) o[i] = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = 0;
  }

  // += a b, for any 256-bit a and b
  __device__ __forceinline__ void mac(const Fr& a, const Fr& b) {
    asm(
        PK_FIRST("%0", "%1", "%20", "%28")
        PK_NEXT("%2", "%3", "%21", "%29")
        PK_NEXT("%4", "%5", "%22", "%30")
        PK_NEXT("%6", "%7", "%23", "%31")
        PK_NEXT("%8", "%9", "%24", "%32")
        PK_NEXT("%10", "%11", "%25", "%33")
        PK_NEXT("%12", "%13", "%26", "%34")
        PK_NEXT("%14", "%15", "%27", "%35")
        PK_COUNT("%19")
        PK_FIRST("%2", "%3", "%22", "%28")
        PK_NEXT("%4", "%5", "%23", "%29")
        PK_NEXT("%6", "%7", "%24", "%30")
        PK_NEXT("%8", "%9", "%25", "%31")
        PK_NEXT("%10", "%11", "%26", "%32")
        PK_NEXT("%12", "%13", "%27", "%33")
        PK_COUNT("%18")
        PK_FIRST("%2", "%3", "%20", "%30")
        PK_NEXT("%4", "%5", "%21", "%31")
        PK_NEXT("%6", "%7", "%22", "%32")
        PK_NEXT("%8", "%9", "%23", "%33")
        PK_NEXT("%10", "%11", "%24", "%34")
        PK_NEXT("%12", "%13", "%25", "%35")
        PK_COUNT("%18")
        PK_FIRST("%4", "%5", "%24", "%28")
        PK_NEXT("%6", "%7", "%25", "%29")
        PK_NEXT("%8", "%9", "%26", "%30")
        PK_NEXT("%10", "%11", "%27", "%31")
        PK_COUNT("%17")
        PK_FIRST("%4", "%5", "%20", "%32")
        PK_NEXT("%6", "%7", "%21", "%33")
        PK_NEXT("%8", "%9", "%22", "%34")
        PK_NEXT("%10", "%11", "%23", "%35")
        PK_COUNT("%17")
        PK_FIRST("%6", "%7", "%26", "%28")
        PK_NEXT("%8", "%9", "%27", "%29")
        PK_COUNT("%16")
        PK_FIRST("%6", "%7", "%20", "%34")
        PK_NEXT("%8", "%9", "%21", "%35")
        PK_COUNT("%16")
        : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]),
          "+r"(e[7]), "+r"(e[8]), "+r"(e[9]), "+r"(e[10]), "+r"(e[11]), "+r"(e[12]),
          "+r"(e[13]), "+r"(e[14]), "+r"(e[15]), "+r"(c[1]), "+r"(c[3]), "+r"(c[5]),
          "+r"(c[7])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
          "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
    asm(
        PK_FIRST("%0", "%1", "%19", "%26")
        PK_NEXT("%2", "%3", "%20", "%27")
        PK_NEXT("%4", "%5", "%21", "%28")
        PK_NEXT("%6", "%7", "%22", "%29")
        PK_NEXT("%8", "%9", "%23", "%30")
        PK_NEXT("%10", "%11", "%24", "%31")
        PK_NEXT("%12", "%13", "%25", "%32")
        PK_COUNT("%17")
        PK_FIRST("%0", "%1", "%18", "%27")
        PK_NEXT("%2", "%3", "%19", "%28")
        PK_NEXT("%4", "%5", "%20", "%29")
        PK_NEXT("%6", "%7", "%21", "%30")
        PK_NEXT("%8", "%9", "%22", "%31")
        PK_NEXT("%10", "%11", "%23", "%32")
        PK_NEXT("%12", "%13", "%24", "%33")
        PK_COUNT("%17")
        PK_FIRST("%2", "%3", "%21", "%26")
        PK_NEXT("%4", "%5", "%22", "%27")
        PK_NEXT("%6", "%7", "%23", "%28")
        PK_NEXT("%8", "%9", "%24", "%29")
        PK_NEXT("%10", "%11", "%25", "%30")
        PK_COUNT("%16")
        PK_FIRST("%2", "%3", "%18", "%29")
        PK_NEXT("%4", "%5", "%19", "%30")
        PK_NEXT("%6", "%7", "%20", "%31")
        PK_NEXT("%8", "%9", "%21", "%32")
        PK_NEXT("%10", "%11", "%22", "%33")
        PK_COUNT("%16")
        PK_FIRST("%4", "%5", "%23", "%26")
        PK_NEXT("%6", "%7", "%24", "%27")
        PK_NEXT("%8", "%9", "%25", "%28")
        PK_COUNT("%15")
        PK_FIRST("%4", "%5", "%18", "%31")
        PK_NEXT("%6", "%7", "%19", "%32")
        PK_NEXT("%8", "%9", "%20", "%33")
        PK_COUNT("%15")
        PK_FIRST("%6", "%7", "%25", "%26")
        PK_COUNT("%14")
        PK_FIRST("%6", "%7", "%18", "%33")
        PK_COUNT("%14")
        : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]),
          "+r"(o[7]), "+r"(o[8]), "+r"(o[9]), "+r"(o[10]), "+r"(o[11]), "+r"(o[12]),
          "+r"(o[13]), "+r"(c[0]), "+r"(c[2]), "+r"(c[4]), "+r"(c[6])
        : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
          "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
          "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  }

  // sum * 2^-256 mod p, fully reduced
  __device__ __forceinline__ Fr finish() const {
    uint32_t t[17];
    t[0] = e[0];
    asm("add.cc.u32  %0, %9,  %17;\n\t"
        "addc.cc.u32 %1, %10, %18;\n\t"
        "addc.cc.u32 %2, %11, %19;\n\t"
        "addc.cc.u32 %3, %12, %20;\n\t"
        "addc.cc.u32 %4, %13, %21;\n\t"
        "addc.cc.u32 %5, %14, %22;\n\t"
        "addc.cc.u32 %6, %15, %23;\n\t"
        "addc.cc.u32 %7, %16, %24;\n\t"
        "addc.u32    %8, 0, 0;"
        : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]),
          "=r"(t[8]), "=r"(t[9])
        : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]),
          "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]));
    // words 8..16: e and o with the carry of the words below, then the counts
    uint32_t h[9] = {t[8], e[9], e[10], e[11], e[12], e[13], e[14], e[15], 0};
    const uint32_t up[8] = {0, o[8], o[9], o[10], o[11], o[12], o[13], 0};
    const uint32_t carry[8] = {0, t[9], 0, 0, 0, 0, 0, 0};
    tc::add9(h, up);
    tc::add9(h, carry);
    const uint32_t low[8] = {0, c[0], c[1], c[2], c[3], c[4], c[5], c[6]};
    tc::add9(h, low);
    h[8] += c[7];
    // (low words + M p) / 2^256 <= p, then S / 2^256 < 2^15 p by one quotient step
    const Fr r = fr_redc(t);
    tc::add9(h, r.v);
    return fr_reduce_once(tc::quotient_step(h));
  }
};

#undef PK_FIRST
#undef PK_NEXT
#undef PK_COUNT

}  // namespace lazy
}  // namespace pk
