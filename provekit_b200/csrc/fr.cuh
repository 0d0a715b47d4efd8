// fr.cuh -- BN254 scalar field (Fr) arithmetic for sm_100a.
//
// An element is 8 x 32-bit little-endian limbs in registers; in memory it is
// the arkworks layout (4 x u64 LE == 8 x u32 LE), 32 bytes, 32-byte aligned.
// Products are Montgomery products with R = 2^256 on the integer pipe, as
// explicit PTX carry chains of 32x32 -> 64-bit multiply-adds.  This replaces
// ark-ff's Fr multiply and bn254_multiplier::scalar_{mul,sqr}
// (skyscraper/bn254-multiplier/src/scalar.rs:12-132); outputs are fully
// reduced, as ark-ff stores them.
#pragma once
#include <cstdint>

namespace pk {

// p = 0x30644e72e131a029b85045b68181585d2833e84879b9709143e1f593f0000001
#define PK_P0 0xf0000001u
#define PK_P1 0x43e1f593u
#define PK_P2 0x79b97091u
#define PK_P3 0x2833e848u
#define PK_P4 0x8181585du
#define PK_P5 0xb85045b6u
#define PK_P6 0xe131a029u
#define PK_P7 0x30644e72u
#define PK_MU 0xefffffffu  // -p^-1 mod 2^32

struct Fr {
  uint32_t v[8];
};

__device__ __forceinline__ Fr fr_zero() {
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = 0;
  return r;
}

// Montgomery form of 1 (2^256 mod p).
__device__ __forceinline__ Fr fr_one_mont() {
  Fr r;
  r.v[0] = 0x4ffffffbu; r.v[1] = 0xac96341cu; r.v[2] = 0x9f60cd29u; r.v[3] = 0x36fc7695u;
  r.v[4] = 0x7879462eu; r.v[5] = 0x666ea36fu; r.v[6] = 0x9a07df2fu; r.v[7] = 0x0e0a77c1u;
  return r;
}

__device__ __forceinline__ Fr fr_load(const uint64_t* base, size_t idx) {
  const uint4* p = reinterpret_cast<const uint4*>(base + 4 * idx);
  uint4 a = p[0], b = p[1];
  Fr r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}

__device__ __forceinline__ Fr fr_load_ro(const uint64_t* base, size_t idx) {
  const uint4* p = reinterpret_cast<const uint4*>(base + 4 * idx);
  uint4 a = __ldg(p), b = __ldg(p + 1);
  Fr r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}

__device__ __forceinline__ void fr_store(uint64_t* base, size_t idx, const Fr& x) {
  uint4* p = reinterpret_cast<uint4*>(base + 4 * idx);
  p[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  p[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

// x - p if x >= p (x < 2^256).
__device__ __forceinline__ Fr fr_reduce_once(const Fr& x) {
  Fr d;
  uint32_t borrow;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d.v[0]), "=r"(d.v[1]), "=r"(d.v[2]), "=r"(d.v[3]), "=r"(d.v[4]), "=r"(d.v[5]),
        "=r"(d.v[6]), "=r"(d.v[7]), "=r"(borrow)
      : "r"(x.v[0]), "r"(x.v[1]), "r"(x.v[2]), "r"(x.v[3]), "r"(x.v[4]), "r"(x.v[5]),
        "r"(x.v[6]), "r"(x.v[7]), "n"(PK_P0), "n"(PK_P1), "n"(PK_P2), "n"(PK_P3), "n"(PK_P4),
        "n"(PK_P5), "n"(PK_P6), "n"(PK_P7));
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = borrow ? x.v[i] : d.v[i];
  return r;
}

// (a + b) mod p for a, b < p.
__device__ __forceinline__ Fr fr_add(const Fr& a, const Fr& b) {
  Fr s;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]),
        "=r"(s.v[6]), "=r"(s.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
        "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
        "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  return fr_reduce_once(s);
}

// (a - b) mod p for a, b < p.
__device__ __forceinline__ Fr fr_sub(const Fr& a, const Fr& b) {
  Fr d;
  uint32_t borrow;
  asm("sub.cc.u32  %0, %9,  %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(d.v[0]), "=r"(d.v[1]), "=r"(d.v[2]), "=r"(d.v[3]), "=r"(d.v[4]), "=r"(d.v[5]),
        "=r"(d.v[6]), "=r"(d.v[7]), "=r"(borrow)
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
        "r"(a.v[6]), "r"(a.v[7]), "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]),
        "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  // add p & borrow-mask
  Fr r;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
        "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(d.v[0]), "r"(d.v[1]), "r"(d.v[2]), "r"(d.v[3]), "r"(d.v[4]), "r"(d.v[5]),
        "r"(d.v[6]), "r"(d.v[7]), "r"(PK_P0 & borrow), "r"(PK_P1 & borrow), "r"(PK_P2 & borrow),
        "r"(PK_P3 & borrow), "r"(PK_P4 & borrow), "r"(PK_P5 & borrow), "r"(PK_P6 & borrow),
        "r"(PK_P7 & borrow));
  return r;
}

// Products are rows of 32x32 -> 64-bit multiply-adds.  A row's partial
// products y_j * b start at consecutive words, so they overlap; the even-index
// ones (words 0-1, 2-3, ..) and the odd-index ones (words 1-2, 3-4, ..) each
// tile their own 8-word accumulator without overlap.  Keeping two
// accumulators -- E at words 0..7, O at words 1..8 of the current row -- makes
// every row one carry chain per accumulator of lo/hi pairs, which compile to
// one 64-bit multiply-add each instead of a low and a high one (B200 issues
// 28 of either kind of 64-bit-wide multiply per SM and cycle, so the pairing
// halves the work).  After a Montgomery row E[0] is 0: the frame moves up one
// word, O becomes the even accumulator, E[2..7] the odd one, and E[1] is
// carried into the next row's first sum.

// O[0..7] = (O[0..5] + y * b), with e0 += c first and its carry entering the chain.
__device__ __forceinline__ void fr_odd_row(uint32_t& e0, uint32_t c, uint32_t* O, uint32_t y1,
                                           uint32_t y3, uint32_t y5, uint32_t y7, uint32_t b) {
  asm("add.cc.u32     %0, %0,  %9;\n\t"
      "madc.lo.cc.u32 %1, %10, %14, %1;\n\t"
      "madc.hi.cc.u32 %2, %10, %14, %2;\n\t"
      "madc.lo.cc.u32 %3, %11, %14, %3;\n\t"
      "madc.hi.cc.u32 %4, %11, %14, %4;\n\t"
      "madc.lo.cc.u32 %5, %12, %14, %5;\n\t"
      "madc.hi.cc.u32 %6, %12, %14, %6;\n\t"
      "madc.lo.cc.u32 %7, %13, %14, 0;\n\t"
      "madc.hi.u32    %8, %13, %14, 0;"
      : "+r"(e0), "+r"(O[0]), "+r"(O[1]), "+r"(O[2]), "+r"(O[3]), "+r"(O[4]), "+r"(O[5]),
        "=r"(O[6]), "=r"(O[7])
      : "r"(c), "r"(y1), "r"(y3), "r"(y5), "r"(y7), "r"(b));
}

// E[0..7] += y * b, the carry into o7 (word 8).
__device__ __forceinline__ void fr_even_row(uint32_t* E, uint32_t& o7, uint32_t y0, uint32_t y2,
                                            uint32_t y4, uint32_t y6, uint32_t b) {
  asm("mad.lo.cc.u32  %0, %9,  %13, %0;\n\t"
      "madc.hi.cc.u32 %1, %9,  %13, %1;\n\t"
      "madc.lo.cc.u32 %2, %10, %13, %2;\n\t"
      "madc.hi.cc.u32 %3, %10, %13, %3;\n\t"
      "madc.lo.cc.u32 %4, %11, %13, %4;\n\t"
      "madc.hi.cc.u32 %5, %11, %13, %5;\n\t"
      "madc.lo.cc.u32 %6, %12, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %12, %13, %7;\n\t"
      "addc.u32       %8, %8, 0;"
      : "+r"(E[0]), "+r"(E[1]), "+r"(E[2]), "+r"(E[3]), "+r"(E[4]), "+r"(E[5]), "+r"(E[6]),
        "+r"(E[7]), "+r"(o7)
      : "r"(y0), "r"(y2), "r"(y4), "r"(y6), "r"(b));
}

// O[0..7] += y * b (the sum fits: the row's total is below 2^288).
__device__ __forceinline__ void fr_odd_acc(uint32_t* O, uint32_t y1, uint32_t y3, uint32_t y5,
                                           uint32_t y7, uint32_t b) {
  asm("mad.lo.cc.u32  %0, %8,  %12, %0;\n\t"
      "madc.hi.cc.u32 %1, %8,  %12, %1;\n\t"
      "madc.lo.cc.u32 %2, %9,  %12, %2;\n\t"
      "madc.hi.cc.u32 %3, %9,  %12, %3;\n\t"
      "madc.lo.cc.u32 %4, %10, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %10, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %11, %12, %6;\n\t"
      "madc.hi.u32    %7, %11, %12, %7;"
      : "+r"(O[0]), "+r"(O[1]), "+r"(O[2]), "+r"(O[3]), "+r"(O[4]), "+r"(O[5]), "+r"(O[6]),
        "+r"(O[7])
      : "r"(y1), "r"(y3), "r"(y5), "r"(y7), "r"(b));
}

// E, O = y * b (first row, nothing to accumulate).
__device__ __forceinline__ void fr_first_row(uint32_t* E, uint32_t* O, const uint32_t* y,
                                             uint32_t b) {
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint64_t e = (uint64_t)y[2 * i] * b, o = (uint64_t)y[2 * i + 1] * b;
    E[2 * i] = (uint32_t)e;
    E[2 * i + 1] = (uint32_t)(e >> 32);
    O[2 * i] = (uint32_t)o;
    O[2 * i + 1] = (uint32_t)(o >> 32);
  }
}

// The frame one word up; returns the word carried into the next row (E[1]).
__device__ __forceinline__ uint32_t fr_next_frame(uint32_t* E, uint32_t* O) {
  const uint32_t c = E[1];
  uint32_t t[6];
#pragma unroll
  for (int i = 0; i < 6; i++) t[i] = E[i + 2];
#pragma unroll
  for (int i = 0; i < 8; i++) E[i] = O[i];
#pragma unroll
  for (int i = 0; i < 6; i++) O[i] = t[i];
  return c;
}

// E at words 0..7 plus c at word 0 plus O[0..5] at words 1..6.
__device__ __forceinline__ Fr fr_join(const uint32_t* E, const uint32_t* O, uint32_t c) {
  Fr r;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, 0;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]),
        "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(E[0]), "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]),
        "r"(c), "r"(O[0]), "r"(O[1]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]));
  return r;
}

// a + b as 256-bit integers (the sum fits).
__device__ __forceinline__ Fr fr_add_raw(const Fr& a, const uint32_t* b) {
  Fr s;
  asm("add.cc.u32  %0, %8,  %16;\n\t"
      "addc.cc.u32 %1, %9,  %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(s.v[0]), "=r"(s.v[1]), "=r"(s.v[2]), "=r"(s.v[3]), "=r"(s.v[4]), "=r"(s.v[5]),
        "=r"(s.v[6]), "=r"(s.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]),
        "r"(a.v[6]), "r"(a.v[7]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]),
        "r"(b[5]), "r"(b[6]), "r"(b[7]));
  return s;
}

// One Montgomery row on the frame: adds m p with m = -E[0] / p mod 2^32.
__device__ __forceinline__ void fr_redc_row(uint32_t* E, uint32_t* O) {
  const uint32_t m = E[0] * PK_MU;
  fr_odd_acc(O, PK_P1, PK_P3, PK_P5, PK_P7, m);
  fr_even_row(E, O[7], PK_P0, PK_P2, PK_P4, PK_P6, m);
}

// Montgomery product a * b * 2^-256 mod p for a, b < 2p: CIOS rows (Koc,
// Acar, Kaliski 1996) over the two accumulators, 128 64-bit multiply-adds and
// 8 low ones.  (a b + M p) / 2^256 < 4 p^2 / 2^256 + p < 1.8 p, so one
// conditional subtraction reduces fully.  Measured on B200: 65.8 G products/s
// (528 multiply cycles per warp of 565), against 44.8 G/s of the binary64
// form (352 instructions) and 42.0 G/s of rows with separate low and high
// chains.
__device__ __forceinline__ Fr fr_mul(const Fr& a, const Fr& b) {
  uint32_t E[8], O[8], c = 0;
  fr_first_row(E, O, a.v, b.v[0]);
  fr_redc_row(E, O);
#pragma unroll
  for (int i = 1; i < 8; i++) {
    c = fr_next_frame(E, O);
    fr_odd_row(E[0], c, O, a.v[1], a.v[3], a.v[5], a.v[7], b.v[i]);
    fr_even_row(E, O[7], a.v[0], a.v[2], a.v[4], a.v[6], b.v[i]);
    fr_redc_row(E, O);
  }
  c = fr_next_frame(E, O);
  return fr_reduce_once(fr_join(E, O, c));
}

// (t + M p) / 2^256 for a 256-bit t: the Montgomery reduction alone, result
// <= p (64 64-bit multiply-adds).
__device__ __forceinline__ Fr fr_redc(const uint32_t* t) {
  uint32_t E[8], O[8], c = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) E[i] = t[i];
  {
    const uint32_t P[8] = {PK_P0, PK_P1, PK_P2, PK_P3, PK_P4, PK_P5, PK_P6, PK_P7};
    const uint32_t m = E[0] * PK_MU;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const uint64_t o = (uint64_t)P[2 * i + 1] * m;
      O[2 * i] = (uint32_t)o;
      O[2 * i + 1] = (uint32_t)(o >> 32);
    }
    fr_even_row(E, O[7], PK_P0, PK_P2, PK_P4, PK_P6, m);
  }
#pragma unroll
  for (int i = 1; i < 8; i++) {
    c = fr_next_frame(E, O);
    const uint32_t m = (E[0] + c) * PK_MU;
    fr_odd_row(E[0], c, O, PK_P1, PK_P3, PK_P5, PK_P7, m);
    fr_even_row(E, O[7], PK_P0, PK_P2, PK_P4, PK_P6, m);
  }
  c = fr_next_frame(E, O);
  return fr_join(E, O, c);
}

// Carry chains over n consecutive products a * y_j into X[0..2n).
__device__ __forceinline__ void fr_chain1(uint32_t* X, uint32_t a, uint32_t y0) {
  asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
      "madc.hi.u32   %1, %2, %3, %1;"
      : "+r"(X[0]), "+r"(X[1])
      : "r"(a), "r"(y0));
}
__device__ __forceinline__ void fr_chain1c(uint32_t* X, uint32_t a, uint32_t y0) {
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32       %2, 0, 0;"
      : "+r"(X[0]), "+r"(X[1]), "=r"(X[2])
      : "r"(a), "r"(y0));
}
__device__ __forceinline__ void fr_chain2(uint32_t* X, uint32_t a, uint32_t y0, uint32_t y1) {
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
      "madc.hi.u32    %3, %4, %6, %3;"
      : "+r"(X[0]), "+r"(X[1]), "+r"(X[2]), "+r"(X[3])
      : "r"(a), "r"(y0), "r"(y1));
}
__device__ __forceinline__ void fr_chain2c(uint32_t* X, uint32_t a, uint32_t y0, uint32_t y1) {
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;"
      : "+r"(X[0]), "+r"(X[1]), "+r"(X[2]), "+r"(X[3]), "=r"(X[4])
      : "r"(a), "r"(y0), "r"(y1));
}
__device__ __forceinline__ void fr_chain3(uint32_t* X, uint32_t a, uint32_t y0, uint32_t y1,
                                          uint32_t y2) {
  asm("mad.lo.cc.u32  %0, %6, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %6, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
      "madc.lo.cc.u32 %4, %6, %9, %4;\n\t"
      "madc.hi.u32    %5, %6, %9, %5;"
      : "+r"(X[0]), "+r"(X[1]), "+r"(X[2]), "+r"(X[3]), "+r"(X[4]), "+r"(X[5])
      : "r"(a), "r"(y0), "r"(y1), "r"(y2));
}
__device__ __forceinline__ void fr_chain3c(uint32_t* X, uint32_t a, uint32_t y0, uint32_t y1,
                                           uint32_t y2) {
  asm("mad.lo.cc.u32  %0, %7, %8, %0;\n\t"
      "madc.hi.cc.u32 %1, %7, %8, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
      "madc.lo.cc.u32 %4, %7, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %7, %10, %5;\n\t"
      "addc.u32       %6, 0, 0;"
      : "+r"(X[0]), "+r"(X[1]), "+r"(X[2]), "+r"(X[3]), "+r"(X[4]), "+r"(X[5]), "=r"(X[6])
      : "r"(a), "r"(y0), "r"(y1), "r"(y2));
}

__device__ __forceinline__ void fr_chain4(uint32_t* X, uint32_t a, uint32_t y0, uint32_t y1,
                                          uint32_t y2, uint32_t y3) {
  asm("mad.lo.cc.u32  %0, %8, %9,  %0;\n\t"
      "madc.hi.cc.u32 %1, %8, %9,  %1;\n\t"
      "madc.lo.cc.u32 %2, %8, %10, %2;\n\t"
      "madc.hi.cc.u32 %3, %8, %10, %3;\n\t"
      "madc.lo.cc.u32 %4, %8, %11, %4;\n\t"
      "madc.hi.cc.u32 %5, %8, %11, %5;\n\t"
      "madc.lo.cc.u32 %6, %8, %12, %6;\n\t"
      "madc.hi.u32    %7, %8, %12, %7;"
      : "+r"(X[0]), "+r"(X[1]), "+r"(X[2]), "+r"(X[3]), "+r"(X[4]), "+r"(X[5]), "+r"(X[6]),
        "+r"(X[7])
      : "r"(a), "r"(y0), "r"(y1), "r"(y2), "r"(y3));
}

// t[0..15] = a^2 for any 256-bit a: the 28 cross products a_i a_j (i < j)
// once, those with i + j even in one accumulator and odd in the other (as in
// a product row, each tiles its words), doubled, plus the 8 squares.
__device__ __forceinline__ void fr_sqr_wide(const uint32_t* a, uint32_t* t) {
  uint32_t o[15], e[14];
#pragma unroll
  for (int j = 1; j < 8; j++) {  // row 0
    const uint64_t w = (uint64_t)a[0] * a[j];
    uint32_t* x = (j & 1) ? o : e;
    x[j] = (uint32_t)w;
    x[j + 1] = (uint32_t)(w >> 32);
  }
  fr_chain3c(o + 3, a[1], a[2], a[4], a[6]);
  e[8] = 0;
  e[9] = 0;
  fr_chain3(e + 4, a[1], a[3], a[5], a[7]);
  o[10] = 0;
  fr_chain3(o + 5, a[2], a[3], a[5], a[7]);
  fr_chain2c(e + 6, a[2], a[4], a[6]);
  fr_chain2c(o + 7, a[3], a[4], a[6]);
  e[11] = 0;
  fr_chain2(e + 8, a[3], a[5], a[7]);
  o[12] = 0;
  fr_chain2(o + 9, a[4], a[5], a[7]);
  fr_chain1c(e + 10, a[4], a[6]);
  fr_chain1c(o + 11, a[5], a[6]);
  e[13] = 0;
  fr_chain1(e + 12, a[5], a[7]);
  o[14] = 0;
  fr_chain1(o + 13, a[6], a[7]);
  uint32_t s[15];  // e + o at words 1..14
  s[1] = o[1];
  asm("add.cc.u32  %0,  %13, %26;\n\t"
      "addc.cc.u32 %1,  %14, %27;\n\t"
      "addc.cc.u32 %2,  %15, %28;\n\t"
      "addc.cc.u32 %3,  %16, %29;\n\t"
      "addc.cc.u32 %4,  %17, %30;\n\t"
      "addc.cc.u32 %5,  %18, %31;\n\t"
      "addc.cc.u32 %6,  %19, %32;\n\t"
      "addc.cc.u32 %7,  %20, %33;\n\t"
      "addc.cc.u32 %8,  %21, %34;\n\t"
      "addc.cc.u32 %9,  %22, %35;\n\t"
      "addc.cc.u32 %10, %23, %36;\n\t"
      "addc.cc.u32 %11, %24, %37;\n\t"
      "addc.u32    %12, %25, 0;"
      : "=r"(s[2]), "=r"(s[3]), "=r"(s[4]), "=r"(s[5]), "=r"(s[6]), "=r"(s[7]), "=r"(s[8]),
        "=r"(s[9]), "=r"(s[10]), "=r"(s[11]), "=r"(s[12]), "=r"(s[13]), "=r"(s[14])
      : "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(o[8]), "r"(o[9]),
        "r"(o[10]), "r"(o[11]), "r"(o[12]), "r"(o[13]), "r"(o[14]), "r"(e[2]), "r"(e[3]),
        "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(e[8]), "r"(e[9]), "r"(e[10]),
        "r"(e[11]), "r"(e[12]), "r"(e[13]));
  t[0] = 0;
  t[1] = s[1] << 1;
#pragma unroll
  for (int i = 2; i < 15; i++) t[i] = __funnelshift_l(s[i - 1], s[i], 1);
  t[15] = s[14] >> 31;
  asm("mad.lo.cc.u32  %0,  %16, %16, %0;\n\t"
      "madc.hi.cc.u32 %1,  %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2,  %17, %17, %2;\n\t"
      "madc.hi.cc.u32 %3,  %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4,  %18, %18, %4;\n\t"
      "madc.hi.cc.u32 %5,  %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6,  %19, %19, %6;\n\t"
      "madc.hi.cc.u32 %7,  %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8,  %20, %20, %8;\n\t"
      "madc.hi.cc.u32 %9,  %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
      "madc.hi.u32    %15, %23, %23, %15;"
      : "+r"(t[0]), "+r"(t[1]), "+r"(t[2]), "+r"(t[3]), "+r"(t[4]), "+r"(t[5]), "+r"(t[6]),
        "+r"(t[7]), "+r"(t[8]), "+r"(t[9]), "+r"(t[10]), "+r"(t[11]), "+r"(t[12]), "+r"(t[13]),
        "+r"(t[14]), "+r"(t[15])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}

// Montgomery square a^2 * 2^-256 mod p for a < 2p: 36 + 64 64-bit
// multiply-adds.  The high half plus the reduced low half is below
// 4 p^2 / 2^256 + p < 1.8 p.  Measured on B200: 78 G squares/s against 55 G/s
// of the binary64 form (296 instructions) and 66 G/s of fr_mul(a, a).
__device__ __forceinline__ Fr fr_sqr(const Fr& a) {
  uint32_t t[16];
  fr_sqr_wide(a.v, t);
  return fr_reduce_once(fr_add_raw(fr_redc(t), t + 8));
}

// canonical -> Montgomery: a * R^2 * R^-1
__device__ __forceinline__ Fr fr_to_mont(const Fr& a) {
  Fr r2;
  r2.v[0] = 0xae216da7u; r2.v[1] = 0x1bb8e645u; r2.v[2] = 0xe35c59e3u; r2.v[3] = 0x53fe3ab1u;
  r2.v[4] = 0x53bb8085u; r2.v[5] = 0x8c49833du; r2.v[6] = 0x7f4e44a5u; r2.v[7] = 0x0216d0b1u;
  return fr_mul(a, r2);
}

// Montgomery -> canonical, a * 2^-256 mod p, for any 256-bit a: the reduction
// alone.  Measured on B200: 121 G/s against 84 G/s with separate low and high
// chains.
__device__ __forceinline__ Fr fr_from_mont(const Fr& a) { return fr_reduce_once(fr_redc(a.v)); }

__device__ __forceinline__ bool fr_eq(const Fr& a, const Fr& b) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) d |= a.v[i] ^ b.v[i];
  return d == 0;
}

}  // namespace pk
