// sky_tc.cuh -- Skyscraper compressions of 128 threads at a time, with the
// Montgomery reduction of every square on the tensor cores.
//
// A square round is l' = l^2 2^-256 + r + rc mod p.  On the integer pipe the
// square takes 36 64-bit multiply-adds and its reduction another 64.  The
// reduction is linear in the bytes of the square T,
//     T 2^-256 = sum_k T_k (2^(8k-256) mod p),
// with the same constants for every element, so it is a matrix product: row =
// element (M = 128, one per thread), K = bytes of T, column n = byte n of the
// constants (N = 32).  tcgen05.mma kind::i8 (u8 x u8 -> s32) does it exactly:
// a column is below 2^22.  What is left on the integer pipe is the square
// itself, assembling 32 columns into 9 words (34 ALU operations), and one
// quotient step back to 8 words (8 multiply-adds).
//
// The product is linear, so the square's two accumulators (even and odd word
// offsets, see fr.cuh) are never added: both go in as they are, the odd one
// against constants for its own offset, and the round constant rides along as
// one more K entry whose A byte is 1.  A and D live in tensor memory: thread i
// writes its bytes to lane i (tcgen05.st) and reads its 32 columns back
// (tcgen05.ld); shared memory holds only the constants.  64 columns of tensor
// memory per CTA:
//     0..31   D
//     32..47  even accumulator E, words 0..15   (K blocks 0 and 1)
//     48..61  odd accumulator O, words 1..14    (K blocks 2 and 3)
//     62      1 (byte 0)  63  unused: its rows of the constants are zero
//
// Bound by the multiplier: 44 64-bit multiply-adds of four issue cycles per
// square round against 100.  Measured on B200: 2^20 leaves of 16 Fr in 2.41 ms
// (6.5 G compressions/s) against 4.10 ms with sky_compress, the multiplier 67 %
// and the tensor pipe 17 % busy; 6 and 7 CTAs per SM take 2.82 and 2.67 ms.  A
// lone CTA takes 6.0 us per compression against 8.0.  Merging E and O first
// and adding T's high half on the ALU (one K block) was 10 % slower.
#pragma once
#include "fr.cuh"
#include "skyscraper.cuh"

namespace pk {
namespace skytc {

constexpr int kThreads = 128;   // one MMA tile: 128 elements
constexpr int kMinCtas = 8;     // CTAs per SM: 64 registers a thread, 8 x 64 columns of 512
constexpr int kBlockBytes = 1024;            // 32 columns x 32 K bytes
constexpr int kSquares = 14;                 // square rounds of a compression
constexpr int kBlocks = 3 + kSquares;

constexpr uint64_t kP64[4] = {0x43e1f593f0000001ULL, 0x2833e84879b97091ULL, 0xb85045b68181585dULL,
                              0x30644e72e131a029ULL};
// 2^-256 mod p
constexpr uint64_t kRinv64[4] = {0xdc5ba0056db1194eULL, 0x090ef5a9e111ec87ULL,
                                 0xc8260de4aeb85d5dULL, 0x15ebf95182c5551cULL};

// index of square round k among the compression's squares
__host__ __device__ constexpr int square_index(int k) {
  return k - (k >= 8 ? 2 : 0) - (k >= 12 ? 2 : 0);
}

// The constants as tcgen05's K-major operand without swizzle: 8 x 16-byte core
// matrices, K halves 512 bytes apart, 8-column groups 128 bytes apart.
struct Image {
  uint32_t w[kBlocks * kBlockBytes / 4];
};

constexpr void image_put(Image& im, int block, int n, int k, uint32_t byte) {
  const int off = block * kBlockBytes + (k / 16) * 512 + (n / 8) * 128 + (n % 8) * 16 + k % 16;
  im.w[off / 4] |= byte << (8 * (off % 4));
}

// block 0: words 0..7 of a square, 1: words 8..15, 2: words 1..8, 3 + s: words
// 9..14 and the round constant of square s.
constexpr Image make_image() {
  Image im{};
  uint64_t v[4] = {kRinv64[0], kRinv64[1], kRinv64[2], kRinv64[3]};
  for (int e = 0; e < 60; e++) {  // v = 2^(8e - 256) mod p, or exactly 2^(8e - 256) from e = 32
    for (int n = 0; n < 32; n++) {
      const uint32_t byte =
          e < 32 ? (uint32_t)((v[n / 8] >> (8 * (n % 8))) & 0xff) : (uint32_t)(n == e - 32);
      if (e < 32) image_put(im, 0, n, e, byte);
      if (e >= 32) image_put(im, 1, n, e - 32, byte);
      if (e >= 4 && e < 36) image_put(im, 2, n, e - 4, byte);
      if (e >= 36)
        for (int s = 0; s < kSquares; s++) image_put(im, 3 + s, n, e - 36, byte);
    }
    for (int b = 0; e < 32 && b < 8; b++) {
      uint64_t top = 0;
      for (int i = 0; i < 4; i++) {
        const uint64_t x = (v[i] << 1) | top;
        top = v[i] >> 63;
        v[i] = x;
      }
      bool ge = true;
      for (int i = 3; i >= 0; i--)
        if (v[i] != kP64[i]) {
          ge = v[i] > kP64[i];
          break;
        }
      uint64_t borrow = 0;
      for (int i = 0; ge && i < 4; i++) {
        const uint64_t d = v[i] - kP64[i];
        const uint64_t out = (uint64_t)(v[i] < kP64[i]) | (uint64_t)(d < borrow);
        v[i] = d - borrow;
        borrow = out;
      }
    }
  }
  // e = 60..63 of block 1: words 15
  for (int e = 60; e < 64; e++) image_put(im, 1, e - 32, e - 32, 1);
  for (int k = 0; k < 18; k++) {
    if (k == 6 || k == 7 || k == 10 || k == 11) continue;
    for (int n = 0; n < 32; n++)
      image_put(im, 3 + square_index(k), n, 24, (kSkyRoundConstants.w[k][n / 4] >> (8 * (n % 4))) & 0xff);
  }
  return im;
}
static __device__ const Image kImage = make_image();

// kind::i8: s32 accumulators, unsigned bytes, K-major, N = 32, M = 128
constexpr uint32_t kInstr = (2u << 4) | ((32u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kColumns = 64;

struct Shared {
  alignas(128) uint4 image[kBlocks * kBlockBytes / 16];
  uint4 park[2 * kThreads];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// X[k..k+2n) += products, a carry chain whose last pair starts from nothing:
// the accumulator words it writes are new.
#define PK_NEW_PAIR(X, k, a, b)                    \
  do {                                             \
    const uint64_t w_ = (uint64_t)(a) * (b);       \
    (X)[k] = (uint32_t)w_;                         \
    (X)[(k) + 1] = (uint32_t)(w_ >> 32);           \
  } while (0)
#define PK_CHAIN3(X, k, a0, b0, a1, b1, a2, b2)                                               \
  asm("mad.lo.cc.u32  %0, %6,  %7,  %0;\n\t"                                                  \
      "madc.hi.cc.u32 %1, %6,  %7,  %1;\n\t"                                                  \
      "madc.lo.cc.u32 %2, %8,  %9,  %2;\n\t"                                                  \
      "madc.hi.cc.u32 %3, %8,  %9,  %3;\n\t"                                                  \
      "madc.lo.cc.u32 %4, %10, %11, 0;\n\t"                                                   \
      "madc.hi.u32    %5, %10, %11, 0;"                                                       \
      : "+r"((X)[k]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]),             \
        "=r"((X)[(k) + 4]), "=r"((X)[(k) + 5])                                                \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2))
#define PK_CHAIN4(X, k, a0, b0, a1, b1, a2, b2, a3, b3)                                       \
  asm("mad.lo.cc.u32  %0, %8,  %9,  %0;\n\t"                                                  \
      "madc.hi.cc.u32 %1, %8,  %9,  %1;\n\t"                                                  \
      "madc.lo.cc.u32 %2, %10, %11, %2;\n\t"                                                  \
      "madc.hi.cc.u32 %3, %10, %11, %3;\n\t"                                                  \
      "madc.lo.cc.u32 %4, %12, %13, %4;\n\t"                                                  \
      "madc.hi.cc.u32 %5, %12, %13, %5;\n\t"                                                  \
      "madc.lo.cc.u32 %6, %14, %15, 0;\n\t"                                                   \
      "madc.hi.u32    %7, %14, %15, 0;"                                                       \
      : "+r"((X)[k]), "+r"((X)[(k) + 1]), "+r"((X)[(k) + 2]), "+r"((X)[(k) + 3]),             \
        "+r"((X)[(k) + 4]), "+r"((X)[(k) + 5]), "=r"((X)[(k) + 6]), "=r"((X)[(k) + 7])        \
      : "r"(a0), "r"(b0), "r"(a1), "r"(b1), "r"(a2), "r"(b2), "r"(a3), "r"(b3))

// a^2 = sum E[i] 2^(32 i) + sum O[i] 2^(32 i) (E: words 0..15, O: words 1..14)
// for a < 2^255.  Cross products take a doubled right operand: the words of
// 2a, with f where the row's first word must not bring in the bit below it.
// Every chain ends on a pair that no earlier one wrote, so no carry is left.
__device__ __forceinline__ void square_words(const uint32_t* a, uint32_t* E, uint32_t* O) {
  uint32_t f[8], g[8];
#pragma unroll
  for (int j = 1; j < 8; j++) {
    f[j] = a[j] << 1;
    g[j] = __funnelshift_l(a[j - 1], a[j], 1);
  }
  PK_NEW_PAIR(O, 1, a[0], f[1]);
  PK_NEW_PAIR(O, 3, a[0], g[3]);
  PK_NEW_PAIR(O, 5, a[0], g[5]);
  PK_NEW_PAIR(O, 7, a[0], g[7]);
  PK_CHAIN4(O, 3, a[1], f[2], a[1], g[4], a[1], g[6], a[2], g[7]);
  PK_CHAIN4(O, 5, a[2], f[3], a[2], g[5], a[3], g[6], a[4], g[7]);
  PK_CHAIN4(O, 7, a[3], f[4], a[4], f[5], a[5], f[6], a[6], f[7]);
  PK_NEW_PAIR(E, 2, a[0], g[2]);
  PK_NEW_PAIR(E, 4, a[0], g[4]);
  PK_NEW_PAIR(E, 6, a[0], g[6]);
  PK_CHAIN3(E, 4, a[1], g[3], a[1], g[5], a[1], g[7]);
  PK_CHAIN3(E, 6, a[2], g[4], a[2], g[6], a[3], g[7]);
  PK_CHAIN3(E, 8, a[3], g[5], a[4], g[6], a[5], g[7]);
  PK_NEW_PAIR(E, 0, a[0], a[0]);
  asm("mad.lo.cc.u32  %0,  %14, %14, %0;\n\t"
      "madc.hi.cc.u32 %1,  %14, %14, %1;\n\t"
      "madc.lo.cc.u32 %2,  %15, %15, %2;\n\t"
      "madc.hi.cc.u32 %3,  %15, %15, %3;\n\t"
      "madc.lo.cc.u32 %4,  %16, %16, %4;\n\t"
      "madc.hi.cc.u32 %5,  %16, %16, %5;\n\t"
      "madc.lo.cc.u32 %6,  %17, %17, %6;\n\t"
      "madc.hi.cc.u32 %7,  %17, %17, %7;\n\t"
      "madc.lo.cc.u32 %8,  %18, %18, %8;\n\t"
      "madc.hi.cc.u32 %9,  %18, %18, %9;\n\t"
      "madc.lo.cc.u32 %10, %19, %19, %10;\n\t"
      "madc.hi.cc.u32 %11, %19, %19, %11;\n\t"
      "madc.lo.cc.u32 %12, %20, %20, 0;\n\t"
      "madc.hi.u32    %13, %20, %20, 0;"
      : "+r"(E[2]), "+r"(E[3]), "+r"(E[4]), "+r"(E[5]), "+r"(E[6]), "+r"(E[7]), "+r"(E[8]),
        "+r"(E[9]), "+r"(E[10]), "+r"(E[11]), "+r"(E[12]), "+r"(E[13]), "=r"(E[14]), "=r"(E[15])
      : "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]));
}

// t = E + O (words 0..15; the sum fits)
__device__ __forceinline__ void merge_words(const uint32_t* E, const uint32_t* O, uint32_t* t) {
  t[0] = E[0];
  asm("add.cc.u32  %0,  %15, %30;\n\t"
      "addc.cc.u32 %1,  %16, %31;\n\t"
      "addc.cc.u32 %2,  %17, %32;\n\t"
      "addc.cc.u32 %3,  %18, %33;\n\t"
      "addc.cc.u32 %4,  %19, %34;\n\t"
      "addc.cc.u32 %5,  %20, %35;\n\t"
      "addc.cc.u32 %6,  %21, %36;\n\t"
      "addc.cc.u32 %7,  %22, %37;\n\t"
      "addc.cc.u32 %8,  %23, %38;\n\t"
      "addc.cc.u32 %9,  %24, %39;\n\t"
      "addc.cc.u32 %10, %25, %40;\n\t"
      "addc.cc.u32 %11, %26, %41;\n\t"
      "addc.cc.u32 %12, %27, %42;\n\t"
      "addc.cc.u32 %13, %28, %43;\n\t"
      "addc.u32    %14, %29, 0;"
      : "=r"(t[1]), "=r"(t[2]), "=r"(t[3]), "=r"(t[4]), "=r"(t[5]), "=r"(t[6]), "=r"(t[7]),
        "=r"(t[8]), "=r"(t[9]), "=r"(t[10]), "=r"(t[11]), "=r"(t[12]), "=r"(t[13]), "=r"(t[14]),
        "=r"(t[15])
      : "r"(E[1]), "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(E[8]),
        "r"(E[9]), "r"(E[10]), "r"(E[11]), "r"(E[12]), "r"(E[13]), "r"(E[14]), "r"(E[15]),
        "r"(O[1]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]), "r"(O[6]), "r"(O[7]), "r"(O[8]),
        "r"(O[9]), "r"(O[10]), "r"(O[11]), "r"(O[12]), "r"(O[13]), "r"(O[14]));
}

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

// S = sum c[n] 2^(8n) for columns below 2^23: c[4j] + c[4j+1] 2^8 is below
// 2^32 and is word j as it is; the other two columns make the same, 16 bits up.
__device__ __forceinline__ void assemble(const uint32_t* c, uint32_t* S) {
  uint32_t x[8], y[8], z[9];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    x[j] = c[4 * j] + (c[4 * j + 1] << 8);
    y[j] = c[4 * j + 2] + (c[4 * j + 3] << 8);
  }
  z[0] = y[0] << 16;
#pragma unroll
  for (int j = 1; j < 8; j++) z[j] = __funnelshift_l(y[j - 1], y[j], 16);
  z[8] = y[7] >> 16;
  asm("add.cc.u32  %0, %9,  %17;\n\t"
      "addc.cc.u32 %1, %10, %18;\n\t"
      "addc.cc.u32 %2, %11, %19;\n\t"
      "addc.cc.u32 %3, %12, %20;\n\t"
      "addc.cc.u32 %4, %13, %21;\n\t"
      "addc.cc.u32 %5, %14, %22;\n\t"
      "addc.cc.u32 %6, %15, %23;\n\t"
      "addc.cc.u32 %7, %16, %24;\n\t"
      "addc.u32    %8, %25, 0;"
      : "=r"(S[0]), "=r"(S[1]), "=r"(S[2]), "=r"(S[3]), "=r"(S[4]), "=r"(S[5]), "=r"(S[6]),
        "=r"(S[7]), "=r"(S[8])
      : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]),
        "r"(z[0]), "r"(z[1]), "r"(z[2]), "r"(z[3]), "r"(z[4]), "r"(z[5]), "r"(z[6]), "r"(z[7]),
        "r"(z[8]));
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

// Any 256-bit value to [0, 1.1 p).
__device__ __forceinline__ Fr reduce_any(const Fr& x) {
  uint32_t S[9];
#pragma unroll
  for (int i = 0; i < 8; i++) S[i] = x.v[i];
  S[8] = 0;
  return quotient_step(S);
}

// The bar's sbox on the 4 bytes of a word, v ^ (~rot1(v) & rot2(v) & rot3(v))
// rotated by 1, with rot2(v) & rot3(v) = rot2(v & rot1(v)).
template <int kBy, uint32_t kMask>
__device__ __forceinline__ uint32_t rot_bytes(uint32_t v) {
  return ((v << kBy) & kMask) | ((v >> (8 - kBy)) & ~kMask);
}
__device__ __forceinline__ uint32_t sbox4(uint32_t v) {
  const uint32_t a = rot_bytes<1, 0xfefefefeu>(v);
  const uint32_t b = rot_bytes<2, 0xfcfcfcfcu>(v & a);
  return rot_bytes<1, 0xfefefefeu>(v ^ (~a & b));
}

// bar(l) + r + rc of round k, in [0, 1.1 p), for r < 1.1 p (r + rc does not
// wait for l).
__device__ __forceinline__ Fr bar_round(const Fr& l, const Fr& r, int k) {
  const Fr x = fr_reduce_once(l), t = fr_add_raw(r, kSkyRC.w[k]);
  uint32_t S[9];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    S[i] = sbox4(x.v[i + 4]);
    S[i + 4] = sbox4(x.v[i]);
  }
  S[8] = 0;
  add9(S, t.v);
  return quotient_step(S);
}

// A square round without the tensor cores (mont_r: r still to be divided by
// 2^256), taken when the wait below runs out.
static __device__ __noinline__ Fr square_round_alone(const Fr l, const Fr r, int k, bool mont_r) {
  const Fr f = fr_sqr(l), c = mont_r ? fr_redc(r.v) : r;
  uint32_t S[9];
#pragma unroll
  for (int i = 0; i < 8; i++) S[i] = f.v[i];
  S[8] = 0;
  add9(S, c.v);
  add9(S, kSkyRC.w[k]);
  return quotient_step(S);
}

__device__ __forceinline__ void tmem_st2(uint32_t t, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(t), "r"(v[0]),
               "r"(v[1])
               : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t t, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(t), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t t, const uint32_t* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(
                   t),
               "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
               "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
      "%11, %12, %13, %14, %15, %16};" ::"r"(t),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
      "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t t, uint32_t* c) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, "
      "%30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]),
        "=r"(c[7]), "=r"(c[8]), "=r"(c[9]), "=r"(c[10]), "=r"(c[11]), "=r"(c[12]), "=r"(c[13]),
        "=r"(c[14]), "=r"(c[15]), "=r"(c[16]), "=r"(c[17]), "=r"(c[18]), "=r"(c[19]), "=r"(c[20]),
        "=r"(c[21]), "=r"(c[22]), "=r"(c[23]), "=r"(c[24]), "=r"(c[25]), "=r"(c[26]), "=r"(c[27]),
        "=r"(c[28]), "=r"(c[29]), "=r"(c[30]), "=r"(c[31])
      : "r"(t)
      : "memory");
}
__device__ __forceinline__ void tmem_written() {
  asm volatile("tcgen05.wait::st.sync.aligned;\n\t"
               "tcgen05.fence::before_thread_sync;" ::
                   : "memory");
}
__device__ __forceinline__ void tmem_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D (+)= A (tensor memory) x constants
__device__ __forceinline__ void mma(uint32_t d, uint32_t a, uint32_t image, int block,
                                    bool accumulate) {
  const uint32_t addr = image + (uint32_t)block * kBlockBytes;
  const uint64_t desc = (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)(512 >> 4) << 16) |
                        ((uint64_t)(128 >> 4) << 32) | (1ULL << 46);
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t"
      "}" ::"r"(d),
      "r"(a), "l"(desc), "r"(kInstr), "r"((uint32_t)accumulate)
      : "memory");
}

// The CTA's barrier; warps may arrive from different places in the code.
__device__ __forceinline__ void cta_sync() { asm volatile("barrier.sync.aligned 0;" ::: "memory"); }

// One lane of a converged warp.  The MMA's operands must be warp-uniform
// values behind this predicate, not behind threadIdx.x == 0: then they come
// from uniform registers, and four MMAs with their completion take 162 cycles
// instead of 368.
__device__ __forceinline__ bool elect_lane() {
  uint32_t e;
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t"
      "}"
      : "=r"(e));
  return e != 0;
}

// The CTA's tensor memory, constants and barrier.  All kThreads threads call
// every member, together.
struct Tile {
  uint32_t cols;   // the CTA's columns of tensor memory
  uint32_t tmem;   // this warp's lanes of them
  uint32_t warp;
  uint32_t image;  // shared address of the constants
  uint32_t mbar;   // shared address of the MMA completion barrier
  uint32_t phase;
  bool alone;      // a wait ran out: this thread squares without the tensor cores
  uint4* park;

  __device__ __forceinline__ void open(Shared& sh) {
    image = smem_addr(sh.image);
    mbar = smem_addr(&sh.mbar);
    park = sh.park + threadIdx.x;
    phase = 0;
    alone = false;
    const uint4* src = reinterpret_cast<const uint4*>(kImage.w);
    for (int i = threadIdx.x; i < kBlocks * kBlockBytes / 16; i += kThreads)
      sh.image[i] = __ldg(src + i);
    if (threadIdx.x == 0)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_addr(&sh.tmem)),
                   "n"(kColumns)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMA reads the constants
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    tmem_after_sync();
    cols = __shfl_sync(0xffffffffu, sh.tmem, 0);
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    tmem = cols + (warp << 21);  // lane 32 * warp in bits 16..31
    const uint32_t one[2] = {1, 0};
    tmem_st2(tmem + 62, one);
    tmem_written();
  }

  __device__ __forceinline__ void close(Shared& sh) {
    if (alone) wait(phase ^ 1);  // the last MMA may still be running
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    tmem_after_sync();
    if (threadIdx.x < 32)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem),
                   "n"(kColumns));
  }

  // The MMA of the phase with this parity has completed; false when the wait
  // ran out.
  __device__ __forceinline__ bool wait(uint32_t parity) const {
    for (int i = 0; i < (1 << 16); i++) {
      uint32_t done;
      asm volatile(
          "{\n\t"
          ".reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t"
          "}"
          : "=r"(done)
          : "r"(mbar), "r"(parity)
          : "memory");
      if (done) return true;
    }
    return false;
  }

  // l^2 2^-256 + r + rc (+ the parked value), in [0, 1.1 p), for l < 2^255 and
  // r < 2^256.  kMontR: r 2^-256 in its place, r as a third K block of the
  // same constants; E and O are merged for it (their columns make room) and
  // the round constant is left out (round 0 has none).
  template <bool kMontR>
  __device__ __forceinline__ Fr square_round(const Fr& l, const Fr& r, int k, bool add_parked) {
    uint32_t E[16], O[16];
    square_words(l.v, E, O);
    const uint32_t A = tmem + 32;
    if (kMontR) {
      uint32_t t[16];
      merge_words(E, O, t);
      tmem_st16(A, t);
      tmem_st8(A + 16, r.v);
    } else {
      tmem_st8(A + 16, O + 1);
      tmem_st4(A + 24, O + 9);
      tmem_st2(A + 28, O + 13);
      tmem_st16(A, E);
    }
    tmem_written();
    cta_sync();
    if (warp == 0 && elect_lane()) {
      tmem_after_sync();
      mma(cols, cols + 32, image, 0, false);
      mma(cols, cols + 40, image, 1, true);
      mma(cols, cols + 48, image, kMontR ? 0 : 2, true);
      if (!kMontR) mma(cols, cols + 56, image, 3 + square_index(k), true);
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
          : "memory");
    }
    if (!alone && !wait(phase)) alone = true;
    phase ^= 1;
    __syncwarp();
    tmem_after_sync();
    uint32_t c[32], S[9];
    tmem_ld32(tmem, c);  // warp-wide: also where a thread squares alone
    if (alone) {
      const Fr n = square_round_alone(l, r, k, kMontR);
#pragma unroll
      for (int i = 0; i < 8; i++) S[i] = n.v[i];
      S[8] = 0;
    } else {
      assemble(c, S);
      if (!kMontR) add9(S, r.v);
    }
    __syncwarp();
    if (add_parked) {
      const uint4 u = park[0], v = park[kThreads];
      const uint32_t t[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
      add9(S, t);
    }
    return quotient_step(S);
  }

  // In place of compress in a warp that has nothing to compress while others of
  // the CTA do.
  __device__ __forceinline__ void sit_out() {
#pragma unroll 1
    for (int i = 0; i < kSquares; i++) cta_sync();  // kSquares completions: phase as it was
  }

  // Skyscraper compress(l, r) in [0, 1.1 p) for l < 1.1 p and r < 2^256
  // (kMontR: of r 2^-256).  Two rounds per turn: the state's halves swap roles
  // instead of registers.
  template <bool kMontR>
  __device__ __forceinline__ Fr compress(Fr l, Fr r) {
    park[0] = make_uint4(l.v[0], l.v[1], l.v[2], l.v[3]);
    park[kThreads] = make_uint4(l.v[4], l.v[5], l.v[6], l.v[7]);
    if (kMontR) {
      r = square_round<true>(l, r, 0, false);
      l = square_round<false>(r, l, 1, false);
    }
#pragma unroll 1
    for (int k = kMontR ? 2 : 0; k < 18; k += 2) {
      if (k == 6 || k == 10) {
        r = bar_round(l, r, k);
        l = bar_round(r, l, k + 1);
      } else {
        r = square_round<false>(l, r, k, false);
        l = square_round<false>(r, l, k + 1, k == 16);
      }
    }
    return l;
  }
};

}  // namespace skytc
}  // namespace pk
