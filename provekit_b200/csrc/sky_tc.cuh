// sky_tc.cuh -- Skyscraper compressions of 128 threads at a time, with the
// Montgomery reduction of every square on the tensor cores (tc_reduce.cuh).
//
// A square round is l' = l^2 2^-256 + r + rc mod p.  On the integer pipe the
// square takes 36 64-bit multiply-adds and its reduction another 64; here 8 of
// the reduction are left.  The round constant rides along as one more K entry
// whose A byte (tensor memory column 62) is 1.
//
// Bound by the multiplier: 44 64-bit multiply-adds of four issue cycles per
// square round against 100.  Measured on B200: 2^20 leaves of 16 Fr in 2.17 ms
// (7.2 G compressions/s) against 4.10 ms with sky_compress.  A lone CTA takes
// 6.1 us per compression against 8.0.  Merging E and O first and adding T's
// high half on the ALU (one K block) was 10 % slower; two K blocks more for T's
// high half and r instead of additions changed nothing.
#pragma once
#include "fr.cuh"
#include "skyscraper.cuh"
#include "tc_reduce.cuh"

namespace pk {
namespace skytc {

using namespace tc;

constexpr int kMinCtas = kMaxCtas;  // 64 registers a thread
constexpr int kSquares = 14;        // square rounds of a compression
constexpr int kBlocks = 3 + kSquares;

// index of square round k among the compression's squares
__host__ __device__ constexpr int square_index(int k) {
  return k - (k >= 8 ? 2 : 0) - (k >= 12 ? 2 : 0);
}

// Blocks 0..2: the accumulators; 3 + s: O's words 9..14 and, against the byte
// of 1, the round constant of square s.
constexpr Image<kBlocks> make_image() {
  Image<kBlocks> im{};
  const Residues r = make_residues();
  image_accumulators(im, r);
  for (int k = 0; k < 18; k++) {
    if (k == 6 || k == 7 || k == 10 || k == 11) continue;
    const int block = 3 + square_index(k);
    image_words(im, r, block, 0, 9, 6);
    for (int n = 0; n < 32; n++)
      image_put(im, block, n, 24, (kSkyRoundConstants.w[k][n / 4] >> (8 * (n % 4))) & 0xff);
  }
  return im;
}
static __device__ const Image<kBlocks> kImage = make_image();

struct Shared {
  alignas(128) uint4 image[kBlocks * kBlockBytes / 16];
  uint4 park[2 * kThreads];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
};

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
  uint32_t y[8];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    y[i] = sbox4(x.v[i + 4]);
    y[i + 4] = sbox4(x.v[i]);
  }
  return quotient_sum(y, t.v, nullptr, 0);
}

// What the tensor cores would hold, without them: l^2 2^-256 + rc of round k,
// (mont_r) plus r 2^-256; below 3 p.
static __device__ __noinline__ Fr square_alone(const Fr l, const Fr r, int k, bool mont_r) {
  Fr f = fr_sqr(l);
  if (mont_r) f = fr_add(f, fr_from_mont(r));
  return fr_add_raw(f, kSkyRC.w[k]);
}

struct SkyTile : Tile {
  uint4* park;

  __device__ __forceinline__ void open(Shared& sh) {
    park = sh.park + threadIdx.x;
    Tile::open(sh, kImage);
    const uint32_t one[2] = {1, 0};
    tmem_st2(tmem + 62, one);
    tmem_written();
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
    start([&] {
      block(0, 0);
      block(1, 1);
      block(2, kMontR ? 0 : 2);
      if (!kMontR) block(3, 3 + square_index(k));
    });
    uint32_t c[32], x[8], z[8], top;
    finish(c);
    if (alone) {
      const Fr n = square_alone(l, r, k, kMontR);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        x[i] = n.v[i];
        z[i] = 0;
      }
      top = 0;
    } else {
      assemble(c, x, z, top);
    }
    __syncwarp();
    if (!add_parked) return quotient_sum(x, z, kMontR ? nullptr : r.v, top);
    uint32_t H[9];
#pragma unroll
    for (int i = 0; i < 8; i++) H[i] = r.v[i];
    H[8] = 0;
    const uint4 u = park[0], v = park[kThreads];
    const uint32_t t[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
    add9(H, t);
    return quotient_sum(x, z, H, top + H[8]);
  }

  // In place of compress or permute in a warp that has nothing to compress while others of
  // the CTA do.
  __device__ __forceinline__ void sit_out() {
#pragma unroll 1
    for (int i = 0; i < kSquares; i++) cta_sync();  // kSquares completions: phase as it was
  }

  // The permutation without the feed-forward (skyscraper/core/src/reference.rs:49-60),
  // l < 2.2 p and r < 1.1 p to both below 1.1 p.
  __device__ __forceinline__ void permute(Fr& l, Fr& r) {
#pragma unroll 1
    for (int k = 0; k < 18; k += 2) {
      if (k == 6 || k == 10) {
        r = bar_round(l, r, k);
        l = bar_round(r, l, k + 1);
      } else {
        r = square_round<false>(l, r, k, false);
        l = square_round<false>(r, l, k + 1, false);
      }
    }
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
