// ntt_tile.cuh -- a transform pass's stages on a tile in shared memory, shared
// by the plain passes (ntt.cu) and the batch's grouped ones (batch.cu).
#pragma once
#include "fr.cuh"
#include "tc_reduce.cuh"

namespace pk {

// A tile of E elements is two planes of 16-byte halves (see ntt.cu).
__device__ __forceinline__ Fr tile_load(const uint4* sm, int E, int i) {
  const uint4 a = sm[i], b = sm[E + i];
  Fr x;
  x.v[0] = a.x; x.v[1] = a.y; x.v[2] = a.z; x.v[3] = a.w;
  x.v[4] = b.x; x.v[5] = b.y; x.v[6] = b.z; x.v[7] = b.w;
  return x;
}
__device__ __forceinline__ void tile_store(uint4* sm, int E, int i, const Fr& x) {
  sm[i] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  sm[E + i] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}
// The product where the tensor cores' wait ran out (w < p, x < 5 p).
static __device__ __noinline__ Fr product_alone(const Fr w, const Fr x) { return fr_mul(w, x); }

// How the T lines of a tile lie (see ntt.cu).
enum : int { kModeA = 0, kModeB = 1, kModeC = 2 };

// `high` of line l in mode C (fewer than 2^32 lines).
__device__ __forceinline__ uint64_t line_high(uint64_t l, uint64_t U) {
  return (uint32_t)l / (uint32_t)U;
}

// Index of tile element e in the data and in shared memory.
__device__ __forceinline__ void pass_index(int mode, int e, int K, int T, int log_t, int log_u,
                                           uint64_t U, uint64_t l0, uint64_t high, uint64_t u0,
                                           uint64_t* g, int* sidx) {
  if (mode == kModeA) {
    const int j = e >> log_t, ll = e & (T - 1);
    *g = ((high << K) + j) * U + u0 + ll;
    *sidx = e;
  } else if (mode == kModeC) {
    const int j = e >> log_t;
    const uint64_t l = l0 + (e & (T - 1)), h = line_high(l, U);
    *g = ((h << K) + j) * U + (l - h * U);
    *sidx = e;
  } else {
    const int j = (e >> log_u) & ((1 << K) - 1);
    const int hl = e >> (log_u + K);
    const int u = e & ((1 << log_u) - 1);
    *g = (((l0 >> log_u) << K) << log_u) + e;
    *sidx = j * T + (hl << log_u) + u;
  }
}

// x0, m -> x0 + m, x0 - m mod p, loosely: for x0 < 5 p and m < 1.1 p both
// results are below 5 p (and 2^256).  2 p is taken from the sum when x0 is
// above it, and added to the difference when it is not (x0 is compared by its
// top word, so the border is up to 2^224 above 2 p).
__device__ __forceinline__ void loose_butterfly(const Fr& x0, const Fr& m, Fr& y0, Fr& y1) {
  asm("{\n\t"
      ".reg .pred b;\n\t"
      "setp.ge.u32 b, %23, 0x60c89ce6;\n\t"
      "add.cc.u32  %0, %16, %24;\n\t"
      "addc.cc.u32 %1, %17, %25;\n\t"
      "addc.cc.u32 %2, %18, %26;\n\t"
      "addc.cc.u32 %3, %19, %27;\n\t"
      "addc.cc.u32 %4, %20, %28;\n\t"
      "addc.cc.u32 %5, %21, %29;\n\t"
      "addc.cc.u32 %6, %22, %30;\n\t"
      "addc.u32    %7, %23, %31;\n\t"
      "sub.cc.u32  %8,  %16, %24;\n\t"
      "subc.cc.u32 %9,  %17, %25;\n\t"
      "subc.cc.u32 %10, %18, %26;\n\t"
      "subc.cc.u32 %11, %19, %27;\n\t"
      "subc.cc.u32 %12, %20, %28;\n\t"
      "subc.cc.u32 %13, %21, %29;\n\t"
      "subc.cc.u32 %14, %22, %30;\n\t"
      "subc.u32    %15, %23, %31;\n\t"
      "@b sub.cc.u32  %0, %0, 0xe0000002;\n\t"
      "@b subc.cc.u32 %1, %1, 0x87c3eb27;\n\t"
      "@b subc.cc.u32 %2, %2, 0xf372e122;\n\t"
      "@b subc.cc.u32 %3, %3, 0x5067d090;\n\t"
      "@b subc.cc.u32 %4, %4, 0x0302b0ba;\n\t"
      "@b subc.cc.u32 %5, %5, 0x70a08b6d;\n\t"
      "@b subc.cc.u32 %6, %6, 0xc2634053;\n\t"
      "@b subc.u32    %7, %7, 0x60c89ce5;\n\t"
      "@!b add.cc.u32  %8,  %8,  0xe0000002;\n\t"
      "@!b addc.cc.u32 %9,  %9,  0x87c3eb27;\n\t"
      "@!b addc.cc.u32 %10, %10, 0xf372e122;\n\t"
      "@!b addc.cc.u32 %11, %11, 0x5067d090;\n\t"
      "@!b addc.cc.u32 %12, %12, 0x0302b0ba;\n\t"
      "@!b addc.cc.u32 %13, %13, 0x70a08b6d;\n\t"
      "@!b addc.cc.u32 %14, %14, 0xc2634053;\n\t"
      "@!b addc.u32    %15, %15, 0x60c89ce5;\n\t"
      "}"
      : "=&r"(y0.v[0]), "=&r"(y0.v[1]), "=&r"(y0.v[2]), "=&r"(y0.v[3]), "=&r"(y0.v[4]),
        "=&r"(y0.v[5]), "=&r"(y0.v[6]), "=&r"(y0.v[7]), "=&r"(y1.v[0]), "=&r"(y1.v[1]),
        "=&r"(y1.v[2]), "=&r"(y1.v[3]), "=&r"(y1.v[4]), "=&r"(y1.v[5]), "=&r"(y1.v[6]),
        "=&r"(y1.v[7])
      : "r"(x0.v[0]), "r"(x0.v[1]), "r"(x0.v[2]), "r"(x0.v[3]), "r"(x0.v[4]), "r"(x0.v[5]),
        "r"(x0.v[6]), "r"(x0.v[7]), "r"(m.v[0]), "r"(m.v[1]), "r"(m.v[2]), "r"(m.v[3]),
        "r"(m.v[4]), "r"(m.v[5]), "r"(m.v[6]), "r"(m.v[7]));
}

// The K stages of a pass over a tile of E = T << K elements in shared memory,
// 128 butterflies at a time (all tc::kThreads threads call it).  first: stage 0
// is stage 0 of the transform, whose twiddles are all 1.  kAhead: the next twiddle is
// loaded beside the matrix product (ntt.cu says where).
template <bool kAhead>
__device__ __forceinline__ void tile_stages(tc::ProductTile& tile, uint4* sm, int mode, int K,
                                            int T, int log_t, int log_u, uint64_t U, uint64_t l0,
                                            uint64_t high_a, bool first,
                                            const uint64_t* __restrict__ roots) {
  const int E = T << K, half = E >> 1;
  Fr ahead = fr_zero();
  // the twiddle of this thread's butterfly from b0 on in stage s
  const auto twiddle = [&](int s, int b0) {
    const int b = b0 + (int)threadIdx.x;
    const int bb = b < half ? b : 0;
    const uint64_t l = l0 + (bb & (T - 1));
    const uint64_t high =
        mode == kModeB ? l >> log_u : (mode == kModeC ? line_high(l, U) : high_a);
    return fr_load_ro(roots, (high << s) | (uint64_t)((bb >> log_t) >> (K - 1 - s)));
  };
  if (kAhead && !first) ahead = twiddle(0, 0);
#pragma unroll 1
  for (int s = 0; s < K; s++) {
    const int log_h = K - 1 - s;
#pragma unroll 1
    for (int b0 = 0; b0 < half; b0 += tc::kThreads) {
      const int b = b0 + (int)threadIdx.x;
      const bool live = b < half;
      const int bb = live ? b : 0;  // others repeat butterfly 0 and store nothing
      const int ll = bb & (T - 1);
      const int pp = bb >> log_t;
      const int grp = pp >> log_h;
      const int j0 = (grp << (log_h + 1)) + (pp & ((1 << log_h) - 1));
      const int i0 = j0 * T + ll, i1 = i0 + (T << log_h);
      const Fr x1 = tile_load(sm, E, i1);
      const bool end = b0 + tc::kThreads >= half;  // of the stage
      const int s2 = end ? s + 1 : s, b2 = end ? 0 : b0 + tc::kThreads;
      Fr m;
      if (first && s == 0) {
        m = fr_reduce_once(x1);
        if (kAhead && end && s2 < K) ahead = twiddle(s2, b2);
      } else {
        Fr w;
        if (kAhead) {
          w = ahead;
        } else {
          const uint64_t l = l0 + ll;
          const uint64_t high =
              mode == kModeB ? l >> log_u : (mode == kModeC ? line_high(l, U) : high_a);
          w = fr_load_ro(roots, (high << s) | (uint64_t)grp);
        }
        tile.start(w, x1);
        if (kAhead && s2 < K) ahead = twiddle(s2, b2);
        m = tile.finish();
        if (tile.alone) m = product_alone(w, x1);
        __syncwarp();
      }
      const Fr x0 = tile_load(sm, E, i0);
      Fr y0, y1;
      loose_butterfly(x0, m, y0, y1);
      if (live) {
        tile_store(sm, E, i0, y0);
        tile_store(sm, E, i1, y1);
      }
    }
    __syncthreads();
  }
}

}  // namespace pk
