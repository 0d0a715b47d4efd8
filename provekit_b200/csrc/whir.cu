// whir.cu -- the data-parallel pieces of WHIR's prove rounds on the device.
//
// The WHIR prover itself lives in the un-vendored `whir` crate (called from
// provekit/prover/src/whir_r1cs.rs:295-301, 378-414).  Its rounds are built
// from the operations below; their arithmetic follows the reference's WHIR
// verifier restated in Go (recursive-verifier/app/utilities/utilities.go,
// recursive-verifier/app/circuit/whir_utilities.go):
//   pkg_whir_fold_coeffs     fold 2^k interleaved messages with the folding
//                            randomness (MultivarPoly weights, utilities.go:16-23)
//   pkg_whir_fold_rows       computeFold over codeword rows (whir_utilities.go:182-188)
//   pkg_poly_eval_many       UnivarPoly at OOD points (utilities.go:25-39)
//   pkg_merkle_open          authentication paths as verifyMerkleTreeProofs
//   pkg_gather_rows          reads them (whir_utilities.go:14-47)
//   pkg_whir_sumcheck_round  one round of the weighted sumcheck, sent as
//                            evaluations at 0, 1, 2 (utilities.go:149-171)
//   pkg_eq_accumulate        w += sum_j c_j eq(p_j, .) for new constraints
//   pkg_stir_indices         getStirChallenges (whir_utilities.go:49-79), host
#include <algorithm>
#include <cstring>
#include <vector>

#include "fr.cuh"
#include "fr_host.hpp"
#include "fr_lazy.cuh"
#include "internal.cuh"
#include "pk_common.cuh"
#include "reduce.cuh"
#include "sumcheck_device.cuh"

namespace pk {

constexpr int kMaxFoldK = 6;

// Montgomery field elements passed by value as kernel parameters.
template <int N>
struct FrParams {
  uint32_t v[N][8];
};

template <int N>
__device__ __forceinline__ Fr param_fr(const FrParams<N>& p, int j) {
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = p.v[j][i];
  return r;
}

template <int N>
static void put_param(FrParams<N>& p, int j, const HostFr& x) {
  memcpy(p.v[j], x.l, 32);
}

// w_j = prod_t alpha[t]^(bit t of j): MultivarPoly's coefficient of row entry j.
static void fold_weights(const uint64_t* alpha, unsigned k, FrParams<1 << kMaxFoldK>& W) {
  std::vector<HostFr> w((size_t)1 << k);
  w[0] = HostFr::one();
  for (unsigned t = 0; t < k; t++) {
    const HostFr a = HostFr::from_limbs(alpha + 4 * t);
    const size_t half = size_t(1) << t;
    for (size_t j = 0; j < half; j++) w[j + half] = HostFr::mul(w[j], a);
  }
  for (size_t j = 0; j < w.size(); j++) put_param(W, (int)j, w[j]);
}

// out[i] = sum_j w_j c[j L + i]  (w_0 = 1).  A product alone (m = 2) is reduced at
// once: 2^21 coefficients 30.8 us, with the unreduced sum 35.5 (rows are the same
// either way, and their larger folds lose registers by it).
__global__ void whir_fold_coeffs_kernel(const uint64_t* __restrict__ c, size_t L, int m,
                                        const __grid_constant__ FrParams<1 << kMaxFoldK> W,
                                        uint64_t* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < L;
       i += (size_t)gridDim.x * blockDim.x) {
    const Fr head = fr_load_ro(c, i);
    Fr tail;
    if (m == 2) {
      tail = fr_mul(param_fr(W, 1), fr_load_ro(c, L + i));
    } else {
      lazy::Acc acc;
      acc.zero();
      for (int j = 1; j < m; j++) acc.mac(param_fr(W, j), fr_load_ro(c, j * L + i));
      tail = acc.finish();
    }
    fr_store(out, i, fr_add(head, tail));
  }
}

// out[i] = sum_j w_j rows[i m + j]
__global__ void whir_fold_rows_kernel(const uint64_t* __restrict__ rows, size_t nrows, int m,
                                      const __grid_constant__ FrParams<1 << kMaxFoldK> W,
                                      uint64_t* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nrows;
       i += (size_t)gridDim.x * blockDim.x) {
    lazy::Acc acc;
    acc.zero();
    for (int j = 1; j < m; j++) acc.mac(param_fr(W, j), fr_load_ro(rows, i * m + j));
    fr_store(out, i, fr_add(fr_load_ro(rows, i * m), acc.finish()));
  }
}

// Up to kMaxEvalPolys polynomials of n coefficients (stride apart) at one point z, a
// run of g CTAs each.  CTA b of a run owns the coefficients [bC, (b + 1)C), C = 256 per;
// its thread j takes bC + j + 256k for k = 0, 1, ..: an unreduced sum (fr_lazy.cuh)
// with the weights y^k, y = z^256, Horner in y^kEvalWeights above that many.  The
// thread's sum is scaled by z^j and the CTA's by z^(bC), each one product of two
// powers that the host computed.  The CTA that takes the last ticket adds the CTAs'
// sums, a warp per polynomial.  Two of 2^21 coefficients: 110 -> 57 us; one of 2^12:
// 18 -> 11 (Horner, a power tree over the CTA and a launch per polynomial before).
constexpr int kMaxEvalPolys = 8;
constexpr int kEvalWeights = 32;
constexpr int kEvalRunBits = 5;  // CTAs per polynomial < 16 * 2^5
struct EvalPowers {
  uint32_t y[kEvalWeights + 1][8];           // z^(256k)
  uint32_t j_lo[16][8], j_hi[16][8];         // z^k, z^(16k)
  uint32_t b_lo[16][8], b_hi[1 << kEvalRunBits][8];  // z^(Ck), z^(16Ck)
};
static_assert(kRedThreads == 256, "a thread's power is two of 16");

__device__ __forceinline__ Fr power(const uint32_t (&w)[8]) {
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = w[i];
  return r;
}

__global__ void __launch_bounds__(kRedThreads, 2) poly_eval_kernel(
    const uint64_t* __restrict__ coeffs, size_t n, size_t stride, int polys, unsigned g, size_t per,
    const __grid_constant__ EvalPowers P, const RedOut ro) {
  const unsigned j = threadIdx.x, b = blockIdx.x % g;
  const uint64_t* c = coeffs + 4 * stride * (blockIdx.x / g);
  const size_t at = b * per * kRedThreads + j;
  const size_t end = n < (b + 1) * per * kRedThreads ? n : (b + 1) * per * kRedThreads;
  const size_t mine = at < end ? (end - at + kRedThreads - 1) / kRedThreads : 0;
  Fr sum[1] = {fr_zero()};
  size_t k0 = mine ? (mine - 1) / kEvalWeights * kEvalWeights : 0;
#pragma unroll 1
  for (size_t left = mine; left > 0; left = k0, k0 -= left ? kEvalWeights : 0) {
    const int terms = (int)(left - k0);
    lazy::Acc acc;
    acc.zero();
#pragma unroll 2
    for (int k = 0; k < terms; k++)
      acc.mac(power(P.y[k]), fr_load_ro(c, at + (k0 + k) * kRedThreads));
    const Fr run = acc.finish();
    sum[0] = left == mine ? run : fr_add(fr_mul(sum[0], power(P.y[kEvalWeights])), run);
  }
  sum[0] = fr_mul(sum[0], fr_mul(power(P.j_lo[j & 15]), power(P.j_hi[j >> 4])));
  block_sum<1>(sum);
  if (j == 0) sum[0] = fr_mul(sum[0], fr_mul(power(P.b_lo[b & 15]), power(P.b_hi[b >> 4])));
  static_assert(kMaxEvalPolys <= kRedThreads / 32, "a warp per polynomial");
  runs_finish(sum[0], ro, polys, (j >> 5) * g, (j >> 5) * g + g);
}

// path[q depth + l] = node (idx[q] >> l) ^ 1 of level l
__global__ void merkle_open_kernel(const uint8_t* __restrict__ layers, size_t num_leaves,
                                   int depth, const uint64_t* __restrict__ idx, size_t nq,
                                   uint8_t* __restrict__ out) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nq * (size_t)depth;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t q = t / depth;
    const int l = (int)(t % depth);
    size_t off = 0, width = num_leaves;
    for (int j = 0; j < l; j++) {
      off += width;
      width >>= 1;
    }
    const uint4* src = reinterpret_cast<const uint4*>(layers + 32 * (off + ((idx[q] >> l) ^ 1)));
    uint4* dst = reinterpret_cast<uint4*>(out + 32 * t);
    dst[0] = src[0];
    dst[1] = src[1];
  }
}

// rows_out[q][e] = codeword[idx[q]][e]
__global__ void gather_rows_kernel(const uint64_t* __restrict__ cw, size_t row_fr,
                                   const uint64_t* __restrict__ idx, size_t nq,
                                   uint64_t* __restrict__ out) {
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nq * row_fr;
       t += (size_t)gridDim.x * blockDim.x) {
    const size_t q = t / row_fr, e = t % row_fr;
    fr_store(out, t, fr_load_ro(cw, idx[q] * row_fr + e));
  }
}

// One WHIR sumcheck round over f, w (quarter layout when folding, as the
// Spartan rounds): pairs (i, i + q); sums f0 w0, f1 w1, (2f1-f0)(2w1-w0).
// The round kernel's seven products go through one out-of-line call, and the
// kernel is bounded to two CTAs per SM (128 registers): with them inlined the
// folding kernel took 172 registers, one CTA of 256 threads per SM.
static __device__ __noinline__ Fr whir_mul(const Fr a, const Fr b) { return fr_mul(a, b); }

template <bool kFold>
__global__ void __launch_bounds__(kRedThreads, 2) whir_round_kernel(
    uint64_t* __restrict__ f, uint64_t* __restrict__ w, size_t q,
    const __grid_constant__ FrParams<1> A, const RedOut ro) {
  Fr acc[3] = {fr_zero(), fr_zero(), fr_zero()};
  const Fr alpha = param_fr(A, 0);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < q;
       i += (size_t)gridDim.x * blockDim.x) {
    Fr f0 = fr_load(f, i), f1 = fr_load(f, i + q), w0 = fr_load(w, i), w1 = fr_load(w, i + q);
    if (kFold) {
      f0 = fr_add(f0, whir_mul(alpha, fr_sub(fr_load(f, i + 2 * q), f0)));
      f1 = fr_add(f1, whir_mul(alpha, fr_sub(fr_load(f, i + 3 * q), f1)));
      w0 = fr_add(w0, whir_mul(alpha, fr_sub(fr_load(w, i + 2 * q), w0)));
      w1 = fr_add(w1, whir_mul(alpha, fr_sub(fr_load(w, i + 3 * q), w1)));
      fr_store(f, i, f0);
      fr_store(f, i + q, f1);
      fr_store(w, i, w0);
      fr_store(w, i + q, w1);
    }
    acc[0] = fr_add(acc[0], whir_mul(f0, w0));
    acc[1] = fr_add(acc[1], whir_mul(f1, w1));
    const Fr f2 = fr_sub(fr_add(f1, f1), f0), w2 = fr_sub(fr_add(w1, w1), w0);
    acc[2] = fr_add(acc[2], whir_mul(f2, w2));
  }
  block_finish<3>(acc, ro);
}

// The same with four lanes per pair (sumcheck_device.cuh).
template <bool kFold>
__global__ void __launch_bounds__(kQuadThreads) whir_quad_kernel(
    uint64_t* __restrict__ f, uint64_t* __restrict__ w, size_t q,
    const __grid_constant__ FrParams<1> A, const RedOut ro) {
  __shared__ FrShared sh;
  const int lane = threadIdx.x & 3, quad = threadIdx.x & ~3;
  uint64_t* const t = lane < 2 ? f : w;  // f0, f1, w0, w1
  const Fr alpha = param_fr(A, 0);
  Fr acc = fr_zero();
  for (size_t base = (size_t)blockIdx.x * kQuadPairs; base < q;
       base += (size_t)gridDim.x * kQuadPairs) {
    const size_t i = base + (threadIdx.x >> 2), at = i + (lane & 1) * q;
    if (i < q) {
      Fr x = fr_load(t, at);
      if (kFold) {
        x = fr_add(x, fr_mul(alpha, fr_sub(fr_load(t, at + 2 * q), x)));
        fr_store(t, at, x);
      }
      sh.put(threadIdx.x, x);
    }
    __syncwarp();
    if (i < q && lane < 3) {
      Fr x = sh.get(quad + (lane == 0 ? 0 : 1)), y = sh.get(quad + (lane == 0 ? 2 : 3));
      if (lane == 2) {
        x = fr_sub(fr_add(x, x), sh.get(quad));
        y = fr_sub(fr_add(y, y), sh.get(quad + 2));
      }
      acc = fr_add(acc, fr_mul(x, y));
    }
    __syncwarp();
  }
  Fr sums[3];
  quad_sums(acc, sums);
  block_finish<3>(sums, ro);
}

// The equality tables of a point (p_0, .., p_nv-1), the top variable first: entry x of
// a run of variables is prod_i (bit i of x ? p_i : 1 - p_i), over the first nhi
// variables times the point's coefficient (hi) and over the rest (lo).
// in: npts coefficients, then the points, each nv coordinates (expanded) or one z
// for p_nv-1-i = z^(2^i) (ExpandFromUnivariate,
// recursive-verifier/app/utilities/utilities.go:183-191).
// A row of CTAs per point.  An entry is one product of two entries of tables over half
// of its variables each, which a CTA builds first: bound by the chain of nv squarings
// and about eight products.  With a launch each for the squarings, the hi and the lo
// tables, and a product per variable, 119 points of 18 variables took 38 us
// and one 30; now 15 and 16.
constexpr int kEqSub = 8;  // variables per half: all of them up to nv = 32
constexpr int kEqMaxVars = 40;

struct EqHalves {  // of k variables: the first `rest` one by one, then a, then b
  int rest, a, b;
  __device__ __forceinline__ explicit EqHalves(int k) {
    a = (k + 1) / 2 < kEqSub ? (k + 1) / 2 : kEqSub;
    b = k - a < kEqSub ? k - a : kEqSub;
    rest = k - a - b;
  }
};

__device__ __forceinline__ Fr eq_factor(const Fr& p, bool bit) {
  return bit ? p : fr_sub(fr_one_mont(), p);
}

__global__ void __launch_bounds__(256) eq_tables_kernel(const uint64_t* __restrict__ in,
                                                        size_t npts, int nv, bool expanded,
                                                        int nhi, uint64_t* __restrict__ hi,
                                                        uint64_t* __restrict__ lo) {
  __shared__ Fr p[kEqMaxVars], sub[4 << kEqSub];
  const size_t j = blockIdx.x;
  if (expanded) {
    for (int i = threadIdx.x; i < nv; i += blockDim.x) p[i] = fr_load_ro(in, npts + j * nv + i);
  } else if (threadIdx.x == 0 && nv) {
    Fr z = fr_load_ro(in, npts + j);
    for (int i = nv - 1; i > 0; i--) {
      p[i] = z;
      z = fr_sqr(z);
    }
    p[0] = z;
  }
  __syncthreads();
  const EqHalves h(nhi), l(nv - nhi);
  // the halves: hi's a and b, then lo's
  const int end0 = 1 << h.a, end1 = end0 + (1 << h.b), end2 = end1 + (1 << l.a),
            end3 = end2 + (1 << l.b);
  for (int t = threadIdx.x; t < end3; t += blockDim.x) {
    int x = t, first = h.rest, k = h.a;
    if (t >= end2) {
      x = t - end2, first = nhi + l.rest + l.a, k = l.b;
    } else if (t >= end1) {
      x = t - end1, first = nhi + l.rest, k = l.a;
    } else if (t >= end0) {
      x = t - end0, first = h.rest + h.a, k = h.b;
    }
    Fr acc = t < end0 ? fr_load_ro(in, j) : fr_one_mont();
    if (k && t >= end0) {
      acc = eq_factor(p[first], (x >> (k - 1)) & 1);
      first++, k--;
    }
#pragma unroll 1
    for (; k > 0; first++, k--) acc = fr_mul(acc, eq_factor(p[first], (x >> (k - 1)) & 1));
    sub[t] = acc;
  }
  __syncthreads();
  const size_t nh = size_t(1) << nhi, nl = size_t(1) << (nv - nhi);
  for (size_t e = blockIdx.y * (size_t)blockDim.x + threadIdx.x; e < nh + nl;
       e += (size_t)gridDim.y * blockDim.x) {
    const bool high = e < nh;
    const size_t x = high ? e : e - nh;
    const EqHalves& s = high ? h : l;
    Fr v = fr_mul(sub[(high ? 0 : end1) + ((x >> s.b) & ((1 << s.a) - 1))],
                  sub[(high ? end0 : end2) + (x & ((1 << s.b) - 1))]);
#pragma unroll 1
    for (int i = 0; i < s.rest; i++)
      v = fr_mul(v, eq_factor(p[(high ? 0 : nhi) + i], (x >> (s.a + s.b + s.rest - 1 - i)) & 1));
    fr_store(high ? hi : lo, j * (high ? nh : nl) + x, v);
  }
}

// w[b] += sum_j hi_j[b >> nlo] lo_j[b & (2^nlo - 1)], the products of an entry
// summed unreduced (fr_lazy.cuh).  2^split threads share an entry's points, so that
// a short table still fills the chip; those of one entry lie 128 / 2^split apart,
// and a warp's loads stay in line.  Bound by the multiplier (256 cycles per warp
// and point): 2^18 entries of 118 points 446 us with binary64 sums, 283 now; 2^14 of
// 40 32 -> 12, 2^21 of two (a product each before) 115 -> 82.
constexpr int kEqThreads = 128;
__global__ void __launch_bounds__(kEqThreads, 4) eq_accumulate_kernel(
    uint64_t* __restrict__ w, size_t n, int nlo, const uint64_t* __restrict__ hi,
    size_t nhi_entries, const uint64_t* __restrict__ lo, size_t npts, int split) {
  __shared__ FrShared sh;
  const size_t nlo_entries = size_t(1) << nlo;
  const unsigned per = kEqThreads >> split, part = threadIdx.x / per;
  const size_t b = blockIdx.x * (size_t)per + threadIdx.x % per;
  Fr sum = fr_zero();
  if (b < n) {
    const size_t bh = b >> nlo, bl = b & (nlo_entries - 1), step = size_t(1) << split;
    size_t j = part;
#pragma unroll 1
    while (j < npts) {
      const size_t left = (npts - j + step - 1) >> split;
      const int terms = left < (size_t)lazy::kMaxTerms ? (int)left : lazy::kMaxTerms;
      lazy::Acc acc;
      acc.zero();
#pragma unroll 2
      for (int i = 0; i < terms; i++, j += step)
        acc.mac(fr_load_ro(hi, j * nhi_entries + bh), fr_load_ro(lo, j * nlo_entries + bl));
      sum = fr_add(sum, acc.finish());
    }
  }
  if (split) {
    sh.put(threadIdx.x, sum);
    __syncthreads();
    if (part) return;
#pragma unroll 1
    for (unsigned k = per; k < kEqThreads; k += per) sum = fr_add(sum, sh.get(threadIdx.x + k));
  }
  if (b < n) fr_store(w, b, fr_add(fr_load(w, b), sum));
}

// Threads per entry: the number (at least kEqMinPoints points each) with the least
// waves of CTAs times products per thread, the reduction of its sum counted as two.
// 2^18 entries of 118 points: one thread 288 us (3.5 waves), two 283; 2^14 entries of
// 40: one 21.8, four 12.4.
constexpr size_t kEqMinPoints = 8;
static int eq_split(size_t n, size_t npts) {
  const size_t resident = 4 * (size_t)sm_count();
  size_t best = 0;
  int split = 0;
  for (int k = 0; k <= 3 && (k == 0 || (npts >> k) >= kEqMinPoints); k++) {
    const size_t per = kEqThreads >> k, ctas = (n + per - 1) / per;
    const size_t cost = (ctas + resident - 1) / resident * ((npts >> k) + 2);
    if (k == 0 || cost < best) {
      best = cost;
      split = k;
    }
  }
  return split;
}

}  // namespace pk

using namespace pk;

extern "C" int pkg_whir_fold_coeffs(const uint64_t* coeffs, size_t n, unsigned k,
                                    const uint64_t* alpha, uint64_t* out, pkg_stream_t stream) {
  PK_REQUIRE(k <= (unsigned)kMaxFoldK, "folding factor %u above %d", k, kMaxFoldK);
  PK_REQUIRE(is_pow2(n) && n >= (size_t(1) << k), "length %zu is not a power of two >= 2^%u", n, k);
  PK_REQUIRE(coeffs && out && (k == 0 || alpha), "null pointer");
  PK_REQUIRE(aligned16(coeffs) && aligned16(out), "device buffers must be 16-byte aligned");
  FrParams<1 << kMaxFoldK> W;
  memset(&W, 0, sizeof W);
  fold_weights(alpha, k, W);
  const size_t L = n >> k;
  whir_fold_coeffs_kernel<<<ew_grid(L), 256, 0, as_stream(stream)>>>(coeffs, L, 1 << k, W, out);
  PK_CHECK_LAUNCH("whir_fold_coeffs_kernel");
  return PKG_OK;
}

extern "C" int pkg_whir_fold_rows(const uint64_t* rows, size_t nrows, unsigned k,
                                  const uint64_t* alpha, uint64_t* out, pkg_stream_t stream) {
  PK_REQUIRE(k <= (unsigned)kMaxFoldK, "folding factor %u above %d", k, kMaxFoldK);
  if (nrows == 0) return PKG_OK;
  PK_REQUIRE(rows && out && (k == 0 || alpha), "null pointer");
  PK_REQUIRE(aligned16(rows) && aligned16(out), "device buffers must be 16-byte aligned");
  FrParams<1 << kMaxFoldK> W;
  memset(&W, 0, sizeof W);
  fold_weights(alpha, k, W);
  whir_fold_rows_kernel<<<ew_grid(nrows), 256, 0, as_stream(stream)>>>(rows, nrows, 1 << k, W, out);
  PK_CHECK_LAUNCH("whir_fold_rows_kernel");
  return PKG_OK;
}

namespace pk {
static void put_powers(uint32_t (*out)[8], size_t count, const HostFr& x) {
  HostFr w = HostFr::one();
  for (size_t k = 0; k < count; k++) {
    memcpy(out[k], w.l, 32);
    w = HostFr::mul(w, x);
  }
}

int poly_eval_device(const uint64_t* coeffs, size_t n, size_t stride, size_t polys,
                     const uint64_t* points, size_t npts, uint64_t* out, cudaStream_t s) {
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  std::vector<uint64_t> vals(4 * kFusedSlotFr);
  for (size_t i0 = 0; i0 < polys; i0 += kMaxEvalPolys) {
    const size_t np = std::min<size_t>(polys - i0, kMaxEvalPolys);
    // all polynomials' CTAs resident at once, at least a coefficient per thread
    const size_t gmax = std::min<size_t>(std::max<size_t>(1, 2 * (size_t)sm_count() / np),
                                         16 << kEvalRunBits);
    const size_t per = (n + kRedThreads * gmax - 1) / (kRedThreads * gmax);
    const size_t C = per * kRedThreads, g = (n + C - 1) / C;
    // a launch per point; their values are read once the slots are full
    const size_t chunk = kFusedSlotFr / np;
    for (size_t j0 = 0; j0 < npts; j0 += chunk) {
      const size_t m = std::min(chunk, npts - j0);
      for (size_t j = 0; j < m; j++) {
        const HostFr z = HostFr::from_limbs(points + 4 * (j0 + j));
        EvalPowers P;
        memset(&P, 0, sizeof P);
        put_powers(P.j_lo, 16, z);
        const HostFr z16 = HostFr::pow_u64(z, 16), y = HostFr::pow_u64(z16, 16);
        put_powers(P.j_hi, 16, z16);
        put_powers(P.y, std::min<size_t>(per, kEvalWeights) + 1, y);
        const HostFr zc = HostFr::pow_u64(y, per);
        put_powers(P.b_lo, std::min<size_t>(g, 16), zc);
        put_powers(P.b_hi, (g + 15) / 16, HostFr::pow_u64(zc, 16));
        const RedOut ro = {fs.part, fs.ticket, fs.dev + 4 * np * j, fused_next_seq()};
        poly_eval_kernel<<<(unsigned)(g * np), kRedThreads, 0, s>>>(
            coeffs + 4 * stride * i0, n, stride, (int)np, (unsigned)g, per, P, ro);
        PK_CHECK_LAUNCH("poly_eval_kernel");
      }
      if ((rc = fused_read(vals.data(), fs, 32 * np * m, s))) return rc;
      for (size_t j = 0; j < m; j++)
        for (size_t i = 0; i < np; i++)
          memcpy(out + 4 * ((i0 + i) * npts + j0 + j), vals.data() + 4 * (np * j + i), 32);
    }
  }
  return PKG_OK;
}
}  // namespace pk

extern "C" int pkg_poly_eval_many(const uint64_t* coeffs, size_t n, const uint64_t* points,
                                  size_t npts, uint64_t* out, pkg_stream_t stream) {
  if (npts == 0) return PKG_OK;
  PK_REQUIRE(points && out, "null pointer");
  if (n == 0) {
    memset(out, 0, 32 * npts);
    return PKG_OK;
  }
  PK_REQUIRE(coeffs && aligned16(coeffs), "null or unaligned coefficients");
  PK_REQUIRE(n < (size_t(1) << 40), "too many coefficients");
  return poly_eval_device(coeffs, n, 0, 1, points, npts, out, as_stream(stream));
}

extern "C" int pkg_merkle_open(const uint8_t* layers, size_t num_leaves, const uint64_t* indices,
                               size_t nq, uint8_t* paths, pkg_stream_t stream) {
  PK_REQUIRE(is_pow2(num_leaves), "num_leaves %zu is not a power of two", num_leaves);
  const int depth = log2_exact(num_leaves);
  if (nq == 0 || depth == 0) return PKG_OK;
  PK_REQUIRE(layers && indices && paths && aligned16(layers), "null or unaligned pointer");
  for (size_t q = 0; q < nq; q++)
    PK_REQUIRE(indices[q] < num_leaves, "index %llu out of range (%zu leaves)",
               (unsigned long long)indices[q], num_leaves);
  cudaStream_t s = as_stream(stream);
  Scratch scr;
  const size_t idx_bytes = (8 * nq + 255) & ~size_t(255);
  int rc = scr.alloc(idx_bytes + 32 * nq * depth, s);
  if (rc) return rc;
  uint64_t* d_idx = static_cast<uint64_t*>(scr.ptr);
  uint8_t* d_out = static_cast<uint8_t*>(scr.ptr) + idx_bytes;
  PK_CUDA(cudaMemcpyAsync(d_idx, indices, 8 * nq, cudaMemcpyHostToDevice, s));
  merkle_open_kernel<<<ew_grid(nq * depth), 256, 0, s>>>(layers, num_leaves, depth, d_idx, nq, d_out);
  PK_CHECK_LAUNCH("merkle_open_kernel");
  PK_CUDA(cudaMemcpyAsync(paths, d_out, 32 * nq * depth, cudaMemcpyDeviceToHost, s));
  PK_CUDA(cudaStreamSynchronize(s));
  return PKG_OK;
}

extern "C" int pkg_gather_rows(const uint64_t* codeword, size_t fr_per_row, size_t num_rows,
                               const uint64_t* indices, size_t nq, uint64_t* rows,
                               pkg_stream_t stream) {
  if (nq == 0 || fr_per_row == 0) return PKG_OK;
  PK_REQUIRE(codeword && indices && rows && aligned16(codeword), "null or unaligned pointer");
  for (size_t q = 0; q < nq; q++)
    PK_REQUIRE(indices[q] < num_rows, "index %llu out of range (%zu rows)",
               (unsigned long long)indices[q], num_rows);
  cudaStream_t s = as_stream(stream);
  Scratch scr;
  const size_t idx_bytes = (8 * nq + 255) & ~size_t(255);
  int rc = scr.alloc(idx_bytes + 32 * nq * fr_per_row, s);
  if (rc) return rc;
  uint64_t* d_idx = static_cast<uint64_t*>(scr.ptr);
  uint64_t* d_out = reinterpret_cast<uint64_t*>(static_cast<uint8_t*>(scr.ptr) + idx_bytes);
  PK_CUDA(cudaMemcpyAsync(d_idx, indices, 8 * nq, cudaMemcpyHostToDevice, s));
  gather_rows_kernel<<<ew_grid(nq * fr_per_row), 256, 0, s>>>(codeword, fr_per_row, d_idx, nq, d_out);
  PK_CHECK_LAUNCH("gather_rows_kernel");
  PK_CUDA(cudaMemcpyAsync(rows, d_out, 32 * nq * fr_per_row, cudaMemcpyDeviceToHost, s));
  PK_CUDA(cudaStreamSynchronize(s));
  return PKG_OK;
}

namespace pk {
// pkg_gather_rows + pkg_merkle_open of the same indices with one upload and
// one synchronisation.
int open_rows_device(const uint64_t* codeword, size_t fr_per_row, size_t num_rows,
                     const uint8_t* layers, const uint64_t* indices, size_t nq, uint64_t* rows,
                     uint8_t* paths, cudaStream_t s, bool sync) {
  if (nq == 0) return PKG_OK;
  const int depth = log2_exact(num_rows);
  for (size_t q = 0; q < nq; q++)
    PK_REQUIRE(indices[q] < num_rows, "index %llu out of range (%zu rows)",
               (unsigned long long)indices[q], num_rows);
  Scratch scr;
  const size_t idx_bytes = (8 * nq + 255) & ~size_t(255);
  const size_t row_bytes = (32 * nq * fr_per_row + 255) & ~size_t(255);
  int rc = scr.alloc(idx_bytes + row_bytes + 32 * nq * (size_t)depth + 32, s);
  if (rc) return rc;
  uint64_t* d_idx = static_cast<uint64_t*>(scr.ptr);
  uint64_t* d_rows = reinterpret_cast<uint64_t*>(static_cast<uint8_t*>(scr.ptr) + idx_bytes);
  uint8_t* d_paths = static_cast<uint8_t*>(scr.ptr) + idx_bytes + row_bytes;
  PK_CUDA(cudaMemcpyAsync(d_idx, indices, 8 * nq, cudaMemcpyHostToDevice, s));
  gather_rows_kernel<<<ew_grid(nq * fr_per_row), 256, 0, s>>>(codeword, fr_per_row, d_idx, nq,
                                                              d_rows);
  PK_CHECK_LAUNCH("gather_rows_kernel");
  if (depth) {
    merkle_open_kernel<<<ew_grid(nq * depth), 256, 0, s>>>(layers, num_rows, depth, d_idx, nq,
                                                           d_paths);
    PK_CHECK_LAUNCH("merkle_open_kernel");
  }
  if (!sync) {
    PK_CUDA(cudaMemcpyAsync(rows, d_rows, 32 * nq * fr_per_row, cudaMemcpyDeviceToHost, s));
    if (depth)
      PK_CUDA(cudaMemcpyAsync(paths, d_paths, 32 * nq * (size_t)depth, cudaMemcpyDeviceToHost, s));
    return PKG_OK;
  }
  const HostRead reads[2] = {{rows, d_rows, 32 * nq * fr_per_row},
                             {paths, d_paths, depth ? 32 * nq * (size_t)depth : 0}};
  return read_small(reads, depth ? 2 : 1, s);
}
}  // namespace pk

extern "C" int pkg_stir_indices(const uint8_t* bytes, size_t folded_domain_size, size_t nq,
                                uint64_t* out) {
  PK_REQUIRE(is_pow2(folded_domain_size), "folded domain size %zu is not a power of two",
             folded_domain_size);
  if (nq == 0) return PKG_OK;
  PK_REQUIRE(bytes && out, "null pointer");
  const int bits = log2_exact(folded_domain_size);
  const size_t nbytes = (size_t)(bits + 7) / 8;
  for (size_t i = 0; i < nq; i++) {
    uint64_t v = 0;
    for (size_t j = 0; j < nbytes; j++) v = (v << 8) | bytes[i * nbytes + j];
    out[i] = bits >= 64 ? v : (v & ((uint64_t(1) << bits) - 1));
  }
  return PKG_OK;
}

extern "C" int pkg_whir_sumcheck_round(uint64_t* f, uint64_t* w, size_t size, const uint64_t* fold,
                                       uint64_t out[12], pkg_stream_t stream) {
  PK_REQUIRE(is_pow2(size) && size >= 2, "table size %zu must be a power of two >= 2", size);
  PK_REQUIRE(!fold || size >= 4, "folding needs size >= 4 (got %zu)", size);
  PK_REQUIRE(f && w && out && aligned16(f) && aligned16(w), "null or unaligned pointer");
  cudaStream_t s = as_stream(stream);
  const size_t q = fold ? size / 4 : size / 2;
  const int g = round_grid(q);
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  uint64_t* part = fs.part;  // g <= 4 CTAs per SM
  FrParams<1> A;
  memset(&A, 0, sizeof A);
  if (fold) memcpy(A.v[0], fold, 32);
  const RedOut ro = {part, fs.ticket, fs.dev, fused_next_seq()};
  const auto kernel = q <= kQuadMaxPairs ? (fold ? whir_quad_kernel<true> : whir_quad_kernel<false>)
                                         : (fold ? whir_round_kernel<true> : whir_round_kernel<false>);
  static_assert(kQuadThreads == kRedThreads, "one CTA size");
  kernel<<<g, kRedThreads, 0, s>>>(f, w, q, A, ro);
  PK_CHECK_LAUNCH("whir_round_kernel");
  return fused_read(out, fs, 96, s);
}

namespace pk {
int eq_accumulate_device(uint64_t* w, size_t nv, const uint64_t* points, const uint64_t* coeffs,
                         size_t npts, cudaStream_t s, bool sync, bool expanded) {
  if (npts == 0) return PKG_OK;
  const int nhi = (int)(nv + 1) / 2, nlo = (int)nv - nhi;
  const size_t nh = size_t(1) << nhi, nl = size_t(1) << nlo, n = size_t(1) << nv;
  Scratch scr;
  // [coefficients | points | hi tables | lo tables], the first two in one copy
  const size_t pts_fr = nv == 0 ? 0 : expanded ? npts * nv : npts, in_fr = npts + pts_fr;
  int rc = scr.alloc(32 * (in_fr + npts * (nh + nl)), s);
  if (rc) return rc;
  uint64_t* d_in = static_cast<uint64_t*>(scr.ptr);
  uint64_t* d_hi = d_in + 4 * in_fr;
  uint64_t* d_lo = d_hi + 4 * npts * nh;
  std::vector<uint64_t> in(4 * in_fr);
  memcpy(in.data(), coeffs, 32 * npts);
  if (pts_fr) memcpy(in.data() + 4 * npts, points, 32 * pts_fr);
  // pageable: staged before the copy returns
  PK_CUDA(cudaMemcpyAsync(d_in, in.data(), 32 * in_fr, cudaMemcpyHostToDevice, s));
  PK_REQUIRE(npts < (size_t(1) << 31), "too many points (%zu)", npts);
  const size_t rows = std::min<size_t>((nh + nl + 1023) / 1024, 65535);
  eq_tables_kernel<<<dim3((unsigned)npts, (unsigned)rows), 256, 0, s>>>(d_in, npts, (int)nv,
                                                                        expanded, nhi, d_hi, d_lo);
  PK_CHECK_LAUNCH("eq_tables_kernel");
  const int split = eq_split(n, npts);
  const size_t per = kEqThreads >> split;
  eq_accumulate_kernel<<<(unsigned)((n + per - 1) / per), kEqThreads, 0, s>>>(w, n, nlo, d_hi, nh,
                                                                             d_lo, npts, split);
  PK_CHECK_LAUNCH("eq_accumulate_kernel");
  if (sync) PK_CUDA(cudaStreamSynchronize(s));
  return PKG_OK;
}
}  // namespace pk

extern "C" int pkg_eq_accumulate(uint64_t* w, size_t nv, const uint64_t* points,
                                 const uint64_t* coeffs, size_t npts, pkg_stream_t stream) {
  PK_REQUIRE(nv < 40, "too many variables (%zu)", nv);
  if (npts == 0) return PKG_OK;
  PK_REQUIRE(w && points && coeffs && aligned16(w), "null or unaligned pointer");
  PK_REQUIRE((nv == 0 || host_readable(points)) && host_readable(coeffs),
             "points and coeffs must be host pointers");
  return eq_accumulate_device(w, nv, points, coeffs, npts, as_stream(stream), true);
}
