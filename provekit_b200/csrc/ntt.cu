// ntt.cu -- BN254 Fr NTT for sm_100a: the ntt crate's ntt_nr / intt_rn
// (ntt/src/ntt.rs:105-348) behind pkg_ntt_nr / pkg_intt_rn.
//
// Algorithm: the same radix-2 DIT, normal-in / bit-reversed-out transform as
// interleaved_ntt_nr (ntt/src/ntt.rs:150-248).  At global stage t there are
// 2^t groups; group k pairs element i with i + half and multiplies the odd
// element by roots[k] from the bit-reversed twiddle table
// (init_roots_reverse_ordered, ntt/src/ntt.rs:275-306).  Stages are fused into
// passes of K <= 8 stages: a pass owns independent 2^K-point sub-transforms
// ("lines": fixed top t row bits and fixed low row bits), stages each line in
// shared memory, and runs its K stages there, so global memory is read and
// written once per pass instead of once per stage.  Exact modular arithmetic
// makes the output bit-identical to the stage-by-stage CPU order.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

#include "fr.cuh"
#include "fr_host.hpp"
#include "ntt_internal.cuh"
#include "ntt_tile.cuh"
#include "host_stage.cuh"
#include "pk_common.cuh"
#include "tc_reduce.cuh"

namespace pk {

// ---------------------------------------------------------------------------
// Device-resident twiddle table (the NTTEngine, ntt/src/ntt.rs:24-95): one
// grow-only table per device, roots[bitrev(i)] = w_order^i for i < order/2.
// By the prefix property (ntt/src/ntt.rs:515-522) the first m/2 entries of
// the table for any order >= m are the order-m table.
// ---------------------------------------------------------------------------
struct RootsTable {
  uint64_t* d = nullptr;
  size_t order = 0;
  std::vector<uint64_t*> retired;
};
static std::mutex g_roots_mu;
static std::vector<RootsTable> g_roots;

__global__ void roots_kernel(uint64_t* __restrict__ roots, const uint64_t* __restrict__ w_lo,
                             const uint64_t* __restrict__ w_hi, int log_half, int s) {
  size_t n = size_t(1) << log_half;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    Fr lo = fr_load_ro(w_lo, i & ((size_t(1) << s) - 1));
    Fr hi = fr_load_ro(w_hi, i >> s);
    Fr w = fr_mul(lo, hi);
    size_t r = __brevll((unsigned long long)i) >> (64 - log_half);
    fr_store(roots, r, w);
  }
}

int roots_reserve(size_t order, const uint64_t** out) {
  if (order < 1024) order = 1024;  // NTTEngine::new() size (ntt/src/ntt.rs:30-33)
  if (!is_pow2(order) || order > (size_t(1) << 28)) {
    set_last_error("twiddle order %zu is not a power of two <= 2^28", order);
    return PKG_ERR_INVALID_ARGUMENT;
  }
  int dev = 0;
  PK_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_roots_mu);
  if ((int)g_roots.size() <= dev) g_roots.resize(dev + 1);
  RootsTable& tab = g_roots[dev];
  if (tab.order >= order) {
    *out = tab.d;
    return PKG_OK;
  }
  // Grow: build the order-`order` table.  Superseded tables stay allocated
  // (kept in `retired`) so that kernels already enqueued on any stream, or
  // pointers already handed to another thread, stay valid; by the prefix
  // property their total size is below the new table's.
  int log_half = log2_exact(order / 2);
  int s = (log_half + 1) / 2;
  size_t nlo = size_t(1) << s, nhi = size_t(1) << (log_half - s);
  HostFr w = HostFr::root_of_unity(order);
  std::vector<uint64_t> h_lo(4 * nlo), h_hi(4 * nhi);
  HostFr acc = HostFr::one();
  for (size_t i = 0; i < nlo; i++) {
    memcpy(&h_lo[4 * i], acc.l, 32);
    acc = HostFr::mul(acc, w);
  }
  HostFr step = acc;  // w^(2^s)
  acc = HostFr::one();
  for (size_t i = 0; i < nhi; i++) {
    memcpy(&h_hi[4 * i], acc.l, 32);
    acc = HostFr::mul(acc, step);
  }
  uint64_t *d_new = nullptr, *d_lo = nullptr, *d_hi = nullptr;
  PK_CUDA(cudaMalloc(&d_new, 32 * (order / 2)));
  cudaError_t e = cudaMalloc(&d_lo, 32 * nlo);
  if (e == cudaSuccess) e = cudaMalloc(&d_hi, 32 * nhi);
  if (e == cudaSuccess) e = cudaMemcpy(d_lo, h_lo.data(), 32 * nlo, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d_hi, h_hi.data(), 32 * nhi, cudaMemcpyHostToDevice);
  // Built on a private stream and waited for, so the table is complete before
  // any caller (on any stream) can see the new pointer.
  cudaStream_t bs = nullptr;
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&bs, cudaStreamNonBlocking);
  if (e == cudaSuccess) {
    int blocks = (int)std::min<size_t>((order / 2 + 255) / 256, (size_t)sm_count() * 16);
    roots_kernel<<<blocks, 256, 0, bs>>>(d_new, d_lo, d_hi, log_half, s);
    e = cudaGetLastError();
    count_launch();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(bs);
  if (bs) cudaStreamDestroy(bs);
  cudaFree(d_lo);
  cudaFree(d_hi);
  if (e != cudaSuccess) {
    cudaFree(d_new);
    return cuda_status(e, "twiddle table");
  }
  if (tab.d) tab.retired.push_back(tab.d);
  tab.d = d_new;
  tab.order = order;
  *out = tab.d;
  return PKG_OK;
}

// ---------------------------------------------------------------------------
// Pass kernel.
//
// Shared memory holds the CTA's E elements as two planes of 16-byte halves
// (plane 0: bytes 0-15 of every element, plane 1: bytes 16-31), so a warp
// touching consecutive elements reads consecutive 16-byte words.
//
// Row r of the transform (codeword position) has log2(N) bits.  A pass over
// global stages [t, t+K) splits r = (high : j : low) with high = top t bits,
// j = next K bits, low = remaining B bits.  With M interleaved columns, the
// element (r, c) sits at r*M + c; "line" = (high, u) with u = low*M + c in
// [0, U), U = 2^B * M, and line element j is at (high*2^K + j)*U + u.
// A CTA owns T consecutive lines.  Mode A (T divides U): the lines share
// `high` and are contiguous per j.  Mode B (U divides T, U a power of two):
// the CTA's lines cover a contiguous memory range.  Mode C (U no power of two):
// each line finds its own `high`, for passes in which mode A's T, at most the
// power-of-two part of U, would leave a tile fewer butterflies than threads.
// Stage s of the pass (global stage t+s) pairs j0 = grp*2h + pos with
// j0 + h (h = 2^(K-1-s)) and uses twiddle roots[(high << s) | grp].
//
// A CTA's 128 threads run a stage's butterflies 128 at a time, their products'
// reductions on the tensor cores (tc_reduce.cuh): 72 64-bit multiply-adds per
// product instead of 128.  Values stay below 5 p between stages and passes.
// Bound by the multiplier and by latency between its phases: 2^24 points take
// 2.86 ms (the multiplier 65-69 % busy, DRAM 13-18 %), with the whole product on
// the integer pipe 3.56 ms, with CTAs that stay for several tiles 3.30 ms, since
// they do not finish together.
// ---------------------------------------------------------------------------
// Where a transform's first pass reads its input.
enum : int { kFromData = 0, kFromEncode = 1, kFromReversed = 2 };

// Element g of the RS-encode layout (see NttSource).
__device__ __forceinline__ Fr encode_load(const NttSource& s, uint64_t g) {
  const uint64_t x = g % s.chunk;
  if (x < s.L * s.M) {
    const uint64_t row = x / s.M, col = x - row * s.M;
    return fr_load(s.messages, col * s.L + row);
  }
  if (x - s.L * s.M < s.mask_len) return fr_load(s.masks, x - s.L * s.M);
  return fr_zero();
}

// Most stages per pass: 8.  2^24 points take 2.89 ms as three 8-stage passes,
// 3.06 as four of 6; 9 (tiles of one line) save a pass at 2^17 and 2^18 points
// (40.5 against 43.2 us) but cost 5 % at 18 stages over 16 columns of 2^20.
constexpr int kPassStages = 8;
// Elements per CTA, log2: two batches of 128 butterflies a stage, or one below
// 2^21 elements, where the batch's latency counts: 2^19 points 94 us with one
// and 105 with two, 2^20 179 and 183, 2^21 352 and 341, 2^22 737 and 692.  Four: 757.
constexpr int kTileElems = 9, kSmallTileElems = 8;
constexpr uint64_t kSmallBelow = uint64_t(1) << 21;

// x 2^-k mod p for x < 5 p and 1 <= k <= 28, below 4 p: p is 1 mod 2^28, so
// (-x mod 2^k) p is what x lacks to a multiple of 2^k.
__device__ __forceinline__ Fr halve(const Fr& x, int k) {
  constexpr uint32_t P[8] = {PK_P0, PK_P1, PK_P2, PK_P3, PK_P4, PK_P5, PK_P6, PK_P7};
  const uint32_t m = (0u - x.v[0]) & ((1u << k) - 1);
  uint32_t E[8], O[8], S[9];
  fr_first_row(E, O, P, m);
#pragma unroll
  for (int i = 0; i < 8; i++) S[i] = E[i];
  S[8] = 0;
  const uint32_t odd[8] = {0, O[0], O[1], O[2], O[3], O[4], O[5], O[6]};
  tc::add9(S, odd);
  S[8] += O[7];
  tc::add9(S, x.v);
  Fr r;
#pragma unroll
  for (int i = 0; i < 8; i++) r.v[i] = __funnelshift_r(S[i], S[i + 1], k);
  return r;
}

// Index i of log_n bits, reversed.
__device__ __forceinline__ uint64_t reversed(uint64_t i, int log_n) {
  return __brevll(i) >> (64 - log_n);
}

struct PassShape {
  uint64_t U;  // lines per `high`
  int log_u, T, log_t, K;
  bool first;      // stage 0 of the pass is stage 0 of the transform: every twiddle is 1
  bool last;       // store fully reduced; other passes leave values below 5 p
  int inverse;     // last pass of an inverse over 2^inverse points, or 0
};

// kMode selects the mode at compile time.  In mode A every line of the CTA
// shares `high`, so stage s reads only the 2^s twiddles roots[(high << s) |
// grp], which stay in L1.
//
// kAhead, for grids that leave two CTAs per SM or fewer: a stage's twiddle is loaded
// during the stage before, with the registers that the missing CTAs leave (2^10 points
// 12.3 -> 11.1 us, 2^16 26.7 -> 24.7); larger grids hide the load behind other CTAs, and eight
// of them have no registers for it (2^24 2.85 -> 2.92 ms).
constexpr int kAheadCtas = 2;
template <int kSrc, int kMode, bool kAhead>
__global__ void __launch_bounds__(tc::kThreads, kAhead ? kAheadCtas : tc::kMaxCtas)
    ntt_pass_kernel(uint64_t* data, uint64_t* out, const uint64_t* __restrict__ roots,
                    const PassShape shape, const NttSource src) {
  extern __shared__ uint4 sm[];
  __shared__ tc::ProductShared sh;
  const int K = shape.K, T = shape.T, log_t = shape.log_t, log_u = shape.log_u;
  const int E = T << K;
  const uint64_t U = shape.U;
  tc::ProductTile tile;
  // kAhead: the loads run beside the allocation (inverse of 2^16 points 26.5 -> 24.6 us);
  // with 64 registers that makes the stages slower (2^24 2.86 -> 2.92 ms)
  if (kAhead)
    tile.begin(sh, tc::kProductImage);
  else
    tile.open(sh, tc::kProductImage);
  const uint64_t l0 = (uint64_t)blockIdx.x * T;
  uint64_t high_a = 0, u0 = 0;
  if (kMode == kModeA) {
    high_a = l0 / U;
    u0 = l0 - high_a * U;
  }
  // ---- load ----
  for (int e = threadIdx.x; e < E; e += tc::kThreads) {
    uint64_t g;
    int sidx;
    pass_index(kMode, e, K, T, log_t, log_u, U, l0, high_a, u0, &g, &sidx);
    if (kSrc != kFromData) {
      // reversed: the inverse's first permutation, v[bitrev((n - g) mod n)]
      const Fr v = kSrc == kFromEncode
                       ? encode_load(src, g)
                       : fr_load(src.messages, reversed((src.L - g) & (src.L - 1), (int)src.M));
      sm[sidx] = make_uint4(v.v[0], v.v[1], v.v[2], v.v[3]);
      sm[E + sidx] = make_uint4(v.v[4], v.v[5], v.v[6], v.v[7]);
    } else {
      const uint4* in = reinterpret_cast<const uint4*>(data + 4 * g);
      sm[sidx] = in[0];      // low 16 bytes: plane 0
      sm[E + sidx] = in[1];  // high 16 bytes: plane 1
    }
  }
  if (kAhead)
    tile.ready(sh);  // a barrier for the loads too
  else
    __syncthreads();
  tile_stages<kAhead>(tile, sm, kMode, K, T, log_t, log_u, U, l0, high_a, shape.first, roots);
  // ---- store ----
  for (int e = threadIdx.x; e < E; e += tc::kThreads) {
    uint64_t g;
    int sidx;
    pass_index(kMode, e, K, T, log_t, log_u, U, l0, high_a, u0, &g, &sidx);
    Fr v = tile_load(sm, E, sidx);
    if (shape.inverse) v = halve(v, shape.inverse);
    if (shape.last) v = fr_reduce_once(tc::reduce_any(v));
    fr_store(out, shape.inverse ? reversed(g, shape.inverse) : g, v);
  }
  tile.close();
}

using PassKernel = void (*)(uint64_t*, uint64_t*, const uint64_t*, PassShape, NttSource);
template <int kSrc, int kMode>
static PassKernel pass_kernel(bool ahead) {
  return ahead ? ntt_pass_kernel<kSrc, kMode, true> : ntt_pass_kernel<kSrc, kMode, false>;
}
template <int kSrc>
static PassKernel pass_kernel(int mode, bool ahead) {
  if (mode == kModeA) return pass_kernel<kSrc, kModeA>(ahead);
  if (kSrc == kFromReversed || mode == kModeB) return pass_kernel<kSrc, kModeB>(ahead);
  return pass_kernel<kSrc == kFromReversed ? kFromData : kSrc, kModeC>(ahead);  // one column: no mode C
}

static inline uint64_t pow2_part(uint64_t x) { return x & (~x + 1); }

// Run global stages [t_begin, t_end) of an N-point transform over M columns;
// t_end is the last stage.  inverse: the stages of an inverse transform, which
// reads and writes `inverse` in the inverse's orders (data is scratch between
// passes; src describes the reads).
static int run_stages(uint64_t* data, size_t N, size_t M, int t_begin, int t_end,
                      const uint64_t* roots, cudaStream_t stream, const NttSource* src,
                      uint64_t* inverse) {
  const int total = t_end - t_begin;
  if (total <= 0) return PKG_OK;
  const int npasses = (total + kPassStages - 1) / kPassStages;
  const int log_elems = N * M < kSmallBelow ? kSmallTileElems : kTileElems;
  // The last pass's lines are cut at the power-of-two part of M.  Where that leaves fewer
  // butterflies than a tile has threads, it takes all the stages it can: 2^18 points of
  // 3 columns take 225 us with a last pass of 6 stages (32 butterflies a tile) and 126
  // with one of 8.
  int last = total / npasses;
  if (!is_pow2(M) && (pow2_part(M) << last) < 2 * tc::kThreads) last = std::min(kPassStages, total);
  int t = t_begin;
  for (int pi = 0; pi < npasses; pi++) {
    const bool final_pass = pi == npasses - 1;
    const int before = total - last - (t - t_begin), left = npasses - 1 - pi;
    const int K = final_pass ? last : (before + left - 1) / left;
    const int B = log2_exact(N) - t - K;
    const uint64_t U = (uint64_t(1) << B) * M;
    const uint64_t num_lines = (uint64_t(1) << t) * U;
    uint64_t T = uint64_t(1) << (K >= log_elems ? 0 : log_elems - K);
    if (T > num_lines) T = pow2_part(num_lines);
    int mode = is_pow2(U) && U < T ? kModeB : kModeA;
    if (mode == kModeA && pow2_part(U) < T) {
      // the last stages of 33 columns of 2^12 points, one and two of them: 360 and 210 us
      // in mode A (2 and 4 elements a CTA), 8.7 and 10.4 in mode C; seven: 22.1 and 18.6
      if (t > 0 && (pow2_part(U) << K) < 2 * tc::kThreads && num_lines >> 32 == 0)
        mode = kModeC, T = std::min(T, pow2_part(num_lines));
      else
        T = pow2_part(U);
    }
    PassShape shape;
    shape.U = U;
    shape.log_u = mode == kModeB ? log2_exact(U) : 0;
    shape.T = (int)T;
    shape.log_t = log2_exact(T);
    shape.K = K;
    shape.first = t == 0;
    shape.last = final_pass;
    shape.inverse = inverse && shape.last ? log2_exact(N) : 0;
    const size_t smem = 32 * (T << K);
    const unsigned grid = (unsigned)(num_lines / T);
    NttSource s;
    memset(&s, 0, sizeof s);
    int kind = kFromData;
    if (src && pi == 0) {
      s = *src;
      kind = inverse ? kFromReversed : kFromEncode;
    }
    uint64_t* const out = inverse && shape.last ? inverse : data;
    const bool ahead = grid <= kAheadCtas * (unsigned)sm_count();
    const PassKernel fn = kind == kFromData     ? pass_kernel<kFromData>(mode, ahead)
                          : kind == kFromEncode ? pass_kernel<kFromEncode>(mode, ahead)
                                                : pass_kernel<kFromReversed>(mode, ahead);
    PK_CUDA(launch_early(fn, grid, tc::kThreads, smem, stream, data, out, roots, shape, s));
    PK_CHECK_LAUNCH("ntt_pass_kernel");
    t += K;
  }
  return PKG_OK;
}

int ntt_stages(uint64_t* data, size_t N, size_t M, int t_begin, int t_end, const uint64_t* roots,
               cudaStream_t stream, const NttSource* src) {
  return run_stages(data, N, M, t_begin, t_end, roots, stream, src, nullptr);
}

// Validation shared by the device and host forms (reference panics ->
// PKG_ERR_INVALID_ARGUMENT).  Returns 1 if there is nothing to do.
int ntt_validate(size_t len, size_t codeword_size, size_t num_groups, int* noop) {
  *noop = 0;
  if (codeword_size <= 1) {  // ntt/src/ntt.rs:161-163
    *noop = 1;
    return PKG_OK;
  }
  PK_REQUIRE(num_groups != 0 && len % num_groups == 0,
             "values.len() must be divisible by num_groups (len=%zu, num_groups=%zu)", len,
             num_groups);
  PK_REQUIRE(is_pow2(codeword_size), "codeword_size %zu is not a power of two", codeword_size);
  PK_REQUIRE(is_pow2(num_groups), "num_groups %zu is not a power of two", num_groups);
  PK_REQUIRE(len > 0 && len % codeword_size == 0,
             "len %zu is not a positive multiple of codeword_size %zu", len, codeword_size);
  PK_REQUIRE(codeword_size <= (size_t(1) << 28), "codeword_size %zu exceeds 2^28", codeword_size);
  if (num_groups >= codeword_size) *noop = 1;
  return PKG_OK;
}

int ntt_nr_device(uint64_t* values, size_t len, size_t codeword_size, size_t num_groups,
                  cudaStream_t stream) {
  int noop = 0;
  int rc = ntt_validate(len, codeword_size, num_groups, &noop);
  if (rc || noop) return rc;
  PK_REQUIRE(values != nullptr, "null values pointer");
  PK_REQUIRE(aligned16(values), "device buffers must be 16-byte aligned");
  const uint64_t* roots = nullptr;
  rc = roots_reserve(codeword_size, &roots);
  if (rc) return rc;
  size_t M = len / codeword_size;
  return ntt_stages(values, codeword_size, M, log2_exact(num_groups), log2_exact(codeword_size),
                    roots, stream);
}

int ntt_nr_from_source(uint64_t* out, size_t len, size_t codeword_size, size_t num_groups,
                       const NttSource& src, cudaStream_t stream) {
  int noop = 0;
  int rc = ntt_validate(len, codeword_size, num_groups, &noop);
  if (rc) return rc;
  PK_REQUIRE(!noop, "no transform stage to read the source");
  PK_REQUIRE(out != nullptr && aligned16(out), "null or unaligned output");
  const uint64_t* roots = nullptr;
  rc = roots_reserve(codeword_size, &roots);
  if (rc) return rc;
  return ntt_stages(out, codeword_size, len / codeword_size, log2_exact(num_groups),
                    log2_exact(codeword_size), roots, stream, &src);
}

// ---------------------------------------------------------------------------
// intt_rn: reverse_order -> values[1..].reverse() -> ntt_nr -> * n^-1 ->
// reverse_order (ntt/src/ntt.rs:326-348): the first pass reads
// v0[bitrev((n - i) mod n)], the last one stores v3[i] n^-1 at bitrev(i).  (As
// two gathers around the transform: 2^16 points 37.5 us; 2^k points' n^-1 is a
// shift, see halve.)
// ---------------------------------------------------------------------------
int intt_rn_device(uint64_t* values, size_t len, cudaStream_t stream) {
  PK_REQUIRE(is_pow2(len), "intt_rn length %zu is not a power of two", len);
  PK_REQUIRE(len <= (size_t(1) << 28), "intt_rn length %zu exceeds 2^28", len);
  PK_REQUIRE(values != nullptr, "null values pointer");
  PK_REQUIRE(aligned16(values), "device buffers must be 16-byte aligned");
  if (len == 1) return PKG_OK;  // both permutations and the scale are identities
  const uint64_t* roots = nullptr;
  int rc = roots_reserve(len, &roots);
  if (rc) return rc;
  const int log_n = log2_exact(len);
  NttSource src;
  memset(&src, 0, sizeof src);
  src.messages = values;
  src.L = len;
  src.M = (uint64_t)log_n;
  // one pass: one CTA holds every value before it stores the first
  static_assert(kPassStages <= kSmallTileElems, "a transform of one pass is one tile");
  Scratch tmp;
  uint64_t* between = values;
  if (log_n > kPassStages) {
    if ((rc = tmp.alloc(32 * len, stream))) return rc;
    between = static_cast<uint64_t*>(tmp.ptr);
  }
  return run_stages(between, len, 1, 0, log_n, roots, stream, &src, values);
}

}  // namespace pk

using namespace pk;

extern "C" int pkg_ntt_nr(uint64_t* values, size_t len, size_t codeword_size, size_t num_groups,
                          pkg_stream_t stream) {
  return ntt_nr_device(values, len, codeword_size, num_groups, as_stream(stream));
}

extern "C" int pkg_intt_rn(uint64_t* values, size_t len, pkg_stream_t stream) {
  return intt_rn_device(values, len, as_stream(stream));
}

extern "C" int pkg_ntt_engine_reserve(size_t order) {
  const uint64_t* r = nullptr;
  return roots_reserve(order, &r);
}

// In-place transform of a host slice through the host stager: one pipelined
// upload, the device transform on the stager's stream, one pipelined download.
static int host_transform(uint64_t* values, size_t len, size_t codeword_size,
                          size_t num_groups, bool inverse) {
  HostStager& hs = HostStager::current();
  std::lock_guard<std::mutex> lk(hs.mutex());
  uint8_t* ws = nullptr;
  int rc = hs.workspace(32 * len, &ws);
  if (rc) return rc;
  rc = hs.h2d(ws, values, 32 * len);
  if (rc) return rc;
  uint64_t* d = reinterpret_cast<uint64_t*>(ws);
  rc = inverse ? intt_rn_device(d, len, hs.stream())
               : ntt_nr_device(d, len, codeword_size, num_groups, hs.stream());
  if (rc) return rc;
  rc = hs.d2h(values, ws, 32 * len);
  if (rc) return rc;
  PK_CUDA(cudaStreamSynchronize(hs.stream()));
  return PKG_OK;
}

extern "C" int pkg_host_ntt_nr(uint64_t* values, size_t len, size_t codeword_size,
                               size_t num_groups) {
  int noop = 0;
  int rc = ntt_validate(len, codeword_size, num_groups, &noop);
  if (rc || noop) return rc;
  PK_REQUIRE(values != nullptr, "null values pointer");
  return host_transform(values, len, codeword_size, num_groups, false);
}

extern "C" int pkg_host_intt_rn(uint64_t* values, size_t len) {
  PK_REQUIRE(is_pow2(len), "intt_rn length %zu is not a power of two", len);
  PK_REQUIRE(values != nullptr, "null values pointer");
  return host_transform(values, len, len, 1, true);
}
