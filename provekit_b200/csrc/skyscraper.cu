// skyscraper.cu -- Skyscraper hashing and the Merkle commit on the device:
//   pkg_skyscraper_compress_many  simple::compress_many (skyscraper/core/src/simple.rs:3-9)
//   pkg_skyscraper_hash_many      SkyscraperHashEngine::hash_many
//                                 (provekit/common/src/skyscraper/whir.rs:42-100)
//   pkg_merkle_tree[_fr]          the binary tree WHIR builds from hash_many
//                                 (leaves: hash_many(leaf_size); nodes: hash_many(64))
//   pkg_skyscraper_pow_solve      generic::solve (skyscraper/core/src/generic.rs:42-71)
//   pkg_whir_commit               RS encode + Merkle tree of one polynomial
//
// One thread owns one compression chain (a leaf's left fold, or one node);
// 32-byte chunks are read as two 128-bit vector loads.  Folds run 128 messages
// at a time with their reductions on the tensor cores (sky_tc.cuh).  Levels
// above kSubtreeMax nodes take one launch each; below it one launch reduces
// 256-node subtrees per CTA by eight levels.
#include <algorithm>
#include <cstring>

#include "fr.cuh"
#include "ntt_internal.cuh"
#include "host_stage.cuh"
#include "internal.cuh"
#include "pk_common.cuh"
#include "reduce.cuh"
#include "rs_internal.cuh"
#include "skyscraper.cuh"
#include "sky_tc.cuh"

namespace pk {

// Plain loads, as everywhere in kernels of launch_early: the previous kernel may
// still be writing when they start, and read-only loads (ld.global.nc) are not
// ordered after griddepcontrol.wait.
__device__ __forceinline__ Fr load_raw(const uint8_t* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 a = q[0], b = q[1];
  Fr r;
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w;
  r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
  return r;
}

__device__ __forceinline__ void store_raw(uint8_t* p, const Fr& x) {
  uint4* q = reinterpret_cast<uint4*>(p);
  q[0] = make_uint4(x.v[0], x.v[1], x.v[2], x.v[3]);
  q[1] = make_uint4(x.v[4], x.v[5], x.v[6], x.v[7]);
}

// ---- compress_many / hash_many -------------------------------------------
__global__ void compress_many_kernel(const uint8_t* __restrict__ in, size_t n,
                                     uint8_t* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    Fr l = load_raw(in + 64 * i), r = load_raw(in + 64 * i + 32);
    store_raw(out + 32 * i, sky_compress(l, r));
  }
}

// Leaves straight from an Fr codeword: leaf i = row i (fr_per_leaf
// consecutive Fr).  Canonical encoding converts each Montgomery element
// (x*2^256 -> x) before hashing; Montgomery encoding hashes the raw limbs.
// A one-element leaf is the element itself (hash_many(32) copies).
// For the leaves that tiles do not pay for (tc_wanted).
constexpr int kLeafMinCtas = 7;  // per SM: 72 registers
template <bool kCanonical>
__global__ void __launch_bounds__(128, kLeafMinCtas)
    leaf_fold_fr_kernel(const uint64_t* __restrict__ cw, size_t fr_per_leaf, size_t count,
                        uint8_t* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < count;
       i += (size_t)gridDim.x * blockDim.x) {
    const size_t base = i * fr_per_leaf;
    Fr acc = fr_load_ro(cw, base);
    if (kCanonical) acc = fr_from_mont(acc);
#pragma unroll 1
    for (size_t k = 1; k < fr_per_leaf; k++) {
      Fr e = fr_load_ro(cw, base + k);
      if (kCanonical) e = fr_from_mont(e);
      acc = sky_compress(acc, e);
    }
    store_raw(out + 32 * i, acc);
  }
}

// ---- the same on the tensor cores (sky_tc.cuh) ---------------------------
// A CTA takes one tile of skytc::kThreads messages; threads past the end work on
// the last one and store nothing.  (CTAs that stayed and took several tiles
// each did not finish together, 25 of 32 warps were active on average: 2^20
// leaves of 16 Fr 2.42 ms against 2.21 then.)
struct ByteMessages {  // chunks of 32 bytes, hashed as they are
  static constexpr bool kMont = false;
  const uint8_t* in;
  size_t size;
  __device__ __forceinline__ Fr first(size_t i) const { return skytc::reduce_any(load_raw(in + i * size)); }
  __device__ __forceinline__ Fr at(size_t i, size_t k) const { return load_raw(in + i * size + 32 * k); }
};
template <bool kCanonical>
struct CodewordRows {  // rows of Fr, in canonical form or as their Montgomery limbs
  static constexpr bool kMont = kCanonical;
  const uint64_t* cw;
  size_t fr_per_leaf;
  __device__ __forceinline__ Fr first(size_t i) const {
    const Fr x = fr_load(cw, i * fr_per_leaf);
    return kCanonical ? fr_from_mont(x) : skytc::reduce_any(x);
  }
  __device__ __forceinline__ Fr at(size_t i, size_t k) const {
    return fr_load(cw, i * fr_per_leaf + k);
  }
};

// Left fold of `chunks` >= 2 chunks of each message.
template <class Messages>
__global__ void __launch_bounds__(skytc::kThreads, skytc::kMinCtas)
    fold_tc_kernel(const Messages msgs, size_t chunks, size_t count, uint8_t* out) {
  __shared__ skytc::Shared sh;
  skytc::SkyTile tile;
  tile.open(sh);
  const size_t i = (size_t)blockIdx.x * skytc::kThreads + threadIdx.x;
  const size_t row = i < count ? i : count - 1;
  Fr acc = msgs.first(row);
#pragma unroll 1
  for (size_t k = 1; k < chunks; k++)
    acc = tile.compress<Messages::kMont>(acc, msgs.at(row, k));
  if (i < count) store_raw(out + 32 * i, fr_reduce_once(acc));
  tile.close();
}

// Folds of three or more chunks always run here: 6.1 us per compression of a
// chain and 2.3 us to set up (5 where that does not run beside the previous
// kernel), against 8 and 2.5 in sky_compress.  A single
// compression each (two chunks) pays from above 2^15 messages on: 2^14 take
// 12.7 us here and 12.6 there, 2^16 20.9 and 24.8.
constexpr size_t kTcMinPairs = (size_t(1) << 15) + 1;
static bool tc_wanted(size_t count, size_t chunks) {
  return chunks >= 3 || (chunks == 2 && count >= kTcMinPairs);
}

template <class Messages>
static int fold_tc(const Messages& msgs, size_t chunks, size_t count, uint8_t* out,
                   cudaStream_t s) {
  const size_t tiles = (count + skytc::kThreads - 1) / skytc::kThreads;
  PK_REQUIRE(tiles <= 0x7fffffffu, "%zu messages exceed one launch", count);
  PK_CUDA(launch_early(fold_tc_kernel<Messages>, (unsigned)tiles, skytc::kThreads, 0, s, msgs,
                       chunks, count, out));
  PK_CHECK_LAUNCH("fold_tc_kernel");
  return PKG_OK;
}

// All the levels above `nodes` (a power of two <= kSubNodes) consecutive nodes
// of a level per CTA, in shared memory, each level's digests also written to
// their slots: the small levels are latency-bound (one compression's latency
// each, whatever their width), so they share one launch.  lvl: the level's
// first node; n: its nodes, the slots of the next level following them.
constexpr int kSubNodes = 2 * skytc::kThreads;
// A level of 2^16 nodes ends in one launch fewer this way (115 -> 113 us for
// the whole tree above it); from 2^17 on eight partly idle levels of that many
// CTAs cost what the launches save (134 and 135 us).
constexpr size_t kSubtreeMax = size_t(1) << 16;

__global__ void __launch_bounds__(skytc::kThreads, 5)
    merkle_subtree_kernel(uint8_t* lvl, size_t n, int nodes) {
  __shared__ skytc::Shared sh;
  __shared__ uint4 buf[2 * kSubNodes];
  skytc::SkyTile tile;
  tile.open(sh);
  const size_t c = blockIdx.x;  // this CTA's nodes: [c nodes, (c + 1) nodes)
  for (int i = threadIdx.x; i < 2 * nodes; i += blockDim.x)
    buf[i] = reinterpret_cast<const uint4*>(lvl + 32 * c * nodes)[i];
  __syncthreads();
  uint8_t* level = lvl;  // first node of the current level
  size_t level_n = n;
#pragma unroll 1
  for (int half = nodes / 2; half > 0; half /= 2) {
    const int i = threadIdx.x;
    Fr h;
    if ((int)tile.warp * 32 < half) {
      const int j = i < half ? i : 0;
      Fr a, b;
      const uint4 x0 = buf[4 * j], x1 = buf[4 * j + 1], y0 = buf[4 * j + 2], y1 = buf[4 * j + 3];
      a.v[0] = x0.x; a.v[1] = x0.y; a.v[2] = x0.z; a.v[3] = x0.w;
      a.v[4] = x1.x; a.v[5] = x1.y; a.v[6] = x1.z; a.v[7] = x1.w;
      b.v[0] = y0.x; b.v[1] = y0.y; b.v[2] = y0.z; b.v[3] = y0.w;
      b.v[4] = y1.x; b.v[5] = y1.y; b.v[6] = y1.z; b.v[7] = y1.w;
      h = fr_reduce_once(tile.compress<false>(skytc::reduce_any(a), b));
    } else {
      tile.sit_out();
    }
    __syncthreads();
    uint8_t* next = level + 32 * level_n;
    if (i < half) {
      buf[2 * i] = make_uint4(h.v[0], h.v[1], h.v[2], h.v[3]);
      buf[2 * i + 1] = make_uint4(h.v[4], h.v[5], h.v[6], h.v[7]);
      store_raw(next + 32 * (c * half + i), h);
    }
    __syncthreads();
    level = next;
    level_n /= 2;
  }
  tile.close();
}

static int grid_for(size_t n, int threads) {
  size_t b = (n + threads - 1) / threads;
  size_t cap = (size_t)sm_count() * 64;
  return (int)std::max<size_t>(1, std::min(b, cap));
}

int compress_many_device(const uint8_t* in, size_t n, uint8_t* out, cudaStream_t s) {
  if (n == 0) return PKG_OK;
  PK_REQUIRE(in && out, "null pointer");
  PK_REQUIRE(aligned16(in) && aligned16(out), "device buffers must be 16-byte aligned");
  if (tc_wanted(n, 2)) return fold_tc(ByteMessages{in, 64}, 2, n, out, s);
  compress_many_kernel<<<grid_for(n, 128), 128, 0, s>>>(in, n, out);
  PK_CHECK_LAUNCH("compress_many_kernel");
  return PKG_OK;
}

int hash_many_device(size_t size, const uint8_t* in, size_t count, uint8_t* out, cudaStream_t s) {
  PK_REQUIRE(size > 0 && size % 32 == 0,
             "skyscraper: unsupported message size %zu (must be a positive multiple of 32)",
             size);
  if (count == 0) return PKG_OK;
  PK_REQUIRE(in && out, "null pointer");
  PK_REQUIRE(aligned16(in) && aligned16(out), "device buffers must be 16-byte aligned");
  if (size == 32) {
    PK_CUDA(cudaMemcpyAsync(out, in, 32 * count, cudaMemcpyDeviceToDevice, s));
    return PKG_OK;
  }
  if (size == 64) return compress_many_device(in, count, out, s);
  return fold_tc(ByteMessages{in, size}, size / 32, count, out, s);
}

// Internal levels above the leaf digests already in layers[0..n) (n a power
// of two): one launch per level while a level has more than kSubtreeMax
// nodes, then eight levels in subtrees of kSubNodes, until one node is left.
int merkle_levels_device(uint8_t* layers, size_t n, cudaStream_t s) {
  uint8_t* cur = layers;
  while (n > kSubtreeMax) {
    uint8_t* next = cur + 32 * n;
    const int rc = compress_many_device(cur, n / 2, next, s);
    if (rc) return rc;
    cur = next;
    n /= 2;
  }
  while (n > 1) {
    const int nodes = (int)std::min<size_t>(n, kSubNodes);
    PK_CUDA(launch_early(merkle_subtree_kernel, (unsigned)(n / nodes), skytc::kThreads, 0, s, cur,
                         n, nodes));
    PK_CHECK_LAUNCH("merkle_subtree_kernel");
    for (int k = nodes; k > 1; k /= 2) {
      cur += 32 * n;
      n /= 2;
    }
  }
  return PKG_OK;
}

int merkle_leaves_fr_device(const uint64_t* cw, size_t fr_per_leaf, size_t num_leaves,
                            int encoding, uint8_t* layers, cudaStream_t s) {
  PK_REQUIRE(is_pow2(num_leaves), "num_leaves %zu is not a power of two", num_leaves);
  PK_REQUIRE(fr_per_leaf >= 1, "fr_per_leaf must be >= 1");
  PK_REQUIRE(encoding == PKG_LEAF_CANONICAL || encoding == PKG_LEAF_MONTGOMERY,
             "unknown leaf encoding %d", encoding);
  PK_REQUIRE(cw && layers, "null pointer");
  PK_REQUIRE(aligned16(cw) && aligned16(layers), "device buffers must be 16-byte aligned");
  if (tc_wanted(num_leaves, fr_per_leaf))
    return encoding == PKG_LEAF_CANONICAL
               ? fold_tc(CodewordRows<true>{cw, fr_per_leaf}, fr_per_leaf, num_leaves, layers, s)
               : fold_tc(CodewordRows<false>{cw, fr_per_leaf}, fr_per_leaf, num_leaves, layers, s);
  int g = grid_for(num_leaves, 128);
  if (encoding == PKG_LEAF_CANONICAL)
    leaf_fold_fr_kernel<true><<<g, 128, 0, s>>>(cw, fr_per_leaf, num_leaves, layers);
  else
    leaf_fold_fr_kernel<false><<<g, 128, 0, s>>>(cw, fr_per_leaf, num_leaves, layers);
  PK_CHECK_LAUNCH("leaf_fold_fr_kernel");
  return PKG_OK;
}

int merkle_tree_fr_device(const uint64_t* cw, size_t fr_per_leaf, size_t num_leaves,
                          int encoding, uint8_t* layers, cudaStream_t s) {
  int rc = merkle_leaves_fr_device(cw, fr_per_leaf, num_leaves, encoding, layers, s);
  if (rc) return rc;
  return merkle_levels_device(layers, num_leaves, s);
}

// ---- PoW -----------------------------------------------------------------
// Candidate nonces base + 128 b .. base + 128 b + 127 in CTA b; kTile: as a tile
// (sky_tc.cuh).
// The CTA that takes the last ticket hands the smallest solution so far to the host
// (reduce.cuh's completion word) and leaves the ticket and *best as they were found.
template <bool kTile>
__global__ void __launch_bounds__(skytc::kThreads, kTile ? 8 : 1)
    pow_kernel(Fr challenge, Fr threshold, uint64_t base, unsigned long long* best, RedOut ro) {
  const uint64_t nonce = base + blockIdx.x * (uint64_t)skytc::kThreads + threadIdx.x;
  Fr r = fr_zero();
  r.v[0] = (uint32_t)nonce;
  r.v[1] = (uint32_t)(nonce >> 32);
  Fr h;
  if constexpr (kTile) {
    __shared__ skytc::Shared sh;
    skytc::SkyTile tile;
    tile.open(sh);
    h = fr_reduce_once(tile.compress<false>(skytc::reduce_any(challenge), r));
    tile.close();
  } else {
    h = sky_compress(challenge, r);
  }
  bool lt = false;
#pragma unroll
  for (int k = 7; k >= 0; k--) {  // less_than, arithmetic.rs:447-456
    if (h.v[k] != threshold.v[k]) {
      lt = h.v[k] < threshold.v[k];
      break;
    }
  }
  if (lt) atomicMin(best, (unsigned long long)nonce);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(ro.ticket, 1u) == gridDim.x - 1) {
      __threadfence();
      *reinterpret_cast<volatile unsigned long long*>(ro.out) = atomicExch(best, ~0ULL);
      announce(ro);
    }
  }
}

// The smallest nonce with compress(challenge, [nonce,0,0,0]) < threshold:
// batches of candidates in increasing order, starting small (a PoW of b
// bits needs about 2^b candidates) and growing four-fold, so the first
// batch that holds a solution holds the smallest one.
int pow_solve_device(const uint64_t challenge[4], const uint64_t threshold[4], cudaStream_t s,
                     uint64_t* nonce_out) {
  Fr c, t;
  memcpy(c.v, challenge, 32);
  memcpy(t.v, threshold, 32);
  bool thr_zero = true;
  for (int i = 0; i < 8; i++) thr_zero &= (t.v[i] == 0);
  PK_REQUIRE(!thr_zero, "threshold 0 admits no nonce");
  // the best nonce in the thread's own PoW word (all ones between searches; after
  // the fused reductions' partials, which it never overlaps): no pool allocation per PoW
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  const unsigned long long none = ~0ULL;
  unsigned long long best = none;
  const uint64_t max_batch = uint64_t(1) << 22;
  uint64_t batch = uint64_t(1) << 13;
  for (uint64_t base = 0; best == none; base += batch, batch = std::min(batch * 4, max_batch)) {
    if (base > (uint64_t(1) << 62)) break;
    // the first batch is one compression's latency either way, and a tile's constants
    // and tensor memory cost more than it saves (proofs 2 us longer per search); a
    // 20-bit search that ends at nonce 582741 takes 324 us, 491 before the tiles
    const unsigned grid = (unsigned)(batch / skytc::kThreads);
    const RedOut ro = {fs.part, fs.ticket, fs.dev, fused_next_seq()};
    if (base == 0)
      pow_kernel<false><<<grid, skytc::kThreads, 0, s>>>(c, t, base, fs.pow, ro);
    else
      PK_CUDA(launch_early(pow_kernel<true>, grid, skytc::kThreads, 0, s, c, t, base, fs.pow, ro));
    PK_CHECK_LAUNCH("pow_kernel");
    if ((rc = fused_read(&best, fs, sizeof best, s))) return rc;
  }
  if (best == none) {
    set_last_error("no nonce found");
    return PKG_ERR_UNSUPPORTED;
  }
  *nonce_out = best;
  return PKG_OK;
}

}  // namespace pk

using namespace pk;

extern "C" int pkg_skyscraper_compress_many(const uint8_t* messages, size_t count,
                                            uint8_t* hashes, pkg_stream_t stream) {
  return compress_many_device(messages, count, hashes, as_stream(stream));
}

extern "C" int pkg_skyscraper_hash_many(size_t size, const uint8_t* input, size_t count,
                                        uint8_t* output, pkg_stream_t stream) {
  return hash_many_device(size, input, count, output, as_stream(stream));
}

extern "C" int pkg_host_skyscraper_hash_many(size_t size, const uint8_t* input, size_t count,
                                             uint8_t* output) {
  PK_REQUIRE(size > 0 && size % 32 == 0,
             "skyscraper: unsupported message size %zu (must be a positive multiple of 32)",
             size);
  if (count == 0) return PKG_OK;
  PK_REQUIRE(input && output, "null pointer");
  const size_t in_span = (size * count + 255) & ~size_t(255);
  HostStager& hs = HostStager::current();
  std::lock_guard<std::mutex> lk(hs.mutex());
  uint8_t* ws = nullptr;
  int rc = hs.workspace(in_span + 32 * count, &ws);
  if (rc) return rc;
  rc = hs.h2d(ws, input, size * count);
  if (rc) return rc;
  rc = hash_many_device(size, ws, count, ws + in_span, hs.stream());
  if (rc) return rc;
  rc = hs.d2h(output, ws + in_span, 32 * count);
  if (rc) return rc;
  PK_CUDA(cudaStreamSynchronize(hs.stream()));
  return PKG_OK;
}

extern "C" int pkg_merkle_tree(const uint8_t* leaves, size_t leaf_size, size_t num_leaves,
                               uint8_t* layers, pkg_stream_t stream) {
  PK_REQUIRE(is_pow2(num_leaves), "num_leaves %zu is not a power of two", num_leaves);
  cudaStream_t s = as_stream(stream);
  int rc = hash_many_device(leaf_size, leaves, num_leaves, layers, s);
  if (rc) return rc;
  return merkle_levels_device(layers, num_leaves, s);
}

extern "C" int pkg_merkle_tree_fr(const uint64_t* codeword, size_t fr_per_leaf,
                                  size_t num_leaves, int leaf_encoding, uint8_t* layers,
                                  pkg_stream_t stream) {
  return merkle_tree_fr_device(codeword, fr_per_leaf, num_leaves, leaf_encoding, layers,
                               as_stream(stream));
}

extern "C" int pkg_merkle_leaves_fr(const uint64_t* codeword, size_t fr_per_leaf,
                                    size_t num_leaves, int leaf_encoding, uint8_t* layers,
                                    pkg_stream_t stream) {
  return merkle_leaves_fr_device(codeword, fr_per_leaf, num_leaves, leaf_encoding, layers,
                                 as_stream(stream));
}

extern "C" int pkg_merkle_levels(uint8_t* layers, size_t num_leaves, pkg_stream_t stream) {
  PK_REQUIRE(is_pow2(num_leaves), "num_leaves %zu is not a power of two", num_leaves);
  PK_REQUIRE(layers && aligned16(layers), "layers must be a 16-byte aligned device pointer");
  return merkle_levels_device(layers, num_leaves, as_stream(stream));
}

extern "C" int pkg_whir_commit(const uint64_t* coeffs, size_t num_coeffs,
                               unsigned folding_factor, unsigned log_inv_rate,
                               const uint64_t* masks, size_t mask_len, int leaf_encoding,
                               uint64_t* codeword_out, uint8_t* layers_out,
                               pkg_stream_t stream) {
  PK_REQUIRE(folding_factor <= 12 && log_inv_rate <= 28, "unsupported folding factor / rate");
  size_t M = size_t(1) << folding_factor;
  PK_REQUIRE(is_pow2(num_coeffs) && num_coeffs >= M,
             "num_coeffs %zu must be a power of two >= 2^folding_factor", num_coeffs);
  size_t L = num_coeffs / M;
  PK_REQUIRE((L << log_inv_rate) <= (size_t(1) << 28),
             "codeword of %zu << %u rows exceeds the largest NTT order 2^28", L, log_inv_rate);
  size_t cw_len = L << log_inv_rate;
  cudaStream_t s = as_stream(stream);
  int rc = rs_encode_device(coeffs, M, L, masks, mask_len, cw_len, codeword_out, s);
  if (rc) return rc;
  return merkle_tree_fr_device(codeword_out, M, cw_len, leaf_encoding, layers_out, s);
}

extern "C" int pkg_skyscraper_pow_solve(const uint64_t challenge[4], const uint64_t threshold[4],
                                        uint64_t* nonce_out) {
  PK_REQUIRE(challenge && threshold && nonce_out, "null pointer");
  cudaStream_t s = nullptr;
  PK_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  const int rc = pow_solve_device(challenge, threshold, s, nonce_out);
  cudaStreamDestroy(s);
  return rc;
}
