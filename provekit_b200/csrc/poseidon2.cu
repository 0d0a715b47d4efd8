// poseidon2.cu -- BN254 Poseidon2, t = 4, rf = 8, rp = 56, on the device:
//   pkg_poseidon2_permutation_many  poseidon2_permutation (poseidon2/src/permutation.rs:134-177)
//   pkg_poseidon2_hash_many         poseidon2_hash (poseidon2/src/hash.rs:17-47)
// One thread per permutation; state and constants in Montgomery form.  The
// constant tables come from the reference's poseidon2/src/constants.rs via
// gen_poseidon2_constants.py and are copied to __constant__ memory once per
// device.
#include <cstring>
#include <mutex>
#include <vector>

#include "fr.cuh"
#include "fr_host.hpp"
#include "pk_common.cuh"
#include "poseidon2_t4_constants.h"
#include "tc_reduce.cuh"

namespace pk {

// One permutation per thread, 128 at a time, every reduction on the tensor
// cores (tc_reduce.cuh).  A partial round is two squares, a product and the
// internal matrix; the matrix is linear, so it is applied to the product
// before that is reduced: each new state element is one sum over the bytes of
// the product's words and of the other three elements, against residues that
// include the matrix entry (7 K blocks), and the product itself is never
// reduced.  The external matrix is one more such sum over the four elements'
// bytes against multiples of 1.  s[1..3] live in tensor memory through the
// partial rounds.  128 columns per CTA, 4 CTAs per SM:
//     0..31, 32..63   two sums at a time
//     64..95          a square's or product's words, or four elements
//     96..119         s[1], s[2], s[3]
// Per partial round 184 64-bit multiply-adds instead of 840: 200003 hashes of 3
// elements take 0.68 ms against 1.64 ms with one thread's products on the
// integer pipe.  Bound by the multiplier and by latency between the phases.
constexpr uint32_t kA = 64, kV = 96, kP2Columns = 128;
constexpr int kP2Ctas = 4;

// K blocks of the constants
enum : int {
  kSq = 0,      // 0..3: words 0..7, 8..15, 1..8, 9..14 of a square
  kOne = 1,     // multiples of an element: 1 (the same as words 8..15) ..
  kTimes3 = 4,  // .. 3, 4, 5, 6, 7
  kTimes4,
  kTimes5,
  kTimes6,
  kTimes7,
  kWord9,       // words 9..14 of a product and its carries
  kD0,          // kD0..kD0 + 3: a product times d0 + 1
  kDi = kD0 + 4,  // kDi + i - 1: an element times di + 1, i = 1..3
  kP2Blocks = kDi + 3
};
using P2Image = tc::Image<kP2Blocks>;

__constant__ uint64_t kP2Rc[64][4][4];
__device__ P2Image kP2Image;
__constant__ uint64_t kP2DiagPlus1[3][4];  // Montgomery d1 + 1 .. d3 + 1, and ..
__constant__ uint64_t kP2D0Plus1[4];       // .. d0 + 1, for a warp that is alone

static std::mutex g_p2_mu;
static std::vector<char> g_p2_ready;

// K bytes [4 at, 4 (at + words)) of a block: v 2^(32 first + 8 i) mod p
static void p2_image_words(P2Image& im, int block, int at, int first, int words, const HostFr& v) {
  HostFr x = v;
  for (int i = 0; i < 32 * first; i++) x = HostFr::add(x, x);
  for (int i = 0; i < 4 * words; i++) {
    for (int n = 0; n < 32; n++)
      tc::image_put(im, block, n, 4 * at + i, (uint32_t)(x.l[n / 8] >> (8 * (n % 8))) & 0xff);
    for (int b = 0; b < 8; b++) x = HostFr::add(x, x);
  }
}

static void p2_make_image(P2Image& im) {
  memset(&im, 0, sizeof im);
  const uint64_t one_limbs[4] = {1, 0, 0, 0};
  const HostFr one = HostFr::from_limbs(one_limbs);
  const HostFr rinv = HostFr::mul(one, one);  // 2^-256
  p2_image_words(im, kSq, 0, 0, 8, rinv);
  p2_image_words(im, kSq + 1, 0, 8, 8, rinv);
  p2_image_words(im, kSq + 2, 0, 1, 8, rinv);
  p2_image_words(im, kSq + 3, 0, 9, 6, rinv);
  const int times[] = {3, 4, 5, 6, 7};
  for (int i = 0; i < 5; i++)
    for (int k = 0; k < 32; k++) tc::image_put(im, kTimes3 + i, k, k, (uint32_t)times[i]);
  const HostFr d0 = HostFr::add(HostFr::from_limbs(POSEIDON2_T4_DIAG[0]), one);
  const HostFr d0r = HostFr::mul(d0, one);
  p2_image_words(im, kD0, 0, 0, 8, d0r);
  p2_image_words(im, kD0 + 1, 0, 8, 8, d0r);
  p2_image_words(im, kD0 + 2, 0, 1, 8, d0r);
  p2_image_words(im, kWord9, 0, 9, 6, rinv);
  p2_image_words(im, kD0 + 3, 0, 9, 6, d0r);
  for (int b : {(int)kWord9, (int)kD0 + 3}) {  // the carries: byte i has the weight of word 9 + i
    P2Image one_word;
    for (int i = 0; i < 7; i++) {
      memset(&one_word, 0, sizeof one_word);
      p2_image_words(one_word, 0, 0, 9 + i, 1, b == kWord9 ? rinv : d0r);
      for (int n = 0; n < 32; n++) {
        const int off = (n / 8) * 128 + (n % 8) * 16;
        tc::image_put(im, b, n, 24 + i, (one_word.w[off / 4] >> (8 * (off % 4))) & 0xff);
      }
    }
  }
  for (int i = 1; i < 4; i++)
    p2_image_words(im, kDi + i - 1, 0, 0, 8,
                   HostFr::add(HostFr::from_limbs(POSEIDON2_T4_DIAG[i]), one));
}

static int p2_upload() {
  int dev = 0;
  PK_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_p2_mu);
  if ((int)g_p2_ready.size() <= dev) g_p2_ready.resize(dev + 1, 0);
  if (!g_p2_ready[dev]) {
    static P2Image image;
    p2_make_image(image);
    PK_CUDA(cudaMemcpyToSymbol(kP2Rc, POSEIDON2_T4_RC_MONT, sizeof kP2Rc));
    PK_CUDA(cudaMemcpyToSymbol(kP2Image, &image, sizeof image));
    HostFr dp[4];
    for (int i = 0; i < 4; i++)
      dp[i] = HostFr::add(HostFr::from_limbs(POSEIDON2_T4_DIAG_MONT[i]), HostFr::one());
    PK_CUDA(cudaMemcpyToSymbol(kP2D0Plus1, dp[0].l, 32));
    for (int i = 1; i < 4; i++)
      PK_CUDA(cudaMemcpyToSymbol(kP2DiagPlus1, dp[i].l, 32, 32 * (size_t)(i - 1)));
    g_p2_ready[dev] = 1;
  }
  return PKG_OK;
}

__device__ __forceinline__ Fr p2_const(const uint64_t* c) {
  Fr r;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    r.v[2 * i] = (uint32_t)c[i];
    r.v[2 * i + 1] = (uint32_t)(c[i] >> 32);
  }
  return r;
}

struct P2Shared {
  alignas(128) uint4 image[kP2Blocks * tc::kBlockBytes / 16];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
};

// matrix_multiplication_4x4 (permutation.rs:101-120) without the tensor cores
static __device__ __noinline__ void p2_ext_alone(Fr* s) {
  for (int i = 0; i < 4; i++) s[i] = fr_reduce_once(fr_reduce_once(s[i]));
  Fr t0 = fr_add(s[0], s[1]);
  Fr t1 = fr_add(s[2], s[3]);
  Fr t2 = fr_add(fr_add(s[1], s[1]), t1);
  Fr t3 = fr_add(fr_add(s[3], s[3]), t0);
  Fr t4 = fr_add(t1, t1);
  t4 = fr_add(fr_add(t4, t4), t3);
  Fr t5 = fr_add(t0, t0);
  t5 = fr_add(fr_add(t5, t5), t2);
  s[0] = fr_add(t3, t5);
  s[1] = t5;
  s[2] = fr_add(t2, t4);
  s[3] = t4;
}
// internal_m_multiplication (permutation.rs:122-127) of (a b, s1, s2, s3)
static __device__ __noinline__ void p2_int_alone(const Fr a, const Fr b, Fr* s) {
  s[0] = fr_mul(fr_reduce_once(a), b);
  for (int i = 1; i < 4; i++) s[i] = fr_reduce_once(s[i]);
  const Fr sum = fr_add(fr_add(s[0], s[1]), fr_add(s[2], s[3]));
  s[0] = fr_sub(fr_add(fr_mul(s[0], p2_const(kP2D0Plus1)), sum), s[0]);
  for (int i = 1; i < 4; i++)
    s[i] = fr_sub(fr_add(fr_mul(s[i], p2_const(kP2DiagPlus1[i - 1])), sum), s[i]);
}
static __device__ __noinline__ Fr p2_sqr_alone(const Fr x) { return fr_sqr(fr_reduce_once(x)); }
static __device__ __noinline__ Fr p2_mul_alone(const Fr a, const Fr b) {
  return fr_mul(fr_reduce_once(a), fr_reduce_once(b));
}

struct P2Tile : tc::TileOf<kP2Columns> {
  // the sum at D columns d as an element below 1.1 p
  __device__ __forceinline__ Fr sum(uint32_t d) const {
    uint32_t c[32];
    tc::tmem_ld32(tmem + d, c);
    return tc::columns_reduce(c);
  }
  // x^2 for x < 2^255
  __device__ __forceinline__ Fr square(const Fr& x) {
    tc::put_square(tmem + kA, x);
    start([&] {
#pragma unroll
      for (int i = 0; i < 4; i++) block(0, kA + 8 * i, kSq + i, i > 0);
    });
    join();
    Fr r = sum(0);
    if (alone) r = p2_sqr_alone(x);
    __syncwarp();
    return r;
  }
  __device__ __forceinline__ Fr mul(const Fr& a, const Fr& b) {
    tc::put_product(tmem + kA, a, b);
    start([&] {
#pragma unroll
      for (int i = 0; i < 4; i++) block(0, kA + 8 * i, i < 3 ? kSq + i : kWord9, i > 0);
    });
    join();
    Fr r = sum(0);
    if (alone) r = p2_mul_alone(a, b);
    __syncwarp();
    return r;
  }
  __device__ __forceinline__ Fr sbox(const Fr& x) {  // x^5
    const Fr x2 = square(x);
    return mul(square(x2), x);
  }

  // The external matrix, rows (5 7 1 3) (4 6 1 1) (1 3 5 7) (1 1 4 6).
  __device__ __forceinline__ void external(Fr (&s)[4]) {
#pragma unroll
    for (int i = 0; i < 4; i++) tc::tmem_st8(tmem + kA + 8 * i, s[i].v);
    start([&] {
      block(0, kA, kTimes5, false);
      block(0, kA + 8, kTimes7, true);
      block(0, kA + 16, kOne, true);
      block(0, kA + 24, kTimes3, true);
      block(32, kA, kTimes4, false);
      block(32, kA + 8, kTimes6, true);
      block(32, kA + 16, kOne, true);
      block(32, kA + 24, kOne, true);
    });
    join();
    const Fr y0 = sum(0), y1 = sum(32);
    start([&] {
      block(0, kA, kOne, false);
      block(0, kA + 8, kTimes3, true);
      block(0, kA + 16, kTimes5, true);
      block(0, kA + 24, kTimes7, true);
      block(32, kA, kOne, false);
      block(32, kA + 8, kOne, true);
      block(32, kA + 16, kTimes4, true);
      block(32, kA + 24, kTimes6, true);
    });
    join();
    const Fr y2 = sum(0), y3 = sum(32);
    if (alone) {
      p2_ext_alone(s);
    } else {
      s[0] = y0;
      s[1] = y1;
      s[2] = y2;
      s[3] = y3;
    }
    __syncwarp();
  }

  // A row of the internal matrix on (the product in A, the three elements in V).
  __device__ __forceinline__ void internal_rows(uint32_t d, int row) const {
#pragma unroll
    for (int i = 0; i < 4; i++)
      block(d, kA + 8 * i, row == 0 ? kD0 + i : (i < 3 ? kSq + i : kWord9), i > 0);
#pragma unroll
    for (int i = 1; i < 4; i++)
      block(d, kV + 8 * (i - 1), i == row ? kDi + i - 1 : kOne, true);
  }
  // (a b, V) through the internal matrix: returns the new s[0], V updated.
  __device__ __forceinline__ Fr product_internal(const Fr& a, const Fr& b) {
    tc::put_product(tmem + kA, a, b);
    start([&] {
      internal_rows(0, 0);
      internal_rows(32, 1);
    });
    join();
    Fr y0 = sum(0), y1 = sum(32);
    start([&] {
      internal_rows(0, 2);
      internal_rows(32, 3);
    });
    join();
    Fr y2 = sum(0), y3 = sum(32);
    if (alone) {
      Fr s[4];
#pragma unroll
      for (int i = 1; i < 4; i++) tc::tmem_ld8(tmem + kV + 8 * (i - 1), s[i].v);
      p2_int_alone(a, b, s);
      y0 = s[0];
      y1 = s[1];
      y2 = s[2];
      y3 = s[3];
    }
    __syncwarp();
    tc::tmem_st8(tmem + kV, y1.v);
    tc::tmem_st8(tmem + kV + 8, y2.v);
    tc::tmem_st8(tmem + kV + 16, y3.v);
    return y0;
  }

  __device__ __forceinline__ Fr add_rc(const Fr& x, int round, int i) const {
    return fr_add_raw(x, p2_const(kP2Rc[round][i]).v);
  }
  __device__ __forceinline__ void full_rounds(Fr (&s)[4], int from) {
#pragma unroll 1
    for (int r = from; r < from + 4; r++) {
#pragma unroll 1
      for (int i = 0; i < 4; i++) {  // the state turns, so that one sbox serves all
        const Fr y = sbox(add_rc(s[0], r, i));
        s[0] = s[1];
        s[1] = s[2];
        s[2] = s[3];
        s[3] = y;
      }
      external(s);
    }
  }
  // s[i] < 2^255; results below 1.1 p
  __device__ __forceinline__ void permute(Fr (&s)[4]) {
    external(s);
    full_rounds(s, 0);
#pragma unroll
    for (int i = 1; i < 4; i++) tc::tmem_st8(tmem + kV + 8 * (i - 1), s[i].v);
#pragma unroll 1
    for (int r = 4; r < 60; r++) {
      const Fr x = add_rc(s[0], r, 0);
      const Fr x2 = square(x);
      s[0] = product_internal(square(x2), x);
    }
    tc::tmem_written();  // V's last writes, before they are read
#pragma unroll
    for (int i = 1; i < 4; i++) tc::tmem_ld8(tmem + kV + 8 * (i - 1), s[i].v);
    full_rounds(s, 60);
  }
};

__global__ void __launch_bounds__(tc::kThreads, kP2Ctas)
    p2_permutation_kernel(uint64_t* __restrict__ states, size_t n) {
  __shared__ P2Shared sh;
  P2Tile tile;
  tile.open(sh, kP2Image);
  const size_t i = (size_t)blockIdx.x * tc::kThreads + threadIdx.x;
  const size_t at = i < n ? i : n - 1;
  Fr s[4];
#pragma unroll
  for (int k = 0; k < 4; k++) s[k] = fr_load(states, 4 * at + k);
  __syncthreads();  // the last state is read by others before it is written
  tile.permute(s);
  if (i < n)
#pragma unroll
    for (int k = 0; k < 4; k++) fr_store(states, 4 * i + k, fr_reduce_once(s[k]));
  tile.close();
}

// Sponge of poseidon2_hash (hash.rs:17-47): rate 3, state[3] = len * 2^64.
__global__ void __launch_bounds__(tc::kThreads, kP2Ctas)
    p2_hash_kernel(const uint64_t* __restrict__ in, size_t len, size_t n, Fr iv,
                   uint64_t* __restrict__ out) {
  __shared__ P2Shared sh;
  P2Tile tile;
  tile.open(sh, kP2Image);
  const size_t i = (size_t)blockIdx.x * tc::kThreads + threadIdx.x;
  const size_t at = i < n ? i : n - 1;
  Fr s[4] = {fr_zero(), fr_zero(), fr_zero(), iv};
  size_t k = 0;
#pragma unroll 1
  do {
#pragma unroll
    for (int j = 0; j < 3; j++)
      if (k + j < len) s[j] = fr_add_raw(s[j], fr_load_ro(in, at * len + k + j).v);
    tile.permute(s);
    k += 3;
  } while (k < len);
  if (i < n) fr_store(out, i, fr_reduce_once(s[0]));
  tile.close();
}

static unsigned p2_grid(size_t n) { return (unsigned)((n + tc::kThreads - 1) / tc::kThreads); }

}  // namespace pk

using namespace pk;

extern "C" int pkg_poseidon2_permutation_many(uint64_t* states, size_t n, pkg_stream_t stream) {
  if (n == 0) return PKG_OK;
  PK_REQUIRE(states && aligned16(states), "states must be a 16-byte aligned device pointer");
  int rc = p2_upload();
  if (rc) return rc;
  p2_permutation_kernel<<<p2_grid(n), tc::kThreads, 0, as_stream(stream)>>>(states, n);
  PK_CHECK_LAUNCH("p2_permutation_kernel");
  return PKG_OK;
}

extern "C" int pkg_poseidon2_hash_many(const uint64_t* inputs, size_t len, size_t n, uint64_t* out,
                                       pkg_stream_t stream) {
  if (n == 0) return PKG_OK;
  PK_REQUIRE(out && aligned16(out) && (len == 0 || (inputs && aligned16(inputs))),
             "null or unaligned device pointer");
  int rc = p2_upload();
  if (rc) return rc;
  HostFr iv = HostFr::mul(HostFr::from_u64(len), HostFr::to_mont(HostFr::from_limbs(
                                                        std::vector<uint64_t>{0, 1, 0, 0}.data())));
  Fr ivd;
  memcpy(ivd.v, iv.l, 32);
  p2_hash_kernel<<<p2_grid(n), tc::kThreads, 0, as_stream(stream)>>>(inputs, len, n, ivd, out);
  PK_CHECK_LAUNCH("p2_hash_kernel");
  return PKG_OK;
}
