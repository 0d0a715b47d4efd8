// tc_reduce.cuh -- Montgomery reductions of 128 threads at a time on the tensor
// cores.
//
// A Montgomery reduction is linear in the bytes of what it reduces,
//     T 2^-256 = sum_k T_k (2^(8k-256) mod p),
// with the same constants for every element, so it is a matrix product: row =
// element (M = 128, one per thread), K = bytes of T, column n = byte n of the
// constants (N = 32).  tcgen05.mma kind::i8 (u8 x u8 -> s32) does it exactly:
// a column of 64 bytes with full residues is below 2^22, the other bytes add
// theirs as they are.  What is left on the integer pipe is the product itself,
// adding the 32 columns up to two 8-word numbers and a top word (assemble), and
// one quotient step over these (8 of the reduction's 64 64-bit multiply-adds).
//
// The sum is linear, so the product's two accumulators (even and odd word
// offsets, see fr.cuh) are never added: both go in as they are, the odd one
// against constants for its own offsets, and so does anything else that has a
// weight, carries and additive constants among them.  A and D live in tensor
// memory: thread i writes its bytes to lane i (tcgen05.st) and reads its 32
// columns back (tcgen05.ld); shared memory holds only the constants.  Columns
// of tensor memory with one product:
//     0..31   D
//     32..47  even accumulator E, words 0..15   (K blocks 0 and 1)
//     48..61  odd accumulator O, words 1..14    (K blocks 2 and 3)
//     62, 63  the caller's                      (K block 3)
#pragma once
#include "fr.cuh"
#include "fr_sum.cuh"

namespace pk {
namespace tc {

constexpr int kThreads = 128;      // one MMA tile: 128 elements
constexpr int kMaxCtas = 8;        // CTAs per SM: 8 x 64 of the 512 columns
constexpr int kBlockBytes = 1024;  // a K block: 32 columns x 32 bytes

constexpr uint64_t kP64[4] = {0x43e1f593f0000001ULL, 0x2833e84879b97091ULL, 0xb85045b68181585dULL,
                              0x30644e72e131a029ULL};
// 2^-256 mod p
constexpr uint64_t kRinv64[4] = {0xdc5ba0056db1194eULL, 0x090ef5a9e111ec87ULL,
                                 0xc8260de4aeb85d5dULL, 0x15ebf95182c5551cULL};

// residue[e] = the bytes of 2^(8e - 256) mod p; from e = 32 on the power itself
struct Residues {
  uint8_t byte[64][32];
};
constexpr Residues make_residues() {
  Residues r{};
  uint64_t v[4] = {kRinv64[0], kRinv64[1], kRinv64[2], kRinv64[3]};
  for (int e = 0; e < 32; e++) {
    for (int n = 0; n < 32; n++) r.byte[e][n] = (uint8_t)(v[n / 8] >> (8 * (n % 8)));
    for (int b = 0; b < 8; b++) {  // v = 2 v mod p
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
  for (int e = 32; e < 64; e++) r.byte[e][e - 32] = 1;
  return r;
}

// K blocks as tcgen05's K-major operand without swizzle: 8 x 16-byte core
// matrices, K halves 512 bytes apart, 8-column groups 128 bytes apart.
template <int kBlocks>
struct Image {
  uint32_t w[kBlocks * kBlockBytes / 4];
};
template <int kBlocks>
constexpr void image_put(Image<kBlocks>& im, int block, int n, int k, uint32_t byte) {
  const int off = block * kBlockBytes + (k / 16) * 512 + (n / 8) * 128 + (n % 8) * 16 + k % 16;
  im.w[off / 4] |= byte << (8 * (off % 4));
}
// K bytes [4 at, 4 (at + words)) of a block: words first.. of a product
template <int kBlocks>
constexpr void image_words(Image<kBlocks>& im, const Residues& r, int block, int at, int first,
                           int words) {
  for (int i = 0; i < 4 * words; i++)
    for (int n = 0; n < 32; n++) image_put(im, block, n, 4 * at + i, r.byte[4 * first + i][n]);
}
// Blocks 0..2 of every image.
template <int kBlocks>
constexpr void image_accumulators(Image<kBlocks>& im, const Residues& r) {
  image_words(im, r, 0, 0, 0, 8);
  image_words(im, r, 1, 0, 8, 8);
  image_words(im, r, 2, 0, 1, 8);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// kind::i8: s32 accumulators, unsigned bytes, K-major, N = 32, M = 128
constexpr uint32_t kInstr = (2u << 4) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

// sum c[n] 2^(8n) = x + z + top 2^256 for columns below 2^23: c[4j] + c[4j+1] 2^8
// is below 2^32 and is word j of x as it is; the other two columns make the
// same, 16 bits up, as z.
__device__ __forceinline__ void assemble(const uint32_t* c, uint32_t* x, uint32_t* z,
                                         uint32_t& top) {
  uint32_t y[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    x[j] = c[4 * j] + (c[4 * j + 1] << 8);
    y[j] = c[4 * j + 2] + (c[4 * j + 3] << 8);
  }
  z[0] = y[0] << 16;
#pragma unroll
  for (int j = 1; j < 8; j++) z[j] = __funnelshift_l(y[j - 1], y[j], 16);
  top = y[7] >> 16;
}

// The element that the columns hold, below 1.1 p.
__device__ __forceinline__ Fr columns_reduce(const uint32_t* c) {
  uint32_t x[8], z[8], top;
  assemble(c, x, z, top);
  return quotient_sum(x, z, nullptr, top);
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
__device__ __forceinline__ void tmem_ld8(uint32_t t, uint32_t* c) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]), "=r"(c[4]), "=r"(c[5]), "=r"(c[6]),
        "=r"(c[7])
      : "r"(t)
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

// Turns of a wait for an MMA (which takes well under one).
constexpr int kWaitTries = 1 << 16;
// Whether this thread takes a wait for one that ran out: an expression, which a
// test's build of the library sets so that some or all warps go on alone.
#ifndef PK_TILE_GIVES_UP
#define PK_TILE_GIVES_UP false
#endif

// The CTA's tensor memory, constants and barrier.  All kThreads threads call
// every member, together.
template <uint32_t kColumns>
struct TileOf {
  uint32_t cols;   // the CTA's columns of tensor memory
  uint32_t tmem;   // this warp's lanes of them
  uint32_t warp;
  uint32_t image;  // shared address of the constants
  uint32_t mbar;   // shared address of the MMA completion barrier
  uint32_t phase;
  // 0, or 2 + the parity of a phase: the wait for it ran out, and this warp reduces
  // without the tensor cores from then on (the same in all lanes).  Warp 0, which
  // issues the MMAs, then issues no more of them; the waits of the others run out
  // after it, each once.
  uint32_t alone;

  // Shared: image (16-byte aligned, as long as src), mbar, tmem.  open() is
  // begin() and ready(); what touches neither tensor memory nor the other
  // threads' data may stand between them, beside the allocation.
  //
  // The order of three steps keeps launch_early (pk_common.cuh) from closing a
  // circle over tensor memory, whatever the kernels' registers allow beside
  // each other and whoever's kernels they are:
  //   wait for the previous kernel, then allocate: a CTA that waits for another
  //     kernel holds no columns that this other kernel may still need;
  //   allocate, then let the next kernel start: once its CTAs can take columns,
  //     every CTA of this kernel has its own.
  // A CTA that waits in the allocation therefore waits only for CTAs that hold
  // everything they need.  Constants and barrier are set up before the wait,
  // beside the previous kernel.  (Allocated before the wait as well, the encode of
  // 12 x 5003 elements, whose second pass starts eight CTAs per SM at once, took
  // 51.8 us instead of 55.0 and a small commitment 126.0 instead of 127.1; but a
  // caller's kernel that triggers its dependents before it allocates could then
  // wait for good.)
  template <class Shared, int kBlocks>
  __device__ __forceinline__ void begin(Shared& sh, const Image<kBlocks>& src) {
    image = smem_addr(sh.image);
    mbar = smem_addr(&sh.mbar);
    phase = 0;
    alone = 0;
    const uint4* from = reinterpret_cast<const uint4*>(src.w);
    for (int i = threadIdx.x; i < kBlocks * kBlockBytes / 16; i += kThreads)
      sh.image[i] = __ldg(from + i);
    if (threadIdx.x == 0)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMA reads the constants
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x < 32) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_addr(&sh.tmem)),
                   "n"(kColumns)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  template <class Shared>
  __device__ __forceinline__ void ready(Shared& sh) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    tmem_after_sync();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    cols = __shfl_sync(0xffffffffu, sh.tmem, 0);
    warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    tmem = cols + (warp << 21);  // lane 32 * warp in bits 16..31
  }
  template <class Shared, int kBlocks>
  __device__ __forceinline__ void open(Shared& sh, const Image<kBlocks>& src) {
    begin(sh, src);
    ready(sh);
  }

  __device__ __forceinline__ void close() {
    if (warp == 0 && alone) wait(alone & 1);  // its last MMA may still be running
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    tmem_after_sync();
    if (threadIdx.x < 32)
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(cols),
                   "n"(kColumns));
  }

  // The MMA of the phase with this parity has completed; false when the wait
  // ran out.
  __device__ __forceinline__ bool wait(uint32_t parity) const {
    for (int i = 0; i < kWaitTries; i++) {
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

  // A is written: reduce it.  issue() (one thread) adds K blocks with block().
  template <class Issue>
  __device__ __forceinline__ void start(Issue&& issue) {
    tmem_written();
    cta_sync();
    if (warp == 0 && !alone && elect_lane()) {
      tmem_after_sync();
      issue();
      asm volatile(
          "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
          : "memory");
    }
  }
  // D at column d (+)= A's K block at column a x block of the constants
  __device__ __forceinline__ void block(uint32_t d, uint32_t a, int image_block,
                                        bool accumulate) const {
    mma(cols + d, cols + a, image, image_block, accumulate);
  }
  // The MMAs of start() are done, or the warp is alone from here on.  Warp 0
  // starts its next MMA only after this one, so at most one is in flight and
  // its parity names it.  (With phase kept instead where the warp is alone,
  // commitments of 2^20 took 1 % longer.)
  __device__ __forceinline__ void join() {
    if (!alone && __any_sync(0xffffffffu, !wait(phase) || PK_TILE_GIVES_UP)) alone = 2 + phase;
    phase ^= 1;
    tmem_after_sync();
  }
};

// 64 columns: D and one product.
struct Tile : TileOf<64> {
  // D (+)= A's K block kblock x block of the constants
  __device__ __forceinline__ void block(int kblock, int image_block) const {
    TileOf<64>::block(0, 32 + 8 * kblock, image_block, kblock > 0);
  }
  // D's columns; meaningless where the warp is alone.
  __device__ __forceinline__ void finish(uint32_t* c) {
    join();
    tmem_ld32(tmem, c);
  }
};

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

// a b = sum E[i] 2^(32 i) + sum O[i] 2^(32 i) + sum C[i] 2^(32 (9 + i)) for any
// 256-bit a, b; E: words 0..15, O: words 1..14, C: seven carries, one a byte.
// A chain runs up from the lowest word where its products are, and ends on a
// pair that no earlier one wrote where there is one; where there is none its
// carry is kept as a term of its own, for the reduction to weigh.
__device__ __forceinline__ void product_words(const uint32_t* a, const uint32_t* b, uint32_t* E,
                                              uint32_t* O, uint32_t* C) {
  PK_NEW_PAIR(E, 0, a[0], b[0]);
  PK_NEW_PAIR(E, 2, a[0], b[2]);
  PK_NEW_PAIR(E, 4, a[0], b[4]);
  PK_NEW_PAIR(E, 6, a[0], b[6]);
  PK_CHAIN4(E, 2, a[1], b[1], a[1], b[3], a[1], b[5], a[1], b[7]);
  PK_CHAIN5(E, 2, a[2], b[0], a[2], b[2], a[2], b[4], a[2], b[6], a[3], b[7]);
  PK_CHAIN5(E, 4, a[3], b[1], a[3], b[3], a[3], b[5], a[4], b[6], a[5], b[7]);
  PK_CHAIN6(E, 4, a[4], b[0], a[4], b[2], a[4], b[4], a[5], b[5], a[6], b[6], a[7], b[7]);
  uint32_t c9, c10, c11, c12, c13, c14, c15;
  PK_CARRY4(E, 6, a[5], b[1], a[5], b[3], a[6], b[4], a[7], b[5], c14);
  PK_CARRY3(E, 6, a[6], b[0], a[6], b[2], a[7], b[3], c12);
  PK_CARRY1(E, 8, a[7], b[1], c10);
  PK_NEW_PAIR(O, 1, a[0], b[1]);
  PK_NEW_PAIR(O, 3, a[0], b[3]);
  PK_NEW_PAIR(O, 5, a[0], b[5]);
  PK_NEW_PAIR(O, 7, a[0], b[7]);
  PK_CHAIN5(O, 1, a[1], b[0], a[1], b[2], a[1], b[4], a[1], b[6], a[2], b[7]);
  PK_CHAIN5(O, 3, a[2], b[1], a[2], b[3], a[2], b[5], a[3], b[6], a[4], b[7]);
  PK_CHAIN6(O, 3, a[3], b[0], a[3], b[2], a[3], b[4], a[4], b[5], a[5], b[6], a[6], b[7]);
  PK_CARRY5(O, 5, a[4], b[1], a[4], b[3], a[5], b[4], a[6], b[5], a[7], b[6], c15);
  PK_CARRY4(O, 5, a[5], b[0], a[5], b[2], a[6], b[3], a[7], b[4], c13);
  PK_CARRY2(O, 7, a[6], b[1], a[7], b[2], c11);
  PK_CARRY1(O, 7, a[7], b[0], c9);
  C[0] = (c9 | (c10 << 8)) | ((c11 << 16) | (c12 << 24));
  C[1] = c13 | (c14 << 8) | (c15 << 16);
}

// The constants of product_words: K block 3 with the carries after O's words.
constexpr int kProductBlocks = 4;
constexpr Image<kProductBlocks> make_product_image() {
  Image<kProductBlocks> im{};
  const Residues r = make_residues();
  image_accumulators(im, r);
  image_words(im, r, 3, 0, 9, 6);
  for (int w = 9; w < 16; w++) image_put(im, 3, 4 * (w - 8), 24 + w - 9, 1);
  return im;
}
static __device__ const Image<kProductBlocks> kProductImage = make_product_image();

// The words of a square or a product to tensor memory, at the columns of A.
__device__ __forceinline__ void put_square(uint32_t A, const Fr& x) {
  uint32_t E[16], O[16];
  square_words(x.v, E, O);
  tmem_st8(A + 16, O + 1);
  tmem_st4(A + 24, O + 9);
  tmem_st2(A + 28, O + 13);
  tmem_st16(A, E);
}
__device__ __forceinline__ void put_product(uint32_t A, const Fr& a, const Fr& b) {
  uint32_t E[16], O[16], t[8];
  product_words(a.v, b.v, E, O, t + 6);
#pragma unroll
  for (int i = 0; i < 6; i++) t[i] = O[9 + i];
  tmem_st8(A + 16, O + 1);
  tmem_st16(A, E);
  tmem_st8(A + 24, t);
}

struct ProductShared {
  alignas(128) uint4 image[kProductBlocks * kBlockBytes / 16];
  alignas(8) uint64_t mbar;
  uint32_t tmem;
};

// Montgomery products through a Tile opened with kProductImage: start() after
// the operands are known, finish() for a b 2^-256 mod p below 1.1 p
// (meaningless where the warp is alone); any 256-bit a, b.
struct ProductTile : Tile {
  __device__ __forceinline__ void start(const Fr& a, const Fr& b) {
    put_product(tmem + 32, a, b);
    Tile::start([&] {
      block(0, 0);
      block(1, 1);
      block(2, 2);
      block(3, 3);
    });
  }
  __device__ __forceinline__ Fr finish() {
    uint32_t c[32];
    Tile::finish(c);
    return columns_reduce(c);
  }
};

}  // namespace tc
}  // namespace pk
