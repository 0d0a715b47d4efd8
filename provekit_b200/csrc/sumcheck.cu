// sumcheck.cu -- the Spartan side of the prover on the device:
//   pkg_spartan_round      one round of run_zk_sumcheck_prover's map-reduce
//                          (provekit/prover/src/whir_r1cs.rs:551-559 over
//                          sumcheck_fold_map_reduce, provekit/common/src/utils/sumcheck.rs:14-102)
//   pkg_spartan_sumcheck   the whole zk-sumcheck (whir_r1cs.rs:519-621), rounds
//                          on the device, round-polynomial bookkeeping and the
//                          transcript on the host
//   pkg_eq_hypercube       calculate_evaluations_over_boolean_hypercube_for_eq (sumcheck.rs:108-153)
//   pkg_spmv_csr           HydratedSparseMatrix * &[Fr] (sparse_matrix.rs:606-627)
//   pkg_csr_transpose      SparseMatrix::transpose (sparse_matrix.rs:409), as a counting sort
//   pkg_hadamard_pad       c = a o b padded with zeros (calculate_witness_bounds, sumcheck.rs:163-179)
//   pkg_dot                whir::algebra::dot (whir_r1cs.rs:614-617, 637, 650)
//   pkg_transcript_*       host Fiat-Shamir transcript stand-in (see the header)
//
// Reductions use the block-wide sums of reduce.cuh.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

#include "fr.cuh"
#include "fr_host.hpp"
#include "fr_lazy.cuh"
#include "internal.cuh"
#include "pk_common.cuh"
#include "reduce.cuh"
#include "sky_host.hpp"
#include "sumcheck_device.cuh"

namespace pk {


struct Tables4 {
  uint64_t* t[4];  // a, b, c, eq
};

// kFold: current size s = 4q, folded in place, then pairs (t[j], t[j+q]);
// !kFold: size s = 2q, pairs (t[j], t[j+q]).
template <bool kFold>
__global__ void __launch_bounds__(kRedThreads) spartan_round_kernel(Tables4 tabs, size_t q,
                                                                     Fr fold, const RedOut ro) {
  Fr acc[3] = {fr_zero(), fr_zero(), fr_zero()};
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < q;
       j += (size_t)gridDim.x * blockDim.x)
    spartan_pair<kFold>(tabs.t, j, q, fold, acc);
  block_finish<3>(acc, ro);
}

// The same with four lanes per pair.
template <bool kFold>
__global__ void __launch_bounds__(kQuadThreads) spartan_quad_kernel(Tables4 tabs, size_t q,
                                                                     Fr fold, const RedOut ro) {
  __shared__ FrShared sh[3];
  Fr sums[3];
  quad_sums(spartan_quads<kFold>(tabs.t, (size_t)blockIdx.x * kQuadPairs,
                                 (size_t)gridDim.x * kQuadPairs, q, fold, sh),
            sums);
  block_finish<3>(sums, ro);
}

// out[x] = prod_i (bit i of x, the top one first ? r_i : 1 - r_i) for x < n <= 2^nr.  A
// CTA takes `per` runs of 256 entries: the product over the last eight variables from a
// table of its own (itself products of two tables of 16), the one over the rest once per
// run, and a product of the two per entry.  Bound by those chains (about 14 products at
// 2^20 entries, eight at 2^14) and from 2^19 on by the products: 2^14 entries 27 -> 7 us,
// 2^20 40 -> 29 (a copy of r, two table kernels and one of products before).
constexpr int kEqMaxVars = 40;
constexpr int kEqRunVars = 8;
constexpr int kEqThreads = 256;
constexpr int kEqMaxRuns = kEqThreads / 2;
struct EqPoint {
  uint32_t r[kEqMaxVars][8];
};

// The factors of variables first .. first + k - 1 for the k low bits of x.
__device__ __forceinline__ Fr eq_product(const EqPoint& P, int first, int k, size_t x) {
  Fr acc = fr_one_mont();
#pragma unroll 1
  for (int i = 0; i < k; i++) {
    Fr f;
#pragma unroll
    for (int w = 0; w < 8; w++) f.v[w] = P.r[first + i][w];
    if (!((x >> (k - 1 - i)) & 1)) f = fr_sub(fr_one_mont(), f);
    acc = i ? fr_mul(acc, f) : f;
  }
  return acc;
}

__global__ void __launch_bounds__(kEqThreads) eq_hypercube_kernel(
    const __grid_constant__ EqPoint P, int nr, size_t n, int per, uint64_t* __restrict__ out) {
  __shared__ Fr high[kEqMaxRuns], part[32];
  const int t = threadIdx.x, low = nr < kEqRunVars ? nr : kEqRunVars, kb = low / 2, ka = low - kb;
  const size_t run0 = blockIdx.x * (size_t)per;
  if (t < 32) {
    const bool a = t < 16;
    if ((t & 15) < 1 << (a ? ka : kb))
      part[t] = eq_product(P, a ? nr - low : nr - kb, a ? ka : kb, (size_t)(t & 15));
  } else if (t >= kEqThreads - kEqMaxRuns && t - (kEqThreads - kEqMaxRuns) < per) {
    const int i = t - (kEqThreads - kEqMaxRuns);
    high[i] = eq_product(P, 0, nr - low, run0 + i);
  }
  __syncthreads();
  Fr mine = fr_zero();
  if (t < 1 << low) mine = fr_mul(part[t >> kb], part[16 + (t & ((1 << kb) - 1))]);
  for (int i = 0; i < per; i++) {
    const size_t x = (run0 + i) * kEqThreads + t;
    if (x < n) fr_store(out, x, fr_mul(high[i], mine));
  }
}

// Column indices >= num_cols are skipped and flagged in *err (the reference
// panics on them); the entry point turns the flag into an error status.
__global__ void spmv_csr_kernel(const uint64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
                                const uint64_t* __restrict__ vals, size_t num_rows, size_t num_cols,
                                const uint64_t* __restrict__ x, uint64_t* __restrict__ y,
                                uint32_t* __restrict__ err) {
  for (size_t row = blockIdx.x * (size_t)blockDim.x + threadIdx.x; row < num_rows;
       row += (size_t)gridDim.x * blockDim.x) {
    Fr acc = fr_zero();
    for (uint64_t k = row_ptr[row]; k < row_ptr[row + 1]; k++) {
      const uint32_t col = cols[k];
      if (col >= num_cols) {
        atomicOr(err, 1u);
        continue;
      }
      acc = fr_add(acc, fr_mul(fr_load_ro(vals, k), fr_load_ro(x, col)));
    }
    fr_store(y, row, acc);
  }
}

// The same product in two balanced passes, for large matrices whose row
// lengths vary (a transposed R1CS matrix: 0 to ~10 entries per witness
// column): one thread per nonzero forms vals[k] * x[cols[k]] into prod[k],
// then one thread per row adds its run of prod -- so a warp's Montgomery
// products no longer wait for its longest row.
__global__ void spmv_products_kernel(const uint32_t* __restrict__ cols,
                                     const uint64_t* __restrict__ vals, size_t nnz,
                                     size_t num_cols, const uint64_t* __restrict__ x,
                                     uint64_t* __restrict__ prod, uint32_t* __restrict__ err) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nnz;
       k += (size_t)gridDim.x * blockDim.x) {
    const uint32_t col = cols[k];
    Fr v = fr_zero();
    if (col >= num_cols)
      atomicOr(err, 1u);
    else
      v = fr_mul(fr_load_ro(vals, k), fr_load_ro(x, col));
    fr_store(prod, k, v);
  }
}

__global__ void spmv_rowsum_kernel(const uint64_t* __restrict__ row_ptr,
                                   const uint64_t* __restrict__ prod, size_t num_rows,
                                   uint64_t* __restrict__ y) {
  for (size_t row = blockIdx.x * (size_t)blockDim.x + threadIdx.x; row < num_rows;
       row += (size_t)gridDim.x * blockDim.x) {
    Fr acc = fr_zero();
    for (uint64_t k = row_ptr[row]; k < row_ptr[row + 1]; k++) acc = fr_add(acc, fr_load_ro(prod, k));
    fr_store(y, row, acc);
  }
}

// calculate_witness_bounds (sumcheck.rs:163-179) in one pass over the rows:
// a_i = <A_i, w>, b_i = <B_i, w>, c_i = a_i b_i for i < num_rows, and zeros
// up to the padded size (the three tables of the zk-sumcheck).  Column
// indices >= num_cols are skipped and flagged in *err.
__global__ void witness_bounds_kernel(const uint64_t* __restrict__ rpa,
                                      const uint32_t* __restrict__ ca,
                                      const uint64_t* __restrict__ va,
                                      const uint64_t* __restrict__ rpb,
                                      const uint32_t* __restrict__ cb,
                                      const uint64_t* __restrict__ vb, size_t num_rows,
                                      size_t num_cols, size_t padded,
                                      const uint64_t* __restrict__ w, uint64_t* __restrict__ ta,
                                      uint64_t* __restrict__ tb, uint64_t* __restrict__ tc,
                                      uint32_t* __restrict__ err) {
  for (size_t row = blockIdx.x * (size_t)blockDim.x + threadIdx.x; row < padded;
       row += (size_t)gridDim.x * blockDim.x) {
    Fr a = fr_zero(), b = fr_zero(), c = fr_zero();
    if (row < num_rows) {
      for (uint64_t k = rpa[row]; k < rpa[row + 1]; k++) {
        const uint32_t col = ca[k];
        if (col >= num_cols) {
          atomicOr(err, 1u);
          continue;
        }
        a = fr_add(a, fr_mul(fr_load_ro(va, k), fr_load_ro(w, col)));
      }
      for (uint64_t k = rpb[row]; k < rpb[row + 1]; k++) {
        const uint32_t col = cb[k];
        if (col >= num_cols) {
          atomicOr(err, 1u);
          continue;
        }
        b = fr_add(b, fr_mul(fr_load_ro(vb, k), fr_load_ro(w, col)));
      }
      c = fr_mul(a, b);
    }
    fr_store(ta, row, a);
    fr_store(tb, row, b);
    fr_store(tc, row, c);
  }
}

__global__ void hadamard_pad_kernel(const uint64_t* __restrict__ a, const uint64_t* __restrict__ b,
                                    size_t n, size_t padded, uint64_t* __restrict__ c) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < padded;
       i += (size_t)gridDim.x * blockDim.x)
    fr_store(c, i, i < n ? fr_mul(fr_load_ro(a, i), fr_load_ro(b, i)) : fr_zero());
}

// Several dot products in one launch, each over its own run of CTAs of `per` entries;
// the products of a thread are summed unreduced (fr_lazy.cuh).  The CTA that takes the
// last ticket (reduce.cuh) adds the CTAs' sums, a warp per dot product.  A proof's
// seven or eight at once (each of its covectors with the witness and with the mask
// polynomial) spare the launches and their tails, a read by the host, and the
// covectors' padding: proofs of 2^14, 300007 and 2^20 constraints 1800 -> 1721,
// 4750 -> 4528 and 11160 -> 10863 us.
struct DotBatch {
  int count;
  size_t per;
  DotJob job[kMaxDots];
  unsigned first[kMaxDots + 1];  // each job's CTAs: first[j] .. first[j + 1]
};

__global__ void __launch_bounds__(kRedThreads, 2) dots_kernel(const __grid_constant__ DotBatch J,
                                                              const RedOut ro) {
  int j = 0;
  while (j + 1 < J.count && blockIdx.x >= J.first[j + 1]) j++;
  const uint64_t* a = J.job[j].a;
  const uint64_t* b = J.job[j].b;
  const size_t start = (blockIdx.x - J.first[j]) * J.per;
  const size_t end = start + J.per < J.job[j].n ? start + J.per : J.job[j].n;
  Fr sum[1] = {fr_zero()};
  size_t i = start + threadIdx.x;
#pragma unroll 1
  while (i < end) {
    const size_t left = (end - i + kRedThreads - 1) / kRedThreads;
    const int terms = left < (size_t)lazy::kMaxTerms ? (int)left : lazy::kMaxTerms;
    lazy::Acc acc;
    acc.zero();
#pragma unroll 2
    for (int k = 0; k < terms; k++, i += kRedThreads)
      acc.mac(fr_load_ro(a, i), fr_load_ro(b, i));
    sum[0] = fr_add(sum[0], acc.finish());
  }
  block_sum<1>(sum);
  static_assert(kMaxDots <= kRedThreads / 32, "a warp per dot product");
  const int w = threadIdx.x >> 5;
  runs_finish(sum[0], ro, J.count, J.first[w], J.first[w + 1]);
}

// ---- CSR transpose: count, exclusive scan, scatter ------------------------
__global__ void csr_count_cols_kernel(const uint32_t* __restrict__ cols, size_t nnz,
                                      size_t num_cols, uint32_t* __restrict__ counts,
                                      uint32_t* __restrict__ err) {
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nnz;
       k += (size_t)gridDim.x * blockDim.x) {
    if (cols[k] >= num_cols) {
      atomicOr(err, 1u);
      continue;
    }
    atomicAdd(&counts[cols[k]], 1u);
  }
}

__global__ void csr_scatter_kernel(const uint64_t* __restrict__ row_ptr, const uint32_t* __restrict__ cols,
                                   const uint64_t* __restrict__ vals, size_t num_rows, size_t num_cols,
                                   unsigned long long* __restrict__ cursor,
                                   uint32_t* __restrict__ cols_t, uint64_t* __restrict__ vals_t) {
  for (size_t row = blockIdx.x * (size_t)blockDim.x + threadIdx.x; row < num_rows;
       row += (size_t)gridDim.x * blockDim.x) {
    for (uint64_t k = row_ptr[row]; k < row_ptr[row + 1]; k++) {
      if (cols[k] >= num_cols) continue;  // flagged by csr_count_cols_kernel
      unsigned long long pos = atomicAdd(&cursor[cols[k]], 1ull);
      cols_t[pos] = (uint32_t)row;
      fr_store(vals_t, pos, fr_load_ro(vals, k));
    }
  }
}

__global__ void widen_kernel(const uint32_t* __restrict__ in, size_t n, unsigned long long* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = in[i];
}


// One Spartan round on device tables; the round kernel writes 3 Fr (f0,
// f(-1), f(inf)) to out (the thread's fused slots, whose ticket it takes).
// part: >= round_grid(q) * 3 Fr of scratch.
int spartan_round_device(uint64_t* a, uint64_t* b, uint64_t* c, uint64_t* eq, size_t size,
                         const uint64_t* fold_host, uint64_t* part, uint64_t* out,
                         cudaStream_t s, unsigned* ticket) {
  Tables4 tabs = {{a, b, c, eq}};
  Fr f;
  memset(&f, 0, sizeof f);
  size_t q;
  int g;
  const RedOut ro = {part, ticket, out, ticket ? fused_next_seq() : 0u};
  if (fold_host) {
    memcpy(f.v, fold_host, 32);
    q = size / 4;
    g = round_grid(q);
    if (q <= kQuadMaxPairs)
      spartan_quad_kernel<true><<<g, kQuadThreads, 0, s>>>(tabs, q, f, ro);
    else
      spartan_round_kernel<true><<<g, kRedThreads, 0, s>>>(tabs, q, f, ro);
  } else {
    q = size / 2;
    g = round_grid(q);
    if (q <= kQuadMaxPairs)
      spartan_quad_kernel<false><<<g, kQuadThreads, 0, s>>>(tabs, q, f, ro);
    else
      spartan_round_kernel<false><<<g, kRedThreads, 0, s>>>(tabs, q, f, ro);
  }
  PK_CHECK_LAUNCH("spartan_round_kernel");
  return PKG_OK;
}

int eq_hypercube_device(const uint64_t* r_host, size_t nr, size_t num_entries, uint64_t* out,
                        cudaStream_t s, bool sync) {
  if (num_entries == 0) return PKG_OK;
  PK_REQUIRE(nr < 40 && num_entries <= (size_t(1) << nr), "num_entries %zu exceeds 2^%zu",
             num_entries, nr);
  PK_REQUIRE(out && aligned16(out), "out must be a 16-byte aligned device pointer");
  if (nr == 0) {  // the single entry 1: a copy takes 15 us with its wait, a launch 18
    const HostFr one = HostFr::one();
    PK_CUDA(cudaMemcpyAsync(out, one.l, 32, cudaMemcpyHostToDevice, s));
    if (sync) PK_CUDA(cudaStreamSynchronize(s));
    return PKG_OK;
  }
  EqPoint P;
  memset(&P, 0, sizeof P);
  memcpy(P.r, r_host, 32 * nr);
  const size_t runs = (num_entries + kEqThreads - 1) / kEqThreads, ctas = 4 * (size_t)sm_count();
  const int per = (int)std::min<size_t>(kEqMaxRuns, (runs + ctas - 1) / ctas);
  eq_hypercube_kernel<<<(unsigned)((runs + per - 1) / per), kEqThreads, 0, s>>>(
      P, (int)nr, num_entries, per, out);
  PK_CHECK_LAUNCH("eq_hypercube_kernel");
  if (sync) PK_CUDA(cudaStreamSynchronize(s));
  return PKG_OK;
}

// err: device word, zeroed by the caller before the launch.
int witness_bounds_device(const pkg_r1cs* r1cs, const uint64_t* w, size_t padded, uint64_t* ta,
                          uint64_t* tb, uint64_t* tc, uint32_t* err, cudaStream_t s) {
  if (padded == 0) return PKG_OK;
  PK_REQUIRE(aligned16(ta) && aligned16(tb) && aligned16(tc) && aligned16(w) &&
                 aligned16(r1cs->vals[0]) && aligned16(r1cs->vals[1]),
             "null or unaligned device pointer");
  witness_bounds_kernel<<<ew_grid(padded), 256, 0, s>>>(
      r1cs->row_ptr[0], r1cs->cols[0], r1cs->vals[0], r1cs->row_ptr[1], r1cs->cols[1],
      r1cs->vals[1], r1cs->num_constraints, r1cs->num_witnesses, padded, w, ta, tb, tc, err);
  PK_CHECK_LAUNCH("witness_bounds_kernel");
  return PKG_OK;
}

// Nonzeros from which the two balanced passes replace the one-row-per-thread
// kernel (below it the product temporary is not worth its traffic).
constexpr size_t kSpmvBalancedNnz = size_t(1) << 16;

// err: device word, zeroed by the caller before the launch.  nnz: the
// matrix's nonzero count (row_ptr[num_rows]), or 0 if the caller does not
// know it (one thread per row then).
int spmv_device(const uint64_t* row_ptr, const uint32_t* cols, const uint64_t* vals,
                size_t num_rows, size_t num_cols, const uint64_t* x, uint64_t* y, uint32_t* err,
                cudaStream_t s, size_t nnz) {
  if (num_rows == 0) return PKG_OK;
  PK_REQUIRE(row_ptr && y && aligned16(y) && aligned16(vals) && aligned16(x),
             "null or unaligned device pointer");
  // rows of at most ~one entry (a transposed C: one constraint per output
  // column) leave nothing to balance
  if (nnz < kSpmvBalancedNnz || nnz <= num_rows) {
    spmv_csr_kernel<<<ew_grid(num_rows), 256, 0, s>>>(row_ptr, cols, vals, num_rows, num_cols, x,
                                                     y, err);
    PK_CHECK_LAUNCH("spmv_csr_kernel");
    return PKG_OK;
  }
  Scratch tmp;
  int rc = tmp.alloc(32 * nnz, s);
  if (rc) return rc;
  uint64_t* prod = static_cast<uint64_t*>(tmp.ptr);
  spmv_products_kernel<<<ew_grid(nnz), 256, 0, s>>>(cols, vals, nnz, num_cols, x, prod, err);
  PK_CHECK_LAUNCH("spmv_products_kernel");
  spmv_rowsum_kernel<<<ew_grid(num_rows), 256, 0, s>>>(row_ptr, prod, num_rows, y);
  PK_CHECK_LAUNCH("spmv_rowsum_kernel");
  return PKG_OK;
}

static int read_err_flag(uint32_t* d_err, cudaStream_t s, const char* what) {
  uint32_t h = 0;
  PK_CUDA(cudaMemcpyAsync(&h, d_err, 4, cudaMemcpyDeviceToHost, s));
  PK_CUDA(cudaStreamSynchronize(s));
  if (h) {
    set_last_error("%s: column index out of range", what);
    return PKG_ERR_INVALID_ARGUMENT;
  }
  return PKG_OK;
}

int dots_device(const DotJob* jobs, int count, uint64_t* out, const FusedSlots& fs,
                cudaStream_t s) {
  PK_REQUIRE(count >= 1 && count <= kMaxDots, "%d dot products in one launch", count);
  DotBatch J;
  memset(&J, 0, sizeof J);
  J.count = count;
  size_t total = 0;
  for (int j = 0; j < count; j++) {
    J.job[j] = jobs[j];
    total += jobs[j].n;
  }
  // as many CTAs as are resident at once, at least an entry per thread
  const size_t share = (total + 2 * (size_t)sm_count() - 1) / (2 * (size_t)sm_count());
  J.per = std::max<size_t>(1, (share + kRedThreads - 1) / kRedThreads) * kRedThreads;
  unsigned ctas = 0;
  for (int j = 0; j < count; j++) {
    J.first[j] = ctas;
    ctas += (unsigned)((jobs[j].n + J.per - 1) / J.per);
  }
  for (int j = count; j <= kMaxDots; j++) J.first[j] = ctas;
  dots_kernel<<<std::max(1u, ctas), kRedThreads, 0, s>>>(
      J, RedOut{fs.part, fs.ticket, out, fused_next_seq()});
  PK_CHECK_LAUNCH("dots_kernel");
  return PKG_OK;
}

// ---- host transcript stand-in ------------------------------------------
struct HostTranscript {
  HostFr l, r;
  void init(const uint64_t domain[4]) {
    l = HostSky::reduce(HostFr::from_limbs(domain));
    r = HostFr::zero();
    HostSky::permute(l, r);
  }
  void absorb(const HostFr& x_mont) {
    l = HostFr::add(l, HostFr::from_mont(x_mont));
    HostSky::permute(l, r);
  }
  HostFr squeeze() {
    HostSky::permute(l, r);
    return HostFr::to_mont(l);
  }
};

static HostFr eval_cubic(const HostFr* c, const HostFr& x) {
  HostFr acc = HostFr::mul(x, c[3]);
  acc = HostFr::mul(HostFr::add(acc, c[2]), x);
  acc = HostFr::mul(HostFr::add(acc, c[1]), x);
  return HostFr::add(acc, c[0]);
}

// 1/2 in Montgomery form, inverted once (an inversion is ~400 products).
static const HostFr& half_mont() {
  static const HostFr h = HostFr::inv(HostFr::add(HostFr::one(), HostFr::one()));
  return h;
}

// g_i(0) + g_i(1) of one blinding cubic
static HostFr cubic_sum01(const HostFr* c) {
  return HostFr::add(eval_cubic(c, HostFr::zero()), eval_cubic(c, HostFr::one()));
}

// The coefficients of compute_blinding_coefficients_for_round for
// cf < n from its two sums: prefix = sum_{i < cf} g_i(alpha_i), suffix =
// sum_{i > cf} (g_i(0) + g_i(1)).
static void blinding_from_sums(const HostFr* g, size_t n, size_t cf, const HostFr& prefix,
                               const HostFr& suffix, HostFr res[4]) {
  HostFr pm = HostFr::one();
  for (size_t i = 0; i < n - 1 - cf; i++) pm = HostFr::add(pm, pm);
  HostFr sm = HostFr::mul(pm, half_mont());
  HostFr cst = HostFr::add(HostFr::mul(pm, prefix), HostFr::mul(sm, suffix));
  const HostFr* cur = g + 4 * cf;
  res[0] = HostFr::add(HostFr::mul(pm, cur[0]), cst);
  for (int k = 1; k < 4; k++) res[k] = HostFr::mul(pm, cur[k]);
}

// compute_blinding_coefficients_for_round (whir_r1cs.rs:427-492)
static void blinding_coeffs(const HostFr* g, size_t n, size_t compute_for, const HostFr* alphas,
                            HostFr out[4]) {
  bool all_fixed = false;
  size_t cf = compute_for;
  if (cf == n) {
    all_fixed = true;
    cf = n - 1;
  }
  HostFr prefix = HostFr::zero(), suffix = HostFr::zero();
  for (size_t i = 0; i < cf; i++) prefix = HostFr::add(prefix, eval_cubic(g + 4 * i, alphas[i]));
  for (size_t i = cf + 1; i < n; i++) suffix = HostFr::add(suffix, cubic_sum01(g + 4 * i));
  if (!all_fixed) {
    blinding_from_sums(g, n, cf, prefix, suffix, out);
    return;
  }
  HostFr pm = HostFr::one();
  for (size_t i = 0; i < n - 1 - cf; i++) pm = HostFr::add(pm, pm);
  HostFr sm = HostFr::mul(pm, half_mont());
  HostFr cst = HostFr::add(HostFr::mul(pm, prefix), HostFr::mul(sm, suffix));
  const HostFr* cur = g + 4 * cf;
  HostFr res[4] = {HostFr::add(HostFr::mul(pm, cur[0]), cst), HostFr::mul(pm, cur[1]),
                   HostFr::mul(pm, cur[2]), HostFr::mul(pm, cur[3])};
  if (all_fixed) {
    out[0] = eval_cubic(res, alphas[cf]);
    out[1] = out[2] = out[3] = HostFr::zero();
    return;
  }
  for (int k = 0; k < 4; k++) out[k] = res[k];
}

// Tables of at most this many entries finish their rounds on the host.
constexpr size_t kHostTailEntries = 64;

// spartan_round_kernel on host tables: with fold, bind the top variable
// first (t[j] += fold (t[j + size/2] - t[j])) and halve size; then the sums
// f(0), f(-1), f(inf) over the pairs (j, j + size/2) (whir_r1cs.rs:552-558),
// as canonical Montgomery limbs into out.
static void host_spartan_round(std::vector<HostFr> (&t)[4], size_t size, const HostFr* fold,
                               uint64_t out[12]) {
  if (fold) {
    const size_t h = size / 2;
    for (auto& v : t)
      for (size_t j = 0; j < h; j++) v[j] = HostFr::add(v[j], HostFr::mul(*fold, HostFr::sub(v[j + h], v[j])));
    size = h;
  }
  const size_t q = size / 2;
  HostFr f0 = HostFr::zero(), fm1 = HostFr::zero(), finf = HostFr::zero();
  for (size_t j = 0; j < q; j++) {
    const HostFr a0 = t[0][j], a1 = t[0][j + q], b0 = t[1][j], b1 = t[1][j + q];
    const HostFr c0 = t[2][j], c1 = t[2][j + q], e0 = t[3][j], e1 = t[3][j + q];
    f0 = HostFr::add(f0, HostFr::mul(e0, HostFr::sub(HostFr::mul(a0, b0), c0)));
    const HostFr a2 = HostFr::sub(HostFr::add(a0, a0), a1), b2 = HostFr::sub(HostFr::add(b0, b0), b1);
    const HostFr c2 = HostFr::sub(HostFr::add(c0, c0), c1), e2 = HostFr::sub(HostFr::add(e0, e0), e1);
    fm1 = HostFr::add(fm1, HostFr::mul(e2, HostFr::sub(HostFr::mul(a2, b2), c2)));
    finf = HostFr::add(finf, HostFr::mul(HostFr::sub(e1, e0),
                                         HostFr::mul(HostFr::sub(a1, a0), HostFr::sub(b1, b0))));
  }
  memcpy(out, f0.l, 32);
  memcpy(out + 4, fm1.l, 32);
  memcpy(out + 8, finf.l, 32);
}

}  // namespace pk

using namespace pk;

static_assert(sizeof(pkg_transcript) == 64, "transcript state is two field elements");

extern "C" int pkg_transcript_init(pkg_transcript* t, const uint64_t domain[4]) {
  PK_REQUIRE(t && domain, "null pointer");
  HostTranscript ht;
  ht.init(domain);
  memcpy(t->l, ht.l.l, 32);
  memcpy(t->r, ht.r.l, 32);
  return PKG_OK;
}

extern "C" int pkg_transcript_absorb(pkg_transcript* t, const uint64_t x[4]) {
  PK_REQUIRE(t && x, "null pointer");
  HostTranscript ht;
  ht.l = HostFr::from_limbs(t->l);
  ht.r = HostFr::from_limbs(t->r);
  ht.absorb(HostFr::from_limbs(x));
  memcpy(t->l, ht.l.l, 32);
  memcpy(t->r, ht.r.l, 32);
  return PKG_OK;
}

extern "C" int pkg_transcript_squeeze_bytes(pkg_transcript* t, uint8_t* out, size_t n) {
  PK_REQUIRE(t && (out || n == 0), "null pointer");
  HostTranscript ht;
  ht.l = HostFr::from_limbs(t->l);
  ht.r = HostFr::from_limbs(t->r);
  for (size_t done = 0; done < n;) {
    const HostFr c = HostFr::from_mont(ht.squeeze());
    const size_t take = std::min<size_t>(31, n - done);
    for (size_t i = 0; i < take; i++) out[done + i] = (uint8_t)(c.l[i / 8] >> (8 * (i % 8)));
    done += take;
  }
  memcpy(t->l, ht.l.l, 32);
  memcpy(t->r, ht.r.l, 32);
  return PKG_OK;
}

extern "C" int pkg_transcript_squeeze(pkg_transcript* t, uint64_t out[4]) {
  PK_REQUIRE(t && out, "null pointer");
  HostTranscript ht;
  ht.l = HostFr::from_limbs(t->l);
  ht.r = HostFr::from_limbs(t->r);
  HostFr v = ht.squeeze();
  memcpy(out, v.l, 32);
  memcpy(t->l, ht.l.l, 32);
  memcpy(t->r, ht.r.l, 32);
  return PKG_OK;
}

extern "C" int pkg_spartan_round(uint64_t* a, uint64_t* b, uint64_t* c, uint64_t* eq, size_t size,
                                 const uint64_t* fold, uint64_t out[12], pkg_stream_t stream) {
  PK_REQUIRE(is_pow2(size) && size >= 2, "table size %zu must be a power of two >= 2", size);
  PK_REQUIRE(!fold || size >= 4, "folding needs size >= 4 (got %zu)", size);
  PK_REQUIRE(a && b && c && eq && out, "null pointer");
  PK_REQUIRE(aligned16(a) && aligned16(b) && aligned16(c) && aligned16(eq),
             "device buffers must be 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  rc = spartan_round_device(a, b, c, eq, size, fold, fs.part, fs.dev, s, fs.ticket);
  if (rc) return rc;
  return fused_read(out, fs, 96, s);
}

extern "C" int pkg_eq_hypercube(const uint64_t* r, size_t nr, size_t num_entries, uint64_t* out,
                                pkg_stream_t stream) {
  PK_REQUIRE(num_entries == 0 || nr == 0 || host_readable(r), "r must be a host pointer");
  return eq_hypercube_device(r, nr, num_entries, out, as_stream(stream), true);
}

extern "C" int pkg_spmv_csr(const uint64_t* row_ptr, const uint32_t* cols, const uint64_t* vals,
                            size_t num_rows, size_t num_cols, const uint64_t* x, uint64_t* y,
                            pkg_stream_t stream) {
  if (num_rows == 0) return PKG_OK;
  cudaStream_t s = as_stream(stream);
  Scratch scr;
  int rc = scr.alloc(256, s);
  if (rc) return rc;
  uint32_t* err = static_cast<uint32_t*>(scr.ptr);
  PK_CUDA(cudaMemsetAsync(err, 0, 4, s));
  PK_REQUIRE(row_ptr, "null row pointers");
  uint64_t nnz = 0;  // row_ptr[num_rows], for the balanced passes
  if ((rc = read_small(&nnz, row_ptr + num_rows, 8, s))) return rc;
  PK_REQUIRE(nnz < (uint64_t(1) << 40), "row_ptr[num_rows] = %llu is not a nonzero count",
             (unsigned long long)nnz);
  rc = spmv_device(row_ptr, cols, vals, num_rows, num_cols, x, y, err, s, (size_t)nnz);
  if (rc) return rc;
  return read_err_flag(err, s, "pkg_spmv_csr");
}

extern "C" int pkg_hadamard_pad(const uint64_t* a, const uint64_t* b, size_t n, size_t padded,
                                uint64_t* c, pkg_stream_t stream) {
  PK_REQUIRE(padded >= n, "padded length %zu < n %zu", padded, n);
  if (padded == 0) return PKG_OK;
  PK_REQUIRE(c && aligned16(c) && aligned16(a) && aligned16(b), "null or unaligned pointer");
  cudaStream_t s = as_stream(stream);
  hadamard_pad_kernel<<<ew_grid(padded), 256, 0, s>>>(a, b, n, padded, c);
  PK_CHECK_LAUNCH("hadamard_pad_kernel");
  return PKG_OK;
}

extern "C" int pkg_dot(const uint64_t* a, const uint64_t* b, size_t n, uint64_t out[4],
                       pkg_stream_t stream) {
  PK_REQUIRE(out, "null output");
  if (n == 0) {
    memset(out, 0, 32);
    return PKG_OK;
  }
  PK_REQUIRE(a && b && aligned16(a) && aligned16(b), "null or unaligned pointer");
  cudaStream_t s = as_stream(stream);
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  const DotJob job = {a, b, n};
  rc = dots_device(&job, 1, fs.dev, fs, s);
  if (rc) return rc;
  return fused_read(out, fs, 32, s);
}

extern "C" int pkg_csr_transpose(const uint64_t* row_ptr, const uint32_t* cols, const uint64_t* vals,
                                 size_t num_rows, size_t num_cols, size_t nnz,
                                 uint64_t* row_ptr_t, uint32_t* cols_t, uint64_t* vals_t,
                                 pkg_stream_t stream) {
  PK_REQUIRE(row_ptr && row_ptr_t, "null row pointer array");
  PK_REQUIRE(num_cols < (size_t(1) << 32) && num_rows < (size_t(1) << 32),
             "matrix dimensions must fit u32 column indices");
  cudaStream_t s = as_stream(stream);
  Scratch scr;
  // counts (u32, num_cols), cursor (u64, num_cols + 1), cub temp
  size_t cub_bytes = 0;
  cub::DeviceScan::ExclusiveSum(nullptr, cub_bytes, (unsigned long long*)nullptr,
                                (unsigned long long*)nullptr, (int)(num_cols + 1), s);
  size_t counts_bytes = ((4 * num_cols + 255) / 256) * 256;
  size_t wide_bytes = ((8 * (num_cols + 1) + 255) / 256) * 256;
  int rc = scr.alloc(counts_bytes + wide_bytes + cub_bytes + 512, s);
  if (rc) return rc;
  uint8_t* base = static_cast<uint8_t*>(scr.ptr);
  uint32_t* counts = reinterpret_cast<uint32_t*>(base);
  unsigned long long* wide = reinterpret_cast<unsigned long long*>(base + counts_bytes);
  void* cub_tmp = base + counts_bytes + wide_bytes;
  uint32_t* err = reinterpret_cast<uint32_t*>(base + counts_bytes + wide_bytes + ((cub_bytes + 255) / 256) * 256);
  PK_CUDA(cudaMemsetAsync(err, 0, 4, s));
  PK_CUDA(cudaMemsetAsync(counts, 0, 4 * num_cols, s));
  PK_CUDA(cudaMemsetAsync(wide, 0, 8 * (num_cols + 1), s));
  if (nnz) {
    csr_count_cols_kernel<<<ew_grid(nnz), 256, 0, s>>>(cols, nnz, num_cols, counts, err);
    PK_CHECK_LAUNCH("csr_count_cols_kernel");
  }
  if (num_cols) {
    widen_kernel<<<ew_grid(num_cols), 256, 0, s>>>(counts, num_cols, wide);
    PK_CHECK_LAUNCH("widen_kernel");
  }
  PK_CUDA(cub::DeviceScan::ExclusiveSum(cub_tmp, cub_bytes, wide,
                                        reinterpret_cast<unsigned long long*>(row_ptr_t),
                                        (int)(num_cols + 1), s));
  count_launch();
  // cursor = row_ptr_t[0..num_cols) (reuse `wide`)
  PK_CUDA(cudaMemcpyAsync(wide, row_ptr_t, 8 * (num_cols + 1), cudaMemcpyDeviceToDevice, s));
  if (nnz && num_rows) {
    csr_scatter_kernel<<<ew_grid(num_rows), 256, 0, s>>>(row_ptr, cols, vals, num_rows, num_cols,
                                                         wide, cols_t, vals_t);
    PK_CHECK_LAUNCH("csr_scatter_kernel");
  }
  return read_err_flag(err, s, "pkg_csr_transpose");
}

extern "C" int pkg_spartan_sumcheck(uint64_t* a, uint64_t* b, uint64_t* c, size_t m0,
                                    const uint64_t* g, const uint64_t* w1_blinding,
                                    pkg_transcript* transcript, uint64_t* r_out, uint64_t rho_out[4],
                                    uint64_t sum_g_out[4], uint64_t* coeffs_out,
                                    uint64_t* alpha_out, uint64_t blinding_eval[4],
                                    pkg_stream_t stream) {
  PK_REQUIRE(m0 >= 1 && m0 <= 30, "m0 %zu out of range [1, 30]", m0);
  PK_REQUIRE(a && b && c && g && w1_blinding && transcript && r_out && rho_out && sum_g_out &&
                 coeffs_out && alpha_out && blinding_eval,
             "null pointer");
  PK_REQUIRE(aligned16(a) && aligned16(b) && aligned16(c), "device buffers must be 16-byte aligned");
  cudaStream_t s = as_stream(stream);
  const size_t n = size_t(1) << m0;
  HostTranscript t;
  t.l = HostFr::from_limbs(transcript->l);
  t.r = HostFr::from_limbs(transcript->r);
  std::vector<HostFr> r(m0), alpha(m0), gv(4 * m0);
  for (size_t i = 0; i < 4 * m0; i++) gv[i] = HostFr::from_limbs(g + 4 * i);
  for (size_t i = 0; i < m0; i++) {  // whir_r1cs.rs:529
    r[i] = t.squeeze();
    memcpy(r_out + 4 * i, r[i].l, 32);
  }
  // scratch: eq table (n Fr), partials; each round's sums go to the
  // thread's fused slots
  const int gmax = std::max(round_grid(n / 2), round_grid(std::min(n / 2, kQuadMaxPairs)));
  FusedSlots fs;
  int rc = fused_slots(&fs);
  if (rc) return rc;
  Scratch scr;
  if ((rc = scr.alloc(32 * (n + 3 * (size_t)gmax), s))) return rc;
  uint64_t* eq = static_cast<uint64_t*>(scr.ptr);
  uint64_t* part = eq + 4 * n;
  rc = eq_hypercube_device(r_out, m0, n, eq, s, false);  // :530; the rounds synchronise
  if (rc) return rc;
  HostFr g0[4];
  blinding_coeffs(gv.data(), m0, 0, nullptr, g0);  // sum_over_hypercube, :494-501
  HostFr sum_g = HostFr::add(eval_cubic(g0, HostFr::zero()), eval_cubic(g0, HostFr::one()));
  memcpy(sum_g_out, sum_g.l, 32);
  t.absorb(sum_g);                  // :541
  HostFr rho = t.squeeze();         // :543
  memcpy(rho_out, rho.l, 32);
  HostFr saved = HostFr::mul(rho, sum_g);
  const HostFr half = half_mont();
  size_t size = n;
  uint64_t h[12];
  // the blinding coefficients' two sums, kept as running sums over the rounds
  HostFr bprefix = HostFr::zero(), bsuffix = HostFr::zero();
  for (size_t i = 1; i < m0; i++) bsuffix = HostFr::add(bsuffix, cubic_sum01(&gv[4 * i]));
  // the last rounds, on tables of at most kHostTailEntries, run on the host
  // (a device round there is launch and round-trip latency)
  std::vector<HostFr> tab[4];
  bool on_host = false;
  for (size_t idx = 0; idx < m0; idx++) {  // :550-610
    if (!on_host && size <= kHostTailEntries) {
      for (int k = 0; k < 4; k++) tab[k].resize(size);
      const HostRead reads[4] = {{tab[0][0].l, a, 32 * size}, {tab[1][0].l, b, 32 * size},
                                 {tab[2][0].l, c, 32 * size}, {tab[3][0].l, eq, 32 * size}};
      if ((rc = read_small(reads, 4, s))) return rc;
      on_host = true;
    }
    if (on_host) {
      host_spartan_round(tab, size, idx ? &alpha[idx - 1] : nullptr, h);
    } else {
      rc = spartan_round_device(a, b, c, eq, size, idx ? alpha[idx - 1].l : nullptr, part, fs.dev,
                                s, fs.ticket);
      if (rc) return rc;
      if ((rc = fused_read(h, fs, 96, s))) return rc;
    }
    if (idx) size /= 2;
    HostFr gp[4];
    if (idx) {
      bprefix = HostFr::add(bprefix, eval_cubic(&gv[4 * (idx - 1)], alpha[idx - 1]));
      bsuffix = HostFr::sub(bsuffix, cubic_sum01(&gv[4 * idx]));
    }
    blinding_from_sums(gv.data(), m0, idx, bprefix, bsuffix, gp);
    HostFr h0 = HostFr::from_limbs(h), hem1 = HostFr::from_limbs(h + 4),
           hinf = HostFr::from_limbs(h + 8);
    HostFr cf[4];
    cf[0] = HostFr::add(h0, HostFr::mul(rho, gp[0]));
    HostFr gem1 = HostFr::sub(HostFr::add(HostFr::sub(gp[0], gp[1]), gp[2]), gp[3]);
    HostFr cem1 = HostFr::add(hem1, HostFr::mul(rho, gem1));
    cf[2] = HostFr::mul(half, HostFr::sub(HostFr::sub(HostFr::sub(HostFr::add(saved, cem1), cf[0]),
                                                      cf[0]),
                                          cf[0]));
    cf[3] = HostFr::add(hinf, HostFr::mul(rho, gp[3]));
    cf[1] = HostFr::sub(HostFr::sub(HostFr::sub(HostFr::sub(saved, cf[0]), cf[0]), cf[3]), cf[2]);
    for (int k = 0; k < 4; k++) {
      memcpy(coeffs_out + 16 * idx + 4 * k, cf[k].l, 32);
      t.absorb(cf[k]);
    }
    alpha[idx] = t.squeeze();
    memcpy(alpha_out + 4 * idx, alpha[idx].l, 32);
    saved = eval_cubic(cf, alpha[idx]);
  }
  // blinding_eval = <expand_powers::<4>(alpha), w1[offset..offset + 4*m0]> (:613-618)
  HostFr acc = HostFr::zero();
  for (size_t i = 0; i < m0; i++) {
    HostFr pw = HostFr::one();
    for (int k = 0; k < 4; k++) {
      acc = HostFr::add(acc, HostFr::mul(pw, HostFr::from_limbs(w1_blinding + 4 * (4 * i + k))));
      pw = HostFr::mul(pw, alpha[i]);
    }
  }
  memcpy(blinding_eval, acc.l, 32);
  t.absorb(acc);  // prover_message(&blinding_eval), :618
  memcpy(transcript->l, t.l.l, 32);
  memcpy(transcript->r, t.r.l, 32);
  return PKG_OK;
}

namespace {
size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
}  // namespace

extern "C" size_t pkg_r1cs_transposes_bytes(const pkg_r1cs* r1cs) {
  if (!r1cs) return 0;
  size_t total = 0;
  for (int k = 0; k < 3; k++) {
    const size_t nnz = r1cs->nnz[k] ? r1cs->nnz[k] : 1;
    total += align256(8 * (r1cs->num_witnesses + 1)) + align256(4 * nnz) + align256(32 * nnz);
  }
  return total;
}

extern "C" int pkg_r1cs_build_transposes(pkg_r1cs* r1cs, void* buf, pkg_stream_t stream) {
  PK_REQUIRE(r1cs && buf, "null pointer");
  PK_REQUIRE((reinterpret_cast<uintptr_t>(buf) & 255) == 0, "buffer must be 256-byte aligned");
  uint8_t* at = static_cast<uint8_t*>(buf);
  const size_t nw = r1cs->num_witnesses, nc = r1cs->num_constraints;
  for (int k = 0; k < 3; k++) {
    const size_t nnz = r1cs->nnz[k] ? r1cs->nnz[k] : 1;
    uint64_t* rp = reinterpret_cast<uint64_t*>(at);
    at += align256(8 * (nw + 1));
    uint32_t* cl = reinterpret_cast<uint32_t*>(at);
    at += align256(4 * nnz);
    uint64_t* vl = reinterpret_cast<uint64_t*>(at);
    at += align256(32 * nnz);
    const int rc = pkg_csr_transpose(r1cs->row_ptr[k], r1cs->cols[k], r1cs->vals[k], nc, nw,
                                     r1cs->nnz[k], rp, cl, vl, stream);
    if (rc) return rc;
    r1cs->row_ptr_t[k] = rp;
    r1cs->cols_t[k] = cl;
    r1cs->vals_t[k] = vl;
  }
  return PKG_OK;
}
