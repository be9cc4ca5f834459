// ls_dgemm_dmma.cu -- grouped FP64 GEMM on the FP64 tensor cores
// (LibShalom_dgemm_batched / _dgemm_stack with LIBSHALOM_DGEMM_DMMA).
//
// Work unit: one run (maximal group of consecutive entries naming the same C)
// whose C block fits a 32 x 32 warp tile.  One warp owns a run from its first
// product to its last: the C block lives in the warp's registers as DMMA
// accumulator fragments, so runs need no atomics and the result does not
// depend on scheduling.  Runs are listed by shape and heaviest first, and dealt round-robin to the warps of the grid.
//
// Operands go from global memory straight into the fragments: a lane of
// mma.sync.m8n8k4 holds A[lane / 4][lane % 4] and B[lane % 4][lane / 4], so a
// warp's load of a fragment reads 32 consecutive bytes of eight rows (64 of
// four rows for op(B) stored K x N), whatever the alignment, and the two
// fragments of a line meet in L1.  A warp loads the fragments of 12 k at a time
// and multiplies them; twelve warps an SM hide each other's latencies.
//
// Arithmetic: mma.sync.m8n8k4 FP64 (tcgen05 has no FP64 kind), only over the
// ceil(M/8) x ceil(N/8) fragments a run's C block covers; k is padded to a
// multiple of 4 with zeros.  Product i of a run computes
// C = beta_i C + (alpha_i A_i) op(B_i) with FP64 accumulation.
//
// Measured on 200,000 products with edges of 5 to 32 in runs of 8: 683 us when
// the operands went through a ring of shared-memory slots (bulk copies, or
// 16-byte cp.async for row windows; 280 M warp instructions, most of them
// addresses and window shifts), 373 us now (142 M), of which the run list and
// the CUDA-core kernel's look at its empty list are 25 us; the products' bytes
// take 174 us.  8,000 products in runs of 8, 1,000 warps' work: 66 -> 42 us.
// What is left is latency: the FP64 tensor pipe is 43 % busy and the issue
// slots 28 %.  More warps an SM lose their cache lines to each other before
// a line's second fragment is read (4 CTAs an SM, 32 x 32 blocks: 158 us
// against 150 with 3).  Loads of 8 k at a time: 405 us; of 16 k, 422; of 16
// or 20 k in the narrow shapes, 405 and 398.  A kernel for each shape let the
// narrow ones have 4 CTAs an SM (82 us instead of 87) but put their tails one
// after the other: 406 us, and 111 us on the 8,000.
#include <cuda_runtime.h>

#include "ls_common.cuh"
#include "ls_dgemm_runs.cuh"
#include "ls_simt_launch.h"

namespace ls {

namespace {

constexpr int DM_WARPS = 4;     // warps per CTA (one run each at a time)
constexpr int DM_KB = 3;        // k-steps of 4 loaded before they are multiplied
constexpr int DM_PER_SM = 3;    // CTAs an SM holds (registers)
// predicated (warp-uniformly): a branch around each would multiply the live
// ranges of the accumulators (1.1 KB of spills)
__device__ __forceinline__ void dmma_if(double &d0, double &d1, double a, double b, bool on) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "@p mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n\t}"
      : "+d"(d0), "+d"(d1)
      : "d"(a), "d"(b), "r"((int)on));
}
__device__ __forceinline__ double ldg_if(const char *p, bool on) {
  double v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
      "@p ld.global.nc.L2::256B.f64 %0, [%1];\n\t}"
      : "=d"(v)
      : "l"(p), "r"((int)on));
  return v;
}

__device__ __forceinline__ double ld_if(const char *p, bool on) {
  double v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
      "@p ld.global.f64 %0, [%1];\n\t}"
      : "=d"(v)
      : "l"(p), "r"((int)on)
      : "memory");
  return v;
}
__device__ __forceinline__ void st_if(char *p, double v, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f64 [%0], %1;\n\t}" ::"l"(p),
               "d"(v), "r"((int)on)
               : "memory");
}

// One product: acc += (alpha A) op(B).  Rows past M and columns past N are
// read as the last one: they reach only fragments' rows and columns that are
// never stored.
template <bool TRANSB, int FM, int FN>
__device__ __forceinline__ void dm_product(double (&acc)[FM][FN][2], const double *A,
                                           const double *B, int M, int N, unsigned K, long lda,
                                           long ldb, double alpha, int lane) {
  const int g = lane >> 2, q = lane & 3;
  const int MF = (M + 7) >> 3, NF = (N + 7) >> 3;
  const bool scale = alpha != 1.0;
  const uint64_t lda8 = 8 * (uint64_t)lda, ldb8 = 8 * (uint64_t)ldb;
  const char *pa = reinterpret_cast<const char *>(A + q);
  const char *pb = TRANSB ? reinterpret_cast<const char *>(B + q)
                          : reinterpret_cast<const char *>(B) + ldb8 * (unsigned)q;
  unsigned ar[FM], bc[FN];
#pragma unroll
  for (int f = 0; f < FM; ++f) ar[f] = min(8 * f + g, M - 1);
#pragma unroll
  for (int f = 0; f < FN; ++f) bc[f] = min(8 * f + g, N - 1);
#pragma unroll 1
  for (unsigned k0 = 0; k0 < K; k0 += 4 * DM_KB) {  // (unsigned: K may be close to 2^31)
    double a[DM_KB][FM], b[DM_KB][FN];
#pragma unroll
    for (int f = 0; f < FM; ++f) {
      const char *s = pa + lda8 * ar[f];
#pragma unroll
      for (int h = 0; h < DM_KB; ++h) a[h][f] = ldg_if(s + 32 * h, f < MF && k0 + 4 * h + q < K);
    }
#pragma unroll
    for (int h = 0; h < DM_KB; ++h) {
      const char *s = TRANSB ? pb + 32 * h : pb + 4 * h * ldb8;
#pragma unroll
      for (int f = 0; f < FN; ++f)
        b[h][f] = ldg_if(s + (TRANSB ? ldb8 : 8) * bc[f], f < NF && k0 + 4 * h + q < K);
    }
    if (scale) {
#pragma unroll
      for (int h = 0; h < DM_KB; ++h)
#pragma unroll
        for (int f = 0; f < FM; ++f) a[h][f] *= alpha;
    }
#pragma unroll
    for (int h = 0; h < DM_KB; ++h) {
      const bool in = k0 + 4 * h < K;
#pragma unroll
      for (int mf = 0; mf < FM; ++mf)
#pragma unroll
        for (int nf = 0; nf < FN; ++nf)
          dmma_if(acc[mf][nf][0], acc[mf][nf][1], a[h][mf], b[h][nf], in && mf < MF && nf < NF);
    }
    pa += 32 * DM_KB;
    pb += TRANSB ? 32 * DM_KB : 4 * DM_KB * ldb8;
  }
}

// what a warp carries from run to run
struct DmWarp {
  const LibShalom_dgemm_entry *entries;
  const unsigned *run_first, *run_len;
  long n_runs, stride, r;
  unsigned first, len;  // run r
  uint32_t w;           // word `lane` of its first entry
};

// the warp's runs below `end`, of C blocks within FM x FN fragments
template <int FM, int FN>
__device__ __forceinline__ void dm_runs(DmWarp &s, long end, int lane) {
  const unsigned FULL = 0xffffffffu;
  const int g = lane >> 2, q = lane & 3;
#pragma unroll 1
  for (; s.r < end; s.r += s.stride) {
    const unsigned at = s.first, n = s.len;
    const bool more = s.r + s.stride < s.n_runs;
    if (more) {  // the next run's place in the list, a run ahead
      s.first = s.run_first[s.r + s.stride];
      s.len = s.run_len[s.r + s.stride];
    }
    auto get = [&](int k) { return __shfl_sync(FULL, s.w, k); };
    auto get64 = [&](int k) { return (uint64_t)get(k + 1) << 32 | get(k); };
    const int M = (int)get(6), N = (int)get(7);  // (M or N <= 0: nothing is read or written)
    const uint64_t C = get64(4);
    const int ldc = (int)get(12);
    const uint64_t ldc8 = 8 * (uint64_t)(ldc > 0 ? ldc : N);
    char *const c0 = reinterpret_cast<char *>(C + ldc8 * g + 16 * q);
    double acc[FM][FN][2];
    const bool have_c = __longlong_as_double((long long)get64(16)) != 0.0;
#pragma unroll
    for (int mf = 0; mf < FM; ++mf)
#pragma unroll
      for (int nf = 0; nf < FN; ++nf)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          acc[mf][nf][h] = ld_if(c0 + 8 * mf * ldc8 + 64 * nf + 8 * h,
                                 have_c && 8 * mf + g < M && 8 * nf + 2 * q + h < N);
#pragma unroll 1
    for (unsigned p = 0; p < n; ++p) {
      const double *A = reinterpret_cast<const double *>(get64(0));
      const double *B = reinterpret_cast<const double *>(get64(2));
      const int K = max(0, (int)get(8)), transb = (int)get(9), lda = (int)get(10),
                ldb = (int)get(11);
      const double alpha = __longlong_as_double((long long)get64(14));
      const double beta = __longlong_as_double((long long)get64(16));
      if (p + 1 < n || more) s.w = entry_word(s.entries + (p + 1 < n ? at + p + 1 : s.first), lane);
      if (beta == 0.0) {
#pragma unroll
        for (int mf = 0; mf < FM; ++mf)
#pragma unroll
          for (int nf = 0; nf < FN; ++nf) acc[mf][nf][0] = acc[mf][nf][1] = 0.0;
      } else if (beta != 1.0) {
#pragma unroll
        for (int mf = 0; mf < FM; ++mf)
#pragma unroll
          for (int nf = 0; nf < FN; ++nf) {
            acc[mf][nf][0] *= beta;
            acc[mf][nf][1] *= beta;
          }
      }
      const long la = lda > 0 ? lda : K, lb = ldb > 0 ? ldb : transb ? K : N;
      if (M <= 0 || N <= 0) continue;
      if (transb) dm_product<true, FM, FN>(acc, A, B, M, N, K, la, lb, alpha, lane);
      else dm_product<false, FM, FN>(acc, A, B, M, N, K, la, lb, alpha, lane);
    }
#pragma unroll
    for (int mf = 0; mf < FM; ++mf)
#pragma unroll
      for (int nf = 0; nf < FN; ++nf)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          st_if(c0 + 8 * mf * ldc8 + 64 * nf + 8 * h, acc[mf][nf][h],
                8 * mf + g < M && 8 * nf + 2 * q + h < N);
  }
}

__global__ void __launch_bounds__(DM_WARPS * 32, DM_PER_SM)
    k_dgemm_dmma(const LibShalom_dgemm_entry *entries, const RunPlan pl) {
  chain_wait();
  chain_next();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long end0 = pl.n_shape[0], end1 = end0 + pl.n_shape[1], end2 = end1 + pl.n_shape[2];
  DmWarp s;
  s.entries = entries;
  s.run_first = pl.small_first;
  s.run_len = pl.small_len;
  s.n_runs = end2;
  s.stride = (long)gridDim.x * DM_WARPS;
  s.r = (long)warp * gridDim.x + blockIdx.x;  // few runs spread over the SMs
  if (s.r >= s.n_runs) return;
  s.first = s.run_first[s.r];
  s.len = s.run_len[s.r];
  s.w = entry_word(entries + s.first, lane);
  dm_runs<4, 4>(s, end0, lane);
  dm_runs<4, 2>(s, end1, lane);
  dm_runs<2, 4>(s, end2, lane);
}

}  // namespace

int run_dgemm_dmma(const LibShalom_dgemm_entry *entries, long count) {
  RunPlan pl;
  int rc = plan_dgemm_runs(entries, count, 0, &pl);
  if (rc) return rc;
  const int per_sm = occupancy_of((const void *)k_dgemm_dmma, DM_WARPS * 32, 0, DM_PER_SM);
  rc = launch_chained(k_dgemm_dmma, grid_for(cdiv(count, DM_WARPS), per_sm), DM_WARPS * 32, 0,
                      state().stream, entries, pl);
  if (rc) return rc;
  return run_dgemm_runs_list(entries, count, pl.n_large, pl.large_first, pl.large_len);
}

}  // namespace ls
