// ls_dgemm.cu -- grouped FP64 GEMM (LibShalom_dgemm_batched) for the
// small-block workloads of atomic-orbital chemistry codes: tens of thousands
// of products with M, N, K of a few to a few dozen, where consecutive products
// accumulate into the same C block (C += A_p B_p).
//
// Runs of consecutive entries naming the same C are found and ordered on the
// device (no host round trip): C blocks of at most 32 x 32 go to
// k_dgemm_small_runs, larger ones to k_dgemm_runs.  In both, one owner holds
// the C block (or tile) in registers from the run's first product to its last
// -- the rule that keeps shared C blocks race-free and the result deterministic
// without atomics.  Each product is a fused multiply-add chain over k in
// increasing order (the reference's KERNEL7x6 order) followed by
// C = fma(beta, C, alpha * acc).
//
// k_dgemm_small_runs: one warp a run, or two (its upper and lower 16 rows) when
// both edges are above 16.  4 x 4 outputs a lane, on a 16 x 32 tile or, for at
// most 16 columns, 32 x 16.  The warp's loads bring 16 k of A and op(B) into
// registers while it multiplies the 16 before from its own piece of shared
// memory, across the ends of products and runs; entries are read one product
// ahead and broadcast.  No barrier but __syncwarp.
//
// Measured on 200,000 products with edges of 5 to 32 in runs of 8: 1069 us with
// a CTA of 64 threads a run (an 8-byte cp.async an element of the 32 x 32 slabs,
// two barriers a slab, entries read again by every thread), 549 us now; as
// single products 1593 -> 615 us.  4,000 in runs of 12, 333 runs for 148 SMs:
// 54.6 -> 48.2 us, the latency of a chain of loads; 8 k at a time made that 60.
// 16 products: 12.3 -> 10.2 us (14.3 before each kernel's blocks were placed
// while the one before runs).
// The shared-memory pipe bounds it (wavefronts 58 % of its peak, FP64 pipe
// 25 %): a lane's outputs lie 4 or 8 apart, so that the 8-byte loads of a warp
// read 4 to 8 neighbouring words; 4 x 4 neighbours with 16-byte loads took 594.
// 4 CTAs an SM (spills, 8 k at a time) 618; 2 CTAs 601.
//
// k_dgemm_runs: a CTA (64 threads, 4 x 4 outputs each, six CTAs per SM) holds a
// 32 x 32 tile of C.  A and op(B) arrive in 32 x 32 slabs through an 8-byte
// cp.async double buffer that prefetches the next slab (of the same product,
// the next product or the next run) while the current one is multiplied,
// staged transposed (A as [k][m]) so the inner loop reads contiguous vectors.
#include <cuda_runtime.h>

#include <algorithm>

#include "ls_common.cuh"
#include "ls_dgemm_runs.cuh"
#include "ls_simt_launch.h"
#include "ls_sizes.h"

namespace ls {

namespace {

constexpr int DR_THREADS = 64;
constexpr int DR_T = 32;       // C tile edge and K slab
constexpr int DR_P = 34;       // padded pitch (doubles) of the staged slabs
constexpr int DR_STAGE = 2 * DR_T * DR_P;  // doubles per stage: A^T and B

// --------------------------------------------------------------------------
// the run list
// --------------------------------------------------------------------------

__device__ __forceinline__ bool run_start(const LibShalom_dgemm_entry *e, long i) {
  return i == 0 || e[i].C != e[i - 1].C;
}

// run starting at entry i: length, and its bin (shape, cost class: operand
// doubles / 256, capped; heavy classes first), or -1 for a C block above 32 x 32.
// Four entries are read at a time: a run's length is a chain of loads.
// Deep runs: where every run has an SM of its own, a run of k_dgemm_small_runs
// takes about 1.8 us for 16 k of a product and one of k_dgemm_runs 3.1 us for
// 32 k (one run of 64 products of 32^3 240 against 209 us, with K = 16 129 against
// 176, with K = 48 348 against 368; a product of 32 x 32 x 512 61 against 55).
// With 148 runs the two are equal, with more the small kernel is faster.  (The
// first product's K stands for the run's.)
__device__ __forceinline__ int run_bin(const LibShalom_dgemm_entry *e, long count, long i,
                                       long *len) {
  const int M = e[i].M, N = e[i].N;
  const double *C = e[i].C;
  const long s16 = (max(0, e[i].K) + 15L) >> 4, s32 = (max(0, e[i].K) + 31L) >> 5;
  long cost = (long)M * N, j = i;
  for (bool in = true; in;) {
    const double *c[4];
    int K[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long at = min(j + u, count - 1);
      c[u] = e[at].C;
      K[u] = max(0, e[at].K);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      in = in && j < count && c[u] == C;
      if (in) {
        cost += (long)K[u] * (M + N);
        ++j;
      }
    }
  }
  *len = j - i;
  if (M > 32 || N > 32) return -1;
  const int shape = M <= 16 ? 2 : N <= 16 ? 1 : 0;
  const bool deep = *len * s16 >= 32 && 7 * s16 > 12 * s32;
  const long cls = deep ? DM_CLASSES - 1 : max(0L, min(cost / 256, DM_CLASSES - 2L));
  return shape * DM_CLASSES + DM_CLASSES - 1 - (int)cls;
}

// Runs are counted per block in shared memory first: thousands of atomics on
// a few words of global memory would take longer than the pass itself.
__global__ void __launch_bounds__(256)
    k_run_count(const LibShalom_dgemm_entry *e, long count, RunPlan pl) {
  __shared__ unsigned n[DM_BINS];
  chain_next();
  if (threadIdx.x < DM_BINS) n[threadIdx.x] = 0;
  __syncthreads();
  for (long i = blockIdx.x * 256L + threadIdx.x; i < count; i += gridDim.x * 256L) {
    long len = 0;
    int bin = DM_BINS;  // not the start of a small run
    if (run_start(e, i)) bin = run_bin(e, count, i, &len);
    pl.entry_bin[i] = (unsigned char)(bin < 0 ? DM_BINS : bin);
    if (bin >= 0 && bin < DM_BINS) {
      pl.entry_len[i] = (unsigned)len;
      atomicAdd(&n[bin], 1u);
    } else if (bin < 0) {
      const unsigned slot = atomicAdd(pl.n_large, 1u);
      pl.large_first[slot] = (unsigned)i;
      pl.large_len[slot] = (unsigned)len;
    }
  }
  __syncthreads();
  if (threadIdx.x < DM_BINS && n[threadIdx.x])
    atomicAdd(&pl.bin_runs[threadIdx.x], n[threadIdx.x]);
}

// bins of the deep runs: the first of each shape
__device__ __forceinline__ bool deep_bin(int bin) { return bin < DM_BINS && bin % DM_CLASSES == 0; }

// off[b]: runs in the bins before b (own: thread b's bin); n_shape: their sums.
// Returns whether the deep ones are left out: there are no more than `few` runs.
__device__ __forceinline__ bool bin_offsets(unsigned own, unsigned few, unsigned *off,
                                            unsigned *n_shape) {
  __shared__ unsigned sums[DM_BINS / 32], deep[DM_SHAPES];
  static_assert(DM_BINS <= 256 && DM_BINS % 32 == 0 && DM_CLASSES % 32 == 0, "one thread a bin");
  const int tid = threadIdx.x, lane = tid & 31;
  unsigned upto = own;
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, upto, s);
    if (lane >= s) upto += v;
  }
  if (tid < DM_BINS && lane == 31) sums[tid >> 5] = upto;
  if (deep_bin(tid)) deep[tid / DM_CLASSES] = own;
  __syncthreads();
  bool leave_out = false;
  if (deep[0] | deep[1] | deep[2]) {
    unsigned all = 0;
#pragma unroll
    for (int i = 0; i < DM_BINS / 32; ++i) all += sums[i];
    leave_out = all <= few;
  }
  if (tid < DM_BINS) {
    for (int i = 0; i < tid >> 5; ++i) upto += sums[i];
    if (leave_out)
      for (int s = 0; s <= tid / DM_CLASSES; ++s) upto -= deep[s];
    off[tid] = upto - own;
  }
  if (n_shape && tid < DM_SHAPES) {
    unsigned runs = leave_out ? 0u - deep[tid] : 0u;
    for (int i = 0; i < DM_CLASSES / 32; ++i) runs += sums[tid * (DM_CLASSES / 32) + i];
    n_shape[tid] = runs;
  }
  return leave_out;
}

// Every block sums the bins itself (192 words, two shuffled scans): a launch
// between the passes would take longer.
__global__ void __launch_bounds__(256)
    k_run_place(long count, RunPlan pl) {
  __shared__ unsigned off[DM_BINS], n[DM_BINS], base[DM_BINS];
  chain_wait();
  chain_next();
  const int tid = threadIdx.x;
  const bool leave_out = bin_offsets(tid < DM_BINS ? pl.bin_runs[tid] : 0, pl.few, off,
                                     blockIdx.x == 0 ? pl.n_shape : nullptr);
  for (long i0 = blockIdx.x * 256L; i0 < count; i0 += gridDim.x * 256L) {
    if (tid < DM_BINS) n[tid] = 0;
    __syncthreads();
    const long i = i0 + tid;
    int bin = i < count ? pl.entry_bin[i] : DM_BINS;
    if (leave_out && deep_bin(bin)) {
      const unsigned slot = atomicAdd(pl.n_large, 1u);
      pl.large_first[slot] = (unsigned)i;
      pl.large_len[slot] = pl.entry_len[i];
      bin = DM_BINS;
    }
    unsigned rank = 0;
    if (bin < DM_BINS) rank = atomicAdd(&n[bin], 1u);
    __syncthreads();
    if (tid < DM_BINS && n[tid]) base[tid] = atomicAdd(&pl.bin_fill[tid], n[tid]);
    __syncthreads();
    if (bin < DM_BINS) {
      const unsigned slot = off[bin] + base[bin] + rank;
      pl.small_first[slot] = (unsigned)i;
      pl.small_len[slot] = pl.entry_len[i];
    }
    __syncthreads();
  }
}

// The same list in one launch of one block, where passes over the whole chip
// cost their launches (16 to 2,000 products: 2 to 3 us less).
constexpr int PLAN_ONE_THREADS = 512, PLAN_ONE_EACH = 4;
__global__ void __launch_bounds__(PLAN_ONE_THREADS)
    k_run_plan_one(const LibShalom_dgemm_entry *e, int count, RunPlan pl) {
  __shared__ unsigned off[DM_BINS], n[DM_BINS], large;
  chain_next();
  const int tid = threadIdx.x;
  if (tid < DM_BINS) n[tid] = 0;
  if (tid == 0) large = 0;
  __syncthreads();
  unsigned rank[PLAN_ONE_EACH], length[PLAN_ONE_EACH];
  int bin[PLAN_ONE_EACH];
#pragma unroll
  for (int u = 0; u < PLAN_ONE_EACH; ++u) {
    const int i = u * PLAN_ONE_THREADS + tid;
    bin[u] = DM_BINS;
    if (i >= count || !run_start(e, i)) continue;
    long len;
    const int b = run_bin(e, count, i, &len);
    length[u] = (unsigned)len;
    if (b >= 0) {
      bin[u] = b;
      rank[u] = atomicAdd(&n[b], 1u);
    } else {
      const unsigned slot = atomicAdd(&large, 1u);
      pl.large_first[slot] = (unsigned)i;
      pl.large_len[slot] = (unsigned)len;
    }
  }
  __syncthreads();
  if (bin_offsets(tid < DM_BINS ? n[tid] : 0, pl.few, off, pl.n_shape)) {
#pragma unroll
    for (int u = 0; u < PLAN_ONE_EACH; ++u) {
      if (!deep_bin(bin[u])) continue;
      const unsigned slot = atomicAdd(&large, 1u);
      pl.large_first[slot] = (unsigned)(u * PLAN_ONE_THREADS + tid);
      pl.large_len[slot] = length[u];
      bin[u] = DM_BINS;
    }
  }
  __syncthreads();
  if (tid == 0) *pl.n_large = large;
#pragma unroll
  for (int u = 0; u < PLAN_ONE_EACH; ++u) {
    if (bin[u] == DM_BINS) continue;
    const unsigned slot = off[bin[u]] + rank[u];
    pl.small_first[slot] = (unsigned)(u * PLAN_ONE_THREADS + tid);
    pl.small_len[slot] = length[u];
  }
}

// --------------------------------------------------------------------------
// C blocks of at most 32 x 32: one warp a run (or half of one)
// --------------------------------------------------------------------------

constexpr int DS_WARPS = 4;
constexpr int DS_PER_SM = 3;
constexpr int DS_KB = 16;              // k staged at a time
constexpr int DS_P16 = 17, DS_P32 = 33;  // odd pitches (doubles): transposed stores meet no bank twice

// Lane's share of one operand's DS_KB x (16 or 32) block: element i is row
// r + i dr (of A, or column of op(B)) at k + i dk, at p + i step in memory and
// s + i sstep in shared memory.
struct DsPart {
  int r, dr, k, dk;
  uint32_t s, sstep;
};
__device__ __forceinline__ DsPart ds_part(bool along_k, bool wide, int lane, uint32_t smem) {
  const int P = wide ? DS_P32 : DS_P16;
  DsPart d;
  if (along_k) {  // memory runs along k: 32 / DS_KB rows a load
    d.r = lane / DS_KB; d.dr = 32 / DS_KB; d.k = lane % DS_KB; d.dk = 0;
  } else if (wide) {
    d.r = lane; d.dr = 0; d.k = 0; d.dk = 1;
  } else {
    d.r = lane & 15; d.dr = 0; d.k = lane >> 4; d.dk = 2;
  }
  d.s = smem + 8 * (d.k * P + d.r);
  d.sstep = 8 * (d.dk * P + d.dr);
  return d;
}
template <int N>
__device__ __forceinline__ void ds_load(double (&v)[N], const DsPart &d, const double *p, long sr,
                                        long sk, int rows, unsigned k0, unsigned K) {
  const char *q = reinterpret_cast<const char *>(p + d.r * sr + (long)(k0 + d.k) * sk);
  const long step = 8 * (d.dr * sr + d.dk * sk);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int on = d.r + i * d.dr < rows && k0 + d.k + i * d.dk < K;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f64 %0, 0d0000000000000000;\n\t"
        "@p ld.global.nc.L2::256B.f64 %0, [%1];\n\t}"
        : "=d"(v[i])
        : "l"(q + i * step), "r"(on));
  }
}
template <int N>
__device__ __forceinline__ void ds_store(const double (&v)[N], const DsPart &d) {
#pragma unroll
  for (int i = 0; i < N; ++i)
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(d.s + i * d.sstep), "d"(v[i]) : "memory");
}

// acc[i][j] += A[i TM] B[j TN], k in increasing order
template <int TM, int PA, int TN, int PB>
__device__ __forceinline__ void ds_multiply(double (&acc)[4][4], const double *a, const double *b,
                                            int kcnt) {
#pragma unroll 4
  for (int k = 0; k < kcnt; ++k, a += PA, b += PB) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = __fma_rn(a[i * TM], b[j * TN], acc[i][j]);
  }
}

__global__ void __launch_bounds__(DS_WARPS * 32, DS_PER_SM)
    k_dgemm_small_runs(const LibShalom_dgemm_entry *entries, const RunPlan pl) {
  chain_wait();
  chain_next();
  constexpr int BLOCK = DS_KB * (DS_P16 + DS_P32);
  __shared__ __align__(16) double smem[DS_WARPS][BLOCK];
  const unsigned FULL = 0xffffffffu;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double *const s16 = smem[warp], *const s32 = s16 + DS_KB * DS_P16;
  const uint32_t a16 = (uint32_t)__cvta_generic_to_shared(s16);
  const uint32_t a32 = (uint32_t)__cvta_generic_to_shared(s32);
  // units: both halves of the shape 0 runs, then the other runs
  const long two = 2L * pl.n_shape[0], units = two + pl.n_shape[1] + pl.n_shape[2];
  const long stride = (long)gridDim.x * DS_WARPS;
  auto run_of = [&](long u) { return u < two ? u >> 1 : u - (two >> 1); };
  long u = (long)warp * gridDim.x + blockIdx.x;  // the unit being loaded
  if (u >= units) return;

  // load side: product `at` (n_left after it) of unit u, its entry in w
  unsigned at = pl.small_first[run_of(u)], n_left = pl.small_len[run_of(u)] - 1;
  unsigned nfirst = 0, nlen = 0;  // the next unit's run
  auto fetch_next_run = [&]() {
    if (u + stride < units) {
      nfirst = pl.small_first[run_of(u + stride)];
      nlen = pl.small_len[run_of(u + stride)];
    }
  };
  fetch_next_run();
  uint32_t w = entry_word(entries + at, lane), w_next = 0;
  auto fetch_next_entry = [&]() {
    if (n_left) w_next = entry_word(entries + at + 1, lane);
    else if (u + stride < units) w_next = entry_word(entries + nfirst, lane);
  };
  fetch_next_entry();
  double v16[DS_KB / 2], v32[DS_KB];
  unsigned k0 = 0;  // (unsigned: K may be close to 2^31)
  auto load = [&]() {  // block k0 of product w
    auto get = [&](int k) { return __shfl_sync(FULL, w, k); };
    auto get64 = [&](int k) { return (uint64_t)get(k + 1) << 32 | get(k); };
    const double *A = reinterpret_cast<const double *>(get64(0));
    const double *B = reinterpret_cast<const double *>(get64(2));
    const int M = (int)get(6), N = (int)get(7), transb = (int)get(9);
    const int K0 = max(0, (int)get(8)), lda = (int)get(10), ldb = (int)get(11);
    const long la = lda > 0 ? lda : K0, lb = ldb > 0 ? ldb : transb ? K0 : N;
    const unsigned K = M > 0 && N > 0 ? K0 : 0;
    const long br = transb ? lb : 1, bk = transb ? 1 : lb;
    if (N > 16) {
      const int m0 = u < two && (u & 1) ? 16 : 0;
      ds_load(v16, ds_part(true, false, lane, a16), A + m0 * la, la, 1, M - m0, k0, K);
      ds_load(v32, ds_part(transb, true, lane, a32), B, br, bk, N, k0, K);
    } else {
      ds_load(v32, ds_part(true, true, lane, a32), A, la, 1, M, k0, K);
      ds_load(v16, ds_part(transb, false, lane, a16), B, br, bk, N, k0, K);
    }
  };
  load();

  double c[4][4], acc[4][4];
  long ldc = 0;  // of the run: its first product's
  bool new_run = true;
#pragma unroll 1
  for (;;) {
    // the block in the registers belongs to this product:
    auto get = [&](int k) { return __shfl_sync(FULL, w, k); };
    auto get64 = [&](int k) { return (uint64_t)get(k + 1) << 32 | get(k); };
    const int M = (int)get(6), N = (int)get(7), transb = (int)get(9);
    const unsigned K = max(0, (int)get(8));
    const bool cols32 = N > 16;
    if (cols32) {
      ds_store(v16, ds_part(true, false, lane, a16));
      ds_store(v32, ds_part(transb, true, lane, a32));
    } else {
      ds_store(v32, ds_part(true, true, lane, a32));
      ds_store(v16, ds_part(transb, false, lane, a16));
    }
    // outputs: rows m + i tm, columns n + j tn (4 x 8 lanes, or 8 x 4)
    const int tm = cols32 ? 4 : 8, tn = cols32 ? 8 : 4;
    const int ml = cols32 ? lane >> 3 : lane >> 2, n = lane & (tn - 1);
    const int m = ml + (cols32 && u < two && (u & 1) ? 16 : 0);
    const double alpha = __longlong_as_double((long long)get64(14));
    const double beta = __longlong_as_double((long long)get64(16));
    double *const C = reinterpret_cast<double *>(get64(4));
    if (new_run) {
      const int ldc0 = (int)get(12);
      ldc = ldc0 > 0 ? ldc0 : N;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[i][j] = 0.0;
          if (beta != 0.0 && m + i * tm < M && n + j * tn < N)
            c[i][j] = C[(m + i * tm) * ldc + n + j * tn];
        }
    }
    const int kcnt = (int)min((unsigned)DS_KB, K - k0);
    if (k0 == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    }
    // move the load side on, and start the next block's loads
    const bool product_done = k0 + DS_KB >= K, run_done = product_done && n_left == 0;
    bool more = true;
    if (!product_done) {
      k0 += DS_KB;
    } else {
      k0 = 0;
      if (n_left) {
        ++at;
        --n_left;
      } else {
        more = u + stride < units;
        u += stride;
        at = nfirst;
        n_left = nlen - 1;
        if (more) fetch_next_run();
      }
      w = w_next;
      if (more) fetch_next_entry();
    }
    __syncwarp();
    if (more) load();
    if (cols32) ds_multiply<4, DS_P16, 8, DS_P32>(acc, s16 + ml, s32 + n, kcnt);
    else ds_multiply<8, DS_P32, 4, DS_P16>(acc, s32 + ml, s16 + n, kcnt);
    if (product_done) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double v = alpha * acc[i][j];
          c[i][j] = beta != 0.0 ? __fma_rn(beta, c[i][j], v) : v;
        }
    }
    if (run_done) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (m + i * tm < M && n + j * tn < N) C[(m + i * tm) * ldc + n + j * tn] = c[i][j];
    }
    new_run = run_done;
    if (!more) break;
    __syncwarp();  // every lane has read this block before it is overwritten
  }
}

// --------------------------------------------------------------------------
// larger C blocks: one CTA a 32 x 32 tile
// --------------------------------------------------------------------------

struct DJob {
  const double *A, *B;
  int M, N, K, lda, ldb, transb;
  double alpha, beta;
};

__device__ __forceinline__ DJob djob(const LibShalom_dgemm_entry &e) {
  DJob j;
  j.A = e.A; j.B = e.B;
  j.M = e.M; j.N = e.N; j.K = max(0, e.K);
  j.transb = e.transb;
  j.lda = e.lda > 0 ? e.lda : j.K;
  j.ldb = e.ldb > 0 ? e.ldb : (e.transb ? j.K : j.N);
  j.alpha = e.alpha; j.beta = e.beta;
  return j;
}

__device__ __forceinline__ void cp_async8(uint32_t saddr, const void *g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Position in this CTA's sequence of slabs: run slot r (round-robin over the
// CTAs), C tile t of the run, product p of the run, K slab k of the product.
struct DCursor {
  long r;
  int t, p, k;
};

__global__ void __launch_bounds__(DR_THREADS, 6)
    k_dgemm_runs(const LibShalom_dgemm_entry *entries, const unsigned *n_runs_p,
                 const unsigned *run_first, const unsigned *run_len) {
  __shared__ __align__(16) double stage[2][DR_STAGE];
  chain_wait();
  const int tid = threadIdx.x;
  const int tx = tid & 7, ty = tid >> 3;  // outputs: rows 4ty..4ty+3; cols 4tx..4tx+3
  const long n_runs = (long)*n_runs_p;

  auto tiles_of = [&](const LibShalom_dgemm_entry &e) {
    return ceil_div(e.M, DR_T) * ceil_div(e.N, DR_T);
  };
  auto slabs_of = [&](const LibShalom_dgemm_entry &e) { return slabs(e.K, DR_T); };

  // advance a cursor to the next slab; returns false past the CTA's last run
  auto advance = [&](DCursor &c) -> bool {
    if (c.r >= n_runs) return false;
    const unsigned f = run_first[c.r], len = run_len[c.r];
    if (++c.k < slabs_of(entries[f + c.p])) return true;
    c.k = 0;
    if (++c.p < (int)len) return true;
    c.p = 0;
    if (++c.t < tiles_of(entries[f])) return true;
    c.t = 0;
    for (c.r += gridDim.x; c.r < n_runs; c.r += gridDim.x)
      if (tiles_of(entries[run_first[c.r]]) > 0) return true;
    return false;
  };
  auto first = [&](DCursor &c) -> bool {
    c.t = c.p = c.k = 0;
    for (c.r = blockIdx.x; c.r < n_runs; c.r += gridDim.x)
      if (tiles_of(entries[run_first[c.r]]) > 0) return true;
    return false;
  };

  // issue the cp.async copies of the slab at cursor c into stage buffer b
  auto load = [&](const DCursor &c, int b) {
    const unsigned f = run_first[c.r];
    const LibShalom_dgemm_entry &e0 = entries[f];
    const DJob jb = djob(entries[f + c.p]);
    const int tiles_n = ceil_div(e0.N, DR_T);
    const int m0 = (c.t / tiles_n) * DR_T, n0 = (c.t % tiles_n) * DR_T, k0 = c.k * DR_T;
    double *As = stage[b];
    double *Bs = stage[b] + DR_T * DR_P;
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(As);
    const uint32_t sb = (uint32_t)__cvta_generic_to_shared(Bs);
#pragma unroll
    for (int q = 0; q < (DR_T * DR_T) / DR_THREADS; ++q) {
      const int e = tid + q * DR_THREADS;
      // A element (m, k): consecutive threads take consecutive k (contiguous in memory)
      const int m = e >> 5, k = e & 31;
      if (m0 + m < jb.M && k0 + k < jb.K)
        cp_async8(sa + (k * DR_P + m) * 8, jb.A + (long)(m0 + m) * jb.lda + k0 + k);
      // B element (k, n) of op(B)
      if (!jb.transb) {
        const int kk = e >> 5, n = e & 31;
        if (k0 + kk < jb.K && n0 + n < jb.N)
          cp_async8(sb + (kk * DR_P + n) * 8, jb.B + (long)(k0 + kk) * jb.ldb + n0 + n);
      } else {
        const int n = e >> 5, kk = e & 31;
        if (k0 + kk < jb.K && n0 + n < jb.N)
          cp_async8(sb + (kk * DR_P + n) * 8, jb.B + (long)(n0 + n) * jb.ldb + k0 + kk);
      }
    }
  };

  DCursor cur, nxt;
  if (!first(cur)) return;
  nxt = cur;
  bool have_next = advance(nxt);
  load(cur, 0);
  cp_commit();

  double c[4][4], acc[4][4];
  int buf = 0;
  for (;;) {
    const unsigned f = run_first[cur.r];
    const LibShalom_dgemm_entry &e0 = entries[f];
    const DJob jb = djob(entries[f + cur.p]);
    const int tiles_n = ceil_div(e0.N, DR_T);
    const int m0 = (cur.t / tiles_n) * DR_T, n0 = (cur.t % tiles_n) * DR_T;
    double *Crow0 = entries[f].C + (long)(m0 + 4 * ty) * (e0.ldc > 0 ? e0.ldc : e0.N) + n0 + 4 * tx;
    const int ldc = e0.ldc > 0 ? e0.ldc : e0.N;
    if (cur.p == 0 && cur.k == 0) {
      // new C tile: load it (the run's first beta decides whether it is read)
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool ok = m0 + 4 * ty + i < e0.M && n0 + 4 * tx + j < e0.N;
          c[i][j] = ok ? Crow0[(long)i * ldc + j] : 0.0;
        }
    }
    if (cur.k == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0;
    }
    // prefetch the next slab into the other buffer, then wait for this one
    if (have_next) load(nxt, buf ^ 1);
    cp_commit();
    cp_wait<1>();
    __syncthreads();
    const double *As = stage[buf];
    const double *Bs = stage[buf] + DR_T * DR_P;
    const int kcnt = min(DR_T, jb.K - cur.k * DR_T);
    for (int k = 0; k < kcnt; ++k) {
      const double2 a0 = *reinterpret_cast<const double2 *>(As + k * DR_P + 4 * ty);
      const double2 a1 = *reinterpret_cast<const double2 *>(As + k * DR_P + 4 * ty + 2);
      const double2 b0 = *reinterpret_cast<const double2 *>(Bs + k * DR_P + 4 * tx);
      const double2 b1 = *reinterpret_cast<const double2 *>(Bs + k * DR_P + 4 * tx + 2);
      const double av[4] = {a0.x, a0.y, a1.x, a1.y};
      const double bv[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __fma_rn(av[i], bv[j], acc[i][j]);
    }
    const bool product_done = cur.k + 1 >= slabs(jb.K, DR_T);
    if (product_done) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double v = jb.alpha * acc[i][j];
          c[i][j] = jb.beta != 0.0 ? __fma_rn(jb.beta, c[i][j], v) : v;
        }
      if (cur.p + 1 == (int)run_len[cur.r]) {
        // run complete for this tile: write it
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (m0 + 4 * ty + i < e0.M && n0 + 4 * tx + j < e0.N) Crow0[(long)i * ldc + j] = c[i][j];
      }
    }
    __syncthreads();  // everyone is done with this buffer before it is refilled
    if (!have_next) break;
    cur = nxt;
    have_next = advance(nxt);
    buf ^= 1;
  }
  cp_wait<0>();
}

}  // namespace

int plan_dgemm_runs(const LibShalom_dgemm_entry *entries, long count, unsigned few, RunPlan *out) {
  State &st = state();
  if (count > (1L << 30)) return LIBSHALOM_ERR_UNSUPPORTED;
  const size_t header = 512;
  static_assert(64 + 2 * DM_BINS <= 512, "header words");
  void *ws = nullptr;
  const int rc = workspace((header + 5 * (size_t)count) * sizeof(unsigned) + (size_t)count, &ws);
  if (rc) return rc;
  unsigned *w = static_cast<unsigned *>(ws);
  RunPlan pl;
  pl.few = few;
  pl.n_large = w;
  pl.n_shape = w + 8;
  pl.bin_runs = w + 64;
  pl.bin_fill = pl.bin_runs + DM_BINS;
  pl.small_first = w + header;
  pl.small_len = pl.small_first + count;
  pl.large_first = pl.small_len + count;
  pl.large_len = pl.large_first + count;
  pl.entry_len = pl.large_len + count;
  pl.entry_bin = reinterpret_cast<unsigned char *>(pl.entry_len + count);
  if (count <= PLAN_ONE_THREADS * PLAN_ONE_EACH) {
    k_run_plan_one<<<1, PLAN_ONE_THREADS, 0, st.stream>>>(entries, (int)count, pl);
  } else {
    LS_CUDA_TRY(cudaMemsetAsync(w, 0, header * sizeof(unsigned), st.stream));
    const int grid = (int)std::max(1L, std::min(cdiv(count, 256), (long)st.num_sms * 8));
    k_run_count<<<grid, 256, 0, st.stream>>>(entries, count, pl);
    LS_CUDA_TRY(cudaGetLastError());
    const int rc = launch_chained(k_run_place, grid, 256, 0, st.stream, count, pl);
    if (rc) return rc;
  }
  LS_CUDA_TRY(cudaGetLastError());
  *out = pl;
  return LIBSHALOM_SUCCESS;
}

// Grouped FP64 batch on the CUDA cores.
int run_dgemm_runs(const LibShalom_dgemm_entry *entries, long count) {
  RunPlan pl;
  int rc = plan_dgemm_runs(entries, count, (unsigned)state().num_sms / 2, &pl);
  if (rc) return rc;
  const int per_sm = occupancy_of((const void *)k_dgemm_small_runs, DS_WARPS * 32, 0, DS_PER_SM);
  rc = launch_chained(k_dgemm_small_runs, grid_for(cdiv(2 * count, DS_WARPS), per_sm),
                      DS_WARPS * 32, 0, state().stream, entries, pl);
  if (rc) return rc;
  return run_dgemm_runs_list(entries, count, pl.n_large, pl.large_first, pl.large_len);
}

// The run kernel over a run list built by another plan (device counts).
int run_dgemm_runs_list(const LibShalom_dgemm_entry *entries, long count, const unsigned *n_runs,
                        const unsigned *run_first, const unsigned *run_len) {
  State &st = state();
  const int per_sm = occupancy_of((const void *)k_dgemm_runs, DR_THREADS, 0, 6);
  const int grid = grid_for(cdiv(count, 1), per_sm);
  return launch_chained(k_dgemm_runs, grid, DR_THREADS, 0, st.stream, entries, n_runs, run_first,
                        run_len);
}

}  // namespace ls
