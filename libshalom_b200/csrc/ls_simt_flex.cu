// ls_simt_flex.cu -- uniform and grouped batches of plain FP32 products
// (LibShalom_sgemm_batched_strided, LibShalom_sgemm_batched) on the tiles of
// ls_flex.cuh: many CTAs of 128 threads per SM, each computing one tile at a
// time.
#include <algorithm>

#include "ls_common.cuh"
#include "ls_flex.cuh"
#include "ls_simt_launch.h"
#include "ls_sizes.h"

namespace ls {

namespace {

using F32 = FlexCfg<32, 32, 3>;
using F64 = FlexCfg<64, 64>;
using F128 = FlexCfg<64, 128>;

// edge of tile t of `tiles` that cover `n` evenly, in steps of 4
__host__ __device__ __forceinline__ int flex_edge(int n, int tiles) {
  return (int)(((long)n + tiles - 1) / tiles + 3) / 4 * 4;
}

// ---------------------------------------------------------------------------
// uniform batches: work item = (product, tile)
// ---------------------------------------------------------------------------
struct FlexUniform {
  const float *A, *B;
  float *C;
  long sA, sB, sC, items;
  int M, N, K, lda, ldb, ldc, transb;
  float alpha, beta;
  int tiles, tiles_n, edge_m, edge_n;
};

// 32 x 32 tiles an SM (as many as it holds) up to which a batch takes them: 64^3
// alone 8.2 -> 5.4 us, 128^3 14.3 -> 8.2, 222 products of 64^3 11.1 -> 9.2
constexpr long FU_FEW = 6;

template <class Cfg, int TM, int TN, int PER_SM>
__global__ void __launch_bounds__(FX_THREADS, PER_SM) k_flex_uniform(const FlexUniform u) {
  extern __shared__ __align__(16) float fsm[];
  FlexJob j;
  j.K = u.K;
  j.lda = u.lda; j.ldb = u.ldb; j.ldc = u.ldc; j.transb = u.transb;
  j.alpha = u.alpha; j.beta = u.beta;
  for (long w = blockIdx.x; w < u.items; w += gridDim.x) {
    const long g = u.tiles == 1 ? w : w / u.tiles;
    const int t = (int)(w - g * u.tiles), tm = u.tiles_n == 1 ? t : t / u.tiles_n;
    const int m0 = tm * u.edge_m, n0 = (t - tm * u.tiles_n) * u.edge_n;
    j.A = u.A + g * u.sA; j.B = u.B + g * u.sB; j.C = u.C + g * u.sC;
    flex_tile<Cfg, TM, TN>(j, m0, n0, min(u.edge_m, u.M - m0), min(u.edge_n, u.N - n0), fsm);
  }
}

// ---------------------------------------------------------------------------
// grouped batches
// ---------------------------------------------------------------------------
constexpr int FG_CLASSES = 64;  // work classes: half octaves of M N K a part
constexpr int FG_PARTS = 16;    // a run's tiles are dealt to at most 16 items
// Wide items a CTA up to which the small list's blocks start beside the wide
// list's: their tails fill each other, but the two share an SM's L1 from then
// on.  Mixed batches of 4..256, beside against behind: 50 products 31 (44) us,
// 1,000 82 (106), 5,000 177 (216), 20,000 604 (599), 35,000 1,035 (996),
// 50,000 1,426 (1,384).
constexpr unsigned FG_BESIDE = 20;
constexpr unsigned FG_LONG = (1u << 28) - 1;  // products of a run an item word can hold

// Plan: every run of entries sharing C becomes min(tiles, parts) items {first
// entry, products << 4 | part}, counting-sorted heaviest first, in two lists:
// C of more than 64 columns and 32 rows takes 64 x 128 tiles of 8 x 8 outputs
// a thread, the rest 64 x 64 tiles of 8 x 4 or 4 x 4 (one list for all took 1.57
// ms on 50,000 products of 4..256 where two took 1.49, now 1.38; one CTA a run on
// 64 x 64 tiles, as before: 4.66 ms).  The lists fill one array from its two ends.
struct FlexPlan {
  unsigned *class_n, *class_fill;  // [2][FG_CLASSES]: small, wide
  unsigned *n_items, *counter;                 // [2]
  uint2 *items;  // [n]: small ones upwards from 0, wide ones downwards from n - 1
  long n;        // parts * count
  int parts;
};

__device__ __forceinline__ bool fg_wide(int M, int N) { return M > 32 && N > 64; }
__device__ __forceinline__ void fg_tiles(int M, int N, int *tiles_m, int *tiles_n) {
  *tiles_m = ceil_div(M, 64);
  *tiles_n = ceil_div(N, fg_wide(M, N) ? 128 : 64);
}

__device__ __forceinline__ FlexJob fg_job(const LibShalom_sgemm_entry &e, int N) {
  FlexJob j;
  j.A = e.A; j.B = e.B; j.C = e.C;
  j.K = max(0, e.K); j.transb = e.transb;
  j.lda = e.lda > 0 ? e.lda : j.K;
  j.ldb = e.ldb > 0 ? e.ldb : (e.transb ? j.K : N);
  j.ldc = e.ldc > 0 ? e.ldc : N;
  j.alpha = e.alpha; j.beta = e.beta;
  return j;
}

// items, class and length of the run starting at entry i (0 items: empty C)
__device__ __forceinline__ int fg_run(const LibShalom_sgemm_entry *e, long count, long i,
                                      int max_parts, long *len, int *cls) {
  const int M = e[i].M, N = e[i].N;
  long k = 0, j = i;
  do {
    k += 16 + max(0, e[j].K);  // each product costs about 16 k of overhead
    ++j;
  } while (j < count && e[j].C == e[i].C);
  *len = j - i;
  *cls = 0;
  if (M <= 0 || N <= 0) return 0;
  int tm, tn;
  fg_tiles(M, N, &tm, &tn);
  const int parts = (int)min((long)tm * tn, (long)max_parts);
  const float work = (float)M * (float)N * (float)k / (float)parts;
  *cls = max(0, min(FG_CLASSES - 1, (int)(2.0f * log2f(fmaxf(work, 1.0f)))));
  if (fg_wide(M, N)) *cls += FG_CLASSES;
  return parts;
}

// Items are counted per block in shared memory first: a call's atomics on the
// few words of the classes took 17 us on 50,000 products.
__global__ void __launch_bounds__(256)
    k_fg_count(const LibShalom_sgemm_entry *e, long count, FlexPlan pl) {
  __shared__ unsigned n[2 * FG_CLASSES];
  chain_next();
  if (threadIdx.x < 2 * FG_CLASSES) n[threadIdx.x] = 0;
  __syncthreads();
  for (long i = blockIdx.x * 256L + threadIdx.x; i < count; i += gridDim.x * 256L) {
    if (i > 0 && e[i].C == e[i - 1].C) continue;
    long len;
    int cls;
    const int parts = fg_run(e, count, i, pl.parts, &len, &cls);
    if (parts) atomicAdd(&n[cls], (unsigned)parts);
  }
  __syncthreads();
  if (threadIdx.x < 2 * FG_CLASSES && n[threadIdx.x])
    atomicAdd(&pl.class_n[threadIdx.x], n[threadIdx.x]);
}

// Every block sums the classes itself: heavy classes of a list come first.
__global__ void __launch_bounds__(256)
    k_fg_place(const LibShalom_sgemm_entry *e, long count, FlexPlan pl) {
  __shared__ unsigned all[2 * FG_CLASSES], off[2 * FG_CLASSES], n[2 * FG_CLASSES],
      base[2 * FG_CLASSES];
  chain_wait();
  chain_next();
  const int tid = threadIdx.x;
  if (tid < 2 * FG_CLASSES) all[tid] = pl.class_n[tid];
  __syncthreads();
  if (tid < 2 * FG_CLASSES) {
    const int lo = tid & ~(FG_CLASSES - 1);
    unsigned before = 0;
    for (int i = lo + FG_CLASSES - 1; i > tid; --i) before += all[i];
    off[tid] = before;
    if (blockIdx.x == 0 && tid == lo) pl.n_items[lo / FG_CLASSES] = before + all[tid];
  }
  for (long i0 = blockIdx.x * 256L; i0 < count; i0 += gridDim.x * 256L) {
    if (tid < 2 * FG_CLASSES) n[tid] = 0;
    __syncthreads();
    const long i = i0 + tid;
    long len = 0;
    int cls = 0, parts = 0;
    if (i < count && (i == 0 || e[i].C != e[i - 1].C))
      parts = fg_run(e, count, i, pl.parts, &len, &cls);
    const unsigned rank = parts ? atomicAdd(&n[cls], (unsigned)parts) : 0;
    __syncthreads();
    if (tid < 2 * FG_CLASSES && n[tid]) base[tid] = atomicAdd(&pl.class_fill[tid], n[tid]);
    __syncthreads();
    const unsigned products = (unsigned)min(len, (long)FG_LONG);
    for (int p = 0; p < parts; ++p) {
      const long at = (long)off[cls] + base[cls] + rank + p;
      pl.items[cls < FG_CLASSES ? at : pl.n - 1 - at] =
          make_uint2((unsigned)i, products << 4 | (unsigned)p);
    }
    __syncthreads();
  }
}

// The lists of a batch of few products in one launch of one block: the memset
// and the passes over the chip cost more than the kernels (256 products of 32^3:
// 15.0 us with them, 10.2 with this).
constexpr int PLAN_THREADS = 512, PLAN_EACH = 4;
__global__ void __launch_bounds__(PLAN_THREADS)
    k_fg_plan_one(const LibShalom_sgemm_entry *e, int count, FlexPlan pl) {
  __shared__ unsigned n[2 * FG_CLASSES], sums[2 * FG_CLASSES / 32];
  static_assert(FG_CLASSES == 64, "two warps a list");
  chain_next();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid < 2 * FG_CLASSES) n[tid] = 0;
  __syncthreads();
  unsigned rank[PLAN_EACH], products[PLAN_EACH];
  int cls[PLAN_EACH], parts[PLAN_EACH];
#pragma unroll
  for (int u = 0; u < PLAN_EACH; ++u) {
    const int i = u * PLAN_THREADS + tid;
    parts[u] = 0;
    if (i >= count || (i > 0 && e[i].C == e[i - 1].C)) continue;
    long len;
    parts[u] = fg_run(e, count, i, pl.parts, &len, &cls[u]);
    products[u] = (unsigned)len;
    if (parts[u]) rank[u] = atomicAdd(&n[cls[u]], (unsigned)parts[u]);
  }
  __syncthreads();
  // first slot of every class, heavy classes of a list first
  const int at = (tid & ~(FG_CLASSES - 1)) + FG_CLASSES - 1 - (tid & (FG_CLASSES - 1));
  const unsigned own = tid < 2 * FG_CLASSES ? n[at] : 0;
  unsigned upto = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d) upto += v;
  }
  if (tid < 2 * FG_CLASSES && lane == 31) sums[warp] = upto;
  __syncthreads();
  if (tid < 2 * FG_CLASSES) {
    if (warp & 1) upto += sums[warp - 1];
    n[at] = upto - own;
    if ((warp & 1) && lane == 31) {
      pl.n_items[warp >> 1] = upto;
      pl.counter[warp >> 1] = 0;
    }
  }
  __syncthreads();
#pragma unroll
  for (int u = 0; u < PLAN_EACH; ++u)
    for (int p = 0; p < parts[u]; ++p) {
      const long slot = (long)n[cls[u]] + rank[u] + p;
      pl.items[cls[u] < FG_CLASSES ? slot : pl.n - 1 - slot] =
          make_uint2((unsigned)(u * PLAN_THREADS + tid), products[u] << 4 | (unsigned)p);
    }
}

// CTAs take items from a counter.  Thread 0 keeps two items ahead: the list
// word of the next item and the counter value after it are in flight while an
// item is computed (inline PTX: the compiler would aggregate an atomicAdd over
// the warp and wait for its result on the spot).
template <bool WIDE>
__global__ void __launch_bounds__(FX_THREADS, WIDE ? 4 : 6)
    k_flex_grouped(const LibShalom_sgemm_entry *entries, long count, FlexPlan pl) {
  extern __shared__ __align__(16) float fsm[];
  __shared__ uint2 s_item[2];
  if constexpr (WIDE) chain_wait();  // the plan
  // Few small items: the four quarters of each 64 x 64 tile are items of their
  // own (a tile's latency is what counts then; B200, 64 products of 64^3 17.5 ->
  // 10.3 us, a run of 128 such products 914 -> 416, 64 of 64 x 64 x 5,000 405 ->
  // 243).
  const unsigned n_tiles = pl.n_items[WIDE];
  const bool quarters = !WIDE && n_tiles <= gridDim.x / 4;
  const unsigned n_items = quarters ? 4 * n_tiles : n_tiles;
  // The small list's blocks may start when all of this kernel's have: the plan
  // is complete then, nothing that either writes is the other's, and the wait
  // at the end keeps what follows in the stream behind both.
  if (WIDE && n_items <= FG_BESIDE * gridDim.x) chain_next();
  uint2 nxt = make_uint2(0, 0);
  unsigned idx = 0;
  auto take = [&]() {
    asm volatile("atom.global.add.u32 %0, [%1], 1;"
                 : "=r"(idx)
                 : "l"(pl.counter + WIDE)
                 : "memory");
  };
  auto at = [&](long i) { return pl.items[WIDE ? pl.n - 1 - i : quarters ? i % n_tiles : i]; };
  if (threadIdx.x == 0) {
    s_item[0] = blockIdx.x < n_items ? at(blockIdx.x) : make_uint2(0, 0);
    const unsigned i1 = blockIdx.x + gridDim.x;
    if (i1 < n_items) {
      nxt = at(i1);
      take();
    }
  }
  __syncthreads();
  for (int it = 0;; it ^= 1) {
    const uint2 item = s_item[it];
    if (item.y == 0) break;  // no products: past the list
    if (threadIdx.x == 0) {
      s_item[it ^ 1] = nxt;
      nxt = make_uint2(0, 0);
      const unsigned long i2 = 2ul * gridDim.x + idx;
      if (i2 < n_items) {
        nxt = at((long)i2);
        take();
      }
    }
    const LibShalom_sgemm_entry *run = entries + item.x;
    const long most = count - item.x;  // (a run as long as FG_LONG: up to its end)
    const unsigned len = item.y >> 4;
    const int M = run->M, N = run->N;
    int tiles_m, tiles_n;
    fg_tiles(M, N, &tiles_m, &tiles_n);
    const int em = flex_edge(M, tiles_m), en = flex_edge(N, tiles_n);
    for (long t = item.y & (FG_PARTS - 1); t < (long)tiles_m * tiles_n; t += pl.parts) {
      const int tm = (int)(t / tiles_n), tn = (int)(t - (long)tm * tiles_n);
      int m0 = tm * em, n0 = tn * en, mrows = min(em, M - m0), ncols = min(en, N - n0);
      if (quarters) {
        const unsigned quarter = blockIdx.x / n_tiles;
        const int dm = quarter & 2 ? 32 : 0, dn = quarter & 1 ? 32 : 0;
        m0 += dm;
        n0 += dn;
        mrows = min(32, mrows - dm);
        ncols = min(32, ncols - dn);
      }
      if (mrows <= 0 || ncols <= 0) continue;
      const bool small = ((mrows + 3) >> 2) * ((ncols + 3) >> 2) <= FX_THREADS;
      for (long p = 0; p < len || (len == FG_LONG && p < most && run[p].C == run->C); ++p) {
        if (p + 1 < len) asm volatile("prefetch.global.L1 [%0];" ::"l"(run + p + 1));
        const FlexJob j = fg_job(run[p], N);
        if constexpr (WIDE) flex_tile<F128, 8, 8>(j, m0, n0, mrows, ncols, fsm);
        else if (quarters) flex_tile<F32, 4, 4>(j, m0, n0, mrows, ncols, fsm);
        else if (small) flex_tile<F64, 4, 4>(j, m0, n0, mrows, ncols, fsm);
        else flex_tile<F64, 8, 4>(j, m0, n0, mrows, ncols, fsm);
      }
    }
    __syncthreads();
  }
  if constexpr (!WIDE) chain_wait();
}

// A batch of few products without lists: FG_PARTS blocks for each entry, which
// deal the tiles of the run that starts there (64 x 128 tiles, or 32 x 32: a
// tile's latency is what counts).  One launch and no scratch: 16 products of 8^3
// 4.4 us, 8.2 with the plan and the list kernels.  More entries than the chip
// holds sixteenfold leave its SMs unevenly loaded (64 products of 100^3: 38.9 us,
// 22.5 with the lists).
constexpr long FG_FEW = 32;
__global__ void __launch_bounds__(FX_THREADS, 4)
    k_flex_few(const LibShalom_sgemm_entry *entries, long count) {
  extern __shared__ __align__(16) float fsm[];
  for (long w = blockIdx.x; w < count * FG_PARTS; w += gridDim.x) {
    const long part = w / count, i = w - part * count, most = count - i;
    const LibShalom_sgemm_entry *run = entries + i;
    if (i > 0 && run->C == run[-1].C) continue;
    const int M = run->M, N = run->N;
    if (M <= 0 || N <= 0) continue;
    const bool wide = fg_wide(M, N);
    const int tiles_m = ceil_div(M, wide ? 64 : 32), tiles_n = ceil_div(N, wide ? 128 : 32);
    const int em = flex_edge(M, tiles_m), en = flex_edge(N, tiles_n);
    for (long t = part; t < (long)tiles_m * tiles_n; t += FG_PARTS) {
      const int tm = (int)(t / tiles_n), tn = (int)(t - (long)tm * tiles_n);
      const int m0 = tm * em, n0 = tn * en, mrows = min(em, M - m0), ncols = min(en, N - n0);
      if (mrows <= 0 || ncols <= 0) continue;
      for (long p = 0; p < most && run[p].C == run->C; ++p) {
        if (p + 1 < most) asm volatile("prefetch.global.L1 [%0];" ::"l"(run + p + 1));
        const FlexJob j = fg_job(run[p], N);
        if (wide) flex_tile<F128, 8, 8>(j, m0, n0, mrows, ncols, fsm);
        else flex_tile<F32, 4, 4>(j, m0, n0, mrows, ncols, fsm);
      }
    }
  }
}

template <class Cfg, int TM, int TN, int PER_SM>
int launch_uniform(FlexUniform &u, long count) {
  const int tiles_m = (int)cdiv(u.M, Cfg::MAXM);
  u.tiles_n = (int)cdiv(u.N, Cfg::MAXN);
  u.edge_m = flex_edge(u.M, tiles_m);
  u.edge_n = flex_edge(u.N, u.tiles_n);
  // edges in steps of 4 can leave the last tile empty
  u.tiles_n = (int)cdiv(u.N, u.edge_n);
  u.tiles = (int)cdiv(u.M, u.edge_m) * u.tiles_n;
  u.items = (long)u.tiles * count;
  auto kern = k_flex_uniform<Cfg, TM, TN, PER_SM>;
  const int per_sm = occupancy_of((const void *)kern, FX_THREADS, Cfg::SMEM, PER_SM);
  kern<<<grid_for(u.items, per_sm), FX_THREADS, Cfg::SMEM, state().stream>>>(u);
  LS_CUDA_TRY(cudaGetLastError());
  return LIBSHALOM_SUCCESS;
}

}  // namespace

int run_flex_strided(const GemmArgs<float> &g, long sA, long sB, long sC, long count) {
  FlexUniform u{};
  u.A = g.A; u.B = g.B; u.C = g.C;
  u.sA = sA; u.sB = sB; u.sC = sC;
  u.M = (int)g.M; u.N = (int)g.N; u.K = (int)g.K;
  u.lda = (int)g.lda; u.ldb = (int)g.ldb; u.ldc = (int)g.ldc;
  u.transb = g.transb;
  u.alpha = g.alpha; u.beta = g.beta;
  // the smallest thread tile that covers a product in one CTA, 8 x 8 (fewest
  // shared-memory loads per FMA) beyond 64 columns.  B200, 10,000 products
  // against the fixed 32 / 64 / 128 tiles before: 24^3 NN 39 (74) us, 104^3 NT
  // 895 (1,241); 3,000 of 64^3 NN 54 (70), of 8 x 100 x 64 40 (184), of 128 x 16 x
  // 64 64 (205), of 300 x 33 x 50 193 (590); 222 of 256^3 177 (197), 16 of 512^3
  // 115 (123)
  // Few products: 32 x 32 tiles, whose latency is what counts.
  if (cdiv(g.M, 32) * cdiv(g.N, 32) * count <= FU_FEW * (long)state().num_sms)
    return launch_uniform<F32, 4, 4, 6>(u, count);
  if (cdiv(g.M, 4) * cdiv(g.N, 4) <= FX_THREADS && g.M <= 64 && g.N <= 64)
    return launch_uniform<F64, 4, 4, 6>(u, count);
  if (g.N <= 64) return launch_uniform<F64, 8, 4, 6>(u, count);
  return launch_uniform<F128, 8, 8, 4>(u, count);
}

int run_grouped_s(const LibShalom_sgemm_entry *entries, long count) {
  State &st = state();
  if (count > UINT32_MAX) return LIBSHALOM_ERR_UNSUPPORTED;
  if (count <= FG_FEW) {
    const int per_sm = occupancy_of((const void *)k_flex_few, FX_THREADS, F128::SMEM, 4);
    k_flex_few<<<grid_for(count * FG_PARTS, per_sm), FX_THREADS, F128::SMEM, st.stream>>>(entries,
                                                                                         count);
    LS_CUDA_TRY(cudaGetLastError());
    return LIBSHALOM_SUCCESS;
  }
  const size_t header = 512;
  FlexPlan pl;
  // one item a run where the items would take much memory
  pl.parts = count <= (1L << 22) ? FG_PARTS : 1;
  void *ws = nullptr;
  int rc = workspace((header + 2 * (size_t)pl.parts * (size_t)count) * sizeof(unsigned), &ws);
  if (rc && pl.parts > 1) {
    pl.parts = 1;
    rc = workspace((header + 2 * (size_t)count) * sizeof(unsigned), &ws);
  }
  if (rc) return rc;
  unsigned *w = static_cast<unsigned *>(ws);
  pl.n = pl.parts * count;
  pl.class_n = w;
  pl.class_fill = w + 2 * FG_CLASSES;
  pl.n_items = w + 4 * FG_CLASSES;
  pl.counter = pl.n_items + 2;
  pl.items = reinterpret_cast<uint2 *>(w + header);
  if (count <= PLAN_THREADS * PLAN_EACH) {
    k_fg_plan_one<<<1, PLAN_THREADS, 0, st.stream>>>(entries, (int)count, pl);
    LS_CUDA_TRY(cudaGetLastError());
  } else {
    LS_CUDA_TRY(cudaMemsetAsync(w, 0, header * sizeof(unsigned), st.stream));
    const int pgrid = (int)std::max(1L, std::min(cdiv(count, 256), (long)st.num_sms * 8));
    k_fg_count<<<pgrid, 256, 0, st.stream>>>(entries, count, pl);
    LS_CUDA_TRY(cudaGetLastError());
    if ((rc = launch_chained(k_fg_place, pgrid, 256, 0, st.stream, entries, count, pl))) return rc;
  }
  const int ps_w = occupancy_of((const void *)k_flex_grouped<true>, FX_THREADS, F128::SMEM, 4);
  const int ps_s = occupancy_of((const void *)k_flex_grouped<false>, FX_THREADS, F64::SMEM, 6);
  rc = launch_chained(k_flex_grouped<true>, grid_for((long)st.num_sms * ps_w, ps_w), FX_THREADS,
                      F128::SMEM, st.stream, entries, count, pl);
  if (rc) return rc;
  rc = launch_chained(k_flex_grouped<false>, grid_for((long)st.num_sms * ps_s, ps_s), FX_THREADS,
                      F64::SMEM, st.stream, entries, count, pl);
  if (rc) return rc;
  return LIBSHALOM_SUCCESS;
}

}  // namespace ls
