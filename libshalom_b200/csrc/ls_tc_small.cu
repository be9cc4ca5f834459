// ls_tc_small.cu -- split-BF16 products of a few to a few hundred rows on the
// tensor cores, several CTAs per SM (LibShalom_sgemm_batched, and uniform
// batches whose rows TMA cannot address).
//
// One CTA of four warps computes one C tile of up to 64 rows x 128 columns at
// a time, and four CTAs share an SM: a small product is a chain of latencies
// (operand loads, split, MMA, TMEM read-back) with little work in each, so
// what fills the machine is several products in flight, not a deep pipeline
// inside one.  Every thread of the CTA takes part in every step:
//   load     global -> registers, eight consecutive k of one row a lane (plain
//            loads: no alignment is asked of rows or leading dimensions)
//   split    registers -> BF16 hi / mid / lo in shared memory, K-major core
//            matrices; only rows, columns and k-steps inside the product
//   MMA      one lane issues tcgen05.mma; the next slab's first loads are in
//            flight meanwhile
//   epilogue TMEM -> registers -> C
// The product computed is C^T = op(B)^T A^T: TMEM lanes are C's columns, so a
// warp stores 32 (or 16) consecutive floats of a C row, whatever C's
// alignment.  Tiles of at most 64 columns use the M = 64 MMA, which reads half
// the operand bytes: an MMA's time here is its operand read, (M + N) * 32
// bytes at 128 bytes a clock (measured: 24 cycles for 64 x 32 x 16, 48 for
// 128 x 64 x 16 with four CTAs issuing).
//
// The tensor core's FP32 accumulation truncates, so K is cut into chunks of
// 128, whose sums are added round to nearest; the products of a chunk are
// issued, and the chunks added, in the order of the other split-BF16 kernels
// (k_tc_sgemm for uniform batches, k_tc_grouped for grouped ones), for their
// bits.  C is updated once, after the last chunk: adding chunk after chunk into
// a C that is large beside the product would round the product away (|C| =
// 1,000, K = 2,048: normwise error 2.2e-7 against 3.7e-8).  Until then the sum
// is kept in C itself by products that do not read C (beta = 0) and have it to
// themselves.  Other products of several chunks have a loop of their own (HOLD) that keeps the
// sum in TMEM beside the accumulators, where there is room for tiles of up to 32
// rows: as a branch of one loop it cost the others 8 % (registers and code), as a
// launch of its own 8 us a call.
//
// Measured on a B200: 50,000 products of 4..256 (log-uniform, one in five
// adding to its predecessor's C) 1.14 ms, against 2.66 ms with k_tc_grouped
// alone; 10,000 products of 45 x 37 x 51 94 us, against 465 us with
// k_tc_sgemm.  Bound by instruction issue and latency (ncu, the mixed batch:
// 55-60 % fewer warp instructions than k_tc_grouped, issue slots 47 % busy,
// L1 55 %, DRAM 22 %, tensor pipe 16 %).  What did not help: eight warps per CTA
// (1.77 ms: per-product work repeated in more warps, 64 registers a thread),
// wider batches of loads (four or six row groups a warp: 1.15 and 1.32 ms,
// the unrolled code leaves the instruction cache), two k a lane with
// 128-byte rows per load (1.32 ms: half the L1 wavefronts, 19 % more
// instructions), a register sum over the K chunks (64 registers and 79 KB of
// code: 2.1 ms).
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "ls_common.cuh"
#include "ls_tc_launch.h"
#include "ls_tc_ptx.cuh"

namespace ls {

namespace {

constexpr int SM_THREADS = 128;
constexpr int SM_WARPS = SM_THREADS / 32;
constexpr int SM_PER_SM = 4;     // TMEM: 4 x 128 columns; registers: 4 x 128 x 128
constexpr int SM_BK = 32;        // k per slab (two MMA k-steps of 16)
constexpr int SM_KC = 4;         // slabs per TMEM accumulation chunk (128 k)
constexpr int SM_TMEM_COLS = 128;  // D_main (64) + D_corr (64)
constexpr int SM_CORR = 64;
constexpr int SM_SUM = 32;  // sum of the chunks so far (tiles of up to 32 rows)
constexpr int SM_BATCH = 3;      // row groups (8 rows x 32 k) a warp loads before it splits them

// BF16 operands, [split][chunk of 8 k][row][16 bytes]
constexpr int SM_L_CHUNK = SM_SMALL_TN * 16;
constexpr int SM_R_CHUNK = SM_SMALL_TM * 16;
constexpr int SM_L_SPLIT = 4 * SM_L_CHUNK;
constexpr int SM_R_SPLIT = 4 * SM_R_CHUNK;
constexpr int SM_OFF_R = 3 * SM_L_SPLIT;
constexpr int SM_OFF_CTL = SM_OFF_R + 3 * SM_R_SPLIT;  // unit slots, mbarrier, flags
constexpr int SM_BYTES = SM_OFF_CTL + 2 * 80 + 16;
static_assert(SM_OFF_CTL % 16 == 0, "slots are read in 16-byte words");
static_assert(SM_KC * SM_BK == SM_SMALL_CHUNK && SM_SUM == SM_SUM_ROWS &&
              SM_SUM + SM_SUM_ROWS <= SM_CORR && 2 * SM_SUM_ROWS == SM_SMALL_TM, "chunk sums");

// Next-unit record in shared memory: the entry and its place in the item.
struct __align__(16) SmallSlot {
  LibShalom_sgemm_entry e;
  int tile;   // tile of the run | hold << 4, -1 past the last item
  int pad[3];
};
static_assert(sizeof(SmallSlot) == 80, "entry words are copied by 16 lanes");

// Takes a number from the work counter.  Inline PTX: for atomicAdd the
// compiler aggregates over the warp and waits for the result on the spot,
// which would put the atomic's round trip into every unit.
__device__ __forceinline__ unsigned fetch_inc(unsigned *p) {
  unsigned v;
  asm volatile("atom.global.add.u32 %0, [%1], 1;" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// UNIFORM_HOLD: uniform batches run the HOLD loop.  Grouped batches run it on the
// items that need it, which come first, and then the other loop.
template <int NSPLIT, bool UNIFORM, bool UNIFORM_HOLD>
__global__ void __launch_bounds__(SM_THREADS, SM_PER_SM) k_tc_small(const TcSmallArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  if constexpr (!UNIFORM) {  // the plan
    chain_wait();
    chain_next();
  }
  // no static shared memory: it would move the operands off their alignment
  SmallSlot *slots = reinterpret_cast<SmallSlot *>(smem + SM_OFF_CTL);
  uint64_t &bar = *reinterpret_cast<uint64_t *>(smem + SM_OFF_CTL + 2 * sizeof(SmallSlot));
  uint32_t &tmem_slot = reinterpret_cast<uint32_t *>(&bar)[2];
  volatile int *s_abort = reinterpret_cast<volatile int *>(&bar) + 3;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = ptx::smem_u32(smem);

  if (tid == 0) {
    ptx::mbar_init(&bar, 1);
    *s_abort = 0;
    ptx::fence_mbar_init();
  }
  if (warp == 0) {
    ptx::tmem_alloc(&tmem_slot, SM_TMEM_COLS);
    ptx::tmem_relinquish();
  }

  const long n_hold = UNIFORM ? 0 : (long)a.n_items_dev[1];
  const long n_items = UNIFORM ? a.n_items : n_hold + (long)a.n_items_dev[0];
  auto list = [&](long i) { return i < n_hold ? a.items[a.n_slots - 1 - i] : a.items[i - n_hold]; };
  long item = blockIdx.x;

  // Item pipeline of warp 1 (grouped batches): the list words of the next two
  // items are loaded a unit ahead of use, the next unit's entry while the
  // current unit's operands are on their way; after the first two rounds the
  // items come from a counter, so that CTAs with heavy items take fewer.
  uint2 it0 = make_uint2(0, 0), it1 = it0;  // current / next item (list words)
  bool have0 = item < n_items, have1 = false;
  int p = 0;  // product of the current item
  unsigned idx2 = 0;
  if (!UNIFORM && warp == 1) {
    if (have0) it0 = list(item);
    const long i1 = item + gridDim.x;
    have1 = i1 < n_items;
    if (have1) it1 = list(i1);
    if (lane == 0) idx2 = fetch_inc(a.counter);
    if (have0 && lane < 16)
      reinterpret_cast<uint32_t *>(&slots[0].e)[lane] =
          reinterpret_cast<const uint32_t *>(a.entries + it0.x)[lane];
    if (lane == 16) slots[0].tile = have0 ? (int)(it0.y & 31) : -1;
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = tmem_slot;

  // lane map of a row group: row `lrow` of 8, chunk `kc8` of 8 k; the 16-byte
  // shared stores of a quarter warp cover 128 consecutive bytes
  const int lrow = lane & 7, kc8 = lane >> 3;

  unsigned js = 0;  // slabs committed so far (mbarrier phase)
  bool stop = false;
  unsigned u = 0;
  auto units = [&](auto hold_loop) {
    constexpr bool HOLD = decltype(hold_loop)::value;
    constexpr int EDGE_M = HOLD ? SM_SUM_ROWS : SM_SMALL_TM;
    for (; !stop; ++u) {
      // ---- the unit: one product on one tile ----
      const float *A, *B;
      float *C, alpha, beta;
      int M, N, K, transb, m0, n0;
      unsigned lda, ldb;
      long ldc;
      bool next_valid = false;
      uint32_t next_word = 0;
      int next_tile = -1;
      if (UNIFORM) {
        if (item >= n_items) break;
        const long g = a.tiles == 1 ? item : item / a.tiles;
        const int t = a.tiles == 1 ? 0 : (int)(item - g * a.tiles);
        A = a.A + g * a.sA; B = a.B + g * a.sB; C = a.C + g * a.sC;
        M = a.M; N = a.N; K = a.K; transb = a.transb;
        lda = a.lda; ldb = a.ldb; ldc = a.ldc; alpha = a.alpha; beta = a.beta;
        const int tm = a.tiles_n == 1 ? t : t / a.tiles_n;
        m0 = tm * EDGE_M;
        n0 = (t - tm * a.tiles_n) * SM_SMALL_TN;
        item += gridDim.x;
      } else {
        const SmallSlot &sl = slots[u & 1];
        if (sl.tile < 0 || (sl.tile >= 16) != HOLD) break;
        const int t = sl.tile & 15;
        A = sl.e.A; B = sl.e.B; C = sl.e.C;
        M = sl.e.M; N = sl.e.N; K = max(0, sl.e.K); transb = sl.e.transb;
        lda = sl.e.lda > 0 ? sl.e.lda : K;
        ldb = sl.e.ldb > 0 ? sl.e.ldb : (transb ? K : N);
        ldc = sl.e.ldc > 0 ? sl.e.ldc : N;
        alpha = sl.e.alpha; beta = sl.e.beta;
        // at most two tile columns (N <= 256)
        const int two = N > SM_SMALL_TN ? 1 : 0;
        m0 = (t >> two) * EDGE_M;
        n0 = (t & two) * SM_SMALL_TN;
      }
      const int mrows = min(EDGE_M, M - m0), ncols = min(SM_SMALL_TN, N - n0);
      const int gR = (mrows + 7) >> 3, gL = (ncols + 7) >> 3;
      const bool m64 = ncols <= 64;
      const uint32_t idesc = m64 ? ptx::idesc_bf16_f32(64, gR * 8)
                                 : ptx::idesc_bf16_f32(128, (mrows + 15) / 16 * 16);
      const int nk = max(1, (K + SM_BK - 1) / SM_BK);
      // per-lane sources and destinations of the two operands (leading
      // dimensions below 2^30: byte strides fit 32 bits)
      const unsigned ldaB = 4 * lda, ldbB = 4 * ldb;
      const char *pR = reinterpret_cast<const char *>(A + 8 * kc8) + (uint64_t)ldaB * (unsigned)m0;
      const char *pL = transb ? reinterpret_cast<const char *>(B + 8 * kc8) + (uint64_t)ldbB * (unsigned)n0
                              : reinterpret_cast<const char *>(B + n0) + (uint64_t)ldbB * (unsigned)(8 * kc8);
      const unsigned rowL = transb ? ldbB : 4u;
      const uint64_t slabL = transb ? 4u * SM_BK : (uint64_t)ldbB * SM_BK;
      const bool vecR = (reinterpret_cast<uintptr_t>(A) & 15) == 0 && (lda & 3) == 0;
      const bool vecL = transb && (reinterpret_cast<uintptr_t>(B) & 15) == 0 && (ldb & 3) == 0;
      const uint32_t dR = sbase + SM_OFF_R + kc8 * SM_R_CHUNK + lrow * 16;
      const uint32_t dL = sbase + kc8 * SM_L_CHUNK + lrow * 16;

      // column of this thread in the accumulator, rows 8 ch .. 8 ch + 7 a chunk
      const int jc = m64 ? warp * 16 + lane : warp * 32 + lane;
      const bool cok = (!m64 || lane < 16) && jc < ncols;
      const bool warp_on = (m64 ? warp * 16 : warp * 32) < ncols;
      const uint32_t acc = tmem + ((uint32_t)(warp * 32) << 16);
      const uint64_t ldcB = 4 * (uint64_t)ldc;
      float *const c0 = C + (long)m0 * ldc + n0 + jc;

      for (int s = 0; s < nk; ++s) {
        const int kleft = K - s * SM_BK;
        const int sh = kleft > 16 ? 1 : 0;  // two k-steps, or one
        const int kv = kleft - 8 * kc8;     // valid k of this lane's chunk
        const int G = gR + gL;
        for (int b = warp; b < G; b += SM_WARPS * SM_BATCH) {
          float x[SM_BATCH][8];
#pragma unroll
          for (int q = 0; q < SM_BATCH; ++q) {
            const int g = b + SM_WARPS * q;
            if (g < G) {
              // rows past the last are read as the last one: they reach only
              // output rows and columns that are never stored
              const bool isL = g >= gR;
              const int gi = isL ? g - gR : g;
              const unsigned row = min(gi * 8 + lrow, (isL ? ncols : mrows) - 1);
              const char *src = (isL ? pL : pR) + (uint64_t)row * (isL ? rowL : ldaB);
              if ((isL ? vecL : vecR) && kleft >= SM_BK) {
                const float4 u0 = __ldg(reinterpret_cast<const float4 *>(src));
                const float4 u1 = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                x[q][0] = u0.x; x[q][1] = u0.y; x[q][2] = u0.z; x[q][3] = u0.w;
                x[q][4] = u1.x; x[q][5] = u1.y; x[q][6] = u1.z; x[q][7] = u1.w;
              } else if (!isL || transb) {
                const float *f = reinterpret_cast<const float *>(src);
                if (kleft >= SM_BK) {
#pragma unroll
                  for (int t = 0; t < 8; ++t) x[q][t] = __ldg(f + t);
                } else {
#pragma unroll
                  for (int t = 0; t < 8; ++t) x[q][t] = t < kv ? __ldg(f + t) : 0.0f;
                }
              } else {
                if (kleft >= SM_BK) {
#pragma unroll
                  for (int t = 0; t < 8; ++t)
                    x[q][t] = __ldg(reinterpret_cast<const float *>(src + (uint64_t)ldbB * t));
                } else {
#pragma unroll
                  for (int t = 0; t < 8; ++t)
                    x[q][t] = t < kv ? __ldg(reinterpret_cast<const float *>(src + (uint64_t)ldbB * t))
                                     : 0.0f;
                }
              }
            }
          }
          if (!UNIFORM && warp == 1 && s == 0 && b == warp) {
            // what comes next: this item's next product, or the next item
            if (++p >= (int)(it0.y >> 5)) {
              it0 = it1;
              have0 = have1;
              p = 0;
              const long i2 = 2L * gridDim.x + __shfl_sync(0xffffffffu, idx2, 0);
              have1 = i2 < n_items;
              if (have1) it1 = list(i2);
              if (lane == 0 && have1) idx2 = fetch_inc(a.counter);
            }
            next_valid = have0;
            next_tile = (int)(it0.y & 31);
            if (have0 && lane < 16)
              next_word = reinterpret_cast<const uint32_t *>(a.entries + it0.x + p)[lane];
          }
          // the previous slab's MMAs have read the operands
          if (b == warp && js > 0) ws_wait(&bar, (js - 1) & 1, s_abort, a.err);
#pragma unroll
          for (int q = 0; q < SM_BATCH; ++q) {
            const int g = b + SM_WARPS * q;
            if (g < G) {
              const bool isL = g >= gR;
              const uint32_t d = isL ? dL + (g - gR) * 128 : dR + g * 128;
              const uint32_t sp = isL ? SM_L_SPLIT : SM_R_SPLIT;
              uint4 h, m, l;
              split8<NSPLIT>(x[q], h, m, l);
              sts128(d, h);
              sts128(d + sp, m);
              if (NSPLIT == 3) sts128(d + 2 * sp, l);
            }
          }
        }
        pR += 4 * SM_BK;
        pL += slabL;
        if (!UNIFORM && s == nk - 1 && warp == 1) {
          SmallSlot &ns = slots[(u + 1) & 1];
          if (lane < 16) reinterpret_cast<uint32_t *>(&ns.e)[lane] = next_word;
          if (lane == 16) ns.tile = next_valid ? next_tile : -1;
        }
        ptx::fence_proxy_async_smem();
        ptx::tc_fence_before();  // TMEM reads of the last epilogue
        __syncthreads();
        if (*s_abort) {
          stop = true;
          break;
        }
        const int s_in = s % SM_KC;
        if (warp == 0) {
          if (ptx::elect_one()) {
            ptx::tc_fence_after();
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
              if (ks > sh) break;
              const uint32_t first = (s_in > 0 || ks > 0) ? 1u : 0u;
              uint64_t da[3], db[3];
#pragma unroll
              for (int sp = 0; sp < NSPLIT; ++sp) {
                da[sp] = ptx::smem_desc(sbase + sp * SM_L_SPLIT + ks * 2 * SM_L_CHUNK, SM_L_CHUNK, 128);
                db[sp] = ptx::smem_desc(sbase + SM_OFF_R + sp * SM_R_SPLIT + ks * 2 * SM_R_CHUNK,
                                        SM_R_CHUNK, 128);
              }
              ptx::mma_bf16(tmem, da[0], db[0], idesc, first);
              // the order of k_tc_sgemm (uniform) / k_tc_grouped, for their bits
              constexpr int P = UNIFORM ? 1 : 0, Q = 1 - P;
              ptx::mma_bf16(tmem + SM_CORR, da[P], db[Q], idesc, first);
              ptx::mma_bf16(tmem + SM_CORR, da[Q], db[P], idesc, 1u);
              if (NSPLIT == 3) {
                ptx::mma_bf16(tmem + SM_CORR, da[2 * P], db[2 * Q], idesc, 1u);
                ptx::mma_bf16(tmem + SM_CORR, da[2 * Q], db[2 * P], idesc, 1u);
                ptx::mma_bf16(tmem + SM_CORR, da[1], db[1], idesc, 1u);
              }
            }
            ptx::mma_commit(&bar);
          }
          __syncwarp();
        }
        ++js;
        if (s_in != SM_KC - 1 && s != nk - 1) continue;

        // ---- epilogue of a K chunk: sum += alpha D (uniform: sum += D), and
        // after the last chunk C = sum + beta C (uniform: alpha sum + beta C).
        // Grouped products with beta == 1 (accumulation, every run's later
        // products) add by fire-and-forget reductions at L2, as in k_tc_grouped;
        // other reads of C (and of a sum kept there) come from L2 and run one
        // step of 8 rows ahead of their use ----
        char *pc = reinterpret_cast<char *>(c0);
        constexpr int ER = 8;  // rows a step
        float c[ER];
        auto load_c = [&](const char *p, int nr) {
#pragma unroll
          for (int w = 0; w < ER; ++w)
            c[w] = ldcg_if(reinterpret_cast<const float *>(p + ldcB * w), w < nr);
        };
        const bool first = s < SM_KC, last = s == nk - 1;
        // 0: store, 1: reduce, 2: read first
        const int how = !UNIFORM && beta == 1.0f && last        ? 1
                        : (!HOLD && !first) || (last && beta != 0.0f) ? 2
                                                                      : 0;
        int nr = cok ? mrows : 0;  // rows of this thread still to come
        if (how == 2) load_c(pc, nr);
        const bool ok = ws_wait(&bar, (js - 1) & 1, s_abort, a.err);
        ptx::tc_fence_after();
        if (!warp_on || !__all_sync(0xffffffffu, ok)) continue;
        const uint64_t alpha2 = pack2(alpha, alpha);
        const uint64_t scale = UNIFORM && nk > SM_KC ? pack2(1.0f, 1.0f) : alpha2;
#pragma unroll 1
        for (int r = 0; r < mrows; r += ER, nr -= ER) {
          float v[ER], dc[ER], sum[ER];
          ptx::tmem_ld8(acc + r, v);
          ptx::tmem_ld8(acc + SM_CORR + r, dc);
          if (HOLD && !first) ptx::tmem_ld8(acc + SM_SUM + r, sum);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int w = 0; w < ER; w += 2) {
            const uint64_t d2 = add2(pack2(v[w], v[w + 1]), pack2(dc[w], dc[w + 1]));
            const uint64_t s2 = first  ? 0ull
                                : HOLD ? pack2(sum[w], sum[w + 1])
                                       : pack2(c[w], c[w + 1]);
            unpack2(fma2(scale, d2, s2), v[w], v[w + 1]);
          }
          if (UNIFORM && HOLD && last) {
#pragma unroll
            for (int w = 0; w < ER; ++w) v[w] *= alpha;
          }
          if (HOLD && !last) {
            ptx::tmem_st8(acc + SM_SUM + r, v);
          } else if (how == 1) {
#pragma unroll
            for (int w = 0; w < ER; ++w)
              red_add_if(reinterpret_cast<float *>(pc + ldcB * w), v[w], w < nr);
          } else {
            if (how == 2) {
              // (C was read for beta; the two forms are one condition, each the
              // faster code in its kernel: 45 x 37 x 51 93.5 us against 96.6)
              if (UNIFORM ? last && beta != 0.0f : HOLD || first) {
#pragma unroll
                for (int w = 0; w < ER; ++w)
                  v[w] = __fmaf_rn(beta, c[w], v[w]);
              } else if (UNIFORM && last) {
#pragma unroll
                for (int w = 0; w < ER; ++w) v[w] *= alpha;
              }
              load_c(pc + ldcB * ER, nr - ER);
            }
#pragma unroll
            for (int w = 0; w < ER; ++w)
              st_if(reinterpret_cast<float *>(pc + ldcB * w), v[w], w < nr);
          }
          pc += ldcB * ER;
        }
        if (HOLD) ptx::tmem_wait_st();
      }
    }
  };
  if constexpr (UNIFORM) {
    units(std::integral_constant<bool, UNIFORM_HOLD>());
  } else {
    units(std::true_type());
    units(std::false_type());
  }

  // every MMA has completed: the last unit's epilogue waited for its commit
  // (after an expired wait: a bounded chance to finish)
  if (*s_abort && js > 0) ptx::mbar_wait_bounded(&bar, (js - 1) & 1);
  ptx::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, SM_TMEM_COLS);
  }
}

template <int NSPLIT>
int small_launch(const TcSmallArgs &a, bool uniform, bool hold) {
  State &st = state();
  auto kern = uniform ? (hold ? k_tc_small<NSPLIT, true, true> : k_tc_small<NSPLIT, true, false>)
                      : k_tc_small<NSPLIT, false, false>;
  (void)occupancy_of((const void *)kern, SM_THREADS, SM_BYTES, SM_PER_SM);
  const int grid = grid_for(uniform ? a.n_items : (long)st.num_sms * SM_PER_SM, SM_PER_SM);
  if (!uniform) return launch_chained(kern, grid, SM_THREADS, SM_BYTES, st.stream, a);
  kern<<<grid, SM_THREADS, SM_BYTES, st.stream>>>(a);
  LS_CUDA_TRY(cudaGetLastError());
  return LIBSHALOM_SUCCESS;
}

}  // namespace

int tc_small_launch(const TcSmallArgs &a, bool uniform, bool hold, int mode) {
  return mode == LIBSHALOM_PREC_BF16X6 ? small_launch<3>(a, uniform, hold)
                                       : small_launch<2>(a, uniform, hold);
}

}  // namespace ls
