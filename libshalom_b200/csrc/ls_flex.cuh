// ls_flex.cuh -- plain FP32 GEMM tile of any size up to MAXM x MAXN for a CTA
// of 128 threads (uniform and grouped batches).
//
// A tile of mrows x ncols is covered by ceil(mrows / TM) x ceil(ncols / TN)
// threads of TM x TN outputs, laid out for the tile at hand, so a 52 x 104
// half of a 104^3 product keeps 7 x 13 of 128 threads busy instead of a
// quarter of a 128 x 128 tile's.  Several CTAs share an SM and hide each
// other's latencies; a tile's K slabs go through a ring of two stages (three on
// 32 x 32 tiles, which are for batches too small to fill the SMs).
//
// Both operands are staged k-major ([k][m], [k][n]) by cp.async straight from
// row-major global memory, whatever its layout: operands whose k runs along
// the row are transposed by the copies themselves (four bytes each: lanes
// take 8 k x 4 rows, 32 consecutive bytes of four rows, and with a pitch of
// 4 mod 32 words the writes fall on 32 different banks).  A k step of a
// thread is then TM / 4 + TN / 4 sixteen-byte loads, and no alignment is asked
// of the operands.
//
// The FMAs are packed along n (fma.rn.f32x2: two IEEE FMAs, the scalar ones'
// bits): the FMA pipe is no wider for it, but half the issue slots are left
// for the shared-memory loads.  Pairing 2 x 2 blocks with swapped columns
// instead of duplicating A values is slower in the kernel (64^3 208 against
// 188 us, 10,000 products).
//
// Bound by the shared-memory pipe (64^3: 74 % busy): the transposing
// four-byte copies take some ten wavefronts each.  Tried instead, on 104^3 NT
// (944 us then) / the mixed batch in one list (1.55 ms then): rows kept as they lie and read along
// k (967 us / 2.86 ms: a register move per pair of columns, more code),
// transposition through registers without (1,533 us / 2.49 ms) and with a
// slab of prefetch (1,341 us / 3.96 ms: spills), two loading warps a CTA
// ahead of four multiplying ones (1,868 us / 4.26 ms: too few loads in
// flight), one barrier a slab instead of two (1,035 us / 1.60 ms), threads
// ordered along m first (1,023 us / 1.58 ms).
//
// Rounding order: one FMA chain per element, k increasing, then
// C = fma(beta, C, alpha * sum), as in simt_tile.
#pragma once

#include "ls_f32x2.cuh"
#include "ls_simt.cuh"
#include "ls_sizes.h"

namespace ls {

constexpr int FX_THREADS = 128;
constexpr int FX_KS = 32;  // k per slab

template <int MAXM_, int MAXN_, int STAGES_ = 2>
struct FlexCfg {
  static constexpr int MAXM = MAXM_, MAXN = MAXN_, STAGES = STAGES_;
  static constexpr int PA = MAXM + 4, PB = MAXN + 4;  // pitches: 4 mod 32 words
  static constexpr int STAGE = FX_KS * (PA + PB);     // floats
  static constexpr int SMEM = STAGES * STAGE * 4;
  // ring position of slab s
  static __device__ __forceinline__ int slot(int s) {
    if constexpr (STAGES == 2) return s & 1;
    else return s % STAGES;
  }
  static_assert(PA % 32 == 4 && PB % 32 == 4, "transposing copies without bank conflicts");
  static_assert(MAXM * PB <= STAGES * STAGE, "the C tile goes through the ring");
};

struct FlexJob {
  const float *A, *B;
  float *C;
  int K, lda, ldb, ldc, transb;
  float alpha, beta;
};

__device__ __forceinline__ void fx_cp4(uint32_t saddr, const float *g, bool on) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "@p cp.async.ca.shared.global [%0], [%1], 4;\n\t}" ::"r"(saddr),
      "l"(g), "r"((int)on)
      : "memory");
}

// k-contiguous operand (rows of k at src, row stride ld) -> [k][row]
template <int PITCH>
__device__ __forceinline__ void fx_stage_k(uint32_t dst, const float *src, int ld, int rows,
                                           int kcnt, int warp, int lane) {
  const int kl = lane & 7, ml = lane >> 3;
  const uint32_t d0 = dst + (uint32_t)(kl * PITCH + ml) * 4;
  const float *s0 = src + kl;
  for (int r = 4 * warp; r < rows; r += FX_THREADS / 8) {
    const bool ok = r + ml < rows;
    const float *s = s0 + (long)(r + ml) * ld;
#pragma unroll
    for (int kb = 0; kb < FX_KS / 8; ++kb)
      fx_cp4(d0 + (uint32_t)(r + kb * 8 * PITCH) * 4, s + kb * 8, ok && kb * 8 + kl < kcnt);
  }
}

// row-contiguous operand (k rows at src, stride ld) -> [k][col]; vec: every k
// row starts on 16 bytes
template <int PITCH, int MAXC>
__device__ __forceinline__ void fx_stage_n(uint32_t dst, const float *src, int ld, int cols,
                                           int kcnt, bool vec, int tid) {
  if (vec) {
    constexpr int U = MAXC / 4, RPI = FX_THREADS / U;  // 16-byte units and k rows a pass
    const int u = tid % U, kr = tid / U, n = min(4, cols - 4 * u);
    if (n > 0) {
#pragma unroll
      for (int k = 0; k < FX_KS; k += RPI)
        if (k + kr < kcnt)
          simt_cp16(dst + (uint32_t)((k + kr) * PITCH + 4 * u) * 4, src + (long)(k + kr) * ld + 4 * u,
                    4 * n);
    }
  } else {
    constexpr int RPI = FX_THREADS / 32;
    const int c = tid & 31, kr = tid >> 5;
    for (int k = kr; k < kcnt; k += RPI) {
      const float *s = src + (long)k * ld + c;
      const uint32_t d = dst + (uint32_t)(k * PITCH + c) * 4;
#pragma unroll
      for (int q = 0; q < MAXC / 32; ++q) fx_cp4(d + q * 128, s + q * 32, c + q * 32 < cols);
    }
  }
}

__device__ __forceinline__ void fx_lds4(uint32_t a, float *v) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
               : "r"(a)
               : "memory");
}

__device__ __forceinline__ float fx_ld(const float *p, bool on) {
  float v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"((int)on)
      : "memory");
  return v;
}

// One product on one tile: C[m0.., n0..] = alpha A op(B) + beta C
template <class Cfg, int TM, int TN>
__device__ __forceinline__ void flex_tile(const FlexJob &j, int m0, int n0, int mrows, int ncols,
                                          float *smem) {
  constexpr int PA = Cfg::PA, PB = Cfg::PB;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
  const int TX = (ncols + TN - 1) / TN, TY = (mrows + TM - 1) / TM;
  const int ty = (int)(((float)tid + 0.5f) * (1.0f / (float)TX)), tx = tid - ty * TX;
  const bool on = ty < TY;
  const float *A = j.A + (long)m0 * j.lda;
  const float *B = j.transb ? j.B + (long)n0 * j.ldb : j.B + n0;
  const bool vec_b = (reinterpret_cast<uintptr_t>(B) & 15) == 0 && (j.ldb & 3) == 0;

  constexpr int AHEAD = Cfg::STAGES - 1;  // slabs on their way while one is multiplied
  auto issue = [&](int s) {
    const int k0 = s * FX_KS, kcnt = min(FX_KS, j.K - k0);
    const uint32_t sa = sbase + Cfg::slot(s) * Cfg::STAGE * 4, sb = sa + FX_KS * PA * 4;
    fx_stage_k<PA>(sa, A + k0, j.lda, mrows, kcnt, warp, lane);
    if (j.transb) fx_stage_k<PB>(sb, B + k0, j.ldb, ncols, kcnt, warp, lane);
    else fx_stage_n<PB, Cfg::MAXN>(sb, B + (long)k0 * j.ldb, j.ldb, ncols, kcnt, vec_b, tid);
  };

  // acc[i][q] = outputs (row i, columns 2 q, 2 q + 1) of the thread: rows
  // 4 ty + 4 TY g + 0..3, columns 4 tx + 4 TX g + 0..3
  uint64_t acc[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int q = 0; q < TN / 2; ++q) acc[i][q] = 0;

  const int nslab = ceil_div(j.K, FX_KS);
#pragma unroll
  for (int s = 0; s < AHEAD; ++s) {
    if (s < nslab) issue(s);
    simt_commit();
  }
  for (int s = 0; s < nslab; ++s) {
    if (s + AHEAD < nslab) issue(s + AHEAD);
    simt_commit();
    simt_wait<AHEAD>();
    __syncthreads();
    if (on) {
      uint32_t pa = sbase + Cfg::slot(s) * Cfg::STAGE * 4 + ty * 16;
      uint32_t pb = sbase + (Cfg::slot(s) * Cfg::STAGE + FX_KS * PA) * 4 + tx * 16;
      const int kcnt = min(FX_KS, j.K - s * FX_KS);
      auto step = [&](uint32_t qa, uint32_t qb) {
        float a[TM], b[TN];
#pragma unroll
        for (int g = 0; g < TM / 4; ++g) fx_lds4(qa + g * TY * 16, a + 4 * g);
#pragma unroll
        for (int g = 0; g < TN / 4; ++g) fx_lds4(qb + g * TX * 16, b + 4 * g);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          const uint64_t a2 = pack2(a[i], a[i]);
#pragma unroll
          for (int q = 0; q < TN / 2; ++q)
            acc[i][q] = fma2(a2, pack2(b[2 * q], b[2 * q + 1]), acc[i][q]);
        }
      };
      int k = 0;
      for (; k + 4 <= kcnt; k += 4, pa += 16 * PA, pb += 16 * PB) {
#pragma unroll
        for (int t = 0; t < 4; ++t) step(pa + t * PA * 4, pb + t * PB * 4);
      }
      for (; k < kcnt; ++k, pa += PA * 4, pb += PB * 4) step(pa, pb);
    }
    __syncthreads();
  }

  // epilogue: through shared memory, so that a warp writes 32 consecutive
  // floats of a C row whatever its alignment
  if (on) {
    const uint32_t pc = sbase + tx * 16;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int r = 4 * ((i / 4) * TY + ty) + i % 4;
#pragma unroll
      for (int g = 0; g < TN / 4; ++g) {
        float c[4];
        unpack2(acc[i][2 * g], c[0], c[1]);
        unpack2(acc[i][2 * g + 1], c[2], c[3]);
        if (r < mrows)
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(pc + g * TX * 16 + r * (PB * 4)),
                       "f"(j.alpha * c[0]), "f"(j.alpha * c[1]), "f"(j.alpha * c[2]),
                       "f"(j.alpha * c[3])
                       : "memory");
      }
    }
  }
  __syncthreads();
  // eight elements a thread at a time, C read for all of them first: one by one,
  // the loads of a 64 x 64 tile were a chain of 32 (a run of 128 products of 64^3
  // 1,454 us instead of 914, 10,000 products of 24^3 49 instead of 39)
  constexpr int W = FX_THREADS / 32, Q = Cfg::MAXN / 32, U = 8 / Q;
  const bool read = j.beta != 0.0f;
  for (int r0 = warp; r0 < mrows; r0 += W * U) {
    float *c0 = j.C + (long)(m0 + r0) * j.ldc + n0 + lane;
    float cv[U][Q];
    if (read) {
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < Q; ++q)
          cv[u][q] = fx_ld(c0 + (long)(u * W) * j.ldc + q * 32,
                           r0 + u * W < mrows && lane + q * 32 < ncols);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (r0 + u * W < mrows && lane + q * 32 < ncols) {
          float v = smem[(r0 + u * W) * PB + lane + q * 32];
          if (read) v = __fmaf_rn(j.beta, cv[u][q], v);
          c0[(long)(u * W) * j.ldc + q * 32] = v;
        }
      }
  }
  __syncthreads();  // the ring is free for the next tile
}

}  // namespace ls
