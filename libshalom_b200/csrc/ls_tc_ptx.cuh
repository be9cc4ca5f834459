// ls_tc_ptx.cuh -- thin inline-PTX wrappers for the sm_100a tensor-core
// path: mbarriers, tcgen05 (TMEM allocation, MMA, commit, loads, fences) and
// the shared-memory / instruction descriptors the MMA consumes.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

#include "ls_f32x2.cuh"

namespace ls {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier --------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Like mbar_try_wait, but the thread may be suspended for up to `ns`
// nanoseconds until the phase completes.
__device__ __forceinline__ bool mbar_try_wait_suspend(uint64_t *bar, uint32_t parity,
                                                      uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait for the phase with the given parity.  Returns false when the
// iteration limit expires (about a second of polling with back-off).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 22); ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if (it > 64) __nanosleep(it < 4096 ? 32 : 256);
  }
  return false;
}

// ---- proxy fences ----------------------------------------------------------
// Makes this thread's generic-proxy shared-memory writes visible to the async
// proxy (the tensor core reads its operands through it).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---- TMA stores (shared -> global, bulk-group completion) --------------------
// 3-D tiled store of the box at smem address `src` to coordinates (c0, c1, c2)
// of the tensor map; elements outside the tensor's bounds are not written.
__device__ __forceinline__ void tma_store_3d(const void *map, uint32_t src, int c0, int c1,
                                             int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(src), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// at most N of this thread's bulk-store groups are still reading their
// shared-memory source
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
// this thread's bulk stores are complete (written to global memory)
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// ---- tcgen05 ---------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc], kind::f16 (bf16 inputs, f32 accumulate)
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same with A in TMEM (row r in lane r, two BF16 a column)
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// True in one lane of a converged warp.  MMAs issued under this predicate
// keep their descriptors in uniform registers: a burst of 12 MMAs of
// 128 x 32 x 16 takes 471 cycles to issue instead of 658 under `lane == 0`
// (64 x 32 x 16: 311 instead of 658).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// Arrives (once) on the mbarrier when all tcgen05 ops issued so far by this
// thread have completed.
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// 32 lanes x 8 consecutive 32-bit columns: thread i of the warp gets lane
// (base lane + i), columns col .. col+7.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float *v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
// thread i of the warp writes columns col .. col+3 of lane (base lane + i)
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint4 &v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr),
               "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float *v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ---- descriptors -------------------------------------------------------------
// Shared-memory matrix descriptor, K-major, no swizzle ("interleaved" core
// matrices of 8 rows x 16 bytes):
//   bits  0-13 start address >> 4
//   bits 16-29 leading byte offset >> 4 (distance between the two 8-element
//              K chunks of one MMA)
//   bits 32-45 stride byte offset >> 4 (distance between 8-row groups)
//   bits 46-47 descriptor version (1 on sm_100)
//   bits 61-63 layout (0 = no swizzle)
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of tcgen05.mma kind::f16: D f32, A and B bf16, both
// K-major; M = 128 with N a multiple of 16, or M = 64 with N a multiple of 8 (N <=
// 256).
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int m, int n) {
  return (1u << 4)                        // D format f32
         | (1u << 7)                      // A format bf16
         | (1u << 10)                     // B format bf16
         | ((uint32_t)(n >> 3) << 17)     // N >> 3
         | ((uint32_t)(m >> 4) << 24);    // M >> 4
}

}  // namespace ptx

// ---- hand-offs shared by the tensor-core kernels -------------------------------
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ptx::smem_u32(bar)) : "memory");
}
// Arrival that publishes no memory.  The default arrive has release
// semantics: it orders this thread's earlier memory operations, the
// epilogue's global C stores included, before the arrival.  Arrivals that
// only say "done reading" (TMEM read back and waited for, a queue slot
// copied into registers) have nothing to publish.
__device__ __forceinline__ void mbar_arrive_relaxed(uint64_t *bar) {
  asm volatile("mbarrier.arrive.relaxed.cta.shared::cta.b64 _, [%0];" ::"r"(ptx::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%1], %0;" ::"r"(bytes),
               "r"(ptx::smem_u32(bar))
               : "memory");
}
// Slow path of ws_wait: the thread suspends in the barrier wait (up to about
// a microsecond per try, woken when the phase completes) instead of polling,
// so waiting roles take no issue slots or shared-memory bandwidth from the
// working ones.  Gives up after `limit` tries or two seconds, whichever
// comes first, or as soon as another role has aborted.  Inlined: a call
// would make the caller save its live registers to local memory around every
// wait.
__device__ __forceinline__ bool ws_wait_slow(uint64_t *bar, uint32_t parity,
                                             volatile int *abort_flag, unsigned *err,
                                             uint32_t limit) {
  const uint64_t t0 = ptx::globaltimer_ns();
  for (uint32_t it = 0; it < limit; ++it) {
    if (ptx::mbar_try_wait_suspend(bar, parity, 1000)) return true;
    if ((it & 15) == 15) {
      if (*abort_flag) return false;
      if (ptx::globaltimer_ns() - t0 > 2000000000ull) break;
    }
  }
  *abort_flag = 1;
  atomicOr(err, 1u);
  return false;
}

// Bounded wait: one test inline, the rest in ws_wait_slow.
__device__ __forceinline__ bool ws_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                        unsigned *err, uint32_t limit = 1u << 22) {
  if (ptx::mbar_try_wait(bar, parity)) return true;
  return ws_wait_slow(bar, parity, abort_flag, err, limit);
}

// C[i] += v at L2 (red.global.add.f32: round to nearest even; subnormal
// inputs and sums flush to zero)
__device__ __forceinline__ void red_add_f32(float *p, float v) {
  asm volatile("red.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

// The split is the busiest step of these kernels' issue slots: the packed
// FMA takes the two subtractions of a pair at once.  x - float(b), both
// halves (exact: b is x rounded to BF16)
__device__ __forceinline__ uint64_t bf16_rest(uint64_t x, uint32_t b) {
  const uint64_t f = (uint64_t)(b & 0xffff0000u) << 32 | (uint64_t)(b << 16);
  return fma2(f, 0xbf800000bf800000ull, x);  // f * -1 + x
}
__device__ __forceinline__ uint32_t bf16_round(uint64_t x) {
  float lo, hi;
  unpack2(x, lo, hi);
  __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t *>(&b);
}

// split 8 floats into hi / mid / lo BF16 (packed pairs, element 0 in the low half)
template <int NSPLIT>
__device__ __forceinline__ void split8(const float *x, uint4 &h, uint4 &m, uint4 &l) {
  uint32_t hh[4], mm[4], ll[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint64_t x2 = pack2(x[2 * i], x[2 * i + 1]);
    hh[i] = bf16_round(x2);
    const uint64_t r2 = bf16_rest(x2, hh[i]);
    mm[i] = bf16_round(r2);
    ll[i] = NSPLIT == 3 ? bf16_round(bf16_rest(r2, mm[i])) : 0u;
  }
  h = make_uint4(hh[0], hh[1], hh[2], hh[3]);
  m = make_uint4(mm[0], mm[1], mm[2], mm[3]);
  l = make_uint4(ll[0], ll[1], ll[2], ll[3]);
}

// predicated global accesses (a predicate, not a branch, per access)
__device__ __forceinline__ void st_if(float *p, float v, bool on) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p),
               "f"(v), "r"((int)on)
               : "memory");
}
__device__ __forceinline__ void red_add_if(float *p, float v, bool on) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p red.global.add.f32 [%0], %1;\n\t}" ::"l"(p),
      "f"(v), "r"((int)on)
      : "memory");
}
__device__ __forceinline__ float ldcg_if(const float *p, bool on) {
  float v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t"
      "@p ld.global.cg.f32 %0, [%1];\n\t}"
      : "=f"(v)
      : "l"(p), "r"((int)on)
      : "memory");
  return v;
}

// 16 bytes to a 16-byte aligned shared-memory address
__device__ __forceinline__ void sts128(uint32_t saddr, const uint4 &v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

}  // namespace ls
