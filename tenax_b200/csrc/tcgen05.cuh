// tcgen05 / TMEM helpers shared by the sm_100a GEMM kernels: bounded
// mbarrier waits on the GPU timer, SWIZZLE_128B K-major smem descriptors,
// MMA issue/commit, TMEM loads and the tcgen05 thread-sync fences.
#pragma once

#include "common.cuh"

namespace tnx {

constexpr uint64_t kTimeoutNs = 2000000000ull;  // 2 s per wait

static __device__ __forceinline__ uint64_t gtimer() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// wait for phase `parity` of `bar`; false on abort (own deadline or another role's abort)
static __device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                              int32_t* err_flag) {
  uint64_t t0 = 0;
  for (uint32_t it = 0;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      uint64_t now = gtimer();
      if (t0 == 0) t0 = now;
      if (now - t0 > kTimeoutNs) {
        *abort_flag = 1;
        if (err_flag) atomicExch(err_flag, 1);
        return false;
      }
    }
  }
}

// One lane of a converged warp, always the same one.  The roles' loops run in
// all lanes of their warp and only the instruction itself is predicated on the
// elected lane (the `on` arguments below), so that addresses and descriptors are
// formed in warp-uniform code.
static __device__ __forceinline__ uint32_t elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p;
}

// wait_or_abort by a whole converged warp, with one answer for all its lanes
static __device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                          int32_t* err_flag) {
  return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, err_flag)) != 0;
}

// a value every lane of the warp holds, marked as such
static __device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }

static __device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);  // start address
  d |= static_cast<uint64_t>(1) << 16;                  // LBO (unused for SW128 K-major)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;          // SBO: 8 rows x 128 B
  d |= static_cast<uint64_t>(1) << 46;                  // descriptor version (sm_100)
  d |= static_cast<uint64_t>(2) << 61;                  // SWIZZLE_128B
  return d;
}

template <bool TF32>
static __device__ __forceinline__ void mma_issue(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  if constexpr (TF32) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
  } else {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
  }
}

// the same from the low words of SWIZZLE_128B descriptors (sw128_lo), whose high word is fixed
constexpr uint32_t kSw128Hi = (1024u >> 4) | (1u << 14) | (2u << 29);
static __device__ __forceinline__ uint32_t sw128_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | (1u << 16); }
template <bool TF32>
static __device__ __forceinline__ void mma_issue_lo(uint32_t d_tmem, uint32_t a, uint32_t b, uint32_t idesc,
                                                    uint32_t acc) {
  if constexpr (TF32) {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\n"
        "mov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(a), "r"(b), "r"(idesc), "r"(acc), "n"(kSw128Hi));
  } else {
    asm volatile(
        "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\n"
        "mov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(d_tmem),
        "r"(a), "r"(b), "r"(idesc), "r"(acc), "n"(kSw128Hi));
  }
}
// one slab's n K steps of A x B, 32 bytes each; acc0: whether the first one accumulates
template <bool TF32>
static __device__ __forceinline__ void mma_slab(uint32_t d_tmem, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc0,
                                                int n) {
  mma_issue_lo<TF32>(d_tmem, a, b, idesc, acc0);
  if (n == 4) {
    mma_issue_lo<TF32>(d_tmem, a + 2, b + 2, idesc, 1u);
    mma_issue_lo<TF32>(d_tmem, a + 4, b + 4, idesc, 1u);
    mma_issue_lo<TF32>(d_tmem, a + 6, b + 6, idesc, 1u);
  } else {
    for (int k = 1; k < n; ++k) mma_issue_lo<TF32>(d_tmem, a + 2 * k, b + 2 * k, idesc, 1u);
  }
}

// expect `bytes` on the barrier at shared address bar, and one bulk copy counted on it
static __device__ __forceinline__ void mbar_expect_tx_on(uint32_t on, uint32_t bar, uint32_t bytes) {
  asm volatile(
      "{\n.reg .pred q;\nsetp.ne.b32 q, %2, 0;\n"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}\n" ::"r"(bar), "r"(bytes), "r"(on)
      : "memory");
}
static __device__ __forceinline__ void bulk_g2s_on(uint32_t on, uint32_t dst, const void* src, uint32_t bytes,
                                                   uint32_t bar) {
  asm volatile(
      "{\n.reg .pred q;\nsetp.ne.b32 q, %4, 0;\n"
      "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n}\n" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "r"(on)
      : "memory");
}

static __device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

static __device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
static __device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

// 32 lanes x 32 consecutive fp32 columns: lane i receives row (quarter*32 + i)
static __device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 lanes x 4 chunks of 8 consecutive 32-bit columns (no wait): in each
// chunk j, thread t holds row t/4 in v[4j], v[4j+1] and row t/4 + 8 in
// v[4j+2], v[4j+3], columns 8j + 2(t%4) and 8j + 2(t%4) + 1
static __device__ __forceinline__ void tmem_ld16x256b_x4(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
static __device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }


// 32 lanes x 1 fp32 column (no wait): lane i receives row (quarter*32 + i)
static __device__ __forceinline__ uint32_t tmem_ld1(uint32_t taddr) {
  uint32_t v;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr));
  return v;
}

}  // namespace tnx
