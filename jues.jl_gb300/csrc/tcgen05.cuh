// PTX wrappers shared by the tcgen05 kernels: bounded mbarrier waits, TMA loads, TMEM, MMA issue.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace jues {
namespace {

constexpr unsigned long long WAIT_LIMIT_NS = 2ull * 1000 * 1000 * 1000;    // 2 s: legitimate waits last microseconds

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// try_wait with a suspend-time hint: a waiting thread sleeps until the phase completes (or up to
// 20 us) instead of polling, which keeps the spinning warps off the shared-memory pipe the
// tensor cores read their operands through
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
// bounded wait; false when the time limit expired, another thread of the CTA aborted, or
// another CTA already raised FLAG_TIMEOUT
__device__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                          const volatile unsigned *gflags) {
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 15u) == 15u) {
            if (*abort_flag || (*gflags & FLAG_TIMEOUT)) return false;
            unsigned long long t = gtimer();
            if (t0 == 0) t0 = t;
            else if (t - t0 > WAIT_LIMIT_NS) return false;
        }
    }
}
// the same by a whole warp in step, with a warp-uniform outcome
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, volatile int *abort_flag,
                                               const volatile unsigned *gflags) {
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (__any_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if ((it & 15u) == 15u) {
            const unsigned long long t = gtimer();
            if (t0 == 0) t0 = t;
            if (__any_sync(0xffffffffu, *abort_flag || (*gflags & FLAG_TIMEOUT) || t - t0 > WAIT_LIMIT_NS)) return false;
        }
    }
}
// bounded wait that ignores the abort flags: used only to let this CTA's own asynchronous
// copies and MMAs settle before it frees TMEM and exits
__device__ __forceinline__ bool mbar_wait_quiet(uint64_t *bar, uint32_t parity) {
    unsigned long long t0 = 0;
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 15u) == 15u) {
            unsigned long long t = gtimer();
            if (t0 == 0) t0 = t;
            else if (t - t0 > WAIT_LIMIT_NS) return false;
        }
    }
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y,
                                            int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem] (+)= A[smem] . B[smem]^T, 16-bit inputs, FP32 accumulation, issued by a whole warp in step (one
// elected lane issues).  Both tiles are K-major as TMA writes them with 128-byte swizzle: the shared-memory
// descriptor has the start address >> 4, LBO unused (1), SBO = 1024 bytes between 8-row groups, version 1 and layout
// type 2 (SWIZZLE_128B).  With warp-uniform loops and
// operands an MMA costs a few issue slots; a loop that one lane runs alone takes about 100 clocks per
// MMA, more than a narrow MMA itself.  alo, blo: low words of sw128 descriptors (sw128_lo); the
// high word is constant.
__device__ __forceinline__ uint32_t sw128_lo(const void *smem) {
    return ((smem_u32(smem) & 0x3FFFFu) >> 4) | (1u << 16);
}
__device__ __forceinline__ void umma_warp(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 a, {%1, 0x40004040};\n\tmov.b64 b, {%2, 0x40004040};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}\n" ::"r"(tmem_d),
        "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate)
        : "memory");
}
// four K = 16 steps (64 K values, one 128-byte swizzle row: 32 bytes a step)
__device__ __forceinline__ void umma_warp_x4(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t.reg .b64 a, b;\n\t.reg .b32 x, y;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "mov.b64 a, {%1, 0x40004040};\n\tmov.b64 b, {%2, 0x40004040};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t"
        "add.u32 x, %1, 2;\n\tadd.u32 y, %2, 2;\n\t"
        "mov.b64 a, {x, 0x40004040};\n\tmov.b64 b, {y, 0x40004040};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
        "add.u32 x, %1, 4;\n\tadd.u32 y, %2, 4;\n\t"
        "mov.b64 a, {x, 0x40004040};\n\tmov.b64 b, {y, 0x40004040};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t"
        "add.u32 x, %1, 6;\n\tadd.u32 y, %2, 6;\n\t"
        "mov.b64 a, {x, 0x40004040};\n\tmov.b64 b, {y, 0x40004040};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, t;\n\t}\n" ::"r"(tmem_d),
        "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate)
        : "memory");
}
// one K = 32 step of 8-bit floats; both tiles 64 bytes a row in TMA's 64-byte swizzle (8-row groups of 512 bytes)
__device__ __forceinline__ void umma_warp_f8(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 a, {%1, 0x80004020};\n\tmov.b64 b, {%2, 0x80004020};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p;\n\t}\n" ::"r"(tmem_d),
        "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit_warp(uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(smem_u32(bar))
        : "memory");
}
// 32 lanes x 32 consecutive 32-bit TMEM columns -> 32 registers per thread
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
          "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
// 32 lanes x 8 consecutive 32-bit TMEM columns -> 8 registers per thread
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// packed FP32 pairs (sm_100+): two round-to-nearest operations per instruction
__device__ __forceinline__ uint64_t pk2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pk2f(float lo, float hi) { return pk2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t fmul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float lo_f(uint64_t x) { return __uint_as_float((uint32_t)x); }
__device__ __forceinline__ float hi_f(uint64_t x) { return __uint_as_float((uint32_t)(x >> 32)); }
__device__ __forceinline__ void red_add_f64(double *p, double v) {
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

}  // namespace
}  // namespace jues
