// sm_100a building blocks shared by the tensor-core kernels: mbarriers with bounded waits, TMA tile
// loads, shared-memory descriptors, tcgen05 MMA / commit / TMEM loads, tensor-map encoding.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "mgq_internal.h"

namespace mgq {

constexpr uint32_t kWaitLimit = 1u << 20;          // try_wait calls before a wait gives up (each may sleep for a short hardware quantum)

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit ran out (the CTA's flag and the device-wide error word are then
// raised) or another role of this CTA already gave up.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity, volatile int *failed, unsigned int *error)
{
    for (uint32_t i = 0; i < kWaitLimit; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*failed) return false;
    }
    *failed = 1;
    atomicExch(error, 1u);
    return false;
}
// A converged warp waits for several barriers at once, a lane (with `mine` set) for each: the try_waits share one latency.
__device__ __forceinline__ bool mbar_wait_lanes(unsigned long long *bar, uint32_t parity, bool mine, volatile int *failed, unsigned int *error)
{
    bool done = !mine;
    for (uint32_t i = 0; i < kWaitLimit; i++) {
        if (!done) done = mbar_try_wait(bar, parity);
        if (__all_sync(0xffffffffu, done)) return true;
        if (__any_sync(0xffffffffu, *failed != 0)) return false;
    }
    *failed = 1;
    atomicExch(error, 1u);
    return false;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, unsigned long long *bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}

// kind::f16 instruction descriptor: D f32, A bf16, B bf16, both K-major.
__host__ __device__ constexpr uint32_t umma_instr(uint32_t m, uint32_t n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24); }

// Operands in shared memory are K-major in the 128-byte swizzle, their descriptors given by the low word: address / 16 in bits 0-13,
// a leading byte offset (unused for a swizzled K-major operand) in bits 16-29.  The high word is a constant, so that a step
// costs one add per operand: stride byte offset (8-row groups, 1024 B) / 16 in bits 32-45, version 1 (Blackwell) in bits 46-47,
// SWIZZLE_128B = 2 in bits 61-63.
constexpr uint32_t kDescHigh = (1024 >> 4) | (1u << 14) | (2u << 29);
template <bool ACC>
__device__ __forceinline__ void umma_step(uint32_t tmem_d, uint32_t a16, uint32_t b16, uint32_t instr)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
                 "setp.ne.b32 p, %5, 0;\n\t"
                 "mov.b64 da, {%1, %4};\n\tmov.b64 db, {%2, %4};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(a16 | 0x10000u), "r"(b16 | 0x10000u), "r"(instr), "r"(kDescHigh), "n"(ACC ? 1 : 0) : "memory");
}
// D[128 lanes, N] (+)= A (f16 pairs in TMEM, 8 columns) . B (shared memory)
template <bool ACC>
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint32_t b16, uint32_t instr)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
                 "setp.ne.b32 p, %5, 0;\n\t"
                 "mov.b64 db, {%2, %4};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b16 | 0x10000u), "r"(instr), "r"(kDescHigh), "n"(ACC ? 1 : 0) : "memory");
}
// D = A . B + D * 2^-SHIFT
template <uint32_t SHIFT>
__device__ __forceinline__ void umma_f16_ts_scaled(uint32_t d, uint32_t a, uint32_t b16, uint32_t instr)
{
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
                 "setp.ne.b32 p, 1, 0;\n\t"
                 "mov.b64 db, {%2, %4};\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p, %5;\n\t}"
                 ::"r"(d), "r"(a), "r"(b16 | 0x10000u), "r"(instr), "r"(kDescHigh), "n"(SHIFT) : "memory");
}
// One lane of a converged warp.
__device__ __forceinline__ bool elect_one()
{
    uint32_t is;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(is));
    return is != 0;
}
__device__ __forceinline__ void umma_commit(unsigned long long *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 columns of this lane's row.
__device__ __forceinline__ void tmem_ld32(uint32_t addr, float (&y)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) y[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&r)[16])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
                 "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t *base_smem, uint32_t columns)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(base_smem)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t columns)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
int encode_fn(EncodeTiledFn &out);                 // mgq_linear_tc.cu

}  // namespace mgq
