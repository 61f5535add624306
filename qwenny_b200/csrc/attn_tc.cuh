// What the attention on the 5th-generation tensor cores needs beside pair_tc.cuh: wide tensor-memory loads and stores, the
// exact int8 -> f16 conversion of cache bytes, the 128-byte swizzle of a K-major tile, and bounded waits that sleep
// instead of polling.
#pragma once
#include "attn_common.cuh"
#include "pair_tc.cuh"

namespace qb {
namespace tc {

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,"
        "%31,%32};\n" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// two code bytes of a cache word -> two halves of their signed values, exactly: 1024 + (q + 128) by prmt, minus 1152
__device__ __forceinline__ uint32_t exact2(uint32_t w, uint32_t sel) {
    const uint32_t off = 0x64806480u;
    uint32_t v = __byte_perm(w, 0x64646464u, sel);
    __half2 r = __hsub2(*(__half2*)&v, *(const __half2*)&off);
    return *(uint32_t*)&r;
}

// byte offset of (row, 16-byte chunk) in a K-major tile with the 128-byte swizzle: 8-row groups of 1 KB
__device__ __forceinline__ uint32_t sw128(int row, int chunk) {
    return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
}

// try_wait with a suspend-time hint: the waiting thread sleeps until the phase completes or the hint (ns) runs out,
// instead of spending issue slots on polls
__device__ __forceinline__ bool mbar_try_wait_hint(uint64_t* bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_sleepy(uint64_t* bar, uint32_t parity) {
    for (uint32_t i = 0; i < (WAIT_LIMIT >> 4); i++)
        if (mbar_try_wait_hint(bar, parity, 2000)) return true;
    return false;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A bounded wait that remembers failure: once a wait ran out the role stops waiting and walks on
struct Waiter {
    int* err;
    int code;
    bool dead = false;
    __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity, int lane) {
        if (dead) return;
        bool ok = true;
        if (lane == 0) ok = mbar_wait_sleepy(bar, parity);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) {
            dead = true;
            if (lane == 0) atomicExch(err, code);
        }
    }
    // two barriers at once, a lane each: about as long as one wait (2048 rows of prompt attention at context 30720: 1917 us
    // without the second wait, 2024 with one after the other, 1930 so)
    __device__ __forceinline__ void wait_both(uint64_t* bar, uint32_t parity, uint64_t* bar1, uint32_t parity1, int lane) {
        if (dead) return;
        bool ok = true;
        if (lane < 2) ok = mbar_wait_sleepy(lane ? bar1 : bar, lane ? parity1 : parity);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            dead = true;
            if (lane == 0) atomicExch(err, code);
        }
        __syncwarp();  // (orders the other lanes' reads behind both)
    }
};

}  // namespace tc
}  // namespace qb
