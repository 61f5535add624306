// What the attention on the 5th-generation tensor cores needs beside pair_tc.cuh: wide tensor-memory loads and stores, the
// exact int8 -> f16 conversion of cache bytes, the 128-byte swizzle of a K-major tile, bounded waits of a warp, and the choice between its two forms.
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

// 2^x, results below 2^-126 as 0 (exp2f spends three more instructions on those; P is rounded to f16 next)
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A bounded wait of a whole warp that remembers failure: once a wait ran out the role stops waiting and walks on. All lanes check: a check by
// one or two of them, with the branch around it, costs more (2048 rows at context 30720 2005 -> 1959 us, 600 at 4000 155.0 -> 151.5)
struct Waiter {
    int* err;
    int code;
    bool dead = false;
    // (the compiler's loop: beside 16 softmax and conversion warps the written-out one of mbar_wait costs 1 %, 2048 rows at context
    // 30720 1997 and 2019 us, 600 at 2000 114.0 and 114.9, in turn)
    __device__ __forceinline__ static bool sleep(uint64_t* bar, uint32_t parity) {
        for (uint32_t i = 0; i < WAIT_LIMIT; i++)
            if (mbar_try_wait(bar, parity)) return true;
        return false;
    }
    __device__ __forceinline__ void wait(uint64_t* bar, uint32_t parity, int lane) {
        if (dead) return;
        const bool ok = __all_sync(0xffffffffu, sleep(bar, parity));
        if (!ok) {
            dead = true;
            if (lane == 0) atomicExch(err, code);
        }
    }
    // two barriers at once, half a warp each: about as long as one wait (2048 rows of prompt attention at context 30720: 1917 us
    // without the second wait, 2024 with one after the other, 1930 so)
    __device__ __forceinline__ void wait_both(uint64_t* bar, uint32_t parity, uint64_t* bar1, uint32_t parity1, int lane) {
        if (dead) return;
        const bool ok = __all_sync(0xffffffffu, sleep(lane & 16 ? bar1 : bar, lane & 16 ? parity1 : parity));
        if (!ok) {
            dead = true;
            if (lane == 0) atomicExch(err, code);
        }
        __syncwarp();  // (orders the other lanes' reads behind both)
    }
};

// ---- Prompt steps with one key split and more than 1664 keys: pairs of blocks (four tiles, attn_prefill_tc.cu) or one block per
// two tiles (attn_prefill_short.cu). A pair passes over its tiles once per RUN of consecutive tiles of one sequence, on two
// SMs, so it wins over long runs (2048 rows at context 30720: 2716 us as blocks, 1920 as pairs) and loses over short ones (40
// sequences of 10 rows at 2000: 176 and 295 us; 30 of 20 at 8000: 290 and 402; 8 of 100 at 8000: 545 and 595).
// The estimate, in units of 100 cycles: a pass costs its stages (5200 cycles per 128 keys over a pair, 3700 per 64 keys)
// and its ends (some 30 us: Q and the gates are read a row per thread); a form takes its passes spread over the SMs, and up
// to its longest unit of work more. Of 33 steps timed as either (single sequences, equal and unequal batches, 38 to 205 tiles)
// it names the faster one for all.
__host__ __device__ __forceinline__ unsigned pair_pass_cost(int keys) { return 52u * (unsigned)((keys + 127) / 128) + 600u; }
__host__ __device__ __forceinline__ unsigned block_pass_cost(int keys) { return 37u * (unsigned)((keys + 63) / 64) + 520u; }
// tile t + 1 continues tile t
__host__ __device__ __forceinline__ bool tile_goes_on(const int* ptile, const int* tok_slot, const int* tok_pos, int t) {
    const int fa = ptile[2 * t], na = ptile[2 * t + 1], fb = ptile[2 * t + 2];
    return fb == fa + na && tok_slot[fb] == tok_slot[fa] && tok_pos[fb] == tok_pos[fa] + na;
}
__host__ __device__ __forceinline__ bool pairs_win(unsigned long long pair_sum, unsigned long long block_sum, unsigned pair_most,
                                                   unsigned block_most, int sms) {
    const unsigned long long pairs = sms > 1 ? sms / 2 : 1;
    return NKV * pair_sum / pairs + pair_most <= NKV * block_sum / (unsigned long long)sms + block_most;
}
// the answer for a step, in every thread of the block (all threads call it, whole warps)
__device__ __forceinline__ bool tiles_on_pairs(const int* ptile, int ntile, const int* tok_slot, const int* tok_pos, int sms) {
    __shared__ unsigned long long part[2][32];
    __shared__ unsigned most[2][32];
    unsigned long long sum[2] = {0ull, 0ull};
    unsigned top[2] = {0u, 0u};
    for (int t0 = 0; t0 < ntile; t0 += blockDim.x) {  // (a unit's tiles are neighbouring lanes of a warp)
        const int t = t0 + threadIdx.x;
        unsigned cost[2] = {0u, 0u};
        if (t < ntile) {
            const bool on = t + 1 < ntile && tile_goes_on(ptile, tok_slot, tok_pos, t);
            const int keys = tok_pos[ptile[2 * t] + ptile[2 * t + 1] - 1] + 1;
            if (!on || (t & 3) == 3) cost[0] = pair_pass_cost(keys);
            if (!on || (t & 1) == 1) cost[1] = block_pass_cost(keys);
        }
#pragma unroll
        for (int f = 0; f < 2; f++) {
            sum[f] += cost[f];
            unsigned unit = cost[f] + __shfl_xor_sync(0xffffffffu, cost[f], 1);
            if (f == 0) unit += __shfl_xor_sync(0xffffffffu, unit, 2);
            top[f] = max(top[f], unit);
        }
    }
#pragma unroll
    for (int f = 0; f < 2; f++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[f] += __shfl_xor_sync(0xffffffffu, sum[f], o);
        top[f] = __reduce_max_sync(0xffffffffu, top[f]);
        if ((threadIdx.x & 31) == 0) { part[f][threadIdx.x >> 5] = sum[f]; most[f][threadIdx.x >> 5] = top[f]; }
    }
    __syncthreads();
    sum[0] = sum[1] = 0ull;
    top[0] = top[1] = 0u;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++)
#pragma unroll
        for (int f = 0; f < 2; f++) { sum[f] += part[f][w]; top[f] = max(top[f], most[f][w]); }
    return pairs_win(sum[0], sum[1], top[0], top[1], sms);
}

}  // namespace tc
}  // namespace qb
