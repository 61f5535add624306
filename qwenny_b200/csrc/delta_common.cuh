// Gated DeltaNet pieces shared by the one-launch decode mixer (deltanet.cu) and the prompt path (delta_rule.cu): the
// rollback plan of a segment's step, and the token form of the delta rule on a thread's slice of the f32 state.
// Slot memory, plan and metadata are the reference's (kernels/qwen_deltanet.cuh:12-82; they are what its host saves,
// loads and rolls back): state [2][48][128 v][128 k] f32, banks [2][16][REP], ring [32][LQKV]; meta {end, ck, ebuf, _}.
#pragma once
#include "common.cuh"

namespace qb {

struct Plan {
    int in, r, from, ck, cbuf, ebuf;
    bool zero, wck;
};

// What a segment's step does with the slot's state: start from zeros or from buffer `in`, replay `r` accepted tokens
// from position `from` out of that buffer's bank, write the checkpoint at position ck into buffer cbuf (when wck) and
// the end state into ebuf.
__device__ __forceinline__ Plan make_plan(const int* meta, int slot, int p0, int len) {
    int end = meta[slot * META], ck = meta[slot * META + 1], eb = meta[slot * META + 2];
    Plan p;
    p.ck = max(p0, p0 + len - KEEP);
    p.r = 0;
    p.from = 0;
    p.zero = p0 == 0 || end < 0;
    if (p.zero) p.in = 0;
    else if (p0 == end) p.in = eb;
    else { p.in = 1 - eb; p.from = ck; p.r = min(max(p0 - ck, 0), KEEP); }
    p.wck = p.zero || p.r > 0 || p.ck > p0;
    p.cbuf = p.wck ? 1 - p.in : p.in;
    p.ebuf = 1 - p.cbuf;
    return p;
}

// Ahead of the kernel before, which may still write them: the slot's state (COLS columns of a head from `row` on) is asked into L2 by a
// block of THREADS. The metadata read here only says which buffer; a stale value costs the hint. (Mixers of many layers in turn, their
// states not in L2, without / with it: 1 row 18.3 / 17.4 us, 12 segments of 2 79.2 / 76.9; on a state in L2 5 segments of 5 44.1 / 44.6.)
template <int COLS, int THREADS>
__device__ __forceinline__ void hint_state(const int* meta, int slot, int p0, const float* sm0, int row) {
    if (p0 == 0) return;
    const int end = __ldcg(meta + slot * META), eb = __ldcg(meta + slot * META + 2);
    const float* s = sm0 + (size_t)((p0 == end ? eb : 1 - eb) & 1) * SLOT_STATE + (size_t)row * LKD;
    for (int x = threadIdx.x; x < COLS * LKD / 32; x += THREADS) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(s + 32 * x));
}

__device__ __forceinline__ float4 ld4(const float* p) { return *(const float4*)p; }

// The state rows of a thread, LPC = 8 lanes per value column, sub = 4 ih + rg: rows 4 (rg + 4 j) + 2 ih + e as x[2 j + e], j < 8, e < 2.
constexpr int LPC = 8, RPT = LKD / LPC;  // lanes per value column, state rows per thread
__device__ __forceinline__ void ld_rows(float* x, const float* src, int sub) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
        float2 v = *(const float2*)(src + 4 * ((sub & 3) + 4 * j) + 2 * (sub >> 2));
        x[2 * j] = v.x; x[2 * j + 1] = v.y;
    }
}
__device__ __forceinline__ void st_rows(float* dst, const float* x, int sub) {
#pragma unroll
    for (int j = 0; j < 8; j++)
        *(float2*)(dst + 4 * ((sub & 3) + 4 * j) + 2 * (sub >> 2)) = make_float2(x[2 * j], x[2 * j + 1]);
}
__device__ __forceinline__ float col_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    return v;
}
// S^T x for the thread's rows: the partial sum of the rows with the same i (row % 4) runs over j in order; then
// (d0 + d1) + (d2 + d3) across the ih lanes, then the column's 4 rg lanes. Replayed and fresh tokens share this function, so a
// replayed state is bit for bit the state one token per step reaches, whichever kernel ran the tokens.
__device__ __forceinline__ float dot_rows(const float* S, const float* x) {
    float d2[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < RPT; j++) d2[j & 1] += S[j] * x[j];
    float s = d2[0] + d2[1];
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    return col_sum(s);
}

}  // namespace qb
