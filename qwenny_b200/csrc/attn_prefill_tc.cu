// Prompt attention over the int8 KV cache on the 5th-generation tensor cores (tcgen05, accumulators in tensor memory).
// Replaces attn_prefill (kernels/attn.cuh:351-553 of the reference) for steps with many prompt tiles.
//
// A PAIR of blocks (a cluster of two, one block per SM; tcgen05 cta_group::2, M = 256 rows) is (up to four prompt tiles =
// 4 x 64 (token, head) rows, kv head) and walks the keys its rows may see in stages of 128. A block's tensor memory (512
// columns x 128 lanes, lane = row) holds what belongs to its 128 rows:
//   columns   0-255  O, the f32 accumulator of the 256 output dims
//   columns 256-511  two score buffers S (128 f32 each); P of a stage overwrites part of its S as f16
// Q (f16, 64 KB) is the A operand of S = Q K^T from shared memory. The f16 keys and values are the B operands, and a pair
// splits those: each block converts and holds half of a stage's keys (for S) and half of the value dims (for P V), so
// the int8 -> f16 conversion and the shared memory per block are half of what one block per tile pair needs.
// Over a pair an instruction takes some 128 cycles whatever its N, so the stage is 128 keys: 2048 rows at context 30720 take 2.79
// ms with one block per two tiles and 64-key stages, 2.66 as pairs with 64-key stages (S then takes 2000 of 3100 cycles
// per stage), 2.02 as pairs with 128, 1.96 with whole warps at the barriers. The pair passes over its tiles once per run of consecutive tiles of one sequence.
//   warps 8-15  read the block's share of a stage's int8 keys and values from the cache (128-bit loads, one stage ahead in
//               registers) and write it as f16 where the tensor core wants it: K as four [64 keys][64 dims] K-major
//               tiles, V transposed as two [128 dims][64 keys] tiles, with the 128-byte swizzle; the codes are
//               converted EXACTLY (1024 + byte via prmt, minus 1152), so no offset has to be folded out afterwards
//   warp 16     of the first block: issues, as a whole warp, S = Q K^T (M 256 rows, N 128 keys, K 256 dims: 16 tcgen05.mma) and
//               O += P V (N 256 dims, K 128 keys: 8 tcgen05.mma, A = P from tensor memory); tcgen05.commit tells both
//               blocks when a product is complete. S of stage i + 1 is issued before P V of stage i, so the tensor core has
//               work while the softmax of stage i runs
//   warps 0-7   softmax: tensor memory hands a THREAD its row of S (tcgen05.ld); two threads (warps w, w + 4) share a
//               row, 64 keys each, and exchange their maxima through shared memory. Scores are scaled by the keys'
//               scales, masked causally where the stage reaches the diagonal, and P = 2^(s - m) times the values'
//               scales goes back as f16 (tcgen05.st), m the row's running maximum: the same rounding points as the
//               reference's kernel; the arithmetic runs on pairs of f32, and half of the scores is read twice: 17 warps leave a
//               thread 96 registers (40 bytes spill even so). A stage in which some row's maximum grows rescales that warp's accumulator rows
//               (tcgen05.ld / st, half of the dims per thread); a lazier rule (rescale only past a threshold) was
//               measured 1 % faster and decorrelates the f16 rounding of P from the reference's, so it is not used
// At the end the softmax threads read their rows of O, divide by the row sum, multiply by the gate and write f32
// (+ f16). Every wait is bounded: a wait that runs out sets the context's error word and the block drains.
#include "attn_tc.cuh"
#include "launch.h"
#include "pair_tc.cuh"

namespace qb {
namespace pft {

constexpr int TROWS = 64;                    // rows of one prompt tile; a block has two, a pair of blocks four
constexpr int SK = 128;                      // keys per stage
constexpr int NST = 2;                       // stages of the key ring and of the value ring
constexpr int K_BYTES = SK / 2 * HD * 2;     // 32 KB: four [64][64] tiles (this block's half of the keys)
constexpr int V_BYTES = HD / 2 * SK * 2;     // 32 KB: two [128][64] tiles (this block's half of the dims)
constexpr int Q_BYTES = 128 * HD * 2;        // 64 KB: four [128][64] tiles
constexpr int NSC = 4;                       // stages of the ring of scales (the softmax reads them after S, the slot of the keys)
constexpr int SC_BYTES = 2 * SK * 4;         // key scales, value scales
constexpr int CTL_BYTES = 1024;
constexpr int ROWS = 128;
constexpr int X_BYTES = 2 * 2 * ROWS * 4;    // the row maxima of the two halves, two stages deep
constexpr int SMEM_BYTES = Q_BYTES + NST * (K_BYTES + V_BYTES) + NSC * SC_BYTES + X_BYTES + CTL_BYTES + 1024;
constexpr int SM_WARPS = 8, CVT_WARP0 = 8, CVT_WARPS = 8, MMA_WARP = 16;
constexpr int THREADS = 32 * (MMA_WARP + 1);
constexpr int TMEM_COLS = 512, O_COL = 0, S_COL = 256;

using namespace tc;

// two f32 at a time (the roundings are those of the single instructions)
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
attn_prefill_tc_kernel(const float* q, const uint8_t* kc, const uint8_t* vc, const float* ks, const float* vs,
                       const int* ptile, int ntile, const int* tok_slot, const int* tok_pos, int cap, float* out,
                       __half* mix, int* err, const int* on_pairs) {
    if (on_pairs) {  // the form behind attn_form_kernel: where the other one does the step, return before anything is taken
        pdl_wait();
        if (!*(const volatile int*)on_pairs) return;
    }
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* qf = smem;                    // [Q_BYTES]
    uint8_t* kf = qf + Q_BYTES;            // [NST][K_BYTES]
    uint8_t* vf = kf + NST * K_BYTES;      // [NST][V_BYTES]
    float* scl = (float*)(vf + NST * V_BYTES);  // [NSC][ksc 128 | vsc 128]
    float* xm = scl + NSC * 2 * SK;        // [2 stages][2 halves][ROWS]
    uint8_t* ctl = (uint8_t*)(xm + 2 * 2 * ROWS);
    uint64_t* k_ready = (uint64_t*)ctl;    // [NST] (first block) a stage's f16 keys and its scales are written in both blocks
    uint64_t* v_ready = k_ready + NST;     // [NST] (first block) its values
    uint64_t* k_free = v_ready + NST;      // [NST] S of the stage in that key slot is complete
    uint64_t* v_free = k_free + NST;       // [NST] O += P V of the stage in that value slot is complete
    uint64_t* s_ready = v_free + NST;     // [2] S of a stage is complete in tensor memory
    uint64_t* p_ready = s_ready + 2;       // [2] (first block) P of a stage is written over its S in both blocks
    uint64_t* o_done = p_ready + 2;        // [2] O += P V of a stage is complete
    uint64_t* sc_ready = o_done + 2;       // [NSC] a stage's scales are written in this block (for its softmax warps)
    uint32_t* tmem_slot = (uint32_t*)(sc_ready + NSC);

    const int g = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)cluster_ctarank();
    if (threadIdx.x == 0) {
        for (int i = 0; i < NST; i++) {
            mbar_init(&k_ready[i], 2 * CVT_WARPS);
            mbar_init(&v_ready[i], 2 * CVT_WARPS);
            mbar_init(&k_free[i], 1);
            mbar_init(&v_free[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&s_ready[i], 1);
            mbar_init(&p_ready[i], 2 * SM_WARPS);
            mbar_init(&o_done[i], 1);
        }
        for (int i = 0; i < NSC; i++) mbar_init(&sc_ready[i], CVT_WARPS);
        mbar_fence_init();
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();

    // the pair's tiles: up to four from 4 quad on (the last ones, with the longest contexts, first), in passes over runs
    // of consecutive tiles of one sequence
    const int quad = (gridDim.x >> 1) - 1 - (blockIdx.x >> 1), t_end = min(ntile, 4 * quad + 4);
    int jbase = 0;  // stages of earlier passes: ring slots and barrier phases run on
    Waiter w_mma{err, 11}, w_sm{err, 12}, w_cv{err, 13};
    const uint32_t k_ready0 = cluster_map(k_ready, 0), v_ready0 = cluster_map(v_ready, 0), p_ready0 = cluster_map(p_ready, 0);

    for (int ta = 4 * quad, run = 1; ta < t_end; ta += run) {
        for (run = 1; ta + run < t_end; run++) {
            const int fa = ptile[2 * (ta + run - 1)], na = ptile[2 * (ta + run - 1) + 1], fb = ptile[2 * (ta + run)];
            if (fb != fa + na || tok_slot[fb] != tok_slot[fa] || tok_pos[fb] != tok_pos[fa] + na) break;
        }
        // tile i of the run: rows 64 i .. of the pair's 256; this block has rows 128 rank ..
        const int tlast = ptile[2 * (ta + run - 1)] + ptile[2 * (ta + run - 1) + 1] - 1;
        const int keys = tok_pos[tlast] + 1, slot = tok_slot[tlast], nstg = (keys + SK - 1) / SK;
        const uint8_t* kh = kc + cache_head(slot, g, cap);
        const uint8_t* vh = vc + cache_head(slot, g, cap);
        const float* ksh = ks + scale_head(slot, g, cap);
        const float* vsh = vs + scale_head(slot, g, cap);
        // the softmax threads' rows (row = 64 group + token * GROUP + head) and halves
        const int qd = warp & 3, half = (warp >> 2) & 1, row = qd * 32 + lane, grp = row / TROWS, lr = row % TROWS;
        const int tok = lr / GROUP, head = g * GROUP + lr % GROUP;
        const int mt = 2 * rank + grp;  // this row's tile of the run
        const int tokn = mt < run && tok < ptile[2 * (ta + mt) + 1] ? ptile[2 * (ta + mt)] + tok : -1;
        const uint32_t trow = tmem + ((uint32_t)(qd * 32) << 16);

        // ---- Q of the 128 rows into shared memory: every softmax thread converts and stores half of its row
        if (warp < SM_WARPS) {
            const float* qp = q + ((size_t)max(tokn, 0) * NH + head) * HD;
#pragma unroll 8  // (16 loads in flight: a thread reads a row of its own)
            for (int c = 128 * half; c < 128 * half + 128; c += 8) {
                float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
                if (tokn >= 0) { v0 = *(const float4*)(qp + c); v1 = *(const float4*)(qp + c + 4); }
                *(uint4*)(qf + (c >> 6) * (128 * 128) + sw128(row, (c & 63) >> 3)) =
                    make_uint4(pack_half2(v0.x, v0.y), pack_half2(v0.z, v0.w), pack_half2(v1.x, v1.y), pack_half2(v1.z, v1.w));
            }
            async_proxy_fence();
        }
        tc_fence_before();
        cluster_sync();  // the products read both blocks' Q
        tc_fence_after();

        if (warp == MMA_WARP) {
          if (rank == 0) {
            // ------------------------------------------------------------ tensor-core issue
            auto issue_s = [&](int i) {
                const int J = jbase + i, b2 = J & 1, rs = J % NST;
                w_mma.wait(&k_ready[rs], (J / NST) & 1, lane);
                // (the S buffer is free: P V of stage J - 2, which read P out of it, was issued before this)
                tc_fence_after();
                if (!w_mma.dead) {
                    const uint64_t kd = smem_desc(uniform(smem_u32(kf + rs * K_BYTES)));
                    const uint32_t sd = uniform(tmem + S_COL + b2 * SK);
#pragma unroll
                    for (int b = 0; b < 4; b++)   // (a [64 keys][64 dims] tile is 8 KB: 512 descriptor units)
                        umma_ss4<2>(sd, smem_desc(uniform(smem_u32(qf))) + b * (128 * 128 / 16), kd + b * (SK / 2 * 128 / 16), idesc_pair(SK), b ? 1u : 0u);
                    umma2_commit(&k_free[rs]);
                    umma2_commit(&s_ready[b2]);
                }
                __syncwarp();
            };
            issue_s(0);
            for (int i = 0; i < nstg; i++) {
                const int J = jbase + i, b2 = J & 1, rs = J % NST;
                if (i + 1 < nstg) issue_s(i + 1);
                w_mma.wait(&v_ready[rs], (J / NST) & 1, lane);
                w_mma.wait(&p_ready[b2], (J >> 1) & 1, lane);
                tc_fence_after();
                if (!w_mma.dead) {
                    const uint64_t vd = smem_desc(uniform(smem_u32(vf + rs * V_BYTES)));
                    const uint32_t pa = uniform(tmem + S_COL + b2 * SK), od = uniform(tmem + O_COL);
                    umma_ts4<2>(od, pa, vd, idesc_pair(HD), i ? 1u : 0u);
                    umma_ts4<2>(od, pa + 64, vd + V_BYTES / 2 / 16, idesc_pair(HD), 1u);
                    umma2_commit(&v_free[rs]);
                    umma2_commit(&o_done[b2]);
                }
                __syncwarp();
            }
          }
        } else if (warp < SM_WARPS) {
            // ------------------------------------------------------------ softmax: two threads per row, 64 keys each
            const int lim = tokn >= 0 ? tok_pos[tokn] + 1 : 1 << 30;  // (rows without a token: Q = 0, nothing masked)
            float m = -INFINITY, l = 0.f;
            for (int i = 0; i < nstg; i++) {
                const int J = jbase + i, b2 = J & 1, kb0 = i * SK + 64 * half;
                // the scales come from the convert warps by plain stores: a barrier of this block orders them (S itself goes by way of
                // the first block's tensor core, which promises nothing about the second block's plain stores)
                w_sm.wait_both(&s_ready[b2], (J >> 1) & 1, &sc_ready[J % NSC], (J / NSC) & 1, lane);
                tc_fence_after();
                const uint32_t ts = trow + S_COL + b2 * SK + 64 * half;
                const float4* ksc4 = (const float4*)(scl + (J % NSC) * 2 * SK + 64 * half);
                const float4* vsc4 = ksc4 + SK / 4;
                const bool edge = __any_sync(0xffffffffu, kb0 + 64 > lim);
                // 32 of this thread's 64 scores times the keys' scales; the causal mask only where the stage reaches past a
                // row's last key (a masked score is a large negative number: 2^(that - m) is 0)
                float sc[32];
                auto scores = [&](int c) {
                    uint32_t sv[32];
                    tmem_ld32(ts + c, sv);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 k4 = ksc4[(c + j) >> 2];
                        const float2 a = unpack2(mul2(pack2(__uint_as_float(sv[j]), __uint_as_float(sv[j + 1])), pack2(k4.x, k4.y)));
                        const float2 b = unpack2(mul2(pack2(__uint_as_float(sv[j + 2]), __uint_as_float(sv[j + 3])), pack2(k4.z, k4.w)));
                        sc[j] = a.x; sc[j + 1] = a.y; sc[j + 2] = b.x; sc[j + 3] = b.y;
                    }
                    if (edge) {
#pragma unroll
                        for (int j = 0; j < 32; j++) sc[j] = kb0 + c + j < lim ? sc[j] : -1e30f;
                    }
                };
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                scores(32);
#pragma unroll
                for (int j = 0; j < 32; j++) mx[j & 3] = fmaxf(mx[j & 3], sc[j]);
                scores(0);  // (kept for the exponentials; the others are read again)
#pragma unroll
                for (int j = 0; j < 32; j++) mx[j & 3] = fmaxf(mx[j & 3], sc[j]);
                const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                // the row's maximum over both halves
                float* xs = xm + (J & 1) * 2 * ROWS;
                xs[half * ROWS + row] = mine;
                named_bar_sync(1 + qd, 64);
                const float both = fmaxf(mine, xs[(1 - half) * ROWS + row]);
                const float mold = m;
                if (both > -1e29f) m = fmaxf(m, both);
                const bool move = m > mold;
                const float factor = mold == -INFINITY ? 0.f : ex2(mold - m);  // 1 where the maximum stays
                const float nref = m == -INFINITY ? 0.f : -m;
                const uint64_t nref2 = pack2(nref, nref);
                uint64_t sum2[2] = {0ull, 0ull};
                // P of 32 keys over 16 columns of scores that this thread has read
                auto probs = [&](int c) {
                    uint32_t ph[16];
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 v4 = vsc4[(c + j) >> 2];
                        const float2 a = unpack2(add2(pack2(sc[j], sc[j + 1]), nref2)), b = unpack2(add2(pack2(sc[j + 2], sc[j + 3]), nref2));
                        const uint64_t p0 = pack2(ex2(a.x), ex2(a.y)), p1 = pack2(ex2(b.x), ex2(b.y));
                        sum2[0] = add2(sum2[0], p0);
                        sum2[1] = add2(sum2[1], p1);
                        const float2 r0 = unpack2(mul2(p0, pack2(v4.x, v4.y))), r1 = unpack2(mul2(p1, pack2(v4.z, v4.w)));
                        ph[j >> 1] = pack_half2(r0.x, r0.y);
                        ph[(j >> 1) + 1] = pack_half2(r1.x, r1.y);
                    }
                    tmem_st16(ts + (c >> 1), ph);
                };
                probs(0);
                scores(32);
                probs(32);
                const float2 sum = unpack2(add2(sum2[0], sum2[1]));
                l = l * factor + (sum.x + sum.y);
                if (i > 0 && __any_sync(0xffffffffu, move)) {
                    // rescale this thread's half of its accumulator row (rows whose maximum stayed multiply by 1) once
                    // the previous stage's product has landed in it
                    w_sm.wait(&o_done[(J - 1) & 1], ((J - 1) >> 1) & 1, lane);
                    tc_fence_after();
#pragma unroll 1
                    for (int c = 128 * half; c < 128 * half + 128; c += 32) {
                        uint32_t ov[32];
                        tmem_ld32(trow + O_COL + c, ov);
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 32; j++) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * factor);
                        tmem_st32(trow + O_COL + c, ov);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_at(p_ready0 + 8 * b2);
            }
            // ---- the rows' results: O / (the two halves' sums) times the gate, half of the dims per thread
            const int Jl = jbase + nstg - 1;
            float* xs = xm + ((Jl + 1) & 1) * 2 * ROWS;
            xs[half * ROWS + row] = l;
            named_bar_sync(1 + qd, 64);
            l += xs[(1 - half) * ROWS + row];
            w_sm.wait(&o_done[Jl & 1], (Jl >> 1) & 1, lane);
            tc_fence_after();
            const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
            for (int c = 128 * half; c < 128 * half + 128; c += 32) {
                uint32_t ov[32];
                tmem_ld32(trow + O_COL + c, ov);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (tokn >= 0 && !w_sm.dead) {
                    float* op = out + (size_t)tokn * MIX + head * HD + c;
                    __half* mp = mix ? mix + (size_t)tokn * MIX + head * HD + c : nullptr;
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        const float4 gt = *(const float4*)(op + j);
                        const float4 res = make_float4(gt.x * __uint_as_float(ov[j]) * inv, gt.y * __uint_as_float(ov[j + 1]) * inv,
                                                       gt.z * __uint_as_float(ov[j + 2]) * inv, gt.w * __uint_as_float(ov[j + 3]) * inv);
                        *(float4*)(op + j) = res;
                        if (mp) *(uint2*)(mp + j) = make_uint2(pack_half2(res.x, res.y), pack_half2(res.z, res.w));
                    }
                }
            }
            tc_fence_before();
        } else if (warp >= CVT_WARP0) {
            // ------------------------------------------------------------ int8 -> f16 tiles, one stage ahead in registers
            // this block's share: keys 64 rank .. of the stage (all dims), dims 128 rank .. of its values (all keys); the
            // scales of all keys. One stage ahead in registers; the keys and the values have rings of their own (a key slot
            // is free when S is complete, long before the values' is).
            const int cw = warp - CVT_WARP0, ct = threadIdx.x - CVT_WARP0 * 32, t4 = lane & 3;
            const int key = 8 * cw + (lane >> 2), d = 32 * (cw & 3) + lane, vt0 = 4 * (cw >> 2);
            uint4 kraw[4], vraw[4];
            float sraw = 0.f;
            // (positions past the cache's end, where its length is no multiple of 128, are not read)
            auto fetch_k = [&](int i) {
                const int kb0 = i * SK;
                // 16-byte groups (b = it, t4) of the key's row
                const uint8_t* kp = kh + (size_t)(kb0 + 64 * rank + key) * HD + t4 * 16;
#pragma unroll
                for (int it = 0; it < 4; it++)
                    kraw[it] = kb0 + 64 * rank < cap ? *(const uint4*)(kp + 64 * it) : make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
                // (scales of positions past the last key are not read: such cache entries may hold anything)
                sraw = kb0 + (ct & (SK - 1)) < keys ? (ct < SK ? ksh : vsh)[kb0 + (ct & (SK - 1))] : 0.f;
            };
            auto fetch_v = [&](int i) {
                const int kb0 = i * SK;
                // 16-key blocks vt0 .. vt0 + 3
                const uint8_t* vp = vh + ((size_t)((kb0 >> 4) + vt0) * HD + 128 * rank + d) * 16;
#pragma unroll
                for (int it = 0; it < 4; it++)
                    vraw[it] = kb0 + 16 * vt0 < cap ? *(const uint4*)(vp + (size_t)it * HD * 16) : make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);
            };
            fetch_k(0);
            fetch_v(0);
            for (int i = 0; i < nstg; i++) {
                const int J = jbase + i, rs = J % NST;
                // the slot's earlier keys are consumed; the scales' slot is two stages older: its softmax came before the
                // product P V that v_free of the stage before has waited for
                if (J >= NST) w_cv.wait(&k_free[rs], (J / NST - 1) & 1, lane);
                uint8_t* kt = kf + rs * K_BYTES;
#pragma unroll
                for (int it = 0; it < 4; it++) {
                    const uint32_t wq[4] = {kraw[it].x, kraw[it].y, kraw[it].z, kraw[it].w};
                    uint8_t* tile = kt + it * (SK / 2 * 128);
#pragma unroll
                    for (int s = 0; s < 4; s++) {
                        // word s: dims 16 s + 2 t4 + {0, 1} (bytes 0, 1) and 16 s + 8 + 2 t4 + {0, 1} (bytes 2, 3)
                        *(uint32_t*)(tile + sw128(key, 2 * s) + 4 * t4) = exact2(wq[s], 0x4140);
                        *(uint32_t*)(tile + sw128(key, 2 * s + 1) + 4 * t4) = exact2(wq[s], 0x4342);
                    }
                }
                scl[(J % NSC) * 2 * SK + ct] = sraw;
                async_proxy_fence();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sc_ready[J % NSC]);
                    mbar_arrive_at(k_ready0 + 8 * rs);
                }
                if (i + 1 < nstg) fetch_k(i + 1);  // (after the fence, which would wait for it)
                if (J >= NST) w_cv.wait(&v_free[rs], (J / NST - 1) & 1, lane);
                uint8_t* vt = vf + rs * V_BYTES + (vt0 >> 2) * (V_BYTES / 2);
#pragma unroll
                for (int it = 0; it < 4; it++) {
                    // word t of a 16-byte group: keys 2 t, 2 t + 1 (bytes 0, 1) and 2 t + 8, 2 t + 9 (bytes 2, 3)
                    const uint32_t wq[4] = {vraw[it].x, vraw[it].y, vraw[it].z, vraw[it].w};
                    *(uint4*)(vt + sw128(d, 2 * it)) = make_uint4(exact2(wq[0], 0x4140), exact2(wq[1], 0x4140),
                                                                 exact2(wq[2], 0x4140), exact2(wq[3], 0x4140));
                    *(uint4*)(vt + sw128(d, 2 * it + 1)) = make_uint4(exact2(wq[0], 0x4342), exact2(wq[1], 0x4342),
                                                                     exact2(wq[2], 0x4342), exact2(wq[3], 0x4342));
                }
                async_proxy_fence();
                __syncwarp();
                if (lane == 0) mbar_arrive_at(v_ready0 + 8 * rs);
                if (i + 1 < nstg) fetch_v(i + 1);
            }
        }
        jbase += nstg;
        tc_fence_before();
        __syncthreads();  // the pass is complete: Q may be rewritten
        tc_fence_after();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

}  // namespace pft
}  // namespace qb

// the many-tile form of qb_attn_prefill (one key split): see attn.cu. on_pairs: null, or a word on the device that says whether
// this form (1) or the other (0) does the step
int qb_attn_prefill_tc_launch(qb_ctx* ctx, cudaStream_t st, const float* q, const void* kc, const void* vc, const float* ks,
                              const float* vs, const int* ptile, int ntile, const int* tok_slot, const int* tok_pos,
                              int cap, float* out, void* mix_f16, const int* on_pairs) {
    using namespace qb;
    return launch(ctx, pft::attn_prefill_tc_kernel, dim3(2 * ((ntile + 3) / 4), NKV), dim3(pft::THREADS), pft::SMEM_BYTES, st, q,
                  (const uint8_t*)kc, (const uint8_t*)vc, ks, vs, ptile, ntile, tok_slot, tok_pos, cap, out,
                  (__half*)mix_f16, ctx->err, on_pairs);
}
