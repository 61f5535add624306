// W4A16 product for 17 .. 64 token rows (several sequences' verify steps, short prompt pieces, the output layer over a
// batch) on the 5th-generation tensor cores: Y = X . W^T with W int4 in Marlin's layout, plain, SwiGLU or argmax epilogue,
// contiguous or gathered rows.
//
// A block owns 128 outputs and the weights go from registers to tensor memory in the layout that a Marlin word already has
// (w4a16_gemm_tc.cu). The floor is the weights' way from HBM (0.52 bytes each, read once): 760 cycles per block and stage, two groups
// of 128 of k. A stage takes some 1350 (40 rows of a 248,320-output matrix, 262 stages a block): the way of a slot of tensor memory
// from "free" to "multiplied" (unpacking 680, the issue of 16 products 800, 130 to 150 per check of a barrier; a group's slot each, 4 to
// 6 of them in turn: with a slot per stage, two in turn, a stage took 1440), and 40 KB through shared memory a stage, 24 of them
// the rows again. What a launch spends beside its stages: 3 us from its first instruction to the first unpacked stage, 3 us from a cut
// tile's last sum to its result (partial sums 0.2, fence and ticket 1.1, parts 0.6, epilogue 0.7).
// From a graph, 40 rows: the MLP 56.5 us (one group per stage, a fence per thread and 64-bit divisions before the ticket, one round
// trip per part, shares whatever the shape: 78.7), 5120 x 6144 12.1 (19.6), the output layer of 248,320 rows 211 (298); 17 and 64
// rows of the MLP 52.7 (72) and 65.7 (86.5). What differs from the prompt-sized product:
//   - the weights are the exact integers q - 8; a group of 128 columns is one accumulation, and the drain warps multiply its
//     f32 sums by the f32 value of the group's scale and add them up in registers (one thread per output, a register per token), as
//     the product for up to 16 rows does (w4a16_gemv.cuh), where f16((q - 8) s) would round every weight. Two pairs of accumulators take
//     turns, so that draining one overlaps the next products, and two warps issue in turn, so that one's checks overlap the other's
//     products
//   - a stage is two groups: a role checks its barriers once for both (with one group per stage a drain warp's chain of check, load,
//     check of the scales and sums took 1000 cycles a group and was what everything waited for)
//   - a drain warp takes 16 tokens: with 32 its threads held 64 values and spilled
//   - gathered rows (the output layer) are copied together first, by a launch of their own: gathered by cp.async in every block they
//     slowed the unpacking from 680 to 1070 cycles a stage (40 rows of 248,320 outputs 269 us against 218 at that time, launch included)
// The (tile, group) list is dealt to at most one block per SM: whole tiles, tiles cut into equal parts, or equal shares; parts of a cut
// tile are added by its last arriver in block order (the bits repeat). Its ticket is taken behind a barrier by one thread with one fence
// (a fence per thread: 2 us; a ticket per warp instead of the barriers: the output layer 241 us against 232).
#include "launch.h"
#include "pair_tc.cuh"

namespace qb {
namespace mid {

using namespace tc;

constexpr int BH = 128;             // outputs per block
constexpr int BK = 128;             // k of a group of scales
constexpr int SG = 2;               // groups per stage
constexpr int NSTAGE = 4;           // stages in shared memory (words, X): a copy takes some 2000 cycles
constexpr int ND = 2;               // stages' accumulators in tensor memory (a column per token and group)
constexpr int NS = 8;               // stages in the ring of scales: those in shared memory and those being drained
constexpr int W_BYTES = BH * BK / 2;  // of a group
constexpr int DQ_WARPS = 8;         // four warps unpack a group of a stage
static_assert(DQ_WARPS == 4 * SG, "four warps per group");
constexpr int DT = 16;              // tokens of a drain warp
constexpr int TMEM_COLS = 512;
constexpr size_t PART_BYTES = 16u << 20;  // of the context's scratch, for the parts of cut tiles; gathered rows come after
template <int NT>
struct Cfg {
    static constexpr int DR_WARPS = 4 * (NT / DT);  // a drain warp: 32 outputs x DT tokens
    static constexpr int COPY_WARP = DQ_WARPS + DR_WARPS, MMA_WARP = COPY_WARP + 1, X_WARP = COPY_WARP + 3;
    static constexpr int THREADS = (X_WARP + 1) * 32;  // (NT = 64: 28 warps leave 72 registers a thread, 29 only 64)
    static constexpr int A_COL = ND * SG * NT, NA = (TMEM_COLS - A_COL) / (BK / 2);  // the groups' weights in tensor memory: 6, 5 or 4 of 64 columns
    static constexpr int XH = NT * 64 * 2, XB = 2 * XH;  // the tokens, 64 of k; a group
    static constexpr int SMEM = NSTAGE * SG * (XB + W_BYTES) + NS * SG * BH * 2 + 1024 + 1024;
    static_assert(XH % 1024 == 0, "swizzled tiles want 1 KB");
};

struct Args {
    const __half* S;     // scales [K/128][N]
    void* Y;             // plain / argmax: f32 [.][N]; silu: f16 [.][N/2]; rows y0 ..
    unsigned long long* keys;
    int m, N, K, y0, n_valid;
    int* err;
    float* part;         // [block][2][NT][BH]
    int* tickets;
    int iters;           // tiles x groups
    int tiles;
    int unit;            // groups that stay together in a share: 1, or a tile's
};

// two values at a time: s x, a + s x (rounded as fmaf rounds it) and a + b
__device__ __forceinline__ void mul2(float& a0, float& a1, float s, uint32_t x0, uint32_t x1) {
    asm("{\n.reg .b64 s, x;\nmov.b64 s, {%2, %2};\nmov.b64 x, {%3, %4};\nmul.rn.f32x2 x, s, x;\nmov.b64 {%0, %1}, x;\n}\n"
        : "=f"(a0), "=f"(a1) : "f"(s), "r"(x0), "r"(x1));
}
__device__ __forceinline__ void add2(float& a0, float& a1, float b0, float b1) {
    asm("{\n.reg .b64 a, b;\nmov.b64 a, {%0, %1};\nmov.b64 b, {%2, %3};\nadd.rn.f32x2 a, a, b;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a0), "+f"(a1) : "f"(b0), "f"(b1));
}
__device__ __forceinline__ void fma2(float& a0, float& a1, float s, uint32_t x0, uint32_t x1) {
    asm("{\n.reg .b64 a, s, x;\nmov.b64 a, {%0, %1};\nmov.b64 s, {%2, %2};\nmov.b64 x, {%3, %4};\nfma.rn.f32x2 a, s, x, a;\nmov.b64 {%0, %1}, a;\n}\n"
        : "+f"(a0), "+f"(a1) : "f"(s), "r"(x0), "r"(x1));
}

template <int NT, int EPI>
__global__ void __launch_bounds__(Cfg<NT>::THREADS, 1)
    w4a16_gemm_mid_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    using C = Cfg<NT>;
    constexpr int XB = C::XB, DR_WARPS = C::DR_WARPS, COPY_WARP = C::COPY_WARP, MMA_WARP = C::MMA_WARP, X_WARP = C::X_WARP;
    uint8_t* wsmem = smem + NSTAGE * SG * XB;
    __half* ssmem = (__half*)(wsmem + NSTAGE * SG * W_BYTES);
    uint64_t* full = (uint64_t*)(ssmem + NS * SG * BH);  // a stage's copies landed in this block
    uint64_t* aready = full + NSTAGE;    // its weights are in tensor memory
    uint64_t* empty = aready + NSTAGE;   // its products are done
    uint64_t* dfull = empty + NSTAGE;    // its accumulators are complete
    uint64_t* dfree = dfull + ND;        // they have been drained
    uint32_t* tmem_slot = (uint32_t*)(dfree + ND);
    int* flag = (int*)(tmem_slot + 1);   // this block finishes the tile; the first of the blocks that hold it, how many

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ngr = a.K / 128;
    Walk<true> walk(a.iters, a.tiles, ngr, gridDim.x, blockIdx.x, a.unit);
    int tile = 0, g0 = 0, g1 = 0;

    // the weights and scales of a stage from group gi of the tile (one lane)
    auto load_weights = [&](int tile, int gi, int g1, uint32_t st) {
        const uint64_t pol = policy_evict_first();
        const int s = (int)(st % NSTAGE), cnt = min(SG, g1 - gi), n0 = tile * BH;
        uint8_t* w = wsmem + s * SG * W_BYTES;
        __half* sc = ssmem + (int)(st % NS) * SG * BH;
        mbar_expect_tx(&full[s], cnt * (W_BYTES + BH * 2));
        for (int i = 0; i < cnt; i++) {
            tma_load_2d(w + i * W_BYTES, &wmap, n0, (gi + i) * (BK / 16), &full[s]);
            bulk_g2s(sc + i * BH, a.S + (size_t)(gi + i) * a.N + n0, BH * 2, &full[s], pol);
        }
    };
    uint32_t begun = 0;
    if (threadIdx.x == COPY_WARP * 32) {
        for (int i = 0; i < NSTAGE; i++) {
            mbar_init(&full[i], 2);
            mbar_init(&aready[i], DQ_WARPS);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < ND; i++) { mbar_init(&dfull[i], 1); mbar_init(&dfree[i], DR_WARPS); }
        mbar_fence_init();
        // the first stage's weights are asked for before the block has come together
        walk.next(tile, g0, g1);
        if (g0 < g1) load_weights(tile, g0, g1, begun++);
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;  // the accumulators, then the weights
    constexpr int NA = C::NA;
    pdl_launch_dependents();

    // every role walks the same segments (tile, groups [g0, g1)) in stages of two groups, the last of a segment maybe of one; st
    // counts stages from the start
    if (warp == COPY_WARP) {
        if (lane == 0) {
            bool ok = true;
            uint32_t st = 0;
            // (the weights do not depend on the kernel before: no wait for it; the first segment is the one begun above)
            for (bool more = g0 < g1; ok && more; more = walk.next(tile, g0, g1)) {
                for (int gi = g0; gi < g1; gi += SG, st++) {
                    // (the scales' slot: the stage NS before this one was drained long ago: this stage waits for products
                    // that came after the reuse of its accumulators)
                    if (st < begun) continue;  // under way
                    if (st >= NSTAGE) {
                        ok = mbar_wait(&empty[st % NSTAGE], ((st / NSTAGE) - 1) & 1);
                        if (!ok) break;
                    }
                    load_weights(tile, gi, g1, st);
                }
            }
            if (!ok) atomicExch(a.err, 14);
        }
        __syncwarp();
    } else if (warp == X_WARP) {
        // ---------------------------------------------------------------- the rows, from a thread of their own (70 cycles per copy)
        if (lane == 0) {
            pdl_wait();
            bool ok = true;
            uint32_t st = 0;
            while (ok && walk.next(tile, g0, g1)) {
                for (int gi = g0; gi < g1; gi += SG, st++) {
                    const int s = (int)(st % NSTAGE), cnt = min(SG, g1 - gi);
                    if (st >= NSTAGE) {
                        ok = mbar_wait(&empty[s], ((st / NSTAGE) - 1) & 1);
                        if (!ok) break;
                    }
                    mbar_expect_tx(&full[s], cnt * XB);
                    for (int i = 0; i < cnt; i++) tma_load_3d(smem + (s * SG + i) * XB, &xmap, 0, 0, (gi + i) * (BK / 64), &full[s]);
                }
            }
            if (!ok) atomicExch(a.err, 14);
        }
        __syncwarp();
    } else if (warp < DQ_WARPS) {
        // ---------------------------------------------------------------- q - 8 into tensor memory
        const int q = warp & 3, h = warp >> 2;
        const uint32_t quarter = (uint32_t)(q * 32) << 16;
        bool dead = false;
        uint32_t st = 0;
        while (walk.next(tile, g0, g1)) {
            for (int gi = g0; gi < g1; gi += SG, st++) {
                const int s = (int)(st % NSTAGE);
                if (!dead) {
                    // (half a warp each; the tensor-memory slot: the products of the group NA before have read it)
                    const int grp = 2 * (int)st + h, us = (grp - NA) >> 1;
                    const bool slot = lane >= 16 && grp >= NA;
                    dead = !warp_wait(slot ? &empty[us % NSTAGE] : &full[s], ((slot ? us : (int)st) / NSTAGE) & 1);
                    if (dead && lane == 0) atomicExch(a.err, 15);
                }
                __syncwarp();
                if (gi + h < g1) {
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t at = tmem + C::A_COL + (2 * st + h) % NA * (BK / 2);
                    const uint8_t* wp = wsmem + (s * SG + h) * W_BYTES + (q >> 1) * 512 + lane * 16 + (q & 1) * 8;
                    uint2 w[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) w[j] = *(const uint2*)(wp + j * 1024);
#pragma unroll
                    for (int bh = 0; bh < 4; bh++) {  // 16-row block b, k half hf of the stage
                        const int b = bh & 1, hf = bh >> 1;
                        uint32_t r[16];
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const uint32_t qw = b ? w[4 * hf + j].y : w[4 * hf + j].x, q8 = qw >> 8;
                            uint32_t lo0, hi0, lo1, hi1;
                            asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;\n" : "=r"(lo0) : "r"(qw));
                            asm("lop3.b32 %0, %1, 0x00f000f0, 0x54005400, 0xea;\n" : "=r"(hi0) : "r"(qw));
                            asm("lop3.b32 %0, %1, 0x000f000f, 0x64006400, 0xea;\n" : "=r"(lo1) : "r"(q8));
                            asm("lop3.b32 %0, %1, 0x00f000f0, 0x54005400, 0xea;\n" : "=r"(hi1) : "r"(q8));
                            const uint32_t SUB_LO = 0x64086408u, SUB_HI = 0x54805480u;
                            __half2 v0 = __hsub2(*(__half2*)&lo0, *(const __half2*)&SUB_LO), v1 = __hsub2(*(__half2*)&lo1, *(const __half2*)&SUB_LO);
                            __half2 v2 = __hsub2(*(__half2*)&hi0, *(const __half2*)&SUB_HI), v3 = __hsub2(*(__half2*)&hi1, *(const __half2*)&SUB_HI);
                            r[4 * j] = *(uint32_t*)&v0; r[4 * j + 1] = *(uint32_t*)&v1;
                            r[4 * j + 2] = *(uint32_t*)&v2; r[4 * j + 3] = *(uint32_t*)&v3;
                        }
                        tmem_st_16x128_x8(at + 32 * hf + quarter + ((uint32_t)(16 * b) << 16), r);
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(&aready[s]);
            }
        }
    } else if (warp < COPY_WARP) {
        // ---------------------------------------------------------------- drain the groups, then the epilogue
        const int q = warp & 3, lrow = q * 32 + lane, t0 = (warp - DQ_WARPS) / 4 * DT;  // this warp's outputs and tokens
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + t0;
        bool dead = false;
        uint32_t st = 0;
        unsigned long long best = 0;  // argmax: lane l holds the best key of token t0 + l over this warp's outputs
        // this thread's output in a group's scales: output 16 b + 8 i + r of a c64 at 8 r + 2 b + i
        const __half* sc = ssmem + (lrow >> 6) * 64 + 8 * (lrow & 7) + ((lrow & 63) >> 3);
        pdl_wait();
        while (walk.next(tile, g0, g1)) {
            const int orow = tile * BH + lrow;
            const bool cut = g0 > 0 || g1 < ngr;
            if (cut && threadIdx.x == DQ_WARPS * 32) walk.parts_of(tile, flag[1], flag[2]);  // (read behind the barriers at the tile's end)
            float acc[DT];
#pragma unroll
            for (int j = 0; j < DT; j++) acc[j] = 0.f;
#pragma unroll 1
            for (int gi = g0; gi < g1; gi += SG, st++) {
                const int p = (int)(st % ND);
                if (!dead) {
                    dead = !warp_wait(&dfull[p], (st / ND) & 1);
                    if (dead && lane == 0) atomicExch(a.err, 16);
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // the second group's sums are on their way while the first's are scaled (in a stage of one group they are whatever the
                // accumulator holds, and not used). A stage's two groups are added to each other first: half as many sums of full size, so that
                // a block that walks a whole tile is no further from 64 bits than equal shares were (16384 x 5120: 1.19e-7 group by group)
                uint32_t v[DT], w[DT];
                tmem_ld16(tq + p * SG * NT, v);
                // (the scales landed with the words: the products that made these sums came after)
                const __half* sp = sc + (int)(st % NS) * SG * BH;
                const float s0 = __half2float(sp[0]), s1 = __half2float(sp[BH]);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                tmem_ld16(tq + (p * SG + 1) * NT, w);
                float t[DT];
#pragma unroll
                for (int j = 0; j < DT; j += 2) mul2(t[j], t[j + 1], s0, v[j], v[j + 1]);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&dfree[p]);
                if (gi + 1 < g1) {
#pragma unroll
                    for (int j = 0; j < DT; j += 2) fma2(t[j], t[j + 1], s1, w[j], w[j + 1]);
                }
#pragma unroll
                for (int j = 0; j < DT; j += 2) add2(acc[j], acc[j + 1], t[j], t[j + 1]);
            }
            bool finish = !dead;
            if (cut) {
                // [4 tokens][output][4]: a thread's sums in 16-byte pieces
                constexpr int PS = BH * 4;
                float* slot = a.part + ((size_t)blockIdx.x * 2 + (g0 == 0 ? 1 : 0)) * (NT * BH) + t0 * BH + lrow * 4;
#pragma unroll
                for (int j = 0; j < DT; j += 4)
                    if (t0 + j < a.m) *(float4*)(slot + (j / 4) * PS) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                named_bar_sync(1, DR_WARPS * 32);
                if (threadIdx.x == DQ_WARPS * 32) {
                    __threadfence();  // (for all warps' sums: the barrier orders them before it)
                    const bool last = atomicAdd(&a.tickets[tile], 1) == flag[2] - 1;
                    *flag = last;
                    if (last) {
                        a.tickets[tile] = 0;
                        __threadfence();
                    }
                }
                named_bar_sync(1, DR_WARPS * 32);
                finish = *flag != 0 && !dead;
                const int first = flag[1], parts = flag[2];
                named_bar_sync(1, DR_WARPS * 32);
                if (finish) {
#pragma unroll
                    for (int j = 0; j < DT; j++) acc[j] = 0.f;
                    // two blocks' parts are on their way at a time
                    const float* o = a.part + ((size_t)first * 2 + 1) * (NT * BH) + t0 * BH + lrow * 4;
#pragma unroll 1
                    for (int pt = 0; pt < parts; pt += 2) {
                        float4 x[2][DT / 4];
#pragma unroll
                        for (int e = 0; e < 2; e++)
#pragma unroll
                            for (int j = 0; j < DT / 4; j++)
                                x[e][j] = pt + e < parts && t0 + 4 * j < a.m ? __ldcg((const float4*)(o + ((size_t)(pt + e) * 2 - (pt + e > 0)) * (NT * BH) + j * PS))
                                                                             : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int e = 0; e < 2; e++)
#pragma unroll
                            for (int j = 0; j < DT / 4; j++) {
                                acc[4 * j] += x[e][j].x; acc[4 * j + 1] += x[e][j].y;
                                acc[4 * j + 2] += x[e][j].z; acc[4 * j + 3] += x[e][j].w;
                            }
                    }
                }
            }
            if (!finish) continue;
            if (EPI == QB_EPI_SILU) {
                // packed rows 16 p + i are gate rows, 16 p + 8 + i their up rows, 8 lanes on
                const bool up_lane = (lane & 8) != 0;
#pragma unroll
                for (int j = 0; j < DT; j += 2) {
                    const float other = __shfl_xor_sync(0xffffffffu, up_lane ? acc[j] : acc[j + 1], 8);
                    const float gate = up_lane ? other : acc[j], up = up_lane ? acc[j + 1] : other;
                    const int tok = t0 + j + (up_lane ? 1 : 0);
                    if (tok < a.m)
                        ((__half*)a.Y)[(size_t)(a.y0 + tok) * (a.N / 2) + (orow >> 4) * 8 + (orow & 7)] = __float2half_rn(silu(gate) * up);
                }
            } else {
#pragma unroll
                for (int j = 0; j < DT; j++)
                    if (t0 + j < a.m) ((float*)a.Y)[(size_t)(a.y0 + t0 + j) * a.N + orow] = acc[j];
                if (EPI == QB_EPI_ARGMAX) {
                    const bool valid = orow < a.n_valid;
                    const unsigned any = __ballot_sync(0xffffffffu, valid);
                    if (any) {
#pragma unroll
                        for (int j = 0; j < DT; j++) {
                            const unsigned u = valid ? ordered(acc[j]) : 0u, mx = __reduce_max_sync(0xffffffffu, u);
                            const int at = __ffs(__ballot_sync(0xffffffffu, valid && u == mx)) - 1;
                            const unsigned long long key =
                                ((unsigned long long)mx << 32) | (0xffffffffu - (uint32_t)(orow - lane + at));
                            if (lane == j && key > best) best = key;
                        }
                    }
                }
            }
        }
        if (EPI == QB_EPI_ARGMAX && best && t0 + lane < a.m) atomicMax(a.keys + a.y0 + t0 + lane, best);
    } else {
        // ---------------------------------------------------------------- the products: two warps take turns
        const int turn = (int)uniform((uint32_t)(warp - MMA_WARP));
        const uint32_t tm = uniform(tmem);
        bool ok = true;
        uint32_t st = 0;
        const uint32_t xs = smem_u32(smem);
        while (ok && walk.next(tile, g0, g1)) {
            for (int gi = g0; gi < g1; gi += SG, st++) {
                if ((int)(st & 1) != turn) continue;
                const int s = (int)(st % NSTAGE), p = (int)(st % ND);
                const uint32_t d = uniform(tm + p * SG * NT), xa = uniform(xs + s * SG * XB);
                const uint32_t at = uniform(tm + C::A_COL + 2 * st % NA * (BK / 2)), at1 = NA % 2 ? uniform(tm + C::A_COL + (2 * st + 1) % NA * (BK / 2)) : at + BK / 2;
                // (whole warps check, one barrier after the other: after a branch for some lanes the products are issued in the slow form)
                if (st >= ND) ok = warp_wait(&dfree[p], ((st / ND) - 1) & 1);
                ok = ok && warp_wait(&aready[s], (st / NSTAGE) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                umma_ts4<1>(d, at, smem_desc(xa), idesc(NT), 0u);
                umma_ts4<1>(d, at + 32, smem_desc(xa + C::XH), idesc(NT), 1u);
                if (gi + 1 < g1) {
                    umma_ts4<1>(d + NT, at1, smem_desc(xa + XB), idesc(NT), 0u);
                    umma_ts4<1>(d + NT, at1 + 32, smem_desc(xa + XB + C::XH), idesc(NT), 1u);
                }
                umma_commit(&empty[s]);
                umma_commit(&dfull[p]);
            }
        }
        if (!ok && lane == 0) atomicExch(a.err, 17);
        __syncwarp();
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

template <int NT>
int go(qb_ctx* ctx, cudaStream_t st, int epi, int G, const CUtensorMap& xmap, const CUtensorMap& wmap, const Args& a) {
    const dim3 grid(G), block(Cfg<NT>::THREADS);
    switch (epi) {
        case QB_EPI_PLAIN: return launch(ctx, w4a16_gemm_mid_kernel<NT, QB_EPI_PLAIN>, grid, block, Cfg<NT>::SMEM, st, xmap, wmap, a);
        case QB_EPI_SILU: return launch(ctx, w4a16_gemm_mid_kernel<NT, QB_EPI_SILU>, grid, block, Cfg<NT>::SMEM, st, xmap, wmap, a);
        default: return launch(ctx, w4a16_gemm_mid_kernel<NT, QB_EPI_ARGMAX>, grid, block, Cfg<NT>::SMEM, st, xmap, wmap, a);
    }
}

}  // namespace mid
}  // namespace qb

using namespace qb;

// whether the scratch has room for the gathered rows of a product beside its parts (64 rows: k up to 170,000)
int qb_gemm_mid_gathers(const qb_ctx* ctx, int m, int k) {
    return (size_t)ctx->sms * 2 * 64 * mid::BH * sizeof(float) <= mid::PART_BYTES && mid::PART_BYTES + (size_t)m * k * 2 <= qb_tc_part_bytes(ctx->sms);
}

// 1 .. 64 rows of X (row0 .., results at the same rows of Y and keys; or xrows[0 .. m), results from row 0 on)
int qb_gemm_mid_launch(qb_ctx* ctx, cudaStream_t st, const void* X, const void* B, void* Y, const void* S, int m, int n, int k,
                       int row0, int epi, const int* xrows, unsigned long long* keys, int n_valid) {
    if (xrows) row0 = 0;
    if (n % mid::BH || k % 128 || m < 1 || m > 64 || !ctx->tc_part) return QB_ERR_ARG;
    EncodeTiled enc = encode_tiled();
    if (!enc) return QB_ERR_UNSUPPORTED;
    const int nt = m <= 32 ? 32 : m <= 48 ? 48 : 64;
    const int tiles = n / mid::BH;
    if (tiles > QB_TC_TICKETS) return QB_ERR_ARG;
    const __half* x = (const __half*)X + (size_t)row0 * k;
    const int y0 = row0;
    if (xrows) {
        const __half* to = (const __half*)((char*)ctx->tc_part + mid::PART_BYTES);
        if (int rc = qb_marlin_gather(ctx, st, X, xrows, (void*)to, k / 8, m)) return rc;
        x = to;
    }
    CUtensorMap xmap, wmap;
    const cuuint32_t one[3] = {1, 1, 1};
    // (k in pieces of 64, a dimension of their own: one copy brings a group's two pieces)
    const cuuint64_t xd[3] = {64, (cuuint64_t)m, (cuuint64_t)(k / 64)}, xs[2] = {(cuuint64_t)k * 2, 128};
    const cuuint32_t xb[3] = {64, (cuuint32_t)nt, mid::BK / 64};
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)x, xd, xs, xb, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    const cuuint64_t wd[2] = {(cuuint64_t)n, (cuuint64_t)(k / 16)}, ws[1] = {(cuuint64_t)n * 8};
    const cuuint32_t wb[2] = {mid::BH, mid::BK / 16};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void*)B, wd, ws, wb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    mid::Args a;
    a.S = (const __half*)S; a.Y = Y; a.keys = keys; a.m = m; a.N = n; a.K = k;
    a.y0 = y0; a.n_valid = n_valid; a.err = ctx->err; a.part = ctx->tc_part;
    a.tickets = ctx->tc_tickets; a.iters = tiles * (k / 128); a.tiles = tiles;
    // How the list is dealt: whole tiles in rounds, each tile cut into c equal parts for as many blocks (few tiles), or equal shares of
    // the list (parts of two tiles a block), by an estimate in ns of the longest block's groups and of joining the parts. Measured at 40
    // rows, us: 16384 x 5120 whole 17.9, shares 20.4; 5120 x 6144 whole 19.3, in two 14.0, in three 12.1, shares 13.3; 5120 x 17408 in
    // three 22.0, shares 21.4; 2048 x 2048 whole 8.8, in two 8.4, four 7.8, six 8.0, shares 10.1; 1024 x 1024 whole 6.0, in two 7.1, shares
    // 7.8. Of these forms (and six parts) the choice is the fastest or within 3 % of it at 17, 40 and 64 rows of those and of 14336 x
    // 5120, 34816 x 5120, 5120 x 10240, 4096 x 4096, 8192 x 2048, 3072 x 8192, 2560 x 5120, 12288 x 4096, 20480 x 2560, 1280 x 17408 and
    // 7168 x 1024, but for 2048 x 2048 at 17 rows, 7.0 where four parts take 6.6.
    const long long ngr = k / 128, sms = ctx->sms, group = 300 + nt * 6 / 5, rounds = (tiles + sms - 1) / sms;
    long long best = a.iters * group / sms + 2000 + 67 * nt, units = a.iters;
    a.unit = 1;
    if (rounds * ngr * group + (rounds - 1) * 700 < best) {
        best = rounds * ngr * group + (rounds - 1) * 700;
        a.unit = (int)ngr;
        units = tiles;
    }
    for (int c = 2; c * tiles <= sms && c <= ngr; c++) {
        const long long cost = (ngr + c - 1) / c * group + 500 + nt * (31 + 5 * c);
        if (cost < best) { best = cost; a.unit = 1; units = (long long)tiles * c; }
    }
    const int G = (int)(units < sms ? units : sms);
    if (nt == 32) return mid::go<32>(ctx, st, epi, G, xmap, wmap, a);
    if (nt == 48) return mid::go<48>(ctx, st, epi, G, xmap, wmap, a);
    return mid::go<64>(ctx, st, epi, G, xmap, wmap, a);
}
