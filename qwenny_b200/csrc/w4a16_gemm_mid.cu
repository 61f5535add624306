// W4A16 product for 17 .. 64 token rows (several sequences' verify steps, short prompt pieces, the output layer over a
// batch) on the 5th-generation tensor cores: Y = X . W^T with W int4 in Marlin's layout, plain, SwiGLU or argmax epilogue,
// contiguous or gathered rows.
//
// A block owns 128 outputs and the weights go from registers to tensor memory in the layout that a Marlin word already has
// (w4a16_gemm_tc.cu). The floor is the weights' way from HBM (0.52 bytes each, read once): 380 cycles per block and 128 of
// k. It takes some 1200 (40 rows of gate_up: 91,500 cycles for 73.5 stages a block): a stage's way from barrier to barrier (copied,
// unpacked, multiplied, drained: each check some 125 cycles) and the issue of 2770 warp instructions a stage (issue slots 64 %
// active there and 60 % in down, 6 warps per scheduler; tensor pipe 17 %, DRAM 23 %).
// A drain warp takes 16 tokens: with 32 its threads held 64 values and spilled (40 rows of the MLP 84.7 -> 78.9 us).
// From a graph the MLP of 17, 40 and 64 rows takes 72, 78 and 86 us, the output layer over 40 rows 299 (316 with other weights in every
// pass); padded to 256 tokens 40 rows of the MLP took 168. What else differs from the prompt-sized product:
//   - the weights are the exact integers q - 8; a group of 128 columns is one accumulation, and the drain warps multiply its
//     f32 sums by the f32 value of the group's scale and add them up in registers (one thread per output, a register
//     per token): one rounding per group, the arithmetic of the product for up to 16 rows (w4a16_gemv.cuh), where
//     f16((q - 8) s) would round every weight. Four accumulators take turns, so that draining one overlaps the next
//     products (with two the products waited 650 of 1100 cycles per stage for them), and two warps issue in turn, so that one's checks
//     overlap the other's products
//   - the rows are few: they are loaded per k block into the swizzled layout by cp.async (which also gathers), or by the
//     tensor map when they are contiguous
// The (tile, group) list is dealt to one block per SM in equal shares; parts of a cut tile are added by its last arriver in
// block order (the bits repeat).
#include "launch.h"
#include "pair_tc.cuh"

namespace qb {
namespace mid {

using namespace tc;

constexpr int BH = 128;             // outputs per block
constexpr int BK = 128;             // k per stage: a group of scales
constexpr int NSTAGE = 8;           // stages in shared memory (words, X): a copy takes some 2000 cycles
constexpr int NA = 4;               // stages in tensor memory (64 columns each)
constexpr int ND = 4;               // accumulators in tensor memory (64 columns each)
constexpr int NS = 16;              // groups in the ring of scales: those of the ring's stages and of the accumulators being drained
constexpr int W_BYTES = BH * BK / 2;
constexpr int DQ_WARPS = 8, DQ_GROUPS = DQ_WARPS / 4;  // a group of four warps unpacks a stage, the groups take turns
constexpr int DT = 16;              // tokens of a drain warp
constexpr int TMEM_COLS = 512;
template <int NT>
struct Cfg {
    static constexpr int DR_WARPS = 4 * (NT / DT);  // a drain warp: 32 outputs x DT tokens
    static constexpr int X_WARPS = NT == 64 ? 1 : 2;  // (28 warps leave 72 registers a thread, 29 only 64)
    static constexpr int COPY_WARP = DQ_WARPS + DR_WARPS, MMA_WARP = COPY_WARP + 1, X_WARP = COPY_WARP + 3;
    static constexpr int THREADS = (X_WARP + X_WARPS) * 32;
    static constexpr int XH = NT * 64 * 2, XB = 2 * XH;  // the tokens, 64 of k; a stage
    static constexpr int SMEM = NSTAGE * (XB + W_BYTES) + NS * BH * 2 + 1024 + 1024;
    static_assert(XH % 1024 == 0, "swizzled tiles want 1 KB");
};

struct Args {
    const __half* X;
    const int* xrows;    // gathered rows of X, or null: rows row0 ..
    const __half* S;     // scales [K/128][N]
    void* Y;             // plain / argmax: f32 [.][N]; silu: f16 [.][N/2]; rows y0 ..
    unsigned long long* keys;
    int m, N, K, row0, y0, n_valid;
    int* err;
    float* part;         // [block][2][NT][BH]
    int* tickets;
    long long iters;     // tiles x groups
    int tiles;
};

template <int NT, int EPI>
__global__ void __launch_bounds__(Cfg<NT>::THREADS, 1)
    w4a16_gemm_mid_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    using C = Cfg<NT>;
    constexpr int XB = C::XB, DR_WARPS = C::DR_WARPS, X_WARPS = C::X_WARPS, COPY_WARP = C::COPY_WARP, MMA_WARP = C::MMA_WARP, X_WARP = C::X_WARP;
    uint8_t* wsmem = smem + NSTAGE * XB;
    __half* ssmem = (__half*)(wsmem + NSTAGE * W_BYTES);
    uint64_t* full = (uint64_t*)(ssmem + NS * BH);  // a stage's copies landed in this block
    uint64_t* aready = full + NSTAGE;    // its weights are in tensor memory
    uint64_t* empty = aready + NSTAGE;   // its products are done
    uint64_t* sfull = empty + NSTAGE;    // a group's scales landed in this block
    uint64_t* dfull = sfull + NS;        // a group's accumulator is complete
    uint64_t* dfree = dfull + ND;         // it has been drained
    uint32_t* tmem_slot = (uint32_t*)(dfree + ND);
    int* flag = (int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ngr = a.K / 128;
    const bool gathered = a.xrows != nullptr;
    Walk<true> walk(a.iters, a.tiles, ngr, gridDim.x, blockIdx.x);
    int tile, g0, g1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NSTAGE; i++) {
            mbar_init(&full[i], gathered ? 1 + X_WARPS : 2);
            mbar_init(&aready[i], 4);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < NS; i++) mbar_init(&sfull[i], 1);
        for (int i = 0; i < ND; i++) { mbar_init(&dfull[i], 1); mbar_init(&dfree[i], DR_WARPS); }
        mbar_fence_init();
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + 256;  // accumulators at columns 0, 64, 128 and 192, weights from 256 on
    pdl_launch_dependents();

    // every role walks the same segments (tile, groups [g0, g1)); st counts stages, gr groups, from the start
    if (warp == COPY_WARP) {
        if (lane == 0) {
            const uint64_t pol = policy_evict_first();
            bool ok = true;
            uint32_t st = 0;
            while (ok && walk.next(tile, g0, g1)) {  // (the weights do not depend on the kernel before: no wait for it)
                const int n0 = tile * BH;
                for (int gi = g0; gi < g1; gi++, st++) {
                    // (the scales' slot: the group NS before this one was drained long ago: this stage waits for products
                    // that came after the reuse of its accumulator)
                    const int s = (int)(st % NSTAGE), sl = (int)(st % NS);
                    if (st >= NSTAGE) {
                        ok = mbar_wait(&empty[s], ((st / NSTAGE) - 1) & 1);
                        if (!ok) break;
                    }
                    mbar_expect_tx(&full[s], W_BYTES);
                    tma_load_2d(wsmem + s * W_BYTES, &wmap, n0, gi * (BK / 16), &full[s]);
                    mbar_expect_tx(&sfull[sl], BH * 2);
                    bulk_g2s(ssmem + sl * BH, a.S + (size_t)gi * a.N + n0, BH * 2, &sfull[sl], pol);
                }
            }
            if (!ok) atomicExch(a.err, 14);
        }
        __syncwarp();
    } else if (warp >= X_WARP) {
        // ---------------------------------------------------------------- gathered rows: cp.async into the swizzled rows
        if (gathered) {
            pdl_wait();
            constexpr int PER = NT * 16 / (X_WARPS * 32);  // 16-byte chunks per lane and stage
            static_assert(PER * X_WARPS * 32 == NT * 16, "chunks divide the loading lanes");
            const int xl = threadIdx.x - X_WARP * 32;
            constexpr int RS = 2 * X_WARPS;        // rows at a time
            const int ch = xl & 15, r0 = xl >> 4;  // this lane: 16-byte chunk ch of rows r0, r0 + RS, ..
            uint32_t row[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) row[i] = (uint32_t)a.xrows[min(RS * i + r0, a.m - 1)];  // (rows past the last are never written)
            const uint32_t line = (uint32_t)((ch >> 3) * C::XH + r0 * 128), piece = (uint32_t)(((ch & 7) ^ r0) << 4);
            bool ok = true;
            uint32_t st = 0;
            // a stage is handed over once the copies of the two after it are under way
            auto hand = [&](uint32_t n) {
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[n % NSTAGE]);
            };
            while (walk.next(tile, g0, g1)) {
                for (int kb = g0; kb < g1; kb++, st++) {
                    const int s = (int)(st % NSTAGE);
                    if (st >= NSTAGE && ok) {
                        if (lane == 0) ok = mbar_wait(&empty[s], ((st / NSTAGE) - 1) & 1);
                        ok = __shfl_sync(0xffffffffu, ok, 0);
                        if (!ok && lane == 0) atomicExch(a.err, 14);
                    }
                    if (ok) {
#pragma unroll
                        for (int i = 0; i < PER; i++) cp_async16(smem + s * XB + RS * i * 128 + line + (piece ^ ((RS * i & 7) << 4)), a.X + (size_t)row[i] * a.K + kb * BK + ch * 8);
                    }
                    cp_async_commit();
                    if (st > 1) {
                        asm volatile("cp.async.wait_group 2;\n" ::: "memory");
                        hand(st - 2);
                    }
                }
            }
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            if (st > 1) hand(st - 2);
            if (st > 0) hand(st - 1);
        } else if (warp == X_WARP && lane == 0) {  // contiguous rows: the tensor map, from a thread of its own (70 cycles per copy)
            pdl_wait();
            bool ok = true;
            uint32_t st = 0;
            while (ok && walk.next(tile, g0, g1)) {
                for (int gi = g0; gi < g1; gi++, st++) {
                    const int s = (int)(st % NSTAGE);
                    if (st >= NSTAGE) {
                        ok = mbar_wait(&empty[s], ((st / NSTAGE) - 1) & 1);
                        if (!ok) break;
                    }
                    mbar_expect_tx(&full[s], XB);
                    tma_load_2d(smem + s * XB, &xmap, gi * BK, 0, &full[s]);
                    tma_load_2d(smem + s * XB + C::XH, &xmap, gi * BK + 64, 0, &full[s]);
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
            for (int kb = g0; kb < g1; kb++, st++) {
                if ((int)(st % DQ_GROUPS) != h) continue;
                const int s = (int)(st % NSTAGE);
                if (!dead) {
                    // (a lane each; the tensor-memory slot: the products of the stage NA before have read it)
                    bool ok = true;
                    if (lane < (st >= NA ? 2 : 1)) ok = mbar_wait(lane ? &empty[(st - NA) % NSTAGE] : &full[s], ((lane ? st - NA : st) / NSTAGE) & 1);
                    dead = !__all_sync(0xffffffffu, ok);
                    if (dead && lane == 0) atomicExch(a.err, 15);
                }
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const int sa = (int)(st % NA);
                const uint8_t* wp = wsmem + s * W_BYTES + (q >> 1) * 512 + lane * 16 + (q & 1) * 8;
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
                    tmem_st_16x128_x8(tmem_a + sa * (BK / 2) + 32 * hf + quarter + ((uint32_t)(16 * b) << 16), r);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&aready[s]);
            }
        }
    } else if (warp < COPY_WARP) {
        // ---------------------------------------------------------------- drain the groups, then the epilogue
        const int q = warp & 3, lrow = q * 32 + lane, t0 = (warp - DQ_WARPS) / 4 * DT;  // this warp's outputs and tokens
        const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + t0;
        bool dead = false;
        uint32_t gr = 0;
        unsigned long long best = 0;  // argmax: lane l holds the best key of token t0 + l over this warp's outputs
        const uint32_t total = (uint32_t)(walk.it1 - walk.it);
        auto scale = [&](uint32_t n) {  // of this thread's output in the share's group n: output 16 b + 8 i + r of a c64 at 8 r + 2 b + i
            if (!dead) {
                dead = !warp_wait(&sfull[n % NS], (n / NS) & 1);
                if (dead && lane == 0) atomicExch(a.err, 16);
            }
            return __half2float(ssmem[(n % NS) * BH + (lrow >> 6) * 64 + 8 * (lrow & 7) + ((lrow & 63) >> 3)]);
        };
        float sc_next = total > 0 ? scale(0) : 0.f;
        pdl_wait();
        while (walk.next(tile, g0, g1)) {
            const int orow = tile * BH + lrow;
            float acc[DT];
#pragma unroll
            for (int j = 0; j < DT; j++) acc[j] = 0.f;
#pragma unroll 1
            for (int gi = g0; gi < g1; gi++, gr++) {
                const int p = (int)(gr % ND);
                if (!dead) {
                    dead = !warp_wait(&dfull[p], (gr / ND) & 1);
                    if (dead && lane == 0) atomicExch(a.err, 16);
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t v[DT];
                tmem_ld16(tq + p * 64, v);
                const float sc = sc_next;
                if (gr + 1 < total) sc_next = scale(gr + 1);  // while the sums are on their way
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&dfree[p]);
#pragma unroll
                for (int j = 0; j < DT; j++) acc[j] = fmaf(sc, __uint_as_float(v[j]), acc[j]);
            }
            bool finish = !dead;
            if (g0 > 0 || g1 < ngr) {
                int parts, first;
                walk.parts_of(tile, first, parts);
                float* slot = a.part + ((size_t)blockIdx.x * 2 + (g0 == 0 ? 1 : 0)) * (NT * BH) + t0 * BH + lrow;
#pragma unroll
                for (int j = 0; j < DT; j++)
                    if (t0 + j < a.m) slot[j * BH] = acc[j];
                __threadfence();
                named_bar_sync(1, DR_WARPS * 32);
                if (threadIdx.x == DQ_WARPS * 32) {
                    const int tk = atomicAdd(&a.tickets[tile], 1);
                    *flag = tk == parts - 1;
                    if (tk == parts - 1) a.tickets[tile] = 0;
                }
                named_bar_sync(1, DR_WARPS * 32);
                finish = *flag != 0 && !dead;
                named_bar_sync(1, DR_WARPS * 32);
                if (finish) {
                    __threadfence();
#pragma unroll
                    for (int j = 0; j < DT; j++) acc[j] = 0.f;
#pragma unroll 1
                    for (int pt = 0; pt < parts; pt++) {
                        const float* o = a.part + ((size_t)(first + pt) * 2 + (pt == 0 ? 1 : 0)) * (NT * BH) + t0 * BH + lrow;
#pragma unroll
                        for (int j = 0; j < DT; j++)
                            if (t0 + j < a.m) acc[j] += __ldcg(o + j * BH);
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
        const int turn = warp - MMA_WARP;
        bool ok = true;
        uint32_t st = 0;
        const uint32_t xs = smem_u32(smem);
        while (ok && walk.next(tile, g0, g1)) {
            for (int gi = g0; gi < g1; gi++, st++) {
                if ((int)(st & 1) != turn) continue;
                const int s = (int)(st % NSTAGE), p = (int)(st % ND);
                const uint32_t d = tmem + p * 64, at = tmem_a + (int)(st % NA) * (BK / 2), xa = xs + s * XB;
                // (whole warps check, one barrier after the other: after a branch for some lanes the products are issued in the slow form)
                if (st >= ND) ok = warp_wait(&dfree[p], ((st / ND) - 1) & 1);
                ok = ok && warp_wait(&aready[s], (st / NSTAGE) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                umma_ts4<1>(d, at, smem_desc(xa), idesc(NT), 0u);
                umma_ts4<1>(d, at + 32, smem_desc(xa + C::XH), idesc(NT), 1u);
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

// 1 .. 64 rows of X (row0 .., or xrows[0 .. m)); results at rows y0 .. of Y; keys[y0 .. y0 + m) for the argmax epilogue
int qb_gemm_mid_launch(qb_ctx* ctx, cudaStream_t st, const void* X, const void* B, void* Y, const void* S, int m, int n, int k,
                       int row0, int epi, const int* xrows, unsigned long long* keys, int n_valid) {
    if (n % mid::BH || k % 128 || m < 1 || m > 64 || !ctx->tc_part) return QB_ERR_ARG;
    EncodeTiled enc = encode_tiled();
    if (!enc) return QB_ERR_UNSUPPORTED;
    const int nt = m <= 32 ? 32 : m <= 48 ? 48 : 64;
    const int tiles = n / mid::BH;
    if (tiles > QB_TC_TICKETS) return QB_ERR_ARG;
    CUtensorMap xmap = {}, wmap;
    const cuuint32_t one[2] = {1, 1};
    if (!xrows) {
        const cuuint64_t xd[2] = {(cuuint64_t)k, (cuuint64_t)m}, xs[1] = {(cuuint64_t)k * 2};
        const cuuint32_t xb[2] = {64, (cuuint32_t)nt};
        if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)((const __half*)X + (size_t)row0 * k), xd, xs, xb, one,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return QB_ERR_ARG;
    }
    const cuuint64_t wd[2] = {(cuuint64_t)n, (cuuint64_t)(k / 16)}, ws[1] = {(cuuint64_t)n * 8};
    const cuuint32_t wb[2] = {mid::BH, mid::BK / 16};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void*)B, wd, ws, wb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    mid::Args a;
    a.X = (const __half*)X; a.xrows = xrows; a.S = (const __half*)S; a.Y = Y; a.keys = keys; a.m = m; a.N = n; a.K = k;
    a.row0 = row0; a.y0 = xrows ? 0 : row0; a.n_valid = n_valid; a.err = ctx->err; a.part = ctx->tc_part;
    a.tickets = ctx->tc_tickets; a.iters = (long long)tiles * (k / 128); a.tiles = tiles;
    const int G = (int)(a.iters < ctx->sms ? a.iters : ctx->sms);
    if (nt == 32) return mid::go<32>(ctx, st, epi, G, xmap, wmap, a);
    if (nt == 48) return mid::go<48>(ctx, st, epi, G, xmap, wmap, a);
    return mid::go<64>(ctx, st, epi, G, xmap, wmap, a);
}
