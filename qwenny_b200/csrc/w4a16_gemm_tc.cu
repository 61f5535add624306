// W4A16 product for prompt-sized steps (more than 64 token rows; zero-point matrices: more than 16) on the 5th-generation
// tensor cores: Y = X . W^T with W int4 in the reference's Marlin layout. Replaces marlin::mul<{1..4},16,4,*> (kernels/marlin.cuh:171-582,
// launched by Gemm::marlin, src/cuda/core.rs:569-612, for n > 16).
//
// A pair of blocks (a cluster of two, one block per SM) computes a tile of 256 outputs x up to 256 tokens with
// tcgen05.mma.cta_group::2: each block holds 128 outputs (its half of the M = 256 rows of A and of the accumulator, in
// its own tensor memory) and half of the tile's tokens (its half of B, in its own shared memory).
// The weights are the A operand and go to TENSOR memory: a Marlin word's lane holds outputs {g, g + 8} x columns
// {2t, 2t + 1, 2t + 8, 2t + 9} of a 16 x 16 block, which is exactly what a lane of tcgen05.st.16x128b writes, so the
// dequantised halves go from registers to tensor memory without touching shared memory. What that buys: the form that
// wrote them to shared memory (one block per tile, two M = 128 halves re-reading the X tile) moved 169 KB through an SM's
// shared memory per 1024 cycles of products and was bound by it (tensor pipe 65 % active); this one moves 80 KB per
// 1024. A stage is 128 of k because the issuing warps are the next limit: a wait, a commit and their like cost 180 cycles per
// stage beside 65 per product, and the copying lane 70 per copy (64 of k per stage: 600 cycles of the 512 at N = 256).
//
// The work is the list of (tile, k block of 128) pairs, tile after tile, on a persistent grid of at most one pair per two SMs. Where
// whole tiles leave pairs idle the list is dealt out in equal contiguous shares (stream-K): a pair that ends or starts inside a tile
// writes that tile's partial accumulators to scratch and takes a ticket; the tile's last arriver adds the parts in pair order and runs
// the epilogue, nobody waits.
// Per (tile, k block):
//   warps 0-7   dequantise: lop3 / hsub2 to q - 8, one hfma2 by the f16 group scale (the reference's rounding:
//               w = f16((q - 8) s), kernels/marlin.cuh:100-124), tcgen05.st into the stage's 64 columns
//   warps 8-15  the accumulators of a finished tile (or part): tcgen05.ld, Y [token][output] f32, or silu(gate) * up as f16 for
//               the interleaved SwiGLU matrices, by way of shared memory and one bulk copy per 16 tokens x 32 outputs; the next tile's
//               weights are unpacked meanwhile
//   warp 16     copies, one lane: the X half tile (tensor map, 128-byte swizzle), the 8 KB of words (tensor map), the
//               group's scales; full/empty mbarriers, a ring of 4 stages
//   warp 17     of the pair's first block: issues the products (K = 16 each) as a whole warp, tcgen05.commit hands the stage
//               back in both blocks when they have read it
// Bound by the tensor pipe and, where it runs for long, by the power it takes. With the epilogue in the unpacking warps, one block per
// tile, 4-byte stores and a fence per thread / as it is, us from a graph: 2048 rows of 16384 x 5120 243 / 226, of 34816 x 5120 545 / 507,
// 333 rows of 5120 x 6144 with zero points 36.0 / 29.8, 100 rows 25.4 / 21.0, 256 rows of 2048 x 2048 39.9 / 32.0, 70 of 1024 x 1024 15.6 / 13.1.
#include "launch.h"
#include "pair_tc.cuh"

namespace qb {

namespace tc {

enum { EPI_PLAIN_TC = 0, EPI_SILU_TC = 1 };
constexpr int BO = 256;             // outputs per pair of blocks
constexpr int BH = BO / 2;          // outputs per block: the 128 lanes of its tensor memory
constexpr int BT = 256;             // most tokens per tile (the product's N); a launch takes the width that divides its rows
constexpr int BK = 128;             // k per stage: two 128-byte swizzle rows of f16, one group of scales
constexpr int NSTAGE = 4;           // ring depth, in shared memory and in tensor memory (4 x 64 columns + 256 = 512)
constexpr int XH_BYTES = BT / 2 * 64 * 2;   // 16 KB: this block's half of the tokens, 64 of k
constexpr int X_BYTES = 2 * XH_BYTES;
constexpr int W_BYTES = BH * BK / 2;        // 8 KB of Marlin words
constexpr int S_BYTES = 512;                // 128 f16 scales, then (zero-point matrices) their offsets (8 - z) * scale
constexpr int DQ_WARPS = 8, DQ_GROUPS = DQ_WARPS / 4;  // a group of four warps dequantises a stage; the groups take turns
constexpr int EP_WARPS = 8, COPY_WARP = DQ_WARPS + EP_WARPS, MMA_WARP = COPY_WARP + 1;
constexpr int THREADS = (MMA_WARP + 1) * 32;
constexpr int OUT_BYTES = 16 * 32 * 4;      // 16 tokens x 32 outputs of an epilogue warp on their way to Y (two of them in turn)
constexpr int SMEM_BYTES = NSTAGE * (X_BYTES + W_BYTES + S_BYTES) + EP_WARPS * 2 * OUT_BYTES + 1024 /* barriers, tmem address */ + 1024 /* alignment slack */;
constexpr int TMEM_COLS = 512;
constexpr int A_COLS = BK / 2;              // tensor-memory columns of a stage's weights

struct Args {
    const __half* S;     // scales [K/128][N]
    void* Y;             // plain: f32 [.][N]; silu: f16 [.][N/2]; rows row0 ..
    int m, N, K, row0;
    int* err;
    int bt, tiles;       // tokens per tile (a multiple of 32, at most BT), tiles
    float* part;         // [pair][2][block][BT / 4][BH][4] partial tiles: [.][0] a share's first tile begun by an earlier pair, [.][1] its last, unfinished one
    int* tickets;        // two per tile (one per block of the pair), zero between launches
    int iters;           // tiles x k blocks
    int direct;          // Y does not start on 16 bytes: plain stores
    int zp;              // S holds a second table [K/128][N] after the scales: the offsets (8 - z) * scale of zero-point matrices
};

template <int EPI, bool SHARES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    w4a16_gemm_tc_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap ymap, const Args a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // swizzled tiles want 1 KB
    uint8_t* wsmem = smem + NSTAGE * X_BYTES;
    uint8_t* ssmem = wsmem + NSTAGE * W_BYTES;
    uint8_t* osmem = ssmem + NSTAGE * S_BYTES;
    uint64_t* full = (uint64_t*)(osmem + EP_WARPS * 2 * OUT_BYTES);  // copies landed in this block
    uint64_t* aready = full + NSTAGE;           // (first block) the weights are in both blocks' tensor memory, X in both's shared memory
    uint64_t* empty = aready + NSTAGE;          // the stage's products are done
    uint64_t* done = empty + NSTAGE;            // all products of a segment are done
    uint64_t* accfree = done + 1;               // (first block) both blocks have read the segment's accumulators
    uint32_t* tmem_slot = (uint32_t*)(accfree + 1);
    // this block finishes its half of the tile (the ticket's answer, for the epilogue warps); the first of the pairs that hold it, how many
    int* flag = (int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)cluster_ctarank(), pair = blockIdx.x >> 1, G = gridDim.x >> 1;
    const int nkb = a.K / BK, ntn = a.N / BO;
    Walk<SHARES> walk(a.iters, a.tiles, nkb, G, pair);
    int tile, kb0, kb1;

    if (threadIdx.x == 0) {
        for (int i = 0; i < NSTAGE; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&aready[i], 2 * 4);
            mbar_init(&empty[i], 1);
        }
        mbar_init(done, 1);
        mbar_init(accfree, 2 * EP_WARPS);
        mbar_fence_init();
    }
    if (warp == MMA_WARP) {  // the product warps own the tensor memory, one in each block
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cluster_sync();  // the other block's barriers are initialised, its tensor memory allocated
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + BT;
    pdl_launch_dependents();
    pdl_wait();

    // Every role walks the pair's share as the same list of segments (tile, k blocks [kb0, kb1)); `ring` counts the
    // stages of the whole share, so the ring's slots and phases run on from one segment to the next.
    if (warp == COPY_WARP) {
        // ---------------------------------------------------------------- copies
        if (lane == 0) {
            const uint64_t pol = policy_evict_last();
            bool ok = true;
            uint32_t ring = 0;  // (a share is far below 2^32 stages)
            const uint32_t bytes = (uint32_t)a.bt / 2 * BK * 2 + W_BYTES + BH * 2 * (1 + a.zp);
            while (ok && walk.next(tile, kb0, kb1)) {
                const int n0 = (tile % ntn) * BO + rank * BH, tok0 = (tile / ntn) * a.bt + rank * (a.bt / 2);
                for (int kb = kb0; kb < kb1; kb++, ring++) {
                    const int s = (int)(ring % NSTAGE);
                    if (ring >= NSTAGE) {
                        ok = mbar_wait(&empty[s], ((ring / NSTAGE) - 1) & 1);
                        if (!ok) break;
                    }
                    mbar_expect_tx(&full[s], bytes);
                    tma_load_2d(smem + s * X_BYTES, &xmap, kb * BK, tok0, &full[s]);
                    tma_load_2d(smem + s * X_BYTES + XH_BYTES, &xmap, kb * BK + 64, tok0, &full[s]);
                    tma_load_2d(wsmem + s * W_BYTES, &wmap, n0, kb * (BK / 16), &full[s]);
                    bulk_g2s(ssmem + s * S_BYTES, a.S + (size_t)kb * a.N + n0, BH * 2, &full[s], pol);
                    if (a.zp)
                        bulk_g2s(ssmem + s * S_BYTES + BH * 2, a.S + (size_t)(a.K / 128 + kb) * a.N + n0, BH * 2, &full[s], pol);
                }
            }
            if (!ok) atomicExch(a.err, 5);
        }
        __syncwarp();
    } else if (warp < DQ_WARPS) {
        // ---------------------------------------------------------------- dequantise into tensor memory
        // a warp writes the 32 tensor-memory lanes of its quarter q (warp % 4): two 16-row blocks of the whole stage
        const int q = warp & 3, h = warp >> 2, g = lane >> 2;
        const uint32_t quarter = (uint32_t)(q * 32) << 16;
        const uint32_t aready0 = cluster_map(aready, 0);
        bool dead = false;
        uint32_t ring = 0;
        while (walk.next(tile, kb0, kb1)) {
            for (int kb = kb0; kb < kb1; kb++, ring++) {
                if ((int)(ring % DQ_GROUPS) != h) continue;
                const int s = (int)(ring % NSTAGE);
                if (!dead) {
                    dead = !mbar_wait(&full[s], (ring / NSTAGE) & 1);
                    if (dead && lane == 0) atomicExch(a.err, 6);
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");  // (the slot's earlier products have read it)
                // words [k16 8][c64 2][lane 32] x 4 blocks; this warp's: c64 q / 2, blocks 2 (q % 2) + b
                const uint8_t* wp = wsmem + s * W_BYTES + (q >> 1) * 512 + lane * 16 + (q & 1) * 8;
                uint2 w[8];
#pragma unroll
                for (int j = 0; j < 8; j++) w[j] = *(const uint2*)(wp + j * 1024);
                // scales of outputs 16 b + g + 8 i of a c64 at 8 g + 2 b + i
                const __half* sp = (const __half*)(ssmem + s * S_BYTES) + (q >> 1) * 64 + 8 * g + 4 * (q & 1);
                const uint2 s4 = *(const uint2*)sp;
                uint2 z4 = make_uint2(0u, 0u);  // the offsets (0: the symmetric form)
                if (a.zp) z4 = *(const uint2*)(sp + BH);
#pragma unroll
                for (int bh = 0; bh < 4; bh++) {  // 16-row block b, k half hf of the stage
                    const int b = bh & 1, hf = bh >> 1;
                    const __half2 sc = *(const __half2*)(b ? &s4.y : &s4.x), zc = *(const __half2*)(b ? &z4.y : &z4.x);
                    const __half2 s0 = __low2half2(sc), s1 = __high2half2(sc), z0 = __low2half2(zc), z1 = __high2half2(zc);
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
                        // (q - 8) * scale + offset, rounded once (scale_z, kernels/marlin.cuh:126-133); with offset 0 the
                        // symmetric form's product
                        __half2 v0 = __hfma2(__hsub2(*(__half2*)&lo0, *(const __half2*)&SUB_LO), s0, z0);  // row g,     k 2t
                        __half2 v1 = __hfma2(__hsub2(*(__half2*)&lo1, *(const __half2*)&SUB_LO), s1, z1);  // row g + 8, k 2t
                        __half2 v2 = __hfma2(__hsub2(*(__half2*)&hi0, *(const __half2*)&SUB_HI), s0, z0);  // row g,     k 2t + 8
                        __half2 v3 = __hfma2(__hsub2(*(__half2*)&hi1, *(const __half2*)&SUB_HI), s1, z1);  // row g + 8, k 2t + 8
                        r[4 * j] = *(uint32_t*)&v0; r[4 * j + 1] = *(uint32_t*)&v1;
                        r[4 * j + 2] = *(uint32_t*)&v2; r[4 * j + 3] = *(uint32_t*)&v3;
                    }
                    tmem_st_16x128_x8(tmem_a + s * A_COLS + 32 * hf + quarter + ((uint32_t)(16 * b) << 16), r);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_at(aready0 + 8 * s);
            }

        }
    } else if (warp < COPY_WARP) {
        // ---------------------------------------------------------------- the segments' accumulators, then the epilogue
        // (the two warps of a quarter share the tokens)
        const int e = warp - DQ_WARPS, q = warp & 3, h = e >> 2, lrow = q * 32 + lane;
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16), accfree_at = cluster_map(accfree, 0);
        const int c_lo = h * (a.bt / 2), c_hi = c_lo + a.bt / 2;
        uint8_t* const stage = osmem + e * 2 * OUT_BYTES;
        constexpr int PS = BH * 4;  // of a part: [4 tokens][output][4], a thread's sums in 16-byte pieces
        constexpr int FIRST_EP = DQ_WARPS * 32;
        bool dead = false;
        uint32_t puts = 0;
        for (int seg = 0; walk.next(tile, kb0, kb1); seg++) {
            const int n0 = (tile % ntn) * BO + rank * BH, tok0 = (tile / ntn) * a.bt, orow = n0 + lrow;
            const bool cut = SHARES && (kb0 > 0 || kb1 < nkb);
            if (cut && threadIdx.x == FIRST_EP) walk.parts_of(tile, flag[1], flag[2]);  // (read behind the barriers at the tile's end)
            if (!dead) {
                dead = !mbar_wait(done, (uint32_t)seg & 1);
                if (dead && lane == 0) atomicExch(a.err, 8);
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            int parts = 1, first = 0;
            bool finish = !dead;
            if (cut) {
                // a part of the tile: store it, take the tile's ticket; the last arriver finishes the tile
                float* slot = a.part + ((size_t)(pair * 2 + (kb0 == 0 ? 1 : 0)) * 2 + rank) * (BT * BH) + lrow * 4;
                if (!dead) {
#pragma unroll 1
                    for (int c = c_lo; c < c_hi; c += 16) {
                        uint32_t v[16];
                        tmem_ld16(tbase + c, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 16; j += 4) *(uint4*)(slot + (size_t)((c + j) / 4) * PS) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                    }
                }
                named_bar_sync(1, EP_WARPS * 32);
                if (threadIdx.x == FIRST_EP) {
                    __threadfence();  // (for all warps' sums: the barrier orders them before it)
                    const bool last = atomicAdd(&a.tickets[2 * tile + rank], 1) == flag[2] - 1;
                    *flag = last;
                    if (last) {
                        a.tickets[2 * tile + rank] = 0;
                        __threadfence();
                    }
                }
                named_bar_sync(1, EP_WARPS * 32);
                finish = *flag != 0 && !dead;
                first = flag[1]; parts = flag[2];
                named_bar_sync(1, EP_WARPS * 32);  // (the flag may be rewritten by the next segment)
            }
            // where pair first + p keeps its part: its last tile's for the first of them, its first one's for the others
            auto part_of = [&](int p) {
                return (const float4*)(a.part + ((size_t)((first + p) * 2 + (p == 0 ? 1 : 0)) * 2 + rank) * (BT * BH) + lrow * 4);
            };
            if (finish) {
                const int mine = pair - first;
                constexpr int UP = 3;  // parts on their way at a time
                float4 x[UP][4];
                auto ask = [&](int u, int p, int c) {
#pragma unroll
                    for (int j = 0; j < 4; j++) x[u][j] = __ldcg(part_of(p) + (c / 4 + j) * (PS / 4));
                };
                if (SHARES && parts == 2) ask(0, 1 - mine, c_lo);
#pragma unroll 1
                for (int c = c_lo; c < c_hi; c += 16) {
                    uint32_t v[16];
                    auto add = [&](int u) {
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            v[4 * j] = __float_as_uint(__uint_as_float(v[4 * j]) + x[u][j].x);
                            v[4 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 1]) + x[u][j].y);
                            v[4 * j + 2] = __float_as_uint(__uint_as_float(v[4 * j + 2]) + x[u][j].z);
                            v[4 * j + 3] = __float_as_uint(__uint_as_float(v[4 * j + 3]) + x[u][j].w);
                        }
                    };
                    if (!SHARES || parts <= 2) {
                        tmem_ld16(tbase + c, v);
                        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                        if (SHARES && parts == 2) {  // own + other = other + own: no order to keep
                            add(0);
                            if (c + 16 < c_hi) ask(0, 1 - mine, c + 16);  // the next ones are on their way meanwhile
                        }
                    } else {  // more parts: all of them from scratch, in pair order
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = 0;
#pragma unroll 1
                        for (int p = 0; p < parts; p += UP) {
#pragma unroll
                            for (int u = 0; u < UP; u++)
                                if (p + u < parts) ask(u, p + u, c);
#pragma unroll
                            for (int u = 0; u < UP; u++)
                                if (p + u < parts) add(u);
                        }
                    }
                    if (tok0 + c >= a.m) continue;
                    // the 16 tokens go through shared memory to one copy of a 32-output box (what lies past the last row is left out)
                    uint8_t* const ob = stage + (puts & 1) * OUT_BYTES;
                    if (!a.direct) {
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
                        __syncwarp();
                    }
                    if (EPI == EPI_SILU_TC) {
                        // packed rows 16 p + i are gate rows, 16 p + 8 + i their up rows, 8 lanes on: the gate lanes take
                        // the even tokens, the up lanes the odd ones, each with the value the other holds
                        const bool up_lane = (lane & 8) != 0;
#pragma unroll
                        for (int j = 0; j < 16; j += 2) {
                            const uint32_t other = __shfl_xor_sync(0xffffffffu, up_lane ? v[j] : v[j + 1], 8);
                            const float gate = __uint_as_float(up_lane ? other : v[j]), up = __uint_as_float(up_lane ? v[j + 1] : other);
                            const int t = j + (up_lane ? 1 : 0);
                            const __half y = __float2half_rn(silu(gate) * up);
                            if (!a.direct)
                                ((__half*)ob)[t * 16 + (lane >> 4) * 8 + (lane & 7)] = y;
                            else if (tok0 + c + t < a.m)
                                ((__half*)a.Y)[(size_t)(a.row0 + tok0 + c + t) * (a.N / 2) + (orow >> 4) * 8 + (orow & 7)] = y;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            if (!a.direct)
                                ((uint32_t*)ob)[j * 32 + lane] = v[j];
                            else if (tok0 + c + j < a.m)
                                ((uint32_t*)a.Y)[(size_t)(a.row0 + tok0 + c + j) * a.N + orow] = v[j];
                        }
                    }
                    if (!a.direct) {
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&ymap, ob, EPI == EPI_SILU_TC ? (n0 + q * 32) / 2 : n0 + q * 32, a.row0 + tok0 + c);
                            asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
                        }
                        puts++;
                    }
                }
            }
            // the accumulator columns may be overwritten by the next segment's first product
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_at(accfree_at);
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // (the writes themselves end with the grid)
    } else if (rank == 0) {
        // ---------------------------------------------------------------- the pair's products (one whole warp)
        bool ok = true;
        uint32_t ring = 0;
        int seg = 0;
        const uint32_t id = idesc_pair(a.bt), xs = smem_u32(smem), d = uniform(tmem);
        for (; ok && walk.next(tile, kb0, kb1); seg++) {
            if (seg > 0) {  // the epilogue warps of both blocks have read the previous segment's accumulators
                ok = warp_wait(accfree, (uint32_t)(seg - 1) & 1);
                if (!ok) break;
            }
            for (int kb = kb0; kb < kb1; kb++, ring++) {
                const int s = (int)(ring % NSTAGE);
                ok = warp_wait(&aready[s], (ring / NSTAGE) & 1);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t at = uniform(tmem_a + s * A_COLS), xa = uniform(xs + s * X_BYTES);
                umma_ts4<2>(d, at, smem_desc(xa), id, kb > kb0 ? 1u : 0u);
                umma_ts4<2>(d, at + 32, smem_desc(xa + XH_BYTES), id, 1u);
                umma2_commit(&empty[s]);
            }
            if (ok) umma2_commit(done);
        }
        if (!ok && lane == 0) atomicExch(a.err, 7);
        __syncwarp();
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    cluster_sync();  // the other block's products read this block's shared and tensor memory until here
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

}  // namespace tc

}  // namespace qb

using namespace qb;

size_t qb_tc_part_bytes(int sms) { return (size_t)(sms / 2) * 2 * tc::BT * tc::BO * sizeof(float); }  // two partial tiles per pair

// Y = X . W^T for many rows: plain (f32 [m][n]) or SwiGLU (f16 [m][n/2]). X f16 [.][k], rows row0 .. row0 + m - 1.
int qb_gemm_tc_launch(qb_ctx* ctx, cudaStream_t st, const void* X, const void* B, void* Y, const void* S, int m, int n,
                      int k, int row0, int epi, int zp) {
    if (n % tc::BO || k % 128 || m < 1) return QB_ERR_ARG;
    qb::EncodeTiled enc = qb::encode_tiled();
    if (!enc) return QB_ERR_UNSUPPORTED;
    // token tiles: as few as possible, all of the same width (a multiple of 32): 333 rows are two tiles of 192, not one
    // of 256 and a mostly empty one
    const int tt = (m + tc::BT - 1) / tc::BT, bt = ((m + tt - 1) / tt + 31) / 32 * 32;
    const long long tiles = (long long)(n / tc::BO) * tt;
    if (tiles > QB_TC_TICKETS / 2) return QB_ERR_ARG;
    CUtensorMap xmap, wmap, ymap = {};
    const cuuint32_t one[2] = {1, 1};
    const cuuint64_t xd[2] = {(cuuint64_t)k, (cuuint64_t)m}, xs[1] = {(cuuint64_t)k * 2};
    const cuuint32_t xb[2] = {64, (cuuint32_t)(bt / 2)};
    void* base = (void*)((const __half*)X + (size_t)row0 * k);
    if (enc(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, base, xd, xs, xb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    // the words: K/16 rows of 2N words = N 8-byte elements; a stage's box: 128 outputs x 8 rows
    const cuuint64_t wd[2] = {(cuuint64_t)n, (cuuint64_t)(k / 16)}, ws[1] = {(cuuint64_t)n * 8};
    const cuuint32_t wb[2] = {tc::BH, tc::BK / 16};
    if (enc(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, (void*)B, wd, ws, wb, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    // Y up to the last row of the call; boxes of 16 rows x 32 outputs (16 after SwiGLU)
    const bool silu = epi == QB_EPI_SILU, direct = ((uintptr_t)Y & 15) != 0;
    const cuuint64_t yd[2] = {(cuuint64_t)(silu ? n / 2 : n), (cuuint64_t)(row0 + m)}, ys[1] = {yd[0] * (silu ? 2 : 4)};
    const cuuint32_t yb[2] = {silu ? 16u : 32u, 16};
    if (!direct && enc(&ymap, silu ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, Y, yd, ys, yb, one,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return QB_ERR_ARG;
    const int pairs = ctx->sms / 2;
    tc::Args a;
    a.S = (const __half*)S; a.Y = Y; a.m = m; a.N = n; a.K = k; a.row0 = row0; a.err = ctx->err;
    a.zp = zp ? 1 : 0; a.part = ctx->tc_part; a.tickets = ctx->tc_tickets; a.iters = (int)tiles * (k / tc::BK);
    a.bt = bt; a.tiles = (int)tiles; a.direct = direct;
    // How the list is dealt: whole tiles, pair by pair in turn, where they fill five sixths of the rounds, else equal shares of the list over
    // all pairs (5120 x 6144, 2048 rows, 2.2 rounds: 97 us as shares, 100 as tiles; 1500 rows, 1.6: 74 and 69; 700 rows, 0.8: 45 and 37).
    // Not by time alone: the tensor core's f32 sums are cut off, not rounded, and lose 1.5e-7 of the result (2-norm) per 128 of k that an
    // accumulator runs over. Shares are the shortest parts there are; a tile that is whole where they are the other choice, or cut into
    // fewer equal parts, is faster with few tiles and further off: 2048 x 2048 at 70 rows 11.3 us and 8.1e-7 in two parts, 15.4 and 3.0e-7 as shares;
    // 5120 x 6144 at 70 16.1 and 2.4e-6 in three, 18.2 and 1.8e-6, at 700 37 and 7.1e-6 whole, 45 and 4.5e-6; with zero points, whose rounding is
    // 4.7e-5, at 333 28.6 and 4.78e-5 whole, 29.8 and 4.74e-5. From five sixths on a tile's error is that of its k: 2.4e-6 for 2048, 2.0e-5 for 17408.
    const long long rounds = (tiles + pairs - 1) / pairs;
    bool whole = 6 * tiles > 5 * rounds * pairs;
    if (ctx->tune_ctas == 1000) whole = false;  // measurement: shares whatever the shape
    if (ctx->tune_ctas == 1001) whole = true;   //              tiles whatever the shape
    if (!ctx->tc_part) whole = true;            // a context without the scratch
    const long long units = whole ? tiles : a.iters;
    const int G = (int)(units < pairs ? units : pairs);
    dim3 grid((unsigned)(2 * G));
    if (epi == QB_EPI_SILU)
        return whole ? launch(ctx, tc::w4a16_gemm_tc_kernel<tc::EPI_SILU_TC, false>, grid, dim3(tc::THREADS), tc::SMEM_BYTES, st, xmap, wmap, ymap, a)
                     : launch(ctx, tc::w4a16_gemm_tc_kernel<tc::EPI_SILU_TC, true>, grid, dim3(tc::THREADS), tc::SMEM_BYTES, st, xmap, wmap, ymap, a);
    return whole ? launch(ctx, tc::w4a16_gemm_tc_kernel<tc::EPI_PLAIN_TC, false>, grid, dim3(tc::THREADS), tc::SMEM_BYTES, st, xmap, wmap, ymap, a)
                 : launch(ctx, tc::w4a16_gemm_tc_kernel<tc::EPI_PLAIN_TC, true>, grid, dim3(tc::THREADS), tc::SMEM_BYTES, st, xmap, wmap, ymap, a);
}
