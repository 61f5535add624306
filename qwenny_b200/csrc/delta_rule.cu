// The gated delta rule of a step's segments (qb_delta_rule), the reference's kernel delta_rule (kernels/qwen_deltanet.cuh:172-288)
// by another algorithm. Segments of 80 tokens and more run in CHUNKS of 64 tokens (the WY form the reference states for its
// MLX backend, src/mlx/delta.rs:6-15,85-137), the last one shorter where need be; the last 16 tokens of a segment, any
// replayed tokens and short segments run in the token form with the operation order of the decode mixer, so the checkpoint, the
// replay bank and a later rollback see the bits a decode step would make. What a segment's tokens run in depends on its length
// alone (given the scratch), so its bits do not depend on what else is in the step.
//
//  delta_chunk_prep_kernel  everything of a chunk that does not depend on the state, all chunks of all segments in parallel: with
//                           G the running sum of the log decays, gam_i = exp(G_i), A_ij = b_i (k_i . k_j) exp(G_i - G_j) (j < i),
//                           T = (I + A)^-1:  W = T diag(b gam) K,  U = T diag(b) V,  P_ij = (q_i . k_j) exp(G_i - G_j) (j <= i).
//  delta_scan_kernel        a block per (64 of a value head's columns, value head, segment) carries its slice of the f32 state
//                           in registers from chunk to chunk: D = U - W S, O = gam Q S + P D,
//                           S' = gam_C S + K^T diag(exp(G_C - G_j)) D: three products on tcgen05, two of them in sequence.
//
// Precision. The tensor cores take every f32 operand x as TWO f16 values of s x, hi = f16(s x) to nearest and lo = f16(s x - hi): 23 bits,
// with s a power of two that brings the largest finite entry of the tile (K, W: 64 x 128; V, the state and D: 16 columns) into
// [2^14, 2^15). f16 ends at 2^-24: what is lost lies 2^-39 below that entry, so values down to 2^-16 of it keep 22 bits, values
// below that fewer (3 x TF32 kept 21 bits of each for twice the instructions). a . b ~ hi_a hi_b + hi_a lo_b + lo_a hi_b,
// summed in f32. Q, P and the D that P meets only feed the step's outputs: one f16 to nearest (11 bits, as TF32 has; P and D down to
// 2^-28 of their tile's largest, D's a bound of it). The scales of the state and of D leave infinities and NaN out, so that those
// stay in their column.
#include "attn_tc.cuh"
#include "delta_common.cuh"
#include "launch.h"

namespace qb {

using namespace tc;

constexpr int CH = 64;                   // tokens per chunk
constexpr int TP_TOK = 2048;             // tokens of a step at most
constexpr int GROUPS = 8, GCOLS = 16;    // a value head's columns in groups of 16: a group shares its scales

// Tokens of a segment that run in chunks: all but the last KEEP (the checkpoint and the bank of the rollback plan are made in the token
// form); the last chunk may be a short one.
__host__ __device__ __forceinline__ int chunked_tokens(int len) { return len < CH + KEEP ? 0 : len - KEEP; }
__host__ __device__ __forceinline__ int chunks_of(int len) { return (chunked_tokens(len) + CH - 1) / CH; }
// the most chunks that `segs` segments of n tokens in all can have: (len + CH - KEEP - 1) / CH of one, for those of CH + KEEP and more
static int chunks_most(int n, int segs) {
    const int k = segs < n / (CH + KEEP) ? segs : n / (CH + KEEP);
    return (n + k * (CH - KEEP - 1)) / CH;
}

// the z-th of a step's segments that run in chunks, or -1; `place`: the chunks of those before it
__device__ __forceinline__ int long_segment(const int* seg_len, int segs, int z, int& place) {
    place = 0;
    const int lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < segs; s0 += 32) {
        const int nc = s0 + lane < segs ? chunks_of(seg_len[s0 + lane]) : 0;
        unsigned any = __ballot_sync(0xffffffffu, nc > 0);
        const bool here = z < __popc(any);
        if (here)
            for (; z > 0; z--) any &= any - 1;
        else
            z -= __popc(any);
        const int at = here ? __ffs(any) - 1 : 32;
        place += __reduce_add_sync(0xffffffffu, lane < at ? nc : 0);
        if (here) return s0 + at;
    }
    return -1;
}

// ---------------------------------------------------------------- a chunk's place in the scratch
// A tile is 64 tokens x 64 halves, a token's 128 bytes in 16-byte pieces swizzled by the token's low three bits: a K-major
// operand with tokens as rows as well as an MN-major one with tokens as k.
constexpr int TILE = CH * 128;
struct Gates {                   // of a chunk and value head
    float gam[CH], dec[CH];      // exp(G_i), exp(G_C - G_i)
    float umax[GROUPS];          // largest |U| of a group of columns
    float winv, qinv, kinv, pinv;  // 1 / scale of the tiles
    float wnorm, decmax, pad[2];   // largest row sum of |W|; largest dec
};
static_assert(sizeof(Gates) % 16 == 0, "bulk copies");
// per key head: K hi (2 tiles: keys 0..63, 64..127), K lo, Q hi; per value head: W hi, W lo, P, then U (f32, groups of 16 columns:
// [group][token][16], 16-byte pieces swizzled by (token >> 1) & 3), then Gates
constexpr int KQ_BYTES = 6 * TILE, VH_BYTES = 9 * TILE + 1024, U_AT = 5 * TILE, GATES_AT = 9 * TILE;
constexpr size_t CHUNK_BYTES = (size_t)LK_HEADS * KQ_BYTES + (size_t)LV_HEADS * VH_BYTES;
static_assert(sizeof(Gates) <= 1024, "the gates' place");
static_assert(CHUNK_BYTES == 4374528, "what the documents say of a context's scratch");
// place: the step's chunks in a row, segment after segment
__device__ __forceinline__ uint8_t* kq_at(uint8_t* tp, int place, int kh) { return tp + (size_t)place * CHUNK_BYTES + (size_t)kh * KQ_BYTES; }
__device__ __forceinline__ uint8_t* vh_at(uint8_t* tp, int place, int h) {
    return tp + (size_t)place * CHUNK_BYTES + (size_t)LK_HEADS * KQ_BYTES + (size_t)h * VH_BYTES;
}
__device__ __forceinline__ uint32_t u_at(int group, int token, int piece) {  // byte offset
    return (uint32_t)(group * (CH * 64) + token * 64 + ((piece ^ ((token >> 1) & 3)) << 4));
}

// ---------------------------------------------------------------- scales and splits
// the larger of m and |x| as an ordered word, infinities and NaN (which wrap around) as almost nothing
__device__ __forceinline__ uint32_t finite_max(uint32_t m, float x) { return max(m, (__float_as_uint(x) << 1) + 0x01000000u); }
__device__ __forceinline__ float finite_value(uint32_t m) { return m < 0x01000000u ? 0.f : __uint_as_float((m - 0x01000000u) >> 1); }
// the power of two that brings m into [2^14, 2^15) (2^126 at most), and its inverse
__device__ __forceinline__ float scale_of(float m) {
    const int e = (int)((__float_as_uint(m) >> 23) & 255);
    return __uint_as_float((uint32_t)min(max(268 - e, 1), 253) << 23);
}
__device__ __forceinline__ float inverse_of(float s) { return __uint_as_float((254u << 23) - __float_as_uint(s)); }
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = *(const uint32_t*)&h;
    lo = pack_half2(a - f.x, b - f.y);
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void ldsm_x4_trans(uint32_t* r, uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void ldsm_x4(uint32_t* r, uint32_t addr) { ldsm_x4(r[0], r[1], r[2], r[3], addr); }

// ------------------------------------------------------------------------------------------------ chunk preparation
// grid (chunks of the longest possible segment, LV_HEADS, segments that may be long enough), block 256, two blocks per SM. The products run on mma.sync (two f16
// per operand). 120 us for 2048 tokens (126 alone and cold), bound by the issue of 34,500 warp instructions a block (43 % of the slots) and
// the latency of its short phases at 3.7 warps per scheduler; the tensor pipe is busy for a fifth of it. W and U are made here, where all chunks run in parallel, so that the
// scan has two products in sequence per chunk instead of three.
constexpr int CP_THREADS = 256, TST = 72;  // TST: row stride of T (a fragment's pairs hit 32 banks)
struct PrepSmem {
    uint8_t k[4][TILE];       // K hi (keys 0..63, 64..127), K lo
    uint8_t x[4][TILE];       // Q hi, Q lo; then V hi, V lo; then W hi, W lo
    uint8_t p[TILE];
    float t[CH][TST];         // A, inverted in place
    float s[32][36];          // a merge's intermediate product
    float g[CH], b[CH], bg[CH];  // G - G_C in base 2, b, b gam
    float rows[4][CH];        // row sums of |W| by quarters of the columns
    uint32_t kmax[8], qmax[8], vmax[8][GROUPS], pmax[4], wmax[8], tmax[8], umax[2][GROUPS];
    float bmax, bgmax;        // largest b, largest b gam
};

__global__ void __launch_bounds__(CP_THREADS, 2)
delta_chunk_prep_kernel(const float* cv, uint8_t* tp, const int* seg_start, const int* seg_len, int segs) {
    extern __shared__ uint8_t cp_raw[];
    PrepSmem& M = *(PrepSmem*)(((uintptr_t)cp_raw + 1023) & ~(uintptr_t)1023);
    pdl_launch_dependents();
    int place;
    const int c = blockIdx.x, h = blockIdx.y, sg = long_segment(seg_len, segs, blockIdx.z, place), kh = h / (LV_HEADS / LK_HEADS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g8 = lane >> 2, t4 = lane & 3;
    const int t0 = sg < 0 ? 0 : seg_start[sg], cnt = sg < 0 ? 0 : min(CH, chunked_tokens(seg_len[sg]) - c * CH);  // the chunk's tokens
    if (cnt <= 0) {
        pdl_wait();  // (the kernel after this one relies on it for the kernels before)
        return;
    }
    const int tok = t0 + c * CH;
    const bool first = h % (LV_HEADS / LK_HEADS) == 0;  // this block stores the key head's tiles
    uint8_t* const kq = kq_at(tp, place + c, kh);
    uint8_t* const vh = vh_at(tp, place + c, h);
    pdl_wait();
    const float* const row0 = cv + (size_t)tok * CVW;
    auto warp_most = [](uint32_t m) { return __reduce_max_sync(0xffffffffu, m); };
    auto most8 = [](const uint32_t* v) {
        uint32_t m = v[0];
#pragma unroll
        for (int i = 1; i < 8; i++) m = max(m, v[i]);
        return finite_value(m);
    };
    // a thread's 32 values of a tile of 64 x 128: row 8 i + warp, columns 4 lane ..; rows past the chunk's last token are zero
    auto tile_load = [&](float4* v, const float* src) {
#pragma unroll
        for (int i = 0; i < 8; i++)
            v[i] = 8 * i + warp < cnt ? ld4(src + (size_t)(8 * i + warp) * CVW + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto tile_most = [&](const float4* v) {
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) m = finite_max(finite_max(finite_max(finite_max(m, v[i].x), v[i].y), v[i].z), v[i].w);
        return warp_most(m);
    };
    auto group_most = [&](const float4* v) {  // of the lane's group of 16 columns: lanes 4 j .. 4 j + 3
        uint32_t m = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) m = finite_max(finite_max(finite_max(finite_max(m, v[i].x), v[i].y), v[i].z), v[i].w);
        m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
        return max(m, __shfl_xor_sync(0xffffffffu, m, 2));
    };
    auto vscale = [&](int group) {
        uint32_t m = M.vmax[0][group];
#pragma unroll
        for (int i = 1; i < 8; i++) m = max(m, M.vmax[i][group]);
        return scale_of(finite_value(m));
    };
    auto tile_store = [&](uint8_t (*to)[TILE], const float4* v, float s) {  // hi into tiles 0 and 1, lo into 2 and 3
#pragma unroll
        for (int i = 0; i < 8; i++) {
            uint2 hi, lo;
            split2(v[i].x * s, v[i].y * s, hi.x, lo.x);
            split2(v[i].z * s, v[i].w * s, hi.y, lo.y);
            const uint32_t at = sw128(8 * i + warp, (lane & 15) >> 1) + 8 * (lane & 1);
            *(uint2*)(to[lane >> 4] + at) = hi;
            *(uint2*)(to[2 + (lane >> 4)] + at) = lo;
        }
    };
    float4 v[8];
    float kscale, qscale;
    {
        float4 q[8];
        tile_load(v, row0 + LK_HEADS * LKD + kh * LKD);
        tile_load(q, row0 + kh * LKD);
        if (warp == 0) {  // the gates and the running sum of the log decays (a decay of 0 counts as 2^-160)
            const float* e0 = row0 + (size_t)(2 * lane) * CVW + LQKV + h;
            const bool in0 = 2 * lane < cnt, in1 = 2 * lane + 1 < cnt;
            float l0 = in0 ? log2f(e0[0]) : 0.f, l1 = in1 ? log2f(e0[CVW]) : 0.f;
            const float b0 = in0 ? e0[LV_HEADS] : 0.f, b1 = in1 ? e0[CVW + LV_HEADS] : 0.f;
            l0 = l0 < -160.f ? -160.f : l0;
            l1 = l1 < -160.f ? -160.f : l1;
            // sums of the log decays from the chunk's start (for gam) and to its end. What else is taken, the difference of two tokens' G,
            // comes from the sums to the end: those are small, and exact, at the tokens that the state behind the chunk still
            // sees (taken from the start's, that state was 2.1e-6 off)
            float run = l0 + l1, back = run;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, run, o), down = __shfl_down_sync(0xffffffffu, back, o);
                if (lane >= o) run += up;
                if (lane + o < 32) back += down;
            }
            back = __shfl_down_sync(0xffffffffu, back, 1);
            const float to1 = lane < 31 ? back : 0.f, to0 = to1 + l1, m0 = exp2f(run - l1), m1 = exp2f(run), d0 = exp2f(to0), d1 = exp2f(to1);
            *(float2*)&M.g[2 * lane] = make_float2(-to0, -to1);
            *(float2*)&M.b[2 * lane] = make_float2(b0, b1);
            *(float2*)&M.bg[2 * lane] = make_float2(b0 * m0, b1 * m1);
            const float bm = warp_max(fmaxf(fabsf(b0), fabsf(b1))), gm = warp_max(fmaxf(fabsf(b0 * m0), fabsf(b1 * m1)));
            const float dm = warp_max(fmaxf(d0, d1));
            Gates* to = (Gates*)(vh + GATES_AT);
            *(float2*)&to->gam[2 * lane] = make_float2(m0, m1);
            *(float2*)&to->dec[2 * lane] = make_float2(d0, d1);
            if (lane == 0) { M.bmax = bm; M.bgmax = gm; to->decmax = dm; }
        }
        const uint32_t km = tile_most(v), qm = tile_most(q);
        if (lane == 0) { M.kmax[warp] = km; M.qmax[warp] = qm; }
        __syncthreads();
        kscale = scale_of(most8(M.kmax));
        qscale = scale_of(most8(M.qmax));
        tile_store(M.k, v, kscale);
        tile_store(M.x, q, qscale);
    }
    const float kinv = inverse_of(kscale);
    async_proxy_fence();
    __syncthreads();
    if (first && tid == 0) {
        bulk_store(kq, M.k, 4 * TILE);
        bulk_store(kq + 4 * TILE, M.x, 2 * TILE);
        bulk_commit();
    }
    // ---- K K^T (warps 0..3, rows 16 m ..) and Q K^T (warps 4..7): the column tiles up to the diagonal, in fragments (a scheduler's
    // two warps have five tiles together)
    const int m = warp < 4 ? warp : 7 - warp;
    float acc[4][2][4];
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 8; e++) acc[j][e >> 2][e & 3] = 0.f;
    {
        const uint32_t a0 = smem_u32(warp < 4 ? M.k : M.x), b0 = smem_u32(M.k);
#pragma unroll 1
        for (int kk = 0; kk < LKD / 16; kk++) {
            const int half = kk >> 2, ch = 2 * (kk & 3);
            uint32_t ah[4], al[4];
            const uint32_t at = half * TILE + sw128(16 * m + (lane & 15), ch + (lane >> 4));
            ldsm_x4(ah, a0 + at);
            ldsm_x4(al, a0 + 2 * TILE + at);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (j > m) continue;
                uint32_t bh[4], bl[4];
                const uint32_t bt = half * TILE + sw128(16 * j + (lane & 7) + ((lane >> 4) << 3), ch + ((lane >> 3) & 1));
                ldsm_x4(bh, b0 + bt);
                ldsm_x4(bl, b0 + 2 * TILE + bt);
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    mma16816(acc[j][e], al, bh[2 * e], bh[2 * e + 1]);
                    mma16816(acc[j][e], ah, bl[2 * e], bl[2 * e + 1]);
                    mma16816(acc[j][e], ah, bh[2 * e], bh[2 * e + 1]);
                }
            }
        }
    }
    tile_load(v, row0 + 2 * LK_HEADS * LKD + h * LVD);  // V is on its way meanwhile
    {
        const float inv = (warp < 4 ? kinv : inverse_of(qscale)) * kinv;
        uint32_t pm = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j > m) continue;
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const int col = 16 * j + 8 * e + 2 * t4;
                const float2 gj = *(const float2*)&M.g[col];
#pragma unroll
                for (int r = 0; r < 2; r++) {  // A, or P for the warps above
                    const int i = 16 * m + g8 + 8 * r;
                    const float gi = M.g[i], f = warp < 4 ? M.b[i] * inv : inv;
                    const int lim = warp < 4 ? i : i + 1;
                    float &a = acc[j][e][2 * r], &b = acc[j][e][2 * r + 1];
                    a = col < lim ? a * f * exp2f(gi - gj.x) : 0.f;
                    b = col + 1 < lim ? b * f * exp2f(gi - gj.y) : 0.f;
                    if (warp < 4) *(float2*)&M.t[i][col] = make_float2(a, b);
                    else pm = finite_max(finite_max(pm, a), b);
                }
            }
        }
        const uint32_t vm = group_most(v);
        pm = warp_most(pm);
        if ((lane & 3) == 0) M.vmax[warp][lane >> 2] = vm;
        if (lane == 0 && warp >= 4) M.pmax[m] = pm;
    }
    if (first && tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");  // V goes where Q was
    __syncthreads();
    // ---- T = (I + A)^-1 in place: the four 16 x 16 diagonal blocks by forward substitution, a thread per column (warps 0, 1);
    // then blocks merge pairwise, 16 -> 32 -> 64: T21 = -T22 (A21 T11)
    uint32_t tm = 0;
    if (warp < 2) {
        const int b0 = (tid >> 4) * 16, col = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float s0 = 0.f, s1 = 0.f;
#pragma unroll
            for (int j4 = 0; j4 < i; j4 += 4) {
                const float4 a = *(const float4*)&M.t[b0 + i][b0 + j4];  // (columns from i on are zero)
                s0 = fmaf(a.x, x[j4], s0);
                if (j4 + 1 < i) s1 = fmaf(a.y, x[j4 + 1], s1);
                if (j4 + 2 < i) s0 = fmaf(a.z, x[j4 + 2], s0);
                if (j4 + 3 < i) s1 = fmaf(a.w, x[j4 + 3], s1);
            }
            x[i] = i < col ? 0.f : i == col ? 1.f : -(s0 + s1);
            tm = finite_max(tm, x[i]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; i++) M.t[b0 + i][b0 + col] = x[i];
    } else if (warp >= 4) {
        const float ps = scale_of(finite_value(max(max(M.pmax[0], M.pmax[1]), max(M.pmax[2], M.pmax[3]))));
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 2; e++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const int i = 16 * m + g8 + 8 * r;
                    *(uint32_t*)(M.p + sw128(i, 2 * j + e) + 4 * t4) = j > m ? 0u : pack_half2(acc[j][e][2 * r] * ps, acc[j][e][2 * r + 1] * ps);
                }
        if (tid == 128) ((Gates*)(vh + GATES_AT))->pinv = inverse_of(ps);
    }
    tile_store(M.x, v, vscale(lane >> 2));
    __syncthreads();
    {
        const int pr = tid >> 7, i = (tid >> 3) & 15, j = 2 * (tid & 7), base = 32 * pr;
        float2 s = make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < 16; b++) {
            const float a = M.t[base + 16 + i][base + b];
            const float2 x = *(const float2*)&M.t[base + b][base + j];
            s.x = fmaf(a, x.x, s.x);
            s.y = fmaf(a, x.y, s.y);
        }
        *(float2*)&M.s[16 * pr + i][j] = s;
        __syncthreads();
        s = make_float2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < 16; b++) {
            const float a = M.t[base + 16 + i][base + 16 + b];
            const float2 x = *(const float2*)&M.s[16 * pr + b][j];
            s.x = fmaf(-a, x.x, s.x);
            s.y = fmaf(-a, x.y, s.y);
        }
        *(float2*)&M.t[base + 16 + i][base + j] = s;
        tm = finite_max(finite_max(tm, s.x), s.y);
        __syncthreads();
    }
    {
        const int i = tid >> 3, j = 4 * (tid & 7);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](float a, float4 x) { s.x = fmaf(a, x.x, s.x); s.y = fmaf(a, x.y, s.y); s.z = fmaf(a, x.z, s.z); s.w = fmaf(a, x.w, s.w); };
#pragma unroll 8
        for (int b = 0; b < 32; b++)  // (above T11's diagonal blocks nothing is stored)
            if (b >= 16 || j < 16) add(M.t[32 + i][b], *(const float4*)&M.t[b][j]);
        *(float4*)&M.s[i][j] = s;
        __syncthreads();
        s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int b = 0; b < 32; b++)
            if (b < 16 || i >= 16) add(-M.t[32 + i][32 + b], *(const float4*)&M.s[b][j]);
        *(float4*)&M.t[32 + i][j] = s;
        tm = finite_max(finite_max(finite_max(finite_max(tm, s.x), s.y), s.z), s.w);
        tm = warp_most(tm);
        if (lane == 0) M.tmax[warp] = tm;
        __syncthreads();
    }
    // ---- U = (T diag(b)) V, then W = (T diag(b gam)) K: a warp has rows 16 ma .. and 16 mb .. (whose triangles add up to five
    // steps of k) and columns 32 nq ..
    const int ma = warp & 1, mb = 3 - ma, nq = warp >> 1;
    const float tmost = most8(M.tmax);
    float w[2][4][4];
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {
        const float* f = pass ? M.bg : M.b;
        const float s = scale_of(tmost * (pass ? M.bgmax : M.bmax)), sinv = inverse_of(s);
        const float inv[2] = {sinv * (pass ? kinv : inverse_of(vscale(2 * nq))), sinv * (pass ? kinv : inverse_of(vscale(2 * nq + 1)))};
        const uint32_t xb = smem_u32(pass ? M.k : M.x);
#pragma unroll
        for (int e = 0; e < 32; e++) w[e >> 4][(e >> 2) & 3][e & 3] = 0.f;
#pragma unroll 1
        for (int kk = 0; kk <= mb; kk++) {
            uint32_t bh[2][4], bl[2][4];
#pragma unroll
            for (int p = 0; p < 2; p++) {
                const uint32_t at = (nq >> 1) * TILE + sw128(16 * kk + (lane & 15), 4 * (nq & 1) + 2 * p + (lane >> 4));
                ldsm_x4_trans(bh[p], xb + at);
                ldsm_x4_trans(bl[p], xb + 2 * TILE + at);
            }
            const int k0 = 16 * kk + 2 * t4;
            float2 f0 = *(const float2*)&f[k0], f1 = *(const float2*)&f[k0 + 8];
            f0.x *= s; f0.y *= s; f1.x *= s; f1.y *= s;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int mm = u ? mb : ma;
                if (kk > mm) continue;
                uint32_t ah[4], al[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {  // rows g8, g8 + 8; columns 2 t4, then 2 t4 + 8
                    const float2 a = *(const float2*)&M.t[16 * mm + g8 + 8 * (e & 1)][k0 + 8 * (e >> 1)];
                    const float2 x = e >> 1 ? f1 : f0;
                    split2(a.x * x.x, a.y * x.y, ah[e], al[e]);
                }
#pragma unroll
                for (int n = 0; n < 4; n++) {
                    const uint32_t *b = &bh[n >> 1][2 * (n & 1)], *l = &bl[n >> 1][2 * (n & 1)];
                    mma16816(w[u][n], al, b[0], b[1]);
                    mma16816(w[u][n], ah, l[0], l[1]);
                    mma16816(w[u][n], ah, b[0], b[1]);
                }
            }
        }
#pragma unroll
        for (int e = 0; e < 32; e++) w[e >> 4][(e >> 2) & 3][e & 3] *= inv[(e >> 3) & 1];
        if (pass) break;
        uint32_t um[2] = {0u, 0u};
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int n = 0; n < 4; n++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const float2 x = make_float2(w[u][n][2 * r], w[u][n][2 * r + 1]);
                    um[n >> 1] = finite_max(finite_max(um[n >> 1], x.x), x.y);
                    const int i = 16 * (u ? mb : ma) + g8 + 8 * r;
                    *(float2*)(vh + U_AT + u_at(2 * nq + (n >> 1), i, 2 * (n & 1) + (t4 >> 1)) + 8 * (t4 & 1)) = x;
                }
        um[0] = warp_most(um[0]);
        um[1] = warp_most(um[1]);
        if (lane == 0) { M.umax[ma][2 * nq] = um[0]; M.umax[ma][2 * nq + 1] = um[1]; }
    }
    {
        uint32_t wm = 0;
#pragma unroll
        for (int u = 0; u < 2; u++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                float s = 0.f;
#pragma unroll
                for (int n = 0; n < 4; n++)
#pragma unroll
                    for (int x = 0; x < 2; x++) {
                        wm = finite_max(wm, w[u][n][2 * r + x]);
                        s += fabsf(w[u][n][2 * r + x]);
                    }
                s = col_sum(s);
                if (t4 == 0) M.rows[nq][16 * (u ? mb : ma) + g8 + 8 * r] = s;
            }
        wm = warp_most(wm);
        if (lane == 0) M.wmax[warp] = wm;
    }
    __syncthreads();  // (every warp is done with V as well)
    const float ws = scale_of(most8(M.wmax));
#pragma unroll
    for (int u = 0; u < 2; u++)
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                uint32_t hi, lo;
                split2(w[u][n][2 * r] * ws, w[u][n][2 * r + 1] * ws, hi, lo);
                const uint32_t at = sw128(16 * (u ? mb : ma) + g8 + 8 * r, 4 * (nq & 1) + n) + 4 * t4;
                *(uint32_t*)(M.x[nq >> 1] + at) = hi;
                *(uint32_t*)(M.x[2 + (nq >> 1)] + at) = lo;
            }
    async_proxy_fence();
    __syncthreads();
    if (tid == 0) {
        bulk_store(vh, M.x, 4 * TILE);
        bulk_store(vh + 4 * TILE, M.p, TILE);
        bulk_commit();
    }
    if (warp == 1) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = lane + 32 * i;
            s = fmaxf(s, (M.rows[0][r] + M.rows[1][r]) + (M.rows[2][r] + M.rows[3][r]));
        }
        s = warp_max(s);
        Gates* to = (Gates*)(vh + GATES_AT);
        if (lane < GROUPS) to->umax[lane] = finite_value(max(M.umax[0][lane], M.umax[1][lane]));
        if (lane == 0) {
            to->wnorm = s;
            to->winv = inverse_of(ws);
            to->qinv = inverse_of(qscale);
            to->kinv = kinv;
        }
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
}

// ------------------------------------------------------------------------------------------------ the scan
// 2048 tokens: some 145 us, 190 with polling waits, spilled registers and tiles from memory, 299 with 3 x TF32 on mma.sync. Bound by a chain per
// chunk, 7900 cycles (clock64 of a state warp that converts D): 2550 until W S is there (the product warp's checks and 16 products, which take
// the tensor core 930), 2750 to convert D beside the other half's outputs of the chunk before, 950 until K^T D is there (8 products), 1150 to
// update the state and hand it on, 400 for U; some 12 us for the last 16 tokens. Issue slots 30 % active, tensor pipe 16 %. 64
// columns a block: a product with N = 128 (hi and lo) takes 66 cycles, with N = 64 50, so narrower blocks would hardly be faster, and two
// blocks per head load each tile twice instead of three times.
constexpr int SC_COLS = 64, SC_THREADS = SC_COLS * 8;  // the state's threads: one per key and 16 columns; token form: 8 per column
constexpr int SC_TAIL = 16;                            // tokens staged per round of the token form
constexpr int KLD = LKD + 4;                           // row stride of the f32 state tile
struct TokenSmem {                                     // the token form's staging
    float q[SC_TAIL][LKD], k[SC_TAIL][LKD], v[SC_TAIL][SC_COLS];
    float te[SC_TAIL], tb[SC_TAIL], tkq[SC_TAIL];
};
struct ScanSmem {
    uint8_t a[2][2][2][TILE];  // [hi, lo][keys 0..63, 64..127][W, Q]: M = 128 rows; lo of Q stays zero
    uint8_t k[4][TILE];        // K hi (2 tiles), K lo
    uint8_t p[TILE];           // P as rows 64..127 of a tile whose upper half is whatever lies before it
    union {
        struct {
            uint8_t s[2][2 * TILE];  // the state [hi, lo][128 keys][64 columns]
            uint8_t dd[2][TILE];     // dec D [hi, lo][64 tokens][64 columns]
            uint8_t d[TILE];         // D
        } o;
        float state[SC_COLS][KLD];   // the f32 state on its way between the registers of the two forms
        TokenSmem t;
    };
    uint8_t u[2][2 * TILE];    // U of a chunk: 4 groups of columns
    Gates g[2];
    float smax[2][4][4];       // [chunk parity][group][warp]
    uint64_t afull, kfull, pfull, ufull[2], sready, dready, g1done, g3done, pdone;
    uint32_t tmem;
};
constexpr int SCAN_SMEM = sizeof(ScanSmem) + 1024;
constexpr int APART_SMEM = 116 * 1024;  // of a block that shares its SM with no other of its kind
static_assert(2 * (APART_SMEM + 1024) > 228 * 1024 && APART_SMEM >= sizeof(TokenSmem), "an SM holds 228 KB, 1 KB of them per block its own");
static_assert(SCAN_SMEM <= 227 * 1024, "shared memory of a block");

// instruction descriptor of tcgen05.mma kind::f16, M = 128, N = n, A / B in MN-major order where asked
__device__ __forceinline__ constexpr uint32_t idesc_mn(int n, bool a_mn, bool b_mn) {
    return idesc(n) | (a_mn ? 1u << 15 : 0u) | (b_mn ? 1u << 16 : 0u);
}
// descriptor of an MN-major operand with the 128-byte swizzle: `stride` bytes from 64 of MN to the next 64 (the leading byte
// offset), 1024 from 8 of k to the next 8
__device__ __forceinline__ uint64_t mn_desc(uint32_t addr, uint32_t stride) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(stride >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// CHUNKS: segment blockIdx.z of those that run in chunks; 16 warps carry the state, one copies, one issues the products. Otherwise
// the segments without chunks (all of them where no chunks were prepared, `all`), PER_SM blocks per SM: two, or one where the SMs hold
// every block so, which then asks for more than half of an SM's shared memory. A token's loop is bound by issue, and early-launched
// blocks of one segment (96 on 148 SMs) pair up on SMs that the kernels before have left while others idle. The mixer, two / one:
// one segment of 30 tokens 47.6 / 36.4 us, 46 62 / 46.5, 64 79 / 59, 79 90 / 66.6; 5 segments of 8 39.4 / 44, 12 of 8 74 / 90, 12 of 40
// 219 / 261.
template <bool CHUNKS, int PER_SM>
__global__ void __launch_bounds__(CHUNKS ? SC_THREADS + 64 : SC_THREADS, PER_SM)
delta_scan_kernel(const float* p, int splits, int n, const float* cv, uint8_t* tp, float* mem, long long sst, const int* meta, float* out,
                  const int* seg_start, const int* seg_len, const int* seg_slot, const int* seg_pos0, int segs, int all, int* err) {
    extern __shared__ __align__(16) uint8_t scan_raw[];
    ScanSmem& M = *(ScanSmem*)(((uintptr_t)scan_raw + 1023) & ~(uintptr_t)1023);
    int place = 0;
    const int vs = blockIdx.x, h = blockIdx.y, sg = CHUNKS && segs > 1 ? long_segment(seg_len, segs, blockIdx.z, place) : blockIdx.z, kh = h / (LV_HEADS / LK_HEADS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int t0 = sg < 0 ? 0 : seg_start[sg], len = sg < 0 ? 0 : seg_len[sg];
    const int l0 = CHUNKS ? chunked_tokens(len) : 0, nc = (l0 + CH - 1) / CH;
    if (CHUNKS ? sg < 0 : !all && chunked_tokens(len) > 0) {  // another kernel's, or nobody's
        pdl_launch_dependents();
        pdl_wait();
        return;
    }
    constexpr int COPY_WARP = SC_THREADS / 32, MMA_WARP = COPY_WARP + 1;
    constexpr int ACC_S = 256, ACC_P = 384, TMEM_COLS = 512;  // accumulators: [W; Q] S (hi, lo) at 0 and 128 in turn, K^T D, P D (two in turn)
    if (nc > 0) {
        if (tid == 0) {
            mbar_init(&M.afull, 1); mbar_init(&M.kfull, 1); mbar_init(&M.pfull, 1); mbar_init(&M.ufull[0], 1); mbar_init(&M.ufull[1], 1);
            mbar_init(&M.sready, SC_THREADS / 32); mbar_init(&M.dready, SC_THREADS / 64);
            mbar_init(&M.g1done, 1); mbar_init(&M.g3done, 1); mbar_init(&M.pdone, 1);
            mbar_fence_init();
        }
        if (warp == MMA_WARP) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&M.tmem)), "r"(TMEM_COLS));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
        }
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }
    // (not before the tensor memory is taken: a block of a later kernel that holds tensor memory and waits for this grid must not
    // come before one of this grid's own)
    pdl_launch_dependents();
    const uint32_t tmem = nc > 0 ? M.tmem : 0u;
    if (CHUNKS && warp == COPY_WARP) {
        pdl_wait();
        if (lane == 0) {
            // a chunk's tiles are asked into L2 two chunks ahead (from memory a copy took up to 3900 cycles, half of a chunk's time), by
            // one of the blocks that read them
            auto ahead = [&](int c) {
                if (c >= nc) return;
                const uint8_t *kq = kq_at(tp, place + c, kh), *vh = vh_at(tp, place + c, h);
                if (vs == 0) bulk_prefetch(vh, 5 * TILE);
                bulk_prefetch(vh + U_AT + vs * 2 * TILE, 2 * TILE);
                if (vs == 0 && h % (LV_HEADS / LK_HEADS) == 0) bulk_prefetch(kq, KQ_BYTES);
            };
            ahead(0);
            ahead(1);
            bool ok = true;
            int na = 0, nk = 0, np = 0;  // chunks whose W, Q and U, whose K and whose P are asked for
            for (int c = 0; c < nc && ok; c++) {
                ahead(c + 2);
                const uint8_t *kq = kq_at(tp, place + c, kh), *vh = vh_at(tp, place + c, h);
                if (c > 0) ok = mbar_wait(&M.g1done, (c - 1) & 1);  // (all state warps are past chunk c - 2 as well)
                if (!ok) break;
                uint64_t* uf = &M.ufull[c & 1];
                mbar_expect_tx(uf, 2 * TILE + sizeof(Gates));
                bulk_load(M.u[c & 1], vh + U_AT + vs * 2 * TILE, 2 * TILE, uf);
                bulk_load(&M.g[c & 1], vh + GATES_AT, sizeof(Gates), uf);
                mbar_expect_tx(&M.afull, 6 * TILE);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    bulk_load(M.a[0][i][0], vh + i * TILE, TILE, &M.afull);
                    bulk_load(M.a[0][i][1], kq + (4 + i) * TILE, TILE, &M.afull);
                    bulk_load(M.a[1][i][0], vh + (2 + i) * TILE, TILE, &M.afull);
                }
                na++;
                if (c > 0) ok = mbar_wait(&M.g3done, (c - 1) & 1);
                if (!ok) break;
                mbar_expect_tx(&M.kfull, 4 * TILE);
                bulk_load(M.k, kq, 4 * TILE, &M.kfull);
                nk++;
                if (c > 0) ok = mbar_wait(&M.pdone, (c - 1) & 1);
                if (!ok) break;
                mbar_expect_tx(&M.pfull, TILE);
                bulk_load(M.p, vh + 4 * TILE, TILE, &M.pfull);
                np++;
            }
            // the block does not end before its copies have landed, also where the warps that use them have given up
            for (int u = max(na - 2, 0); u < na; u++) mbar_wait(&M.ufull[u & 1], (u >> 1) & 1);
            if (na) mbar_wait(&M.afull, (na - 1) & 1);
            if (nk) mbar_wait(&M.kfull, (nk - 1) & 1);
            if (np) mbar_wait(&M.pfull, (np - 1) & 1);
            if (!ok) atomicExch(err, 20);
        }
        __syncwarp();
    } else if (CHUNKS && warp == MMA_WARP) {
        const uint32_t a = smem_u32(M.a), k = smem_u32(M.k), s = smem_u32(M.o.s), dd = smem_u32(M.o.dd), d = smem_u32(M.o.d),
                       pt = smem_u32(M.p) - TILE;
        constexpr uint32_t W128 = idesc_mn(128, false, true), W64 = idesc_mn(64, false, true), K128 = idesc_mn(128, true, true),
                           K64 = idesc_mn(64, true, true);
        const uint32_t tm = uniform(tmem);
        bool ok = true;
        int n1 = 0, n3 = 0, np = 0;  // products committed
        for (int c = 0; c < nc; c++) {
            ok = warp_wait(&M.afull, c & 1) && warp_wait(&M.sready, c & 1);
            if (!ok) break;
            tc_fence_after();
            // [W; Q] S: hi x (hi, lo), then lo x hi
#pragma unroll
            for (int i = 0; i < 8; i++)
                umma_ss<1>(tm + (c & 1) * 128, smem_desc(a + (i >> 2) * 2 * TILE + (i & 3) * 32), mn_desc(s + i * 2048, 2 * TILE), W128, i > 0);
#pragma unroll
            for (int i = 0; i < 8; i++)
                umma_ss<1>(tm + (c & 1) * 128, smem_desc(a + 4 * TILE + (i >> 2) * 2 * TILE + (i & 3) * 32), mn_desc(s + i * 2048, 2 * TILE), W64, 1);
            umma_commit(&M.g1done);
            n1++;
            ok = warp_wait(&M.kfull, c & 1) && warp_wait(&M.dready, c & 1);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < 4; i++) umma_ss<1>(tm + ACC_S, mn_desc(k + i * 2048, TILE), mn_desc(dd + i * 2048, TILE), K128, i > 0);
#pragma unroll
            for (int i = 0; i < 4; i++) umma_ss<1>(tm + ACC_S, mn_desc(k + 2 * TILE + i * 2048, TILE), mn_desc(dd + i * 2048, TILE), K64, 1);
            umma_commit(&M.g3done);
            n3++;
            ok = warp_wait(&M.pfull, c & 1);
            if (!ok) break;
#pragma unroll
            for (int i = 0; i < 4; i++) umma_ss<1>(tm + ACC_P + (c & 1) * 64, smem_desc(pt + i * 32), mn_desc(d + i * 2048, TILE), W64, i > 0);
            umma_commit(&M.pdone);
            np++;
        }
        // (nor before its products are done: this warp gives the tensor memory back)
        if (n1) warp_wait(&M.g1done, (n1 - 1) & 1);
        if (n3) warp_wait(&M.g3done, (n3 - 1) & 1);
        if (np) warp_wait(&M.pdone, (np - 1) & 1);
        if (!ok && lane == 0) atomicExch(err, 21);
        __syncwarp();
    } else {
        const int lc = tid >> 3, sub = tid & 7, col = vs * SC_COLS + lc;  // token form: 8 lanes per value column
        int slot = seg_slot[sg], p0 = seg_pos0[sg];
        float* sm0 = mem + slot * sst;
        if (!CHUNKS) hint_state<SC_COLS, SC_THREADS>(meta, slot, p0, sm0, h * LVD + vs * SC_COLS);  // (beside the chunks its registers spill)
        pdl_wait();
        Plan pl = make_plan(meta, slot, p0, len);
        auto sbuf = [&](int b) { return sm0 + (size_t)b * SLOT_STATE + ((size_t)h * LVD + col) * LKD; };
        auto entry = [&](int b, int pos) { return sm0 + 2 * SLOT_STATE + (size_t)b * SLOT_BANK + (size_t)(pos % KEEP) * REP; };
        auto sync = [] { named_bar_sync(1, SC_THREADS); };
        // ---- the state, and the replay of accepted tokens from the bank
        float S[RPT];
        if (pl.zero) {
#pragma unroll
            for (int i = 0; i < RPT; i++) S[i] = 0.f;
        } else {
            ld_rows(S, sbuf(pl.in), sub);
        }
        for (int i = 0; i < pl.r; i++) {
            const float* e = entry(pl.in, pl.from + i);
            float k[RPT];
            ld_rows(k, e + kh * LKD, sub);
            const float dk = dot_rows(S, k);
            const float ex = e[LK_HEADS * LKD + LV_HEADS * LVD + h], be = e[LK_HEADS * LKD + LV_HEADS * LVD + LV_HEADS + h];
            const float delta = (e[LK_HEADS * LKD + h * LVD + col] - ex * dk) * be;
#pragma unroll
            for (int j = 0; j < RPT; j++) S[j] = ex * S[j] + k[j] * delta;
        }

        if (nc > 0) {
            // ============================================================ chunks: thread = key, 16 columns
            const int q = warp & 3, cg = warp >> 2, key = 32 * q + lane, i = key & 63;  // i: the token whose row of [W; Q] S is this lane's
            const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16), c16 = cg * GCOLS;
            bool dead = false;
            auto wait = [&](uint64_t* bar, int parity) {
                if (dead) return;
                dead = !warp_wait(bar, parity);
                if (dead && lane == 0) atomicExch(err, 22);
            };
            auto arrive = [&](uint64_t* bar) {  // what was written for the tensor core is complete
                async_proxy_fence();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar);
            };
            // 8 sums: hi x hi + lo x hi in the first columns, hi x lo 64 columns on. (The 16 columns go in two halves and Q S stays in
            // tensor memory until the output: a thread has 96 registers.)
            auto sums = [&](uint32_t at, float* x) {
                uint32_t a[8], b[8];
                tmem_ld8(at, a);
                tmem_ld8(at + 64, b);
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] = __uint_as_float(a[j]) + __uint_as_float(b[j]);
            };
            // 8 columns of a row of a tile of 64 columns, as hi and lo
            auto put = [&](uint8_t* hi, uint8_t* lo, int row, int ch, const float* x, float s) {
                uint4 a, b;
                split2(x[0] * s, x[1] * s, a.x, b.x);
                split2(x[2] * s, x[3] * s, a.y, b.y);
                split2(x[4] * s, x[5] * s, a.z, b.z);
                split2(x[6] * s, x[7] * s, a.w, b.w);
                const uint32_t at = sw128(row, 2 * cg + ch);
                *(uint4*)(hi + at) = a;
                *(uint4*)(lo + at) = b;
            };
            float st[16], smax, sinv;
            auto publish = [&](int c) {  // the state of chunk c for the tensor core
                float mx = 0.f;
#pragma unroll
                for (int j = 0; j < 16; j++) mx = fmaxf(mx, fabsf(st[j]));
                uint32_t mw = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
                if (mw >= 0x7f800000u) {  // an infinity: the largest finite entry
                    uint32_t f = 0;
#pragma unroll
                    for (int j = 0; j < 16; j++) f = finite_max(f, st[j]);
                    mw = __float_as_uint(finite_value(__reduce_max_sync(0xffffffffu, f)));
                }
                if (lane == 0) M.smax[c & 1][cg][q] = __uint_as_float(mw);
                named_bar_sync(2 + cg, 128);
                const float4 m4 = *(const float4*)M.smax[c & 1][cg];
                smax = fmaxf(fmaxf(m4.x, m4.y), fmaxf(m4.z, m4.w));
                const float s = scale_of(smax);
                sinv = inverse_of(s);
#pragma unroll
                for (int ch = 0; ch < 2; ch++) put(M.o.s[0], M.o.s[1], key, ch, st + 8 * ch, s);
                arrive(&M.sready);
            };
            st_rows(&M.state[lc][0], S, sub);
            for (int x = tid; x < 2 * TILE / 16; x += SC_THREADS)  // the rows of Q's lo tiles
                *(uint4*)(M.a[1][x / (TILE / 16)][1] + (x % (TILE / 16)) * 16) = make_uint4(0u, 0u, 0u, 0u);
            sync();
#pragma unroll
            for (int j = 0; j < 16; j++) st[j] = M.state[c16 + j][key];
            sync();
            publish(0);
            for (int c = 0; c < nc; c++) {
                wait(&M.ufull[c & 1], (c >> 1) & 1);
                const Gates& g = M.g[c & 1];
                const float bound = g.umax[vs * (SC_COLS / GCOLS) + cg] + g.wnorm * smax;  // of |D|
                const float ds = scale_of(bound), dds = scale_of(bound * g.decmax), gc = g.gam[CH - 1];
                const float kinv = g.kinv * inverse_of(dds), pinv = g.pinv * inverse_of(ds);
                if (q < 2) {  // D = U - W S
                    const float inv = g.winv * sinv, dec = g.dec[i] * dds;
                    wait(&M.g1done, c & 1);
                    tc_fence_after();
#pragma unroll
                    for (int ch = 0; ch < 2; ch++) {
                        float x[8], u[8];
                        *(float4*)u = *(const float4*)(M.u[c & 1] + u_at(cg, i, 2 * ch));
                        *(float4*)(u + 4) = *(const float4*)(M.u[c & 1] + u_at(cg, i, 2 * ch + 1));
                        sums(lanes + (c & 1) * 128 + c16 + 8 * ch, x);
#pragma unroll
                        for (int j = 0; j < 8; j++) u[j] = fmaf(-inv, x[j], u[j]);
                        put(M.o.dd[0], M.o.dd[1], i, ch, u, dec);
                        *(uint4*)(M.o.d + sw128(i, 2 * cg + ch)) = make_uint4(pack_half2(u[0] * ds, u[1] * ds), pack_half2(u[2] * ds, u[3] * ds),
                                                                              pack_half2(u[4] * ds, u[5] * ds), pack_half2(u[6] * ds, u[7] * ds));
                    }
                    arrive(&M.dready);
                }
                const float qinv = g.qinv * sinv * g.gam[i];
#pragma unroll
                for (int j = 0; j < 16; j++) st[j] *= gc;
                wait(&M.g3done, c & 1);
                tc_fence_after();
#pragma unroll
                for (int ch = 0; ch < 2; ch++) {
                    float x[8];
                    sums(lanes + ACC_S + c16 + 8 * ch, x);
#pragma unroll
                    for (int j = 0; j < 8; j++) st[8 * ch + j] = fmaf(kinv, x[j], st[8 * ch + j]);
                }
                if (c + 1 < nc) publish(c + 1);
                if (q >= 2) {  // O = gam Q S + P D
                    wait(&M.pdone, c & 1);
                    tc_fence_after();
                    float* to = out + (size_t)(t0 + c * CH + i) * MIX + h * LVD + vs * SC_COLS + c16;
#pragma unroll
                    for (int ch = 0; ch < 2; ch++) {
                        float x[8];
                        uint32_t pd[8];
                        tmem_ld8(lanes + ACC_P + (c & 1) * 64 + c16 + 8 * ch, pd);
                        sums(lanes + (c & 1) * 128 + c16 + 8 * ch, x);
                        if (c * CH + i < l0) {
#pragma unroll
                            for (int j = 0; j < 8; j += 2)
                                *(float2*)(to + 8 * ch + j) =
                                    make_float2(fmaf(pinv, __uint_as_float(pd[j]), qinv * x[j]), fmaf(pinv, __uint_as_float(pd[j + 1]), qinv * x[j + 1]));
                        }
                    }
                }
            }
            sync();  // (the last products have read their operands: every warp has waited for them)
#pragma unroll
            for (int j = 0; j < 16; j++) M.state[c16 + j][key] = st[j];
            sync();
            ld_rows(S, &M.state[lc][0], sub);
            // (read anew: kept across the chunks they would spill)
            t0 = __ldcg(seg_start + sg);
            len = __ldcg(seg_len + sg);
            slot = __ldcg(seg_slot + sg);
            p0 = __ldcg(seg_pos0 + sg);
            pl = make_plan(meta, slot, p0, len);
            sm0 = mem + slot * sst;
        }

        // ================================================================ the token form: tokens l0 .. len - 1
        TokenSmem& T = CHUNKS ? M.t : *(TokenSmem*)scan_raw;
        for (int c0 = l0; c0 < len; c0 += SC_TAIL) {
            const int m = min(SC_TAIL, len - c0);
            sync();  // the previous round (or the chunks) is done with the staging area
            for (int x = tid; x < m * (LKD / 4); x += SC_THREADS) {
                const int r = x / (LKD / 4), dd = (x % (LKD / 4)) * 4;
                const float* row = cv + (size_t)(t0 + c0 + r) * CVW + kh * LKD + dd;
                *(float4*)&T.q[r][dd] = ld4(row);
                *(float4*)&T.k[r][dd] = ld4(row + LK_HEADS * LKD);
            }
            for (int x = tid; x < m * (SC_COLS / 4); x += SC_THREADS) {
                const int r = x / (SC_COLS / 4), dd = (x % (SC_COLS / 4)) * 4;
                *(float4*)&T.v[r][dd] = ld4(cv + (size_t)(t0 + c0 + r) * CVW + 2 * LK_HEADS * LKD + h * LVD + vs * SC_COLS + dd);
            }
            if (tid < 2 * m) {
                const int r = tid >> 1, which = tid & 1;
                (which ? T.tb : T.te)[r] = cv[(size_t)(t0 + c0 + r) * CVW + LQKV + which * LV_HEADS + h];
            }
            sync();
            for (int r = warp; r < m; r += SC_THREADS / 32) {  // k . q of each token
                const float4 a = ld4(&T.q[r][lane * 4]), b = ld4(&T.k[r][lane * 4]);
                const float x = warp_sum(a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w);
                if (lane == 0) T.tkq[r] = x;
            }
            // the inputs of the tokens from the new checkpoint on go to its bank, for a later restart: k once per key head,
            // v by each block for its columns, the gates once per value head
            for (int r = max(0, pl.ck - (p0 + c0)); r < m; r++) {
                float* e = entry(pl.cbuf, p0 + c0 + r);
                if (vs == 0 && h % (LV_HEADS / LK_HEADS) == 0 && tid < LKD) e[kh * LKD + tid] = T.k[r][tid];
                if (tid >= 128 && tid < 128 + SC_COLS) e[LK_HEADS * LKD + h * LVD + vs * SC_COLS + tid - 128] = T.v[r][tid - 128];
                if (vs == 0 && tid == 256) {
                    e[LK_HEADS * LKD + LV_HEADS * LVD + h] = T.te[r];
                    e[LK_HEADS * LKD + LV_HEADS * LVD + LV_HEADS + h] = T.tb[r];
                }
            }
            sync();
            for (int r = 0; r < m; r++) {
                if (pl.wck && p0 + c0 + r == pl.ck) st_rows(sbuf(pl.cbuf), S, sub);
                float k[RPT], qv[RPT];
                ld_rows(k, T.k[r], sub);
                ld_rows(qv, T.q[r], sub);
                const float dk = dot_rows(S, k), dq = dot_rows(S, qv);
                const float ex = T.te[r], delta = (T.v[r][lc] - ex * dk) * T.tb[r];
                if (sub == 0) out[(size_t)(t0 + c0 + r) * MIX + h * LVD + col] = ex * dq + delta * T.tkq[r];
#pragma unroll
                for (int j = 0; j < RPT; j++) S[j] = ex * S[j] + k[j] * delta;
            }
        }
        st_rows(sbuf(pl.ebuf), S, sub);
        // ---- the conv ring: the conv inputs of the segment's last CR tokens, this block's share of the channels (after
        // delta_prep, which read the ring, has finished: it is an earlier kernel of the stream)
        const int nb = gridDim.x * gridDim.y, share = (LQKV + nb - 1) / nb;
        const int cb = (h * gridDim.x + vs) * share, cnt = max(0, min(share, LQKV - cb)), mm = min(len, CR);
        for (int x = tid; x < mm * cnt; x += SC_THREADS) {
            const int r = len - mm + x / cnt, cc = cb + x % cnt;
            float v = 0.f;
            for (int s = 0; s < splits; s++) v += p[((size_t)s * n + t0 + r) * DELTA_IN + cc];
            sm0[SLOT_RING + (size_t)((p0 + r) & (CR - 1)) * LQKV + cc] = v;
        }
    }
    if (nc > 0) {
        tc_fence_before();
        __syncthreads();
        if (warp == MMA_WARP)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

}  // namespace qb

using namespace qb;

size_t qb_delta_tp_bytes(int chunks) { return (size_t)chunks * CHUNK_BYTES; }
static_assert(TP_TOK / (CH + KEEP) * (CH - KEEP - 1) + TP_TOK < (QB_DELTA_CHUNKS + 1) * CH, "room for the chunks of any step");

// of the longest segment that the step can hold
static int chunked_of(const qb_ctx* ctx, int n, int segs) { return chunks_most(n, segs) <= ctx->delta_chunks ? chunked_tokens(n) : 0; }

int qb_delta_rule_launches(const qb_ctx* ctx, int n, int segs) { return chunked_of(ctx, n, segs) == 0 ? 1 : segs > 1 ? 3 : 2; }

extern "C" {

// The chunked form's scratch (the chunks' tiles) belongs to the context; a step that may have more chunks than its context has room
// for runs every segment in the token form.
int qb_delta_rule(qb_ctx* ctx, void* stream, const float* p, int splits, int n, const float* cv, float* mem,
                  long long sst, const int* meta, float* out, const int* seg_start, const int* seg_len,
                  const int* seg_slot, const int* seg_pos0, int segs) {
    if (!ctx || !p || !cv || !mem || !meta || !out || !seg_start || !seg_len || !seg_slot || !seg_pos0 || n <= 0 ||
        segs <= 0 || splits < 1)
        return QB_ERR_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (n > TP_TOK) return QB_ERR_TOO_LARGE;
    const int l0 = chunked_of(ctx, n, segs);
    const int most = segs < n / (CH + KEEP) ? segs : n / (CH + KEEP);  // segments that can run in chunks
    if (l0 > 0) {
        int rc = launch(ctx, delta_chunk_prep_kernel, dim3((l0 + CH - 1) / CH, LV_HEADS, most), dim3(CP_THREADS), sizeof(PrepSmem) + 1024, st, cv,
                        (uint8_t*)ctx->delta_tp, seg_start, seg_len, segs);
        if (rc) return rc;
    }
    // the segments in the token form, unless the step's only one may run in chunks
    if (l0 == 0 || segs > 1) {
        const bool apart = (LVD / SC_COLS) * LV_HEADS * segs <= ctx->sms;
        int rc = launch(ctx, apart ? delta_scan_kernel<false, 1> : delta_scan_kernel<false, 2>, dim3(LVD / SC_COLS, LV_HEADS, segs), dim3(SC_THREADS),
                        apart ? APART_SMEM : sizeof(TokenSmem), st, p, splits, n, cv, (uint8_t*)nullptr, mem, sst, meta, out, seg_start, seg_len,
                        seg_slot, seg_pos0, segs, l0 == 0, ctx->err);
        if (rc || l0 == 0) return rc;
    }
    return launch(ctx, delta_scan_kernel<true, 1>, dim3(LVD / SC_COLS, LV_HEADS, most), dim3(SC_THREADS + 64), SCAN_SMEM, st, p, splits, n, cv,
                  (uint8_t*)ctx->delta_tp, mem, sst, meta, out, seg_start, seg_len, seg_slot, seg_pos0, segs, 0, ctx->err);
}

}  // extern "C"
