// Gated GQA attention of a decode / verify step over the int8 KV cache.
//  attn_prep    per token: sum of the in-projection parts, q/k RMSNorm(1+w), partial RoPE, q scaled to base-2 scores,
//               sigmoid gate -> out, k and v quantised into the cache in the reference's byte order
//               (replaces attn_prep + kv_store, kernels/qwen.cu:156-202, kernels/attn.cuh:50-64)
//  attn_decode  split-K flash-decode: a block per (segment, kv head, key split), or with many of those a block per SM that
//               takes a run of them, streams a split's keys and values with
//               bulk async copies into a shared-memory ring (keys are [pos][256] and values [pos/16][256][16] bytes
//               per head, both contiguous per run) while RT x 4 warps compute S = Q K^T and O += P V on tensor cores
//               with a warp-level base-2 online softmax, straight from the int8 bytes (prmt to 1152 + q halves, the
//               offset folded out through the row sums as the reference does, kernels/attn.cuh:38-40,198-234)
//               (replaces attn_mq_tc<RT>, kernels/attn.cuh:77-261)
//  attn_combine merges the splits of a (token, head) in split order, multiplies into the gated output and can write
//               the f16 copy the out-projection reads (replaces attn_combine + to_xin, kernels/attn.cuh:271-325,
//               kernels/qwen.cu:136-138)
// The size of a key split is a function of the key count alone (dec_chunk), so a token's sums are the same whether
// it runs alone or with drafts.
#include "attn_tc.cuh"
#include "dec_ring.h"
#include "launch.h"
#include "measure.h"

namespace qb {

// ------------------------------------------------------------------------------------------------ attn_prep
// grid (n tokens, 2): block (t, 0) makes the 24 query heads and their gates (a warp per head), block (t, 1) the 4 key
// and 4 value heads and stores them in the cache. A warp's lane owns dims lane + 32 j of its head: the RoPE pair
// (d, d + 32) of the 64 rotated dims is then elements 0 and 1 of one lane, and the sum of squares adds the lane's eight
// values in dim order, then the lanes as a butterfly: the order that makes the int8 codes the reference's, bit for bit.
constexpr int HEAD_VALS = HD / 32;

struct HeadRow {
    float v[HEAD_VALS];
};

// the head row at `col` of token t's in-projection, summed over the split-K parts
__device__ __forceinline__ HeadRow head_row(const float* part, int splits, int n, int t, int col, int lane) {
    HeadRow r;
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) r.v[j] = 0.f;
    for (int sp = 0; sp < splits; sp++) {
        const float* p = part + ((size_t)sp * n + t) * ATTN_IN + col + lane;
#pragma unroll
        for (int j = 0; j < HEAD_VALS; j++) r.v[j] += p[32 * j];
    }
    return r;
}

// RMSNorm with the head's weight (pre-biased 1 + w), then the rotation of the first 64 dims by pos * inv_freq
__device__ __forceinline__ void norm_and_rotate(HeadRow& r, const float* w_lane, float angle) {
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) ss += r.v[j] * r.v[j];
    const float rms = rsqrtf(warp_sum(ss) / HD + EPS);
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) r.v[j] = w_lane[j] * (r.v[j] * rms);
    float sn, cs;
    sincosf(angle, &sn, &cs);
    const float a = r.v[0], b = r.v[1];
    r.v[0] = a * cs - b * sn;
    r.v[1] = b * cs + a * sn;
}

// One head row into the int8 cache: a scale per (position, head) = max |v| / 127, code = round(v * 127 / max) + 128.
// KEY: the row's place is [pos][256] in kslot order; else the 16-position block [pos / 16][256][16] in vslot order.
template <bool KEY>
__device__ __forceinline__ void store_quantised(const HeadRow& r, uint8_t* head_cache, float* head_scales, int pos, int lane) {
    float mx = 0.f;
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) mx = fmaxf(mx, fabsf(r.v[j]));
    mx = warp_max(mx);
    const float inv = mx > 0.f ? 127.f / mx : 0.f;
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) {
        const int d = lane + 32 * j;
        const uint8_t code = (uint8_t)(__float2int_rn(r.v[j] * inv) + 128);
        head_cache[KEY ? (size_t)pos * HD + kslot(d) : vslot(pos, d)] = code;
    }
    if (lane == 0) head_scales[pos] = mx / 127.f;
}

__global__ void __launch_bounds__(32 * NH)
attn_prep_kernel(const float* part, int splits, int n, const float* q_norm, const float* k_norm, const float* inv_freq,
                 float qscale, float* q, float* out, uint8_t* kc, uint8_t* vc, float* ks, float* vs,
                 const int* tok_slot, const int* tok_pos, int cap) {
    pdl_launch_dependents();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool cache_block = blockIdx.y == 1;
    if (cache_block && warp >= 2 * NKV) return;
    // the norm weight of the lane's dims and its rotation frequency do not depend on earlier kernels
    const bool normed = !cache_block || warp < NKV;
    float w_lane[HEAD_VALS];
#pragma unroll
    for (int j = 0; j < HEAD_VALS; j++) w_lane[j] = normed ? (cache_block ? k_norm : q_norm)[lane + 32 * j] : 0.f;
    const float freq = inv_freq[lane];
    pdl_wait();
    const int pos = tok_pos[t];
    if (!cache_block) {
        // query head `warp`: rows [q; gate] of the head are adjacent in the in-projection
        HeadRow qr = head_row(part, splits, n, t, warp * 2 * HD, lane);
        const HeadRow gate = head_row(part, splits, n, t, warp * 2 * HD + HD, lane);
        norm_and_rotate(qr, w_lane, (float)pos * freq);
        float* qo = q + ((size_t)t * NH + warp) * HD + lane;
        float* go = out + (size_t)t * MIX + warp * HD + lane;
#pragma unroll
        for (int j = 0; j < HEAD_VALS; j++) {
            qo[32 * j] = qr.v[j] * qscale;
            go[32 * j] = 1.f / (1.f + expf(-gate.v[j]));
        }
        return;
    }
    const int slot = tok_slot[t], g = warp % NKV;
    if (warp < NKV) {
        HeadRow kr = head_row(part, splits, n, t, QG_ROWS + g * HD, lane);
        norm_and_rotate(kr, w_lane, (float)pos * freq);
        store_quantised<true>(kr, kc + cache_head(slot, g, cap), ks + scale_head(slot, g, cap), pos, lane);
    } else {
        const HeadRow vr = head_row(part, splits, n, t, QG_ROWS + NKV * HD + g * HD, lane);
        store_quantised<false>(vr, vc + cache_head(slot, g, cap), vs + scale_head(slot, g, cap), pos, lane);
    }
}

// ------------------------------------------------------------------------------------------------ prompt tiles
__device__ __forceinline__ uint32_t kv_half2(uint32_t w, uint32_t sel) { return __byte_perm(w, 0x64646464u, sel); }

// Prompt tiles: z key splits of a whole number of 64-key blocks (z from tile_splits on the host: one value per step).
__host__ __device__ __forceinline__ int tile_chunk(int keys, int z) { return max(64, ((keys + z - 1) / z + 63) / 64 * 64); }
// About two blocks per SM and no split shorter than 256 keys, or more splits where an estimate says that they take a seventh less: a block has
// an SM to itself, starts and ends in 3 us and takes 2 us per 32 keys, the combine some 0.1 per split. Never fewer: for one sequence a
// single round of blocks can take less (20 rows at context 30000 126 us, 146 so), but of several the shorter ones then leave their SMs early
// (8 of 20 rows up to 30000 930 us, 761 so), and that the host does not know here. Nor more than a round of blocks of less than 384 keys
// (100 rows at 1000, 6 splits of 192 52.5 us, 51 with 4 of 320: partials). Where the first rule says one split the tcgen05 forms do the
// step. Tiles x splits stay below 75: with the 64 decode tokens that may stand before a step's tiles (partials are kept by the step's
// token) that is (64 + 10 tiles) x splits, 2700 partials a head at most. 148 SMs whatever the part: the caller sizes its scratch by this
// count, and names no device.
// By the first rule alone / now, one sequence, with attn_prep and the combine, us: 10 rows at context 600 34.7 / 21.0, at 1000 46.5 / 21.4, at
// 4000 46.1 / 27.1; 20 at 1000 48.4 / 22.4; 40 at 1000 37.2 / 26.3; 64 at 30000 494 / 404; 100 at 4000 153 / 111, at 30000 928 / 574; 200 at 30000
// 1880 / 1289. Of several sequences of unequal lengths: 3 of 20 rows up to 9000 111 / 103, 6 of 10 up to 30000 305 / 275, 2 of
// 100 up to 9000 354 / 279; slower are 3 of 40 up to 9000 188.5 / 189.4, 4 of 30 up to 5000 119.5 / 124.7 (one sequence of 100 rows gains a quarter).
constexpr int TSMS = 148;
__host__ inline int tile_splits(int ntile, int max_keys) {
    int z = 1;
    while (z < TSPLITS && ntile * NKV * z * 2 <= 2 * TSMS && max_keys / (z * 2) >= 256) z *= 2;
    int best = z;
    long long least = 0;
    for (int y = z; z > 1 && y <= TSPLITS && ntile * y < 75; y++) {
        const int chunk = tile_chunk(max_keys, y), ns = (max_keys + chunk - 1) / chunk, rounds = (ntile * NKV * ns + TSMS - 1) / TSMS;
        const long long cost = rounds * (3000 + 2050ll * (chunk / 32)) + 100 * ns;
        if (y == z) least = cost - cost / 7;
        else if (cost < least && (rounds == 1 || chunk >= 384)) { least = cost; best = y; }
    }
    return best;
}

// RT row tiles of 16 (token, head) rows; KW warps per row tile, one 16-key block of a stage each; NS ring stages
template <int RT, int KW, int NS>
struct TileCfg {
    static constexpr int KWARPS = KW, NSTG = NS;
    static constexpr int SK = 16 * KW;                // keys per ring stage
    static constexpr int STG_BYTES = SK * HD * 2 + SK * 4 * 2;  // keys, values, key scales, value scales
    static constexpr int CW = RT * KW;                // warps (warp 0 also issues the copies)
    static constexpr int THREADS = CW * 32;
    static constexpr int Q_BYTES = RT * 16 * SROW * 2;
    static constexpr int BAR_BYTES = 128;
    static constexpr int SMEM = BAR_BYTES + Q_BYTES + NS * STG_BYTES;
    static constexpr int MERGE_FLOATS = 32 * (HD / 8 * 4 + 6);  // one warp's o, m, l, ps
    static_assert(RT * (KW / 2) * MERGE_FLOATS * 4 <= NS * STG_BYTES, "the merge buffers reuse the ring");
};

// 128 dims of two keys, 8 apart, as a lane's words of the key fragments. Keys are 256 bytes apart, all in the same banks, so the lanes of
// odd keys (odd) read the two halves the other way round.
__device__ __forceinline__ void key_words(const uint8_t* kp, bool odd, uint32_t* w0, uint32_t* w1) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const uint8_t* k = kp + i * 8 * HD;
        const uint4 a = *(const uint4*)(k + (odd ? 64 : 0)), b = *(const uint4*)(k + (odd ? 0 : 64));
        const uint4 lo = odd ? b : a, hi = odd ? a : b;
        uint32_t* w = i ? w1 : w0;
        w[0] = lo.x; w[1] = lo.y; w[2] = lo.z; w[3] = lo.w;
        w[4] = hi.x; w[5] = hi.y; w[6] = hi.z; w[7] = hi.w;
    }
}

// Block (prompt tile, kv head, key split) of the prompt attention of a few tiles: ptile is the host's array of tiles (first token, count) of
// consecutive tokens.
template <int RT, int KW, int NS>
__global__ void __launch_bounds__(TileCfg<RT, KW, NS>::THREADS, 1)
attn_tile_kernel(const float* q, const uint8_t* kc, const uint8_t* vc, const float* ks, const float* vs, const int* ptile,
                 const int* tok_slot, const int* tok_pos, int cap, int z, float* part_ml, float* part_acc, float* out, int* err) {
    using C = TileCfg<RT, KW, NS>;
    constexpr int KWARPS = C::KWARPS, NSTG = C::NSTG, SK = C::SK, STG_BYTES = C::STG_BYTES;
    constexpr int NTD = HD / 8;  // n8 dim tiles of the output
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;
    uint64_t* empty = full + NSTG;
    __half* qsh = (__half*)(smem + C::BAR_BYTES);
    uint8_t* ring = smem + C::BAR_BYTES + C::Q_BYTES;

    const int tile = gridDim.x - 1 - blockIdx.x;  // the longest contexts first
    const int g = blockIdx.y, s = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < NSTG; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], C::CW); }
        mbar_fence_init();
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();  // the step's own keys and values are written by attn_prep just before

    const int first = ptile[2 * tile], nt = ptile[2 * tile + 1];
    const int tlast = first + nt - 1, keys = tok_pos[tlast] + 1;
    const int chunk = tile_chunk(keys, z), ns = (keys + chunk - 1) / chunk;
    if (s >= ns) return;
    const int kbeg = s * chunk, ke = min(keys, kbeg + chunk), nstg = (ke - kbeg + SK - 1) / SK;
    const int slot = tok_slot[tlast];

    // ---- the copies: warp 0 issues stage j two stages ahead of its own consumption (three stages in flight, four
    // slots: the slot it refills was released two iterations ago by everyone who keeps pace), one lane per region
    const uint64_t pol = policy_evict_first();
    const uint8_t* kh = kc + cache_head(slot, g, cap);
    const uint8_t* vh = vc + cache_head(slot, g, cap);
    const float* ksh = ks + scale_head(slot, g, cap);
    const float* vsh = vs + scale_head(slot, g, cap);
    bool copy_ok = true;
    auto issue = [&](int j) {
        const int sl = j % NSTG;
        if (j >= NSTG) {
            bool ok = true;
            if (lane == 0) ok = mbar_wait(&empty[sl], ((j / NSTG) - 1) & 1);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) {
                if (lane == 0 && copy_ok) atomicExch(err, 3);
                copy_ok = false;
                return;
            }
        }
        uint8_t* base = ring + sl * STG_BYTES;
        const int kb = kbeg + j * SK;
        if (lane == 0) mbar_expect_tx(&full[sl], STG_BYTES);
        __syncwarp();
        if (lane == 0) bulk_g2s(base, kh + (size_t)kb * HD, SK * HD, &full[sl], pol);
        if (lane == 1) bulk_g2s(base + SK * HD, vh + (size_t)kb * HD, SK * HD, &full[sl], pol);
        if (lane == 2) bulk_g2s(base + 2 * SK * HD, ksh + kb, SK * 4, &full[sl], pol);
        if (lane == 3) bulk_g2s(base + 2 * SK * HD + SK * 4, vsh + kb, SK * 4, &full[sl], pol);
    };
    if (warp == 0) {
        issue(0);
        if (nstg > 1) issue(1);
    }

    // ---------------------------------------------------------------- compute warps
    const int wt = warp / KWARPS, kw = warp % KWARPS, r = lane >> 2, t4 = lane & 3;
    // Q of the segment's rows (row = token * GROUP + head) as f16
    for (int x = threadIdx.x; x < RT * 16 * HD / 4; x += C::CW * 32) {
        int row = x / (HD / 4), d = (x % (HD / 4)) * 4, tok = row / GROUP;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tok < nt) v = *(const float4*)(q + ((size_t)(first + tok) * NH + g * GROUP + row % GROUP) * HD + d);
        *(uint2*)&qsh[row * SROW + d] = make_uint2(pack_half2(v.x, v.y), pack_half2(v.z, v.w));
    }
    named_bar_sync(1, C::CW * 32);
    // this lane's rows wt * 16 + r and + 8: the keys they may see end at lim; KV_OFF times the sums of their Q
    int lim[2];
    float qoff[2];
    {
        float qs = 0.f;
        const __half* qr = qsh + (wt * 16 + (lane & 15)) * SROW + (lane >> 4) * (HD / 2);
        for (int d = 0; d < HD / 2; d += 2) {
            float2 f = __half22float2(*(const __half2*)(qr + d));
            qs += f.x + f.y;
        }
        qs += __shfl_xor_sync(0xffffffffu, qs, 16);
        qoff[0] = KV_OFF * __shfl_sync(0xffffffffu, qs, r);
        qoff[1] = KV_OFF * __shfl_sync(0xffffffffu, qs, r + 8);
    }
#pragma unroll
    for (int h2 = 0; h2 < 2; h2++) {
        int tok = (wt * 16 + r + 8 * h2) / GROUP;
        lim[h2] = tok < nt ? min(ke, tok_pos[first + tok] + 1) : 0;
    }
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, ps[2] = {0.f, 0.f}, o[NTD][4];
#pragma unroll
    for (int j = 0; j < NTD; j++) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
    const uint32_t qa = smem_u32(qsh + (wt * 16 + (lane & 15)) * SROW + (lane >> 4) * 8);

    int sl = 0;
    uint32_t par = 0;
    bool dead = false;
    for (int i = 0; i < nstg; i++) {
        if (warp == 0 && i + 2 < nstg && copy_ok) issue(i + 2);
        if (!dead) {
            dead = !mbar_wait(&full[sl], par);
            if (dead && lane == 0) atomicExch(err, 4);
        } else {
            for (int k = 0; k < 1024 && !mbar_try_wait(&full[sl], par); k++) {}
        }
        const uint8_t* base = ring + sl * STG_BYTES;
        const int kb = kbeg + i * SK + 16 * kw;  // this warp's 16 keys of the stage
        if (kb < ke) {
            const uint8_t* kp = base + (16 * kw + r) * HD + 16 * t4;
            const uint8_t* vp = base + SK * HD + kw * 16 * HD + r * 16 + t4 * 4;
            const float* ksc_s = (const float*)(base + 2 * SK * HD) + 16 * kw;
            const float* vsc_s = ksc_s + SK;
            float ksc[2][2], vsc[2][2];
#pragma unroll
            for (int nn = 0; nn < 2; nn++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    int kk = 8 * nn + 2 * t4 + e;
                    bool in = kb + kk < ke;
                    ksc[nn][e] = in ? ksc_s[kk] : 0.f;
                    vsc[nn][e] = in ? vsc_s[kk] : 0.f;
                }
            // S = Q K^T
            float sacc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int b2 = 0; b2 < HD / 128; b2++) {
                uint32_t w0[8], w1[8];
                key_words(kp + 128 * b2, r & 1, w0, w1);
#pragma unroll
                for (int st = 0; st < 8; st++) {
                    uint32_t a[4];
                    ldsm_x4(a[0], a[1], a[2], a[3], qa + (b2 * 128 + st * 16) * 2);
                    mma16816(sacc[0], a, kv_half2(w0[st], 0x4140), kv_half2(w0[st], 0x4342));
                    mma16816(sacc[1], a, kv_half2(w1[st], 0x4140), kv_half2(w1[st], 0x4342));
                }
            }
            // scale, mask, online softmax per row; P times the value scales as the A fragments of P V
            float pv[2][4];
            bool grew = false;
            float corr[2];
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                float v[2][2], mx = -INFINITY;
#pragma unroll
                for (int nn = 0; nn < 2; nn++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        int k = kb + 8 * nn + 2 * t4 + e;
                        v[nn][e] = k < lim[h2] ? (sacc[nn][2 * h2 + e] - qoff[h2]) * ksc[nn][e] : -INFINITY;
                        mx = fmaxf(mx, v[nn][e]);
                    }
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
                float mn = fmaxf(m[h2], mx);
                corr[h2] = mn == -INFINITY ? 1.f : exp2f(m[h2] - mn);
                m[h2] = mn;
                float sum = 0.f;
#pragma unroll
                for (int nn = 0; nn < 2; nn++)
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        float p = v[nn][e] == -INFINITY ? 0.f : exp2f(v[nn][e] - mn);
                        sum += p;
                        pv[nn][2 * h2 + e] = p * vsc[nn][e];
                    }
                l[h2] = l[h2] * corr[h2] + sum;
                ps[h2] *= corr[h2];
                grew |= corr[h2] != 1.f;
            }
            if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
                for (int j = 0; j < NTD; j++) {
                    o[j][0] *= corr[0]; o[j][1] *= corr[0];
                    o[j][2] *= corr[1]; o[j][3] *= corr[1];
                }
            }
            uint32_t pa[4] = {pack_half2(pv[0][0], pv[0][1]), pack_half2(pv[0][2], pv[0][3]),
                              pack_half2(pv[1][0], pv[1][1]), pack_half2(pv[1][2], pv[1][3])};
            // the P the products see (f16): rows r (words 0, 2) and r + 8 (1, 3)
            float2 f0 = __half22float2(*(__half2*)&pa[0]), f2 = __half22float2(*(__half2*)&pa[2]);
            float2 f1 = __half22float2(*(__half2*)&pa[1]), f3 = __half22float2(*(__half2*)&pa[3]);
            ps[0] += f0.x + f0.y + f2.x + f2.y;
            ps[1] += f1.x + f1.y + f3.x + f3.y;
            // O += P V
#pragma unroll
            for (int j = 0; j < NTD; j++) {
                uint32_t vw = *(const uint32_t*)(vp + j * 8 * 16);
                mma16816(o[j], pa, kv_half2(vw, 0x4140), kv_half2(vw, 0x4342));
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[sl]);
        if (++sl == NSTG) { sl = 0; par ^= 1; }
    }

    // ---- the warps of a row tile merge pairwise in two rounds (1 -> 0 and 3 -> 2, then 2 -> 0) through the ring, which
    // is free: every stage was consumed
    named_bar_sync(1, C::CW * 32);
    for (int round = 1; round < KWARPS; round <<= 1) {
        const bool sender = (kw & (2 * round - 1)) == round, receiver = (kw & (2 * round - 1)) == 0;
        float* mb = (float*)ring + (size_t)(wt * (KWARPS / 2) + (kw >> 1) / round % (KWARPS / 2)) * C::MERGE_FLOATS;
        if (sender) {
#pragma unroll
            for (int j = 0; j < NTD; j++)
                *(float4*)(mb + (j * 32 + lane) * 4) = make_float4(o[j][0], o[j][1], o[j][2], o[j][3]);
            float* t = mb + NTD * 32 * 4 + lane * 6;
            t[0] = m[0]; t[1] = m[1]; t[2] = l[0]; t[3] = l[1]; t[4] = ps[0]; t[5] = ps[1];
        }
        named_bar_sync(1, C::CW * 32);
        if (receiver) {
            const float* t = mb + NTD * 32 * 4 + lane * 6;
            float c0[2], c1[2];
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                float m1 = t[h2], mn = fmaxf(m[h2], m1);
                c0[h2] = mn == -INFINITY ? 1.f : exp2f(m[h2] - mn);
                c1[h2] = mn == -INFINITY ? 1.f : exp2f(m1 - mn);
                m[h2] = mn;
                l[h2] = l[h2] * c0[h2] + t[2 + h2] * c1[h2];
                ps[h2] = ps[h2] * c0[h2] + t[4 + h2] * c1[h2];
            }
#pragma unroll
            for (int j = 0; j < NTD; j++) {
                float4 v = *(const float4*)(mb + (j * 32 + lane) * 4);
                o[j][0] = o[j][0] * c0[0] + v.x * c1[0]; o[j][1] = o[j][1] * c0[0] + v.y * c1[0];
                o[j][2] = o[j][2] * c0[1] + v.z * c1[1]; o[j][3] = o[j][3] * c0[1] + v.w * c1[1];
            }
        }
        named_bar_sync(1, C::CW * 32);
    }
    if (kw != 0) return;
#pragma unroll
    for (int h2 = 0; h2 < 2; h2++) {
        float L = l[h2], P = ps[h2];
        L += __shfl_xor_sync(0xffffffffu, L, 1);
        L += __shfl_xor_sync(0xffffffffu, L, 2);
        P += __shfl_xor_sync(0xffffffffu, P, 1);
        P += __shfl_xor_sync(0xffffffffu, P, 2);
        int row = wt * 16 + r + 8 * h2, tok = row / GROUP;
        if (tok >= nt) continue;
        int t = first + tok, head = g * GROUP + row % GROUP;
        if (ns == 1) {
            float f = 1.f / L;
            float* op = out + (size_t)t * MIX + head * HD + 2 * t4;
#pragma unroll
            for (int j = 0; j < NTD; j++) {
                float2 gt = *(float2*)(op + j * 8);
                *(float2*)(op + j * 8) = make_float2(gt.x * (o[j][2 * h2] - KV_OFF * P) * f, gt.y * (o[j][2 * h2 + 1] - KV_OFF * P) * f);
            }
        } else {
            size_t pi = ((size_t)t * NH + head) * z + s;
            float* pp = part_acc + pi * HD + 2 * t4;
#pragma unroll
            for (int j = 0; j < NTD; j++)
                *(float2*)(pp + j * 8) = make_float2(o[j][2 * h2] - KV_OFF * P, o[j][2 * h2 + 1] - KV_OFF * P);
            if (t4 == 0) { part_ml[pi * 2] = m[h2]; part_ml[pi * 2 + 1] = L; }
        }
    }
}

// ------------------------------------------------------------------------------------------------ decode attention
// Block (short segment, kv head, key split) of the decode / verify attention: 2 or 4 QUADS of four warps. The keys and values of the
// split arrive in 64-key stages through a ring fed by bulk copies; the quads take the stages in turn. Inside a quad the work
// of a stage is dealt so that no byte is converted twice:
//   scores   warp w multiplies all the rows (RT tiles of 16 (token, head) rows) by the keys 16 w .. 16 w + 15 of the
//            stage over the whole head dimension: one conversion of a key serves every row tile;
//   softmax  the four warps agree on the rows' running maxima through shared memory, so that all of them scale by the same
//            power of two, and exchange their 16-key slices of P (as f16 mma fragments); a lane keeps the sums of its own keys
//            to the end. (P relative to a reference that moves only near f16's end: one barrier per stage instead of two, but P
//            is made twice where it moves and rounded to other values: no faster, 5 rows at 32000 29.4 us, 28.9 so; 8 sequences of 4 rows up to
//            32000 are the exception, 112 and 117);
//   values   warp w accumulates the output dims 64 w .. 64 w + 63 over all 64 keys of the stage (for every row tile),
//            so the output accumulators of a row are spread over four warps (RT x 32 registers each).
// The int8 codes go to the tensor cores as 1152 + q halves (one prmt per pair) and the offset is folded out through the
// row sums, as in the reference (kernels/attn.cuh:38-40,198-234). The quads' partial results meet in shared memory
// at the end; the block writes one (m, l, acc) partial per row, or the finished rows when the segment has one split.
// Bound by latency, with two warps per scheduler (four at one row tile). From a graph with attn_prep and the combine, us, before (a copy
// warp, Q row by row, keys with bank conflicts) / now: 5 rows at 100 keys 13.7 / 11.0, at 4000 18.3 / 14.9, at 32000 34.8 / 28.9; 1 row at
// 32000 26.3 / 24.3; 8 rows 50.4 / 38.3 (registers spilled before); 8 sequences of 4 rows at 972 to 7777 66.7 / 47.8 (57.7 with a block per
// split), at 4000 to 32000 139.9 / 117 (126.6).
// Many splits (MANY): a block per split would pay for each one's start (its segment's tokens, Q, the first stages' way from memory: half of
// the 11 us that a split of four stages took) and leave the last round of the SMs partly idle. So a block per SM takes a run of them, equal
// shares of the line on which each split is as long as its stages and SPLIT_COST: Q stays where the run stays with a segment's kv head,
// and the next split's first stages are under way while the quads merge. The sums of a split are the same in both forms.
constexpr int DEC_SEGS = 64;         // segments of a step whose splits are dealt out: the table's size
constexpr unsigned SPLIT_COST = 3;   // what a split costs beside its stages, in stages (measured: 1830 cycles a stage, 5000 a split)

template <int RT, int NQ>
struct Dec4Cfg {
    static constexpr int QUADS = NQ, CW = 4 * QUADS, THREADS = CW * 32;
    static constexpr int SK = 64, NSTG = NQ > 2 ? 6 : 5;  // keys per stage, ring depth
    static constexpr int STG_BYTES = SK * HD * 2 + SK * 8;
    static constexpr int Q_BYTES = RT * 16 * SROW * 2;
    // per quad: the warps' row maxima [4][RT][16], their P fragments [4][RT][32 lanes] x 16 B, their (sum, ps) [4][RT][16][2]
    static constexpr int X_MAX = 4 * RT * 16 * 4, X_P = 4 * RT * 32 * 16, X_SUM = 4 * RT * 16 * 8;
    static constexpr int X_BYTES = X_MAX + X_P + X_SUM;
    static constexpr int BAR_BYTES = 128;
    static constexpr int SMEM = BAR_BYTES + Q_BYTES + QUADS * X_BYTES + NSTG * STG_BYTES;
    static constexpr int SMEM_MANY = SMEM + DEC_SEGS * (16 + 8 + 4);  // and the step's segments
    static constexpr int MERGE_BYTES = 8 * 32 * (RT * 8 * 4 + RT * 6) * 4;   // two quads' registers at a time
    static_assert(MERGE_BYTES <= NSTG * STG_BYTES, "the merge buffers reuse the ring");
    static constexpr int MERGE_SLOTS = (MERGE_BYTES + STG_BYTES - 1) / STG_BYTES;
    static_assert(SMEM_MANY <= 227 * 1024, "shared memory");
};

template <int RT, int NQ, bool MANY>
__global__ void __launch_bounds__(Dec4Cfg<RT, NQ>::THREADS, 1)
attn_dec4_kernel(const float* q, const uint8_t* kc, const uint8_t* vc, const float* ks, const float* vs, const int* dseg,
                 const int* dtok, const int* tok_slot, const int* tok_pos, int cap, int z, int dsplits, int old_margin, int ndseg,
                 float* part_ml, float* part_acc, float* out, int* err) {
    using C = Dec4Cfg<RT, NQ>;
    constexpr int NSTG = C::NSTG, SK = C::SK, STG_BYTES = C::STG_BYTES;
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t* full = (uint64_t*)smem;
    volatile int* issued = (volatile int*)(full + NSTG);  // per slot: the stage whose copies were asked for last
    __half* qsh = (__half*)(smem + C::BAR_BYTES);
    uint8_t* xch = smem + C::BAR_BYTES + C::Q_BYTES;
    uint8_t* ring = xch + C::QUADS * C::X_BYTES;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int seg = blockIdx.x, g = blockIdx.y, s = blockIdx.z;
    if (threadIdx.x == 32) {
        for (int i = 0; i < NSTG; i++) { mbar_init(&full[i], 1); issued[i] = 0; }
        mbar_fence_init();
    }
    // The step's token lists are uploaded before its first kernel, so they are read ahead of the kernel before (this
    // step's attn_prep), and so, where the caller vouches for them, are the stages of keys and values that earlier steps wrote: whatever
    // ends `old_margin` positions or more before the segment's last key (0: nothing is read ahead, the first stages are only
    // asked into L2).
    int4* segs = (int4*)(ring + NSTG * STG_BYTES);  // MANY: per segment its first token's place, tokens, keys and slot,
    int2* how = (int2*)(segs + DEC_SEGS);           // keys per split and splits,
    unsigned* cum = (unsigned*)(how + DEC_SEGS);    // and where its splits end on the line that the blocks share
    unsigned at = 0, until = 0;                     // where this split begins there, and where the block's share ends
    if constexpr (MANY) {
        if (warp == 0) {
            unsigned sum = 0;
            for (int i0 = 0; i0 < ndseg; i0 += 32) {
                const int i = i0 + lane;
                unsigned c = 0;
                if (i < ndseg) {
                    const int first = dseg[2 * i], nt = dseg[2 * i + 1], tlast = dtok[first + nt - 1], keys = tok_pos[tlast] + 1;
                    segs[i] = make_int4(first, nt, keys, tok_slot[tlast]);
                    const int chunk = dec_chunk(keys, dsplits), ns = min((keys + chunk - 1) / chunk, z);  // (more: more keys than the caller said)
                    how[i] = make_int2(chunk, ns);
                    c = NKV * ((min(keys, ns * chunk) + SK - 1) / SK + SPLIT_COST * ns);
                }
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned x = __shfl_up_sync(0xffffffffu, c, d);
                    if (lane >= d) c += x;
                }
                if (i < ndseg) cum[i] = sum + c;
                sum += __shfl_sync(0xffffffffu, c, 31);
            }
        }
        __syncthreads();
        // the first split that begins in the block's share
        const unsigned total = cum[ndseg - 1], part = total / gridDim.x, over = total % gridDim.x;
        const unsigned from = blockIdx.x * part + blockIdx.x * over / gridDim.x;
        until = (blockIdx.x + 1) * part + (blockIdx.x + 1) * over / gridDim.x;
        if (from >= total) {  // (fewer units than blocks)
            pdl_launch_dependents();
            return;
        }
        seg = 0;
#pragma unroll
        for (int i0 = 0; i0 < DEC_SEGS; i0 += 32)
            seg += __popc(__ballot_sync(0xffffffffu, i0 + lane < ndseg && cum[min(i0 + lane, ndseg - 1)] <= from));
        const unsigned begin_at = seg ? cum[seg - 1] : 0, head = (cum[seg] - begin_at) / NKV, rest = from - begin_at, each = how[seg].x / SK + SPLIT_COST;
        g = rest / head;
        s = (rest - g * head + each - 1) / each;
        if (s >= how[seg].y) { s = 0; g++; }
        at = begin_at + g * head + s * each;
        if (g == NKV) { g = 0; seg++; }
        pdl_launch_dependents();
        if (at >= until) return;  // (also where seg is ndseg)
    } else {
        __syncthreads();
        pdl_launch_dependents();
    }
    int first, nt, my_tok, my_pos, keys, chunk, ns, kbeg, ke, nstg, slot;
    auto splits = [&]() {  // how the segment is split
        chunk = MANY ? how[seg].x : dec_chunk(keys, dsplits);
        ns = MANY ? how[seg].y : (keys + chunk - 1) / chunk;
    };
    auto split = [&]() {  // what this split is
        kbeg = s * chunk;
        ke = min(keys, kbeg + chunk);
        nstg = (ke - kbeg + SK - 1) / SK;
    };
    if constexpr (MANY) {
        const int4 x = segs[seg];
        first = x.x; nt = x.y; keys = x.z; slot = x.w;
        my_tok = dtok[first + min(lane, nt - 1)];
        my_pos = tok_pos[my_tok];
    } else {
        first = dseg[2 * seg]; nt = dseg[2 * seg + 1];
        my_tok = dtok[first + min(lane, nt - 1)]; my_pos = tok_pos[my_tok];  // lane i: the segment's token i
        const int tlast = __shfl_sync(0xffffffffu, my_tok, nt - 1);
        keys = __shfl_sync(0xffffffffu, my_pos, nt - 1) + 1;
        slot = tok_slot[tlast];
    }
    splits();
    if (!MANY && s >= ns) return;
    split();

    // ---- the copies of a stage, its keys, values and scales, are shared out among the warps, at the start among all and later among a
    // quad's (by one warp they take 690 cycles, which the others would wait for), behind a barrier of the warps before which the stage's
    // own is armed. (A copy warp would be a third warp of one scheduler, and leave the others 168 registers instead of 255.)
    const int quad = warp >> 2, w = warp & 3, r = lane >> 2, t4 = lane & 3;
    constexpr int NCW = C::THREADS;
    // (with many splits the slots at the front are those that the quads merge through, and a split's first stages go behind them)
    constexpr int OFF = MANY ? C::MERGE_SLOTS : 0;
    using Ring = DecRing<C::QUADS, NSTG, OFF>;
    Ring order;
    const uint64_t pol = policy_evict_first();
    auto copy = [&](int j, int part) {
        const uint8_t* from = part == 0 ? kc + cache_head(slot, g, cap) + (size_t)kbeg * HD : part == 1 ? vc + cache_head(slot, g, cap) + (size_t)kbeg * HD
                              : (const uint8_t*)((part == 2 ? ks : vs) + scale_head(slot, g, cap) + kbeg);
        const uint32_t bytes = part < 2 ? SK * HD : SK * 4, to = part < 2 ? part * SK * HD : 2 * SK * HD + (part - 2) * SK * 4;
        bulk_g2s(ring + Ring::slot(j) * STG_BYTES + to, from + (size_t)j * bytes, bytes, &full[Ring::slot(j)], pol);
    };
    auto arm = [&](int j) {
        mbar_expect_tx(&full[Ring::slot(j)], STG_BYTES);
        issued[Ring::slot(j)] = order.number(j);
    };
    int begin = min(nstg, NSTG);
    if (warp < begin && lane == 0) arm(warp);
    named_bar_sync(1, NCW);
    auto ask = [&](bool ahead) {  // the first stages
        for (int x = warp; x < 4 * begin; x += C::CW) {
            const bool old = old_margin > 0 && kbeg + ((x >> 2) + 1) * SK <= keys - old_margin;
            if (old == ahead && lane == 0) copy(x >> 2, x & 3);
        }
        __syncwarp();
    };
    if (old_margin > 0)
        ask(true);
    else if (warp < begin && lane < 2)
        bulk_prefetch((lane ? vc : kc) + cache_head(slot, g, cap) + (size_t)(kbeg + warp * SK) * HD, SK * HD);
    pdl_wait();  // q, the gates and the step's own keys and values come from its attn_prep
    // Q of the segment's rows (row = token * GROUP + head) as f16, and each row's sum of those. All of a thread's loads are under way
    // together: one after the other, behind the token's own load, they took 4 us.
    float* xmax = (float*)(xch + quad * C::X_BYTES);                 // [4][RT][16]
    uint4* xp = (uint4*)(xch + quad * C::X_BYTES + C::X_MAX);        // [4][RT][32]
    float2* xsum = (float2*)(xch + quad * C::X_BYTES + C::X_MAX + C::X_P);  // [4][RT][16]
    float* qsum = (float*)(xch + C::X_BYTES + C::X_MAX + C::X_P);  // [RT * 16], in the second quad's place for sums, which it never uses
    auto load_q = [&](bool begins) {
        constexpr int PER = RT * 16 * HD / 4 / NCW, RSTEP = NCW / (HD / 4);  // float4 per thread, rows at a time
        const int r0 = threadIdx.x / (HD / 4), d = (threadIdx.x % (HD / 4)) * 4;
        float4 v[PER];
#pragma unroll
        for (int i = 0; i < PER; i++) {
            const int row = r0 + i * RSTEP, tok = row / GROUP;
            const int t = __shfl_sync(0xffffffffu, my_tok, min(tok, nt - 1));
            v[i] = tok < nt ? *(const float4*)(q + ((size_t)t * NH + g * GROUP + row % GROUP) * HD + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (begins) ask(false);
#pragma unroll
        for (int i = 0; i < PER; i++)
            *(uint2*)&qsh[(r0 + i * RSTEP) * SROW + d] = make_uint2(pack_half2(v[i].x, v[i].y), pack_half2(v[i].z, v[i].w));
        named_bar_sync(1, NCW);
        if (warp < RT) {  // a lane sums half a row
            const uint4* from = (const uint4*)(qsh + (warp * 16 + (lane & 15)) * SROW + (lane >> 4) * (HD / 2));
            float sum = 0.f;
#pragma unroll 4
            for (int i = 0; i < HD / 16; i++) {
                const uint4 x = from[i];
                const uint32_t h[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const float2 f = __half22float2(*(const __half2*)&h[e]);
                    sum += f.x + f.y;
                }
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 16);
            if (lane < 16) qsum[warp * 16 + lane] = sum;
        }
    };
    // KV_OFF times the sums of Q of this lane's rows 16 rt + r and + 8
    float qoff[RT][2];
    uint32_t qa[RT];
#pragma unroll
    for (int rt = 0; rt < RT; rt++) qa[rt] = smem_u32(qsh + (rt * 16 + (lane & 15)) * SROW + (lane >> 4) * 8);
    bool fresh = true, dead = false;  // fresh: these rows' Q is not in place yet
    for (;;) {  // MANY: the block's splits; else the one
        if (fresh) {
            load_q(order.j0 == 0);
            named_bar_sync(1, NCW);
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int h2 = 0; h2 < 2; h2++) qoff[rt][h2] = KV_OFF * qsum[rt * 16 + r + 8 * h2];
        }
        // the keys that the rows may see end at lim
        int lim[RT][2], all_see = ke;  // (keys below all_see are seen by every row of the segment)
#pragma unroll
        for (int rt = 0; rt < RT; rt++)
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                const int tok = (rt * 16 + r + 8 * h2) / GROUP;
                const int p = __shfl_sync(0xffffffffu, my_pos, min(tok, nt - 1));
                lim[rt][h2] = tok < nt ? min(ke, p + 1) : 0;
            }
        all_see = min(all_see, __reduce_min_sync(0xffffffffu, my_pos) + 1);
        // m: the rows' largest score so far; -inf until a key was seen
        float m[RT][2], l[RT][2], ps[RT][2], o[RT][8][4];
#pragma unroll
        for (int rt = 0; rt < RT; rt++) {
            m[rt][0] = m[rt][1] = -INFINITY;
            l[rt][0] = l[rt][1] = ps[rt][0] = ps[rt][1] = 0.f;
#pragma unroll
            for (int j = 0; j < 8; j++) o[rt][j][0] = o[rt][j][1] = o[rt][j][2] = o[rt][j][3] = 0.f;
        }

        for (int j = quad; j < nstg; j += C::QUADS) {
            const int sl = Ring::slot(j);
            const uint32_t par = order.parity(j);
            if (!dead) {
                uint32_t polls = 0;
                if (Ring::looks(j))
                    while (issued[sl] != order.number(j) && polls < WAIT_LIMIT) polls++;
                dead = polls == WAIT_LIMIT || !mbar_wait(&full[sl], par);
                if (dead && lane == 0) atomicExch(err, 4);
            } else {
                for (int k = 0; k < 1024 && !mbar_try_wait(&full[sl], par); k++) {}
            }
            const int refill = Ring::in_the_middle(j, nstg);  // the slot of the quad's stage before this one is filled again
            if (refill >= 0 && w == 0 && lane == 0) arm(refill);
            const uint8_t* base = ring + sl * STG_BYTES;
            const int kb = kbeg + j * SK + 16 * w;  // this warp's 16 keys of the stage
            const uint8_t* kp = base + (16 * w + r) * HD + 16 * t4;
            const float* ksc_s = (const float*)(base + 2 * SK * HD) + 16 * w;
            const float* vsc_s = ksc_s + SK;
            const bool whole = kbeg + (j + 1) * SK <= all_see;  // every row sees every key of the stage
            float ksc[2][2], vsc[2][2];
#pragma unroll
            for (int nn = 0; nn < 2; nn++)
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int kk = 8 * nn + 2 * t4 + e;
                    const bool in = kb + kk < ke;
                    ksc[nn][e] = in ? ksc_s[kk] : 0.f;
                    vsc[nn][e] = in ? vsc_s[kk] : 0.f;
                }
            // ---- scores: S = Q K^T for every row tile, this warp's 16 keys
            float v[RT][2][4];
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int nn = 0; nn < 2; nn++) v[rt][nn][0] = v[rt][nn][1] = v[rt][nn][2] = v[rt][nn][3] = 0.f;
#pragma unroll
            for (int b2 = 0; b2 < HD / 128; b2++) {
                // (the halves turned round: 5 rows at context 32000 30.35 -> 29.67 us; not with one row tile, whose warps had no registers left
                // for it: 8 sequences of one row 42.3 -> 44.8)
                uint32_t w0[8], w1[8];
                key_words(kp + 128 * b2, RT > 1 && (r & 1), w0, w1);
#pragma unroll
                for (int st = 0; st < 8; st++) {
                    const uint32_t b00 = kv_half2(w0[st], 0x4140), b01 = kv_half2(w0[st], 0x4342);
                    const uint32_t b10 = kv_half2(w1[st], 0x4140), b11 = kv_half2(w1[st], 0x4342);
#pragma unroll
                    for (int rt = 0; rt < RT; rt++) {
                        uint32_t a[4];
                        ldsm_x4(a[0], a[1], a[2], a[3], qa[rt] + (b2 * 128 + st * 16) * 2);
                        mma16816(v[rt][0], a, b00, b01);
                        mma16816(v[rt][1], a, b10, b11);
                    }
                }
            }
            // ---- the scores proper
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int nn = 0; nn < 2; nn++)
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        float& sv = v[rt][nn][x];
                        sv = (sv - qoff[rt][x >> 1]) * ksc[nn][x & 1];
                        if (!whole && kb + 8 * nn + 2 * t4 + (x & 1) >= lim[rt][x >> 1]) sv = -INFINITY;
                    }
            // ---- the rows' maxima over this warp's keys, then over the quad's
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int h2 = 0; h2 < 2; h2++) {
                    float x = fmaxf(fmaxf(v[rt][0][2 * h2], v[rt][0][2 * h2 + 1]), fmaxf(v[rt][1][2 * h2], v[rt][1][2 * h2 + 1]));
                    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 1));
                    x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, 2));
                    if (t4 == 0) xmax[(w * RT + rt) * 16 + r + 8 * h2] = x;
                }
            named_bar_sync(2 + quad, 128);
            // (all of the quad is done with its stage before this one, and the slot's barrier is armed)
            if (refill >= 0 && lane == 0) copy(refill, w);
            float corr[RT][2];
            bool grew = false;
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int h2 = 0; h2 < 2; h2++) {
                    float mn = m[rt][h2];
#pragma unroll
                    for (int ww = 0; ww < 4; ww++) mn = fmaxf(mn, xmax[(ww * RT + rt) * 16 + r + 8 * h2]);
                    corr[rt][h2] = mn == -INFINITY ? 1.f : exp2f(m[rt][h2] - mn);
                    m[rt][h2] = mn;
                    grew |= corr[rt][h2] != 1.f;
                }
            // ---- P of this warp's keys (times the value scales, rounded to f16 as the products see it) and its row sums
#pragma unroll
            for (int rt = 0; rt < RT; rt++) {
                float pv[2][4], sum[2];
#pragma unroll
                for (int h2 = 0; h2 < 2; h2++) {
                    const float mm = m[rt][h2] == -INFINITY ? 0.f : m[rt][h2];
                    sum[h2] = 0.f;
#pragma unroll
                    for (int nn = 0; nn < 2; nn++)
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            const float pp = tc::ex2(v[rt][nn][2 * h2 + e] - mm);
                            sum[h2] += pp;
                            pv[nn][2 * h2 + e] = pp * vsc[nn][e];
                        }
                }
                uint4 pa;
                pa.x = pack_half2(pv[0][0], pv[0][1]); pa.y = pack_half2(pv[0][2], pv[0][3]);
                pa.z = pack_half2(pv[1][0], pv[1][1]); pa.w = pack_half2(pv[1][2], pv[1][3]);
                xp[(w * RT + rt) * 32 + lane] = pa;
                const float2 f0 = __half22float2(*(const __half2*)&pa.x), f1 = __half22float2(*(const __half2*)&pa.y);
                const float2 f2 = __half22float2(*(const __half2*)&pa.z), f3 = __half22float2(*(const __half2*)&pa.w);
                const float pr[2] = {f0.x + f0.y + f2.x + f2.y, f1.x + f1.y + f3.x + f3.y};
                // (a lane sums its own keys; lanes and warps are added up once, after the last stage)
#pragma unroll
                for (int h2 = 0; h2 < 2; h2++) {
                    l[rt][h2] = fmaf(l[rt][h2], corr[rt][h2], sum[h2]);
                    ps[rt][h2] = fmaf(ps[rt][h2], corr[rt][h2], pr[h2]);
                }
            }
            named_bar_sync(2 + quad, 128);
            if (__any_sync(0xffffffffu, grew)) {
#pragma unroll
                for (int rt = 0; rt < RT; rt++)
#pragma unroll
                    for (int jd = 0; jd < 8; jd++) {
                        o[rt][jd][0] *= corr[rt][0]; o[rt][jd][1] *= corr[rt][0];
                        o[rt][jd][2] *= corr[rt][1]; o[rt][jd][3] *= corr[rt][1];
                    }
            }
            // ---- values: O += P V over the stage's 64 keys, this warp's 64 output dims
#pragma unroll
            for (int kbk = 0; kbk < 4; kbk++) {
                uint32_t pa[RT][4];
#pragma unroll
                for (int rt = 0; rt < RT; rt++) {
                    const uint4 x = xp[(kbk * RT + rt) * 32 + lane];
                    pa[rt][0] = x.x; pa[rt][1] = x.y; pa[rt][2] = x.z; pa[rt][3] = x.w;
                }
                const uint8_t* vp = base + SK * HD + kbk * 16 * HD + (64 * w + r) * 16 + t4 * 4;
#pragma unroll
                for (int jd = 0; jd < 8; jd++) {
                    const uint32_t vw = *(const uint32_t*)(vp + jd * 8 * 16);
                    const uint32_t b0 = kv_half2(vw, 0x4140), b1 = kv_half2(vw, 0x4342);
#pragma unroll
                    for (int rt = 0; rt < RT; rt++) mma16816(o[rt][jd], pa[rt], b0, b1);
                }
            }
            const int behind = Ring::at_the_end(j, nstg);  // (few stages more than quads: the next stage's barrier would be late)
            if (behind >= 0) {
                if (w == 0 && lane == 0) arm(behind);
                named_bar_sync(2 + quad, 128);
                if (lane == 0) copy(behind, w);
            }
        }

        // ---- the quads merge pairwise through the ring, which is free (every stage was consumed): 1 -> 0 and 3 -> 2, then
        // 2 -> 0. A warp's registers go to the warp of the same index in the other quad (same rows, same dims).
        named_bar_sync(1, NCW);
        // With many splits a quad that has handed its registers over asks for the next one's first stages meanwhile, those that go behind the
        // slots of the merge; the others when the merge is done, and then it goes on. (Where the results of this one go: `was`.)
        const int4 was = make_int4(first, nt, g, s);
        const int was_ns = ns;
        bool more = false;
        auto go_on = [&]() {
            at += nstg + SPLIT_COST;
            more = at < until;
            if (!more) return;
            order.next_split(nstg);
            fresh = false;
            if (++s == ns) {
                s = 0;
                fresh = true;
                if (++g == NKV) {
                    g = 0;
                    const int4 x = segs[++seg];
                    first = x.x; nt = x.y; keys = x.z; slot = x.w;
                    my_tok = dtok[first + min(lane, nt - 1)];
                    my_pos = tok_pos[my_tok];
                    splits();
                }
            }
            split();
            begin = min(nstg, NSTG);
        };
        auto begin_with = [&](int a, int b) {  // stages a up to b: a warp of the second quad each
            const int j = a + w;
            if (j < min(b, begin) && lane == 0) {
                arm(j);
                for (int part = 0; part < 4; part++) copy(j, part);
            }
            __syncwarp();
        };
        static_assert(!MANY || (NSTG - OFF <= 4 && OFF <= 4), "a warp of a quad per stage");
        constexpr int MF = RT * 8 * 4 + RT * 6;  // floats per lane
        for (int round = 1; round < C::QUADS; round <<= 1) {
            const bool sender = (quad & (2 * round - 1)) == round;
            const bool receiver = (quad & (2 * round - 1)) == 0 && quad + round < C::QUADS;
            float* mb = (float*)ring + (size_t)(((quad >> 1) / round % 2) * 4 + w) * 32 * MF + lane;
            if (sender) {
#pragma unroll
                for (int rt = 0; rt < RT; rt++) {
#pragma unroll
                    for (int jd = 0; jd < 8; jd++)
#pragma unroll
                        for (int e = 0; e < 4; e++) mb[((rt * 8 + jd) * 4 + e) * 32] = o[rt][jd][e];
#pragma unroll
                    for (int h2 = 0; h2 < 2; h2++) {
                        mb[(RT * 32 + rt * 6 + h2) * 32] = m[rt][h2];
                        mb[(RT * 32 + rt * 6 + 2 + h2) * 32] = l[rt][h2];
                        mb[(RT * 32 + rt * 6 + 4 + h2) * 32] = ps[rt][h2];
                    }
                }
            }
            if (MANY && sender) tc::async_proxy_fence();  // (copies are written there next)
            named_bar_sync(1, NCW);
            if (MANY && round == 1 && quad == 1) {
                go_on();
                if (more) begin_with(0, NSTG - OFF);
            }
            if (receiver) {
#pragma unroll
                for (int rt = 0; rt < RT; rt++) {
                    float c0[2], c1[2];
#pragma unroll
                    for (int h2 = 0; h2 < 2; h2++) {
                        const float m1 = mb[(RT * 32 + rt * 6 + h2) * 32], mn = fmaxf(m[rt][h2], m1);
                        c0[h2] = mn == -INFINITY ? 1.f : exp2f(m[rt][h2] - mn);
                        c1[h2] = mn == -INFINITY ? 1.f : exp2f(m1 - mn);
                        m[rt][h2] = mn;
                        l[rt][h2] = l[rt][h2] * c0[h2] + mb[(RT * 32 + rt * 6 + 2 + h2) * 32] * c1[h2];
                        ps[rt][h2] = ps[rt][h2] * c0[h2] + mb[(RT * 32 + rt * 6 + 4 + h2) * 32] * c1[h2];
                    }
#pragma unroll
                    for (int jd = 0; jd < 8; jd++)
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            o[rt][jd][e] = o[rt][jd][e] * c0[e >> 1] + mb[((rt * 8 + jd) * 4 + e) * 32] * c1[e >> 1];
                }
            }
            named_bar_sync(1, NCW);
        }
        if (MANY && quad == 1 && more) begin_with(NSTG - OFF, NSTG);
        if (quad == 0) {
        // the rows' sums: over a row's four lanes, then over the four warps in order
#pragma unroll
        for (int rt = 0; rt < RT; rt++)
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                float a = l[rt][h2], b = ps[rt][h2];
                a += __shfl_xor_sync(0xffffffffu, a, 1); b += __shfl_xor_sync(0xffffffffu, b, 1);
                a += __shfl_xor_sync(0xffffffffu, a, 2); b += __shfl_xor_sync(0xffffffffu, b, 2);
                if (t4 == 0) xsum[(w * RT + rt) * 16 + r + 8 * h2] = make_float2(a, b);
            }
        named_bar_sync(2, 128);
#pragma unroll
        for (int rt = 0; rt < RT; rt++)
#pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                float L = 0.f, P = 0.f;
#pragma unroll
                for (int ww = 0; ww < 4; ww++) {
                    const float2 x = xsum[(ww * RT + rt) * 16 + r + 8 * h2];
                    L += x.x;
                    P += x.y;
                }
                const int row = rt * 16 + r + 8 * h2, tok = row / GROUP, head = was.z * GROUP + row % GROUP;
                const bool in = tok < was.y;
                if (was_ns == 1) {
                    if (!in) continue;
                    const float f = 1.f / L;
                    float* op = out + (size_t)dtok[was.x + tok] * MIX + head * HD + 64 * w + 2 * t4;
#pragma unroll
                    for (int jd = 0; jd < 8; jd++) {
                        const float2 gt = *(float2*)(op + jd * 8);
                        *(float2*)(op + jd * 8) = make_float2(gt.x * (o[rt][jd][2 * h2] - KV_OFF * P) * f,
                                                              gt.y * (o[rt][jd][2 * h2 + 1] - KV_OFF * P) * f);
                    }
                } else {
                    // (neighbours swap, so that a lane writes 16 bytes and a row's four 64)
                    const size_t pi = ((size_t)(was.x + tok) * NH + head) * z + was.w;
                    float* pp = part_acc + pi * HD + 64 * w + (t4 & 1) * 8 + (t4 & 2) * 2;
#pragma unroll
                    for (int jd = 0; jd < 8; jd += 2) {
                        const bool odd = t4 & 1;
                        const float2 a = make_float2(o[rt][jd][2 * h2] - KV_OFF * P, o[rt][jd][2 * h2 + 1] - KV_OFF * P);
                        const float2 b = make_float2(o[rt][jd + 1][2 * h2] - KV_OFF * P, o[rt][jd + 1][2 * h2 + 1] - KV_OFF * P);
                        const float x = __shfl_xor_sync(0xffffffffu, odd ? a.x : b.x, 1), y = __shfl_xor_sync(0xffffffffu, odd ? a.y : b.y, 1);
                        if (in) *(float4*)(pp + jd * 8) = odd ? make_float4(x, y, b.x, b.y) : make_float4(a.x, a.y, x, y);
                    }
                    if (in && w == 0 && t4 == 0) { part_ml[pi * 2] = m[rt][h2]; part_ml[pi * 2 + 1] = L; }
                }
            }
        }
        if constexpr (MANY) {
            if (quad != 1) go_on();
        }
        if (!more) return;
    }
}

// Merge the ns key splits of one (token, head) in split order; *op *= result (the gate is there); optionally also the
// f16 copy of the product. HD threads, thread d owns dim d; the splits' maxima and sums go through shared memory once
// so that the accumulator loads of all splits are independent and in flight together.
__device__ __forceinline__ void combine_row(const float* part_ml, const float* part_acc, size_t base, int ns, float* op,
                                            __half* mp) {
    static_assert(DSPLITS <= 64 && TSPLITS <= 64, "two splits per lane");
    __shared__ float se[64];
    __shared__ float sL;
    const int d = threadIdx.x;
    float res;
    if (ns == 1) {
        res = *op;  // the attention kernel finished it
    } else {
        if (d < 32) {  // lane d: splits d and d + 32
            const float ms0 = d < ns ? part_ml[(base + d) * 2] : -INFINITY;
            const float ls0 = d < ns ? part_ml[(base + d) * 2 + 1] : 0.f;
            const float ms1 = d + 32 < ns ? part_ml[(base + d + 32) * 2] : -INFINITY;
            const float ls1 = d + 32 < ns ? part_ml[(base + d + 32) * 2 + 1] : 0.f;
            const float M = warp_max(fmaxf(ms0, ms1));
            const float e0 = ms0 == -INFINITY ? 0.f : exp2f(ms0 - M), e1 = ms1 == -INFINITY ? 0.f : exp2f(ms1 - M);
            se[d] = e0;
            se[d + 32] = e1;
            // the sum over splits in split order (not a tree: the same order whatever the lane count)
            float L = 0.f;
            for (int s = 0; s < ns; s++) L += __shfl_sync(0xffffffffu, s < 32 ? e0 * ls0 : e1 * ls1, s & 31);
            if (d == 0) sL = L;
        }
        __syncthreads();
        float A = 0.f;
        const float* pa = part_acc + base * HD + d;
#pragma unroll 8
        for (int s = 0; s < ns; s++) A += se[s] * pa[(size_t)s * HD];
        res = *op * A * (1.f / sL);
        *op = res;
    }
    if (mp) *mp = __float2half_rn(res);
}

// block (decode token, head)
__global__ void __launch_bounds__(HD)
attn_combine_kernel(const float* part_ml, const float* part_acc, const int* dtok, const int* dkeys, int z, int dsplits,
                    float* out, __half* mix) {
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x, h = blockIdx.y, t = dtok[i], d = threadIdx.x;
    const size_t o = (size_t)t * MIX + h * HD + d;
    combine_row(part_ml, part_acc, ((size_t)i * NH + h) * z, dec_splits(dkeys[i], dsplits), out + o, mix ? mix + o : nullptr);
}

// block (prompt tile * PTILE + row, head)
__global__ void __launch_bounds__(HD)
attn_combine_tiles_kernel(const float* part_ml, const float* part_acc, const int* ptile, const int* tok_pos, int z,
                          float* out, __half* mix) {
    pdl_launch_dependents();
    pdl_wait();
    const int tile = blockIdx.x / PTILE, row = blockIdx.x % PTILE, h = blockIdx.y, d = threadIdx.x;
    const int t0 = ptile[2 * tile], len = ptile[2 * tile + 1];
    if (row >= len) return;
    const int keys = tok_pos[t0 + len - 1] + 1, chunk = tile_chunk(keys, z), t = t0 + row;
    const size_t o = (size_t)t * MIX + h * HD + d;
    combine_row(part_ml, part_acc, ((size_t)t * NH + h) * z, (keys + chunk - 1) / chunk, out + o, mix ? mix + o : nullptr);
}

// one block: which form the two tcgen05 kernels behind it take
constexpr int FORM_THREADS = 512;
__global__ void __launch_bounds__(FORM_THREADS)
attn_form_kernel(const int* ptile, int ntile, const int* tok_slot, const int* tok_pos, int sms, int* on_pairs) {
    pdl_launch_dependents();
    pdl_wait();
    const bool p = tc::tiles_on_pairs(ptile, ntile, tok_slot, tok_pos, sms);
    if (threadIdx.x == 0) {
        on_pairs[0] = p;
        on_pairs[1] = 0;
    }
}

}  // namespace qb

using namespace qb;

extern "C" {

int qb_attn_prep(qb_ctx* ctx, void* stream, const float* part, int splits, int n, const float* q_norm,
                 const float* k_norm, const float* inv_freq, float qscale, float* q, float* out, void* kc, void* vc,
                 float* ks, float* vs, const int* tok_slot, const int* tok_pos, int cap) {
    if (!ctx || !part || !q_norm || !k_norm || !inv_freq || !q || !out || !kc || !vc || !ks || !vs || !tok_slot ||
        !tok_pos || n <= 0 || splits < 1 || cap <= 0 || cap % 64)
        return QB_ERR_ARG;
    return launch(ctx, attn_prep_kernel, dim3(n, 2), dim3(32 * NH), 0, (cudaStream_t)stream, part, splits, n,
                  q_norm, k_norm, inv_freq, qscale, q, out, (uint8_t*)kc, (uint8_t*)vc, ks, vs, tok_slot, tok_pos, cap);
}

int qb_attn_dec_splits(int keys) { return keys > 0 ? dec_splits(keys, DSPLITS) : 0; }
int qb_attn_dec_splits_sm(int keys, int sms) { return keys > 0 && sms > 0 ? dec_splits(keys, dsplits_for(sms)) : 0; }

int qb_attn_dec_grid(int max_keys, int sms) { return max_keys > 0 && sms > 0 ? dec_splits_upto(max_keys, dsplits_for(sms)) : 0; }

// One block per split where they are few; blocks that keep running where they would be more than four rounds of the SMs, or more than
// three with the last at most half full, if all sequences were as long as the longest. Block per split against that, us:
// 8 sequences x 4 rows, up to context 7777 57.7 / 47.9; 8 x 8 at 8000 96.0 / 87.1; 8 x 1 at 3000 35.7 / 33.8; 4 x 4 up to 8000
// (3.4 rounds) 36.0 / 32.7; but 6 x 8 at 3000 (3.9) 42.5 / 44.5, 4 x 4 up to 3000 (2.6) 21.5 / 22.5, 2 x 4 up to 3000 14.1 / 14.9, 3 x 8 at
// 3000 25.0 / 32.2: the table of the segments costs a microsecond before the first split. (Left: 8 x 4 at 2048, 3.7 rounds, 34.1 / 29.1.)
int qb_attn_dec_dealt(int ndseg, int max_keys, int sms) {
    if (ndseg <= 0 || ndseg > DEC_SEGS || max_keys <= 0 || sms <= 0) return 0;
    const long long most = (long long)ndseg * NKV * dec_splits(max_keys, dsplits_for(sms));
    return most > 4 * sms || (most > 3 * sms && 2 * most <= 7 * sms);
}

// (a captured step is replayed for every step that it serves, so whatever the launches are chosen by is here)
int qb_attn_step_form(int ndseg, int dec_keys, int ntile, int tile_keys, int sms) {
    return qb_attn_dec_grid(dec_keys, sms) + 128 * (ntile > 0 ? qb_attn_tile_splits(ntile, tile_keys) : 0) + 8192 * qb_attn_dec_dealt(ndseg, dec_keys, sms);
}

// ndseg short segments (dseg: first index into dtok, token count; at most 8 tokens each), ndec = their tokens in
// all, dmax = the longest segment's tokens, max_keys = the largest key count among them (sizes the grid).
int qb_attn_decode(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks,
                   const float* vs, const int* dseg, const int* dtok, const int* dkeys, const int* tok_slot,
                   const int* tok_pos, int cap, int ndseg, int ndec, int dmax, int max_keys, float* part_ml,
                   float* part_acc, float* out, void* mix_f16) {
    return qb_attn_decode_as(ctx, stream, q, kc, vc, ks, vs, dseg, dtok, dkeys, tok_slot, tok_pos, cap, ndseg, ndec, dmax, max_keys,
                             part_ml, part_acc, out, mix_f16, 0);
}

}  // extern "C"

int qb_attn_decode_as(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks, const float* vs,
                      const int* dseg, const int* dtok, const int* dkeys, const int* tok_slot, const int* tok_pos, int cap, int ndseg,
                      int ndec, int dmax, int max_keys, float* part_ml, float* part_acc, float* out, void* mix_f16, int ahead) {
    if (!ctx || !q || !kc || !vc || !ks || !vs || !dseg || !dtok || !dkeys || !tok_slot || !tok_pos || !part_ml ||
        !part_acc || !out || ndseg <= 0 || ndec <= 0 || dmax <= 0 || dmax > 8 || max_keys <= 0 || cap % 64 ||
        max_keys > cap)
        return QB_ERR_ARG;
    const int dsplits = dsplits_for(ctx->sms);
    const int z = dec_splits_upto(max_keys, dsplits), rt = (dmax * GROUP + 15) / 16;
    cudaStream_t st = (cudaStream_t)stream;
    dim3 grid(ndseg, NKV, z);
    // (the model's steps have at most 64 decode tokens: whatever lies 64 positions or more before a segment's last key is from
    // earlier steps)
    const int old_margin = ahead && ndec <= 64 ? 64 : 0;
    const bool many = qb_attn_dec_dealt(ndseg, max_keys, ctx->sms);
    int rc;
#define QB_DEC(RT, NQ)                                                                                          \
    {                                                                                                           \
        using C = Dec4Cfg<RT, NQ>;                                                                              \
        rc = many ? launch(ctx, attn_dec4_kernel<RT, NQ, true>, dim3(ctx->sms), dim3(C::THREADS), C::SMEM_MANY, st, q, (const uint8_t*)kc, \
                           (const uint8_t*)vc, ks, vs, dseg, dtok, tok_slot, tok_pos, cap, z, dsplits, old_margin, ndseg, part_ml,   \
                           part_acc, out, ctx->err)                                                                             \
                  : launch(ctx, attn_dec4_kernel<RT, NQ, false>, grid, dim3(C::THREADS), C::SMEM, st, q, (const uint8_t*)kc, \
                           (const uint8_t*)vc, ks, vs, dseg, dtok, tok_slot, tok_pos, cap, z, dsplits, old_margin, ndseg, part_ml,   \
                           part_acc, out, ctx->err);                                                                             \
    }
    // quads per block: as many as leave every warp its registers (a warp holds RT x 32 output accumulators per lane);
    // measured at 5 rows with a copy warp beside them: 2 quads 33.4 us, 3 quads (spills) 36.6 us, 4 quads 43.2 us
    if (rt == 1) QB_DEC(1, 4) else if (rt == 2) QB_DEC(2, 2) else QB_DEC(3, 2)
#undef QB_DEC
    if (rc) return rc;
    return launch(ctx, attn_combine_kernel, dim3(ndec, NH), dim3(HD), 0, st, (const float*)part_ml,
                  (const float*)part_acc, dtok, dkeys, z, dsplits, out, (__half*)mix_f16);
}

extern "C" {

int qb_attn_tile_splits(int ntile, int max_keys) { return ntile > 0 && max_keys > 0 ? tile_splits(ntile, max_keys) : 0; }

// Prompt attention: ntile tiles of up to 10 consecutive tokens of one segment (the host's ptile array: first token,
// count), each against all the keys up to its last token; max_keys = the largest key count among them. `out` holds
// the gate on entry and the gated attention output on return; mix_f16 (optional) gets its f16 copy. One block per
// (tile, kv head, key split); part_ml / part_acc: scratch for n * 24 * qb_attn_tile_splits(ntile, max_keys) (m, l)
// pairs and accumulators of 256 floats, n = the step's tokens (unused with one split).
int qb_attn_prefill(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks,
                    const float* vs, const int* ptile, const int* tok_slot, const int* tok_pos, int cap, int ntile,
                    int max_keys, float* part_ml, float* part_acc, float* out, void* mix_f16) {
    return qb_attn_prefill_as(ctx, stream, q, kc, vc, ks, vs, ptile, tok_slot, tok_pos, cap, ntile, max_keys, part_ml, part_acc, out,
                              mix_f16, -1);
}

// what attn_form_kernel says, from the arrays on the host
int qb_attn_tiles_on_pairs(const int* h_ptile, int ntile, const int* h_tok_slot, const int* h_tok_pos, int sms) {
    if (!h_ptile || !h_tok_slot || !h_tok_pos || ntile <= 0 || sms <= 0) return 0;
    unsigned long long sum[2] = {0ull, 0ull};
    unsigned top[2] = {0u, 0u}, unit[2] = {0u, 0u};
    for (int t = 0; t < ntile; t++) {
        const bool on = t + 1 < ntile && tc::tile_goes_on(h_ptile, h_tok_slot, h_tok_pos, t);
        const int keys = h_tok_pos[h_ptile[2 * t] + h_ptile[2 * t + 1] - 1] + 1;
        for (int f = 0; f < 2; f++) {
            const int of = f ? 2 : 4;
            if (t % of == 0) unit[f] = 0u;
            if (!on || t % of == of - 1) {
                const unsigned c = f ? tc::block_pass_cost(keys) : tc::pair_pass_cost(keys);
                sum[f] += c;
                unit[f] += c;
            }
            if (unit[f] > top[f]) top[f] = unit[f];
        }
    }
    return tc::pairs_win(sum[0], sum[1], top[0], top[1], sms);
}

}  // extern "C"

namespace {
// One key split: two tiles per block or four per pair of blocks. Up to 1664 keys as blocks: a stage of 128 keys and the pair's
// set-up cost more there than the faster stages give (100 rows at context 0 40.1 us as blocks, 43.7 as pairs; 1500 at 100
// 200 and 210; 2048 at 0 289 and 277; 1024 at 2000 257 and 225). Beyond, the runs of the tiles decide (attn_tc.cuh): 0
// blocks, 1 pairs. A caller that has the tiles on the host says which; for the others (2) a small kernel works it out and
// both forms are launched, one of which returns before it takes anything (with attn_prep, in a graph: 600 rows at 2000
// 106 -> 112 us, 400 at 4000 136.6 -> 138.6, 2048 at 1700 370 -> 376, 2048 at 8000 734 -> 734; each of the blocks working it
// out for itself: 4 to 6 % throughout).
int prefill_form(const qb_ctx* ctx, int max_keys, int as) {
    if (ctx->tune_ctas == 1002 || ctx->tune_ctas == 1003) return ctx->tune_ctas - 1002;  // measurement
    return max_keys <= 1664 ? 0 : as < 0 ? 2 : as;
}
}  // namespace

int qb_attn_prefill_launches(const qb_ctx* ctx, int ntile, int max_keys, int as) {
    if (tile_splits(ntile, max_keys) > 1) return 2;
    return prefill_form(ctx, max_keys, as) == 2 ? 3 : 1;
}

int qb_attn_prefill_as(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks,
                       const float* vs, const int* ptile, const int* tok_slot, const int* tok_pos, int cap, int ntile,
                       int max_keys, float* part_ml, float* part_acc, float* out, void* mix_f16, int as) {
    if (!ctx || !q || !kc || !vc || !ks || !vs || !ptile || !tok_slot || !tok_pos || !out || ntile <= 0 || cap % 64 ||
        max_keys <= 0 || max_keys > cap)
        return QB_ERR_ARG;
    const int z = tile_splits(ntile, max_keys);
    if (z > 1 && (!part_ml || !part_acc)) return QB_ERR_ARG;
    if (z == 1) {
        const int form = prefill_form(ctx, max_keys, as);
        int* word = form == 2 ? ctx->form : nullptr;
        cudaStream_t st = (cudaStream_t)stream;
        int rc = QB_OK;
        if (word) rc = launch(ctx, attn_form_kernel, dim3(1), dim3(FORM_THREADS), 0, st, ptile, ntile, tok_slot, tok_pos, ctx->sms, ctx->form);
        if (!rc && form != 0) rc = qb_attn_prefill_tc_launch(ctx, st, q, kc, vc, ks, vs, ptile, ntile, tok_slot, tok_pos, cap, out, mix_f16, word);
        if (!rc && form != 1) rc = qb_attn_prefill_short_launch(ctx, st, q, kc, vc, ks, vs, ptile, ntile, tok_slot, tok_pos, cap, out, mix_f16, word);
        return rc;
    }
    using C = TileCfg<4, 2, 5>;  // 10 tokens x 6 heads = 60 rows: 4 row tiles; 2 warps each; 5 stages of 32 keys
    static_assert(PTILE * GROUP <= 64, "a prompt tile fills at most 4 row tiles");
    cudaStream_t st = (cudaStream_t)stream;
    int rc = launch(ctx, attn_tile_kernel<4, 2, 5>, dim3(ntile, NKV, z), dim3(C::THREADS), C::SMEM, st, q, (const uint8_t*)kc,
                    (const uint8_t*)vc, ks, vs, ptile, tok_slot, tok_pos, cap, z, part_ml, part_acc, out, ctx->err);
    if (rc) return rc;
    return launch(ctx, attn_combine_tiles_kernel, dim3(ntile * PTILE, NH), dim3(HD), 0, st, (const float*)part_ml,
                  (const float*)part_acc, ptile, tok_pos, z, out, (__half*)mix_f16);
}
