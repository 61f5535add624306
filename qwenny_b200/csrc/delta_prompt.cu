// Gated DeltaNet for steps whose segments are not decode-sized (prompt chunks, long verify steps, and every step that
// does not take the one-launch mixer of deltanet.cu). Same entry points and buffers as the reference's three kernels
// (kernels/qwen_deltanet.cuh: delta_conv :84-131, delta_rule :172-288, delta_norm :295-315); the rule itself is in
// delta_rule.cu. Here:
//
//  delta_prep_kernel, delta_prep_run_kernel (128 tokens and more)
//                           the causal depthwise conv, SiLU, the L2 norms of the q and k heads and the two gates. A
//                           lane owns FOUR channels and slides along the tokens with the conv's four inputs in
//                           registers (each input row is read once, not four times); the 128 channels of a warp are
//                           one q, k or v head, so the head's norm is a warp reduction per token.
//  delta_gate_norm_kernel   RMSNorm(w) * SiLU(z) per value head -> f16, then the slots' metadata.
#include "delta_common.cuh"
#include "launch.h"

namespace qb {

// ------------------------------------------------------------------------------------------------ delta_prep

// exp(g) and beta per value head of cnt tokens from tb on, by 128 threads
__device__ __forceinline__ void gates(int tb, int cnt, int n, const float* ba, int ba_splits, const float* a_log, const float* dt_bias, float* cv) {
    for (int x = threadIdx.x; x < cnt * LV_HEADS; x += 128) {
        const int t = tb + x / LV_HEADS, v = x % LV_HEADS;
        float b = 0.f, a = 0.f;
        for (int s = 0; s < ba_splits; s++) {
            const float* r = ba + ((size_t)s * n + t) * (2 * LV_HEADS);
            b += r[v];
            a += r[LV_HEADS + v];
        }
        a += dt_bias[v];
        const float sp = a > 20.f ? a : log1pf(expf(a));
        cv[(size_t)t * CVW + LQKV + v] = expf(-expf(a_log[v]) * sp);
        cv[(size_t)t * CVW + LQKV + LV_HEADS + v] = 1.f / (1.f + expf(-b));
    }
}

// a lane's four channels of a token: the conv over the three tokens before (h) and itself, SiLU, and for a q or k head the L2 norm over
// its 128 channels, q also / sqrt(128)
__device__ __forceinline__ float4 conv_token(const float4* taps, const float4* h, float4 v, int head) {
    auto conv = [&](float4 w, float a0, float a1, float a2, float a3) {
        float a = w.x * a0;
        a = fmaf(w.y, a1, a);
        a = fmaf(w.z, a2, a);
        a = fmaf(w.w, a3, a);
        return silu(a);
    };
    float4 y;
    y.x = conv(taps[0], h[0].x, h[1].x, h[2].x, v.x);
    y.y = conv(taps[1], h[0].y, h[1].y, h[2].y, v.y);
    y.z = conv(taps[2], h[0].z, h[1].z, h[2].z, v.z);
    y.w = conv(taps[3], h[0].w, h[1].w, h[2].w, v.w);
    if (head < 2 * LK_HEADS) {
        float sc = rsqrtf(warp_sum((y.x * y.x + y.y * y.y) + (y.z * y.z + y.w * y.w)) + 1e-6f);
        if (head < LK_HEADS) sc *= rsqrtf((float)LKD);
        y.x *= sc; y.y *= sc; y.z *= sc; y.w *= sc;
    }
    return y;
}

// grid (LQKV / 512 + 1, ceil(n / PREP_TOK)), block 128: a warp is one head, a lane four of its channels; the last column of
// blocks makes the gates. Bound by the rows' way from memory and back (n x 80 KB): every row of the tile is requested
// before anything is used, 16 bytes per lane, and the head's norm is a warp reduction (2048 tokens, one part: 53 us; 76 us with
// a channel per thread, four bytes per request and the gates behind the first head's channels).
// VEC: p and cv start on 16 bytes, as a device allocation does; elsewhere (any float address is allowed) a lane moves its four
// channels one by one.
// 8 tokens per block leave room for five blocks per SM; 16 read less history but take 9.4 us for 129 tokens (8: 5.8), 10.5 for
// 333 (10.3), 17.5 for 512 (11.9), 61 for 2048 (53), and gain only around 420 (10.6, 11.0).
constexpr int PREP_TOK = 8;  // tokens a block slides along
template <bool VEC>
__global__ void __launch_bounds__(128, 5)
delta_prep_kernel(const float* p, int splits, int n, const float* ba, int ba_splits, const float* cw,
                  const float* a_log, const float* dt_bias, const float* mem, long long sst, float* cv,
                  const int* tok_slot, const int* tok_pos) {
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tb = blockIdx.y * PREP_TOK, cnt = min(PREP_TOK, n - tb);
    if (blockIdx.x == LQKV / 512) {  // the gates of the tile's tokens: exp(g) and beta per value head
        pdl_wait();
        gates(tb, cnt, n, ba, ba_splits, a_log, dt_bias, cv);
        return;
    }
    const int head = blockIdx.x * 4 + warp, ch = head * 128 + lane * 4;
    float4 taps[4];  // of the lane's four channels
#pragma unroll
    for (int c = 0; c < 4; c++) taps[c] = ld4(cw + (size_t)(ch + c) * CONV_K);
    pdl_wait();
    const size_t stride = (size_t)n * DELTA_IN;
    auto row4 = [](const float* r) { return VEC ? ld4(r) : make_float4(r[0], r[1], r[2], r[3]); };
    // lane i < PREP_TOK: token tb + i's slot and position; the next three: the slots of the three tokens before the tile
    const int mt = min(lane < PREP_TOK ? tb + lane : max(tb - PREP_TOK - 3 + lane, 0), n - 1);
    const int my_slot = tok_slot[mt], my_pos = tok_pos[mt];
    float4 x[PREP_TOK], h[3];  // h: the conv inputs at the three positions before the current token
#pragma unroll
    for (int i = 0; i < 3; i++) h[i] = row4(p + (size_t)max(tb - 3 + i, 0) * DELTA_IN + ch);
#pragma unroll
    for (int i = 0; i < PREP_TOK; i++) x[i] = row4(p + (size_t)min(tb + i, n - 1) * DELTA_IN + ch);
    // (the other partial sums in a loop of their own: one inside the row's load makes the loads wait for one another)
    for (int s = 1; s < splits; s++) {
        const float* ps = p + s * stride + ch;
        auto add = [](float4& v, float4 w) { v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w; };
#pragma unroll
        for (int i = 0; i < 3; i++) add(h[i], row4(ps + (size_t)max(tb - 3 + i, 0) * DELTA_IN));
#pragma unroll
        for (int i = 0; i < PREP_TOK; i++) add(x[i], row4(ps + (size_t)min(tb + i, n - 1) * DELTA_IN));
    }
    int prev_slot = -1;
#pragma unroll
    for (int i = 0; i < PREP_TOK; i++) {
        if (i < cnt) {
            const int t = tb + i, slot = __shfl_sync(0xffffffffu, my_slot, i), pos = __shfl_sync(0xffffffffu, my_pos, i);
            if (slot != prev_slot) {
                // a segment starts in this tile (or the tile starts): the history comes from the step's own rows of the same
                // sequence (at the tile's start those are loaded already), from the slot's ring, or is zero
                float4 f[3];
#pragma unroll
                for (int b = 0; b < 3; b++) {
                    const int back = 3 - b, qp = pos - back, tt = t - back;
                    const bool own = i == 0 && tt >= 0 && __shfl_sync(0xffffffffu, my_slot, PREP_TOK + b) == slot;
                    f[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (qp >= 0) {
                        const float* r = mem + slot * sst + SLOT_RING + (size_t)(qp & (CR - 1)) * LQKV + ch;  // (sst may be odd)
                        if (own) f[b] = h[b];
                        else f[b] = make_float4(r[0], r[1], r[2], r[3]);
                    }
                }
                h[0] = f[0]; h[1] = f[1]; h[2] = f[2];
                prev_slot = slot;
            }
            const float4 v = x[i];
            const float4 y = conv_token(taps, h, v, head);
            h[0] = h[1]; h[1] = h[2]; h[2] = v;
            float* to = cv + (size_t)t * CVW + ch;
            if (VEC) *(float4*)to = y;
            else { to[0] = y.x; to[1] = y.y; to[2] = y.z; to[3] = y.w; }
        }
    }
}

// The same for prompt steps (one part, 16-byte aligned): a block keeps 512 channels and runs along `run` tokens, so that it starts
// once and reads each row once, and a lane's 16 bytes of the next RUN_ROWS - 1 rows are on their way into shared memory, where they take
// no registers and no other thread waits for them. grid (LQKV / 512, runs + the gates' blocks of PREP_TOK tokens), block 128.
// Against the tiles of 8 tokens, us: 128 tokens 6.2 / 5.4, 200 7.6 / 6.1, 220 7.7 / 8.0, 256 8.4 / 8.4, 333 13.4 / 9.1, 512 16.7 / 12.8, 1024
// 29.2 / 20.5, 2048 53.3 / 35.2 (168 MB: 4.8 TB/s). More rows under way are slower (2048 tokens: 16 rows 39.2, 8 rows 37.0), so are fewer blocks
// (5 of 8 rows 40.8); 7 or 8 blocks per SM are alike above 700 tokens and worse below (333: 9.7, 10.3).
constexpr int RUN_ROWS = 4, RUN_PER_SM = 6;
constexpr int RUN_FROM = 128;  // tokens: a run has four tokens then, and below the tiles fill the SMs as well
__global__ void __launch_bounds__(128, RUN_PER_SM)
delta_prep_run_kernel(const float* p, int n, int run, int runs, const float* ba, int ba_splits, const float* cw,
                      const float* a_log, const float* dt_bias, const float* mem, long long sst, float* cv,
                      const int* tok_slot, const int* tok_pos) {
    __shared__ float4 ring[RUN_ROWS][128];
    pdl_launch_dependents();
    if (blockIdx.y >= runs) {
        const int tb = ((blockIdx.y - runs) * gridDim.x + blockIdx.x) * PREP_TOK;
        pdl_wait();
        if (tb < n) gates(tb, min(PREP_TOK, n - tb), n, ba, ba_splits, a_log, dt_bias, cv);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tb = blockIdx.y * run, cnt = min(run, n - tb);
    const int head = blockIdx.x * 4 + warp, ch = head * 128 + lane * 4;
    float4 taps[4], h[3];  // of the lane's four channels; h: the conv inputs at the three positions before the current token
#pragma unroll
    for (int c = 0; c < 4; c++) taps[c] = ld4(cw + (size_t)(ch + c) * CONV_K);
    pdl_wait();
    const float* from = p + (size_t)tb * DELTA_IN + ch;
    auto fetch = [&](int i) {
        if (i < cnt) cp_async16(&ring[i % RUN_ROWS][threadIdx.x], from + (size_t)i * DELTA_IN);
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < RUN_ROWS - 1; i++) fetch(i);
#pragma unroll
    for (int i = 0; i < 3; i++) h[i] = ld4(p + (size_t)max(tb - 3 + i, 0) * DELTA_IN + ch);
    const int before = tok_slot[max(tb - 3 + min(lane, 2), 0)];  // lane i < 3: the slot of the token 3 - i before the run
    int prev_slot = -1, my_slot = 0, my_pos = 0;
#pragma unroll 4
    for (int i = 0; i < cnt; i++) {
        if (i % 32 == 0) {
            my_slot = tok_slot[min(tb + i + lane, n - 1)];
            my_pos = tok_pos[min(tb + i + lane, n - 1)];
        }
        const int t = tb + i, slot = __shfl_sync(0xffffffffu, my_slot, i % 32), pos = __shfl_sync(0xffffffffu, my_pos, i % 32);
        if (slot != prev_slot) {
            // a segment starts here (or the run does): the history as above
            float4 f[3];
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const int back = 3 - b, qp = pos - back, tt = t - back;
                const bool own = i == 0 && tt >= 0 && __shfl_sync(0xffffffffu, before, b) == slot;
                f[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (qp >= 0) {
                    const float* r = mem + slot * sst + SLOT_RING + (size_t)(qp & (CR - 1)) * LQKV + ch;  // (sst may be odd)
                    if (own) f[b] = h[b];
                    else f[b] = make_float4(r[0], r[1], r[2], r[3]);
                }
            }
            h[0] = f[0]; h[1] = f[1]; h[2] = f[2];
            prev_slot = slot;
        }
        asm volatile("cp.async.wait_group %0;\n" ::"n"(RUN_ROWS - 2) : "memory");
        const float4 v = ring[i % RUN_ROWS][threadIdx.x];
        fetch(i + RUN_ROWS - 1);  // (in the place of the row before this one)
        const float4 y = conv_token(taps, h, v, head);
        h[0] = h[1]; h[1] = h[2]; h[2] = v;
        *(float4*)(cv + (size_t)t * CVW + ch) = y;
    }
}

// ------------------------------------------------------------------------------------------------ delta_gate_norm
// grid (n), block 384: warp w normalises value heads 4 w .. 4 w + 3 of the token, a lane four columns of each
constexpr int GN_THREADS = 384;
__global__ void __launch_bounds__(GN_THREADS)
delta_gate_norm_kernel(const float* p, int splits, int n, const float* nw, const float* o, __half* y, int* meta,
                       const int* seg_len, const int* seg_slot, const int* seg_pos0, int segs) {
    pdl_launch_dependents();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float4 w = ld4(nw + lane * 4);
    pdl_wait();
    const size_t stride = (size_t)n * DELTA_IN;
#pragma unroll
    for (int i = 0; i < LV_HEADS / (GN_THREADS / 32); i++) {
        const int h = warp * (LV_HEADS / (GN_THREADS / 32)) + i;
        const size_t at = (size_t)t * MIX + h * LVD + lane * 4;
        const float4 v = ld4(o + at);
        const float* zp = p + (size_t)t * DELTA_IN + LQKV + h * LVD + lane * 4;
        float4 z = ld4(zp);
        for (int s = 1; s < splits; s++) {
            const float4 x = ld4(zp + s * stride);
            z.x += x.x; z.y += x.y; z.z += x.z; z.w += x.w;
        }
        const float r = rsqrtf(warp_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w) / LVD + EPS);
        *(uint2*)(y + at) = make_uint2(pack_half2(w.x * (v.x * r) * silu(z.x), w.y * (v.y * r) * silu(z.y)),
                                       pack_half2(w.z * (v.z * r) * silu(z.z), w.w * (v.w * r) * silu(z.w)));
    }
    if (t == 0) {  // the step is recorded in the slots' metadata (every reader of the old values ran in earlier kernels)
        for (int s = threadIdx.x; s < segs; s += GN_THREADS) {
            const int slot = seg_slot[s], p0 = seg_pos0[s], len = seg_len[s];
            const Plan pl = make_plan(meta, slot, p0, len);
            meta[slot * META] = p0 + len;
            meta[slot * META + 1] = pl.ck;
            meta[slot * META + 2] = pl.ebuf;
        }
    }
}

}  // namespace qb

using namespace qb;

extern "C" {

int qb_delta_conv(qb_ctx* ctx, void* stream, const float* p, int splits, int n, const float* ba, int ba_splits,
                  const float* cw, const float* a_log, const float* dt_bias, const float* mem, long long sst,
                  float* cv, const int* tok_slot, const int* tok_pos) {
    if (!ctx || !p || !ba || !cw || !a_log || !dt_bias || !mem || !cv || !tok_slot || !tok_pos || n <= 0 ||
        splits < 1 || ba_splits < 1)
        return QB_ERR_ARG;
    const dim3 grid(LQKV / 512 + 1, (n + PREP_TOK - 1) / PREP_TOK);
    const bool vec = (((uintptr_t)p | (uintptr_t)cv) & 15) == 0;
    if (vec && splits == 1 && n >= RUN_FROM) {
        const int most = max(1, ctx->sms * RUN_PER_SM / (LQKV / 512)), run = (n + most - 1) / most, runs = (n + run - 1) / run;
        const int per = LQKV / 512 * PREP_TOK;
        return launch(ctx, delta_prep_run_kernel, dim3(LQKV / 512, runs + (n + per - 1) / per), dim3(128), 0, (cudaStream_t)stream, p, n, run,
                      runs, ba, ba_splits, cw, a_log, dt_bias, mem, sst, cv, tok_slot, tok_pos);
    }
    auto kern = vec ? delta_prep_kernel<true> : delta_prep_kernel<false>;
    return launch(ctx, kern, grid, dim3(128), 0, (cudaStream_t)stream, p, splits, n, ba, ba_splits, cw, a_log, dt_bias, mem, sst, cv,
                  tok_slot, tok_pos);
}

int qb_delta_norm(qb_ctx* ctx, void* stream, const float* p, int splits, int n, const float* nw, const float* out,
                  void* y, int* meta, const int* seg_len, const int* seg_slot, const int* seg_pos0, int segs) {
    if (!ctx || !p || !nw || !out || !y || !meta || !seg_len || !seg_slot || !seg_pos0 || n <= 0 || segs <= 0 ||
        splits < 1)
        return QB_ERR_ARG;
    return launch(ctx, delta_gate_norm_kernel, dim3(n), dim3(GN_THREADS), 0, (cudaStream_t)stream, p, splits, n, nw, out,
                  (__half*)y, meta, seg_len, seg_slot, seg_pos0, segs);
}

}  // extern "C"
