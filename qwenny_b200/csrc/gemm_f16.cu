// Dense f16 skinny product for the few matrices a checkpoint keeps in 16 bits (the DeltaNet in_proj_b / in_proj_a
// pair, 96 x 5120): Y[split][t][r] = W[r] . X[t] over the split's k range. Replaces gemm_dec<16, NTT, EPI_PLAIN>
// (kernels/gemm.cuh:222-304 of the reference). W arrives in the reference's packed form: tiles of 16 rows, per k16
// step the 32 lanes' mma A fragments (8 halves each), so a warp's 128-bit loads are the fragments themselves.
// A block is one (tile, k split, block of 8 NTT tokens); its 4 warps take alternate k16 steps and add up in shared memory in warp order.
#include "common.cuh"
#include "launch.h"
#include "measure.h"

namespace qb {

template <int NTT>
__global__ void __launch_bounds__(128) gemm_f16_plain_kernel(const uint4* __restrict__ W, const __half* __restrict__ X,
                                                             const int* __restrict__ xrows, int K, int ntiles, int n,
                                                             int kper, float* __restrict__ Y, int ldy) {
    __shared__ float4 red[3][NTT][32];
    pdl_launch_dependents();
    const int tile = blockIdx.x, split = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3, tok0 = blockIdx.z * (8 * NTT);
    const int k0 = split * kper, k1 = min(K, k0 + kper);
    const uint4* wp = W + ((size_t)tile * (K / 16) + k0 / 16) * 32 + lane;
    const int steps = (k1 - k0) / 16;
    // the weights do not depend on the previous kernel: all of this warp's fragments (up to MAXF k16 steps) are in
    // flight before it waits for that kernel; longer ranges fetch the rest as they go
    constexpr int MAXF = 16;
    uint4 wf[MAXF];
#pragma unroll
    for (int i = 0; i < MAXF; i++) {
        int sidx = warp + 4 * i;
        wf[i] = sidx < steps ? __ldg(wp + (size_t)sidx * 32) : make_uint4(0, 0, 0, 0);
    }
    pdl_wait();
    float acc[NTT][4];
#pragma unroll
    for (int j = 0; j < NTT; j++) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    const __half* xr[NTT];
#pragma unroll
    for (int j = 0; j < NTT; j++) {
        int tok = tok0 + 8 * j + g;
        xr[j] = tok < n ? X + (size_t)(xrows ? xrows[tok] : tok) * K + k0 + 2 * t : nullptr;
    }
    auto step = [&](int s, const uint4& w) {
        uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < NTT; j++) {
            uint32_t b0 = 0, b1 = 0;
            if (xr[j]) {
                b0 = *(const uint32_t*)(xr[j] + s * 16);
                b1 = *(const uint32_t*)(xr[j] + s * 16 + 8);
            }
            mma16816(acc[j], a, b0, b1);
        }
    };
#pragma unroll
    for (int i = 0; i < MAXF; i++)
        if (warp + 4 * i < steps) step(warp + 4 * i, wf[i]);
    for (int s = warp + 4 * MAXF; s < steps; s += 4) step(s, __ldg(wp + (size_t)s * 32));
    if (warp > 0) {
#pragma unroll
        for (int j = 0; j < NTT; j++) red[warp - 1][j][lane] = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
    }
    __syncthreads();
    if (warp == 0) {
        float* y = Y + (size_t)split * n * ldy;
#pragma unroll
        for (int j = 0; j < NTT; j++) {
#pragma unroll
            for (int w = 0; w < 3; w++) {
                float4 v = red[w][j][lane];
                acc[j][0] += v.x; acc[j][1] += v.y; acc[j][2] += v.z; acc[j][3] += v.w;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                int tok = tok0 + 8 * j + 2 * t + (i & 1), r = tile * 16 + g + (i >> 1) * 8;
                if (tok < n) y[(size_t)tok * ldy + r] = acc[j][i];
            }
        }
    }
}

// The same for prompt steps: a block multiplies its 32 tokens by TILES tiles, so that a fragment of X, which is gathered in
// 4-byte pieces, is loaded once for all of them (qb_gemm_f16_block_tiles says where). Same order of additions per output.
template <int TILES>
__global__ void __launch_bounds__(128) gemm_f16_wide_kernel(const uint4* __restrict__ W, const __half* __restrict__ X,
                                                            const int* __restrict__ xrows, int K, int ntiles, int n,
                                                            int kper, float* __restrict__ Y, int ldy) {
    constexpr int NTT = 4;
    __shared__ float4 red[3][TILES][NTT][32];
    pdl_launch_dependents();
    const int tile0 = blockIdx.x * TILES, split = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3, tok0 = blockIdx.z * (8 * NTT);
    const int k0 = split * kper, k1 = min(K, k0 + kper), steps = (k1 - k0) / 16;
    const uint4* wp = W + ((size_t)tile0 * (K / 16) + k0 / 16) * 32 + lane;
    pdl_wait();
    float acc[TILES][NTT][4];
#pragma unroll
    for (int i = 0; i < TILES; i++)
#pragma unroll
        for (int j = 0; j < NTT; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
    const __half* xr[NTT];
#pragma unroll
    for (int j = 0; j < NTT; j++) {
        const int tok = min(tok0 + 8 * j + g, n - 1);  // (a token past the last repeats it and is not written)
        xr[j] = X + (size_t)(xrows ? xrows[tok] : tok) * K + k0 + 2 * t;
    }
#pragma unroll 2
    for (int s = warp; s < steps; s += 4) {
        uint4 w[TILES];
        uint32_t b0[NTT], b1[NTT];
#pragma unroll
        for (int j = 0; j < NTT; j++) {
            b0[j] = *(const uint32_t*)(xr[j] + s * 16);
            b1[j] = *(const uint32_t*)(xr[j] + s * 16 + 8);
        }
#pragma unroll
        for (int i = 0; i < TILES; i++) w[i] = __ldg(wp + ((size_t)i * (K / 16) + s) * 32);
#pragma unroll
        for (int i = 0; i < TILES; i++) {
            const uint32_t a[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
            for (int j = 0; j < NTT; j++) mma16816(acc[i][j], a, b0[j], b1[j]);
        }
    }
    if (warp > 0) {
#pragma unroll
        for (int i = 0; i < TILES; i++)
#pragma unroll
            for (int j = 0; j < NTT; j++)
                red[warp - 1][i][j][lane] = make_float4(acc[i][j][0], acc[i][j][1], acc[i][j][2], acc[i][j][3]);
    }
    __syncthreads();
    if (warp == 0) {
        float* y = Y + (size_t)split * n * ldy;
#pragma unroll
        for (int i = 0; i < TILES; i++)
#pragma unroll
            for (int j = 0; j < NTT; j++) {
#pragma unroll
                for (int w = 0; w < 3; w++) {
                    const float4 v = red[w][i][j][lane];
                    acc[i][j][0] += v.x; acc[i][j][1] += v.y; acc[i][j][2] += v.z; acc[i][j][3] += v.w;
                }
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int tok = tok0 + 8 * j + 2 * t + (e & 1), r = (tile0 + i) * 16 + g + (e >> 1) * 8;
                    if (tok < n) y[(size_t)tok * ldy + r] = acc[i][j][e];
                }
            }
    }
}

// That, where X lets a row be copied in 16-byte pieces: weights and the block's 32 rows come through shared memory, 64 columns at a time
// and three such pieces under way in each of three blocks per SM (of registers a warp has room for one k16 step ahead, and 16 steps of it
// are 16 times the way from L2). Same order of additions per output.
constexpr int ST_PIECE = 64, ST_NP = 4, ST_ROW = ST_PIECE * 2 + 16;  // columns per piece, pieces, bytes per row of one (no bank conflicts)
template <int TILES>
struct StagedCfg {
    static constexpr int W_BYTES = TILES * 4 * 512, BYTES = W_BYTES + 32 * ST_ROW;
    static constexpr int RING = ST_NP * BYTES, RED = 3 * TILES * 4 * 32 * 16, SMEM = RING > RED ? RING : RED;
};
template <int TILES>
__global__ void __launch_bounds__(128, 3) gemm_f16_staged_kernel(const uint4* __restrict__ W, const __half* __restrict__ X,
                                                                 const int* __restrict__ xrows, int K, int ntiles, int n,
                                                                 int kper, float* __restrict__ Y, int ldy) {
    using C = StagedCfg<TILES>;
    constexpr int NTT = 4;
    extern __shared__ __align__(16) uint8_t st_raw[];
    pdl_launch_dependents();
    const int tile0 = blockIdx.x * TILES, split = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3, tok0 = blockIdx.z * (8 * NTT);
    const int k0 = split * kper, k1 = min(K, k0 + kper), steps = (k1 - k0) / 16, pieces = (steps + 3) / 4;
    const uint4* wp = W + ((size_t)tile0 * (K / 16) + k0 / 16 + warp) * 32 + lane;
    auto fetch_w = [&](int pc) {  // a warp fetches the steps that it will multiply
        if (pc * 4 + warp < steps)
#pragma unroll
            for (int i = 0; i < TILES; i++)
                cp_async16(st_raw + (pc % ST_NP) * C::BYTES + (i * 4 + warp) * 512 + lane * 16, wp + ((size_t)i * (K / 16) + pc * 4) * 32);
    };
    for (int pc = 0; pc < ST_NP - 1; pc++) fetch_w(pc);  // (they do not depend on the kernel before)
    pdl_wait();
    const int c = threadIdx.x & 7, r0 = threadIdx.x >> 3;
    const __half* row[2];  // the thread's 16 bytes of two rows
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int tok = min(tok0 + r0 + 16 * i, n - 1);  // (a token past the last repeats it and is not written)
        row[i] = X + (size_t)(xrows ? xrows[tok] : tok) * K + k0 + c * 8;
    }
    auto fetch_x = [&](int pc) {
        if (pc * ST_PIECE + c * 8 < k1 - k0)
#pragma unroll
            for (int i = 0; i < 2; i++)
                cp_async16(st_raw + (pc % ST_NP) * C::BYTES + C::W_BYTES + (r0 + 16 * i) * ST_ROW + c * 16, row[i] + pc * ST_PIECE);
    };
    for (int pc = 0; pc < ST_NP - 1; pc++) {
        fetch_x(pc);
        cp_async_commit();
    }
    float acc[TILES][NTT][4];
#pragma unroll
    for (int i = 0; i < TILES; i++)
#pragma unroll
        for (int j = 0; j < NTT; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;
    const int xat = C::W_BYTES + ((lane & 7) + (lane >> 4) * 8) * ST_ROW + ((lane >> 3) & 1) * 16 + warp * 32;
    for (int pc = 0; pc < pieces; pc++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(ST_NP - 2) : "memory");
        __syncthreads();  // (the piece is there, and all are done with the one before it)
        fetch_w(pc + ST_NP - 1);
        fetch_x(pc + ST_NP - 1);
        cp_async_commit();
        if (pc * 4 + warp < steps) {
            const uint8_t* base = st_raw + (pc % ST_NP) * C::BYTES;
            uint32_t b[NTT][2];
            ldsm_x4(b[0][0], b[0][1], b[1][0], b[1][1], smem_u32(base) + xat);
            ldsm_x4(b[2][0], b[2][1], b[3][0], b[3][1], smem_u32(base) + xat + 16 * ST_ROW);
#pragma unroll
            for (int i = 0; i < TILES; i++) {
                const uint4 w = *(const uint4*)(base + (i * 4 + warp) * 512 + lane * 16);
                const uint32_t a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int j = 0; j < NTT; j++) mma16816(acc[i][j], a, b[j][0], b[j][1]);
            }
        }
    }
    cp_async_wait_all();
    __syncthreads();
    float4(*red)[TILES][NTT][32] = (float4(*)[TILES][NTT][32])st_raw;
    if (warp > 0) {
#pragma unroll
        for (int i = 0; i < TILES; i++)
#pragma unroll
            for (int j = 0; j < NTT; j++)
                red[warp - 1][i][j][lane] = make_float4(acc[i][j][0], acc[i][j][1], acc[i][j][2], acc[i][j][3]);
    }
    __syncthreads();
    if (warp == 0) {
        float* y = Y + (size_t)split * n * ldy;
#pragma unroll
        for (int i = 0; i < TILES; i++)
#pragma unroll
            for (int j = 0; j < NTT; j++) {
#pragma unroll
                for (int ww = 0; ww < 3; ww++) {
                    const float4 v = red[ww][i][j][lane];
                    acc[i][j][0] += v.x; acc[i][j][1] += v.y; acc[i][j][2] += v.z; acc[i][j][3] += v.w;
                }
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int tok = tok0 + 8 * j + 2 * t + (e & 1), r = (tile0 + i) * 16 + g + (e >> 1) * 8;
                    if (tok < n) y[(size_t)tok * ldy + r] = acc[i][j][e];
                }
            }
    }
}

}  // namespace qb

using namespace qb;

// Tiles per block. More than one from the row count on at which one per block fills the SMs (5/6 of a block each): below that, more
// blocks in flight are worth more than X loaded once. 96 x 5120 in 5 splits, one tile per block against six (X gathered): 33 rows 5.9
// and 7.8 us, 128 rows (120 blocks) 7.1 and 8.0, 160 rows (150) 8.5 and 8.0, 333 rows 11.3 and 8.7, 2048 rows 37.0 and 17.0.
// Six tiles of a split of less than 256 columns leave a warp a few steps: there four blocks of one tile per SM are as good
// (40 splits, 64 rows, 480 blocks: 3.1 and 3.3 us; 96 rows, 720 blocks: 4.8 and 3.5). Blocks of two save little work each
// and lose where their second wave is partly filled (5 splits of 1024: 160 outputs, 200 rows, 175 blocks of two 11.4 and
// 9.8; 333 rows, 275 blocks 11.7 and 15.2; 512 rows, 400 blocks 18.0 and 17.6; 1024 rows 31.8 and 19.6).
extern "C" int qb_gemm_f16_block_tiles(int ntiles, int splits, int kper, int n, int sms) {
    const int per = ntiles % 6 == 0 ? 6 : ntiles % 4 == 0 ? 4 : ntiles % 2 == 0 ? 2 : 1;
    const long long blocks = (long long)ntiles * splits * ((n + 31) / 32);
    if (n <= 32 || 6 * blocks <= 5ll * sms) return 1;
    if (per == 6 && kper < 256 && blocks <= 4ll * sms) return 1;
    if (per == 2 && 2 * blocks > 5ll * sms && 5 * blocks < 26ll * sms) return 1;
    return per;
}

extern "C" int qb_gemm_f16_plain(qb_ctx* ctx, void* stream, const void* W, const void* X, const int* xrows, int K,
                                 int ntiles, int n, int kper, float* Y, int ldy) {
    if (!ctx || !W || !X || !Y || K <= 0 || K % 16 || ntiles <= 0 || n <= 0 || n > 65535 * 32 || kper <= 0 || kper % 16 ||
        ldy < ntiles * 16)
        return QB_ERR_ARG;
    int split = (K + kper - 1) / kper;
    dim3 grid(ntiles, split, n <= 32 ? 1 : (n + 31) / 32);
    cudaStream_t st = (cudaStream_t)stream;
    const uint4* w = (const uint4*)W;
    const __half* x = (const __half*)X;
    if (n <= 8) return launch(ctx, gemm_f16_plain_kernel<1>, grid, dim3(128), 0, st, w, x, xrows, K, ntiles, n, kper, Y, ldy);
    if (n <= 16) return launch(ctx, gemm_f16_plain_kernel<2>, grid, dim3(128), 0, st, w, x, xrows, K, ntiles, n, kper, Y, ldy);
    const int per = qb_gemm_f16_block_tiles(ntiles, split, kper, n, ctx->sms);
    if (per > 1) {
        grid.x = ntiles / per;
        // Copied in 16-byte pieces, where X starts on such: three blocks per SM instead of two, but a round of them takes a tenth longer (and
        // a block on its own a twentieth over a long k). So not where both forms take as many rounds and the last one is fairly full, unless X
        // no longer stays in L2 beside the rest (from 12 MB on, taken from four buffers in turn). X gathered against copied, us: 96 x 5120 in 5 splits,
        // 160 rows (25 blocks) 8.1 and 7.8, 512 9.9 and 8.3, 955 (150) 10.4 and 10.0, 1024 (160) 10.8 and 11.0, 2048 (320) 23.7 and 12.3; 160
        // outputs, 1024 rows (800) 19.8 and 12.6; 384 x 2048 in 2 splits, 640 rows (160) 10.5 and 11.0, 1184 (296) 10.8 and 12.0, 1408 (352)
        // 18.0 and 11.9; in 4 of 256, 832 rows (208) 5.1 and 4.9, 955 (240) 5.1 and 5.3; 768 x 2048 in 2, 1024 rows (512) 19.3 and 20.0; 768 x
        // 5120 in one, 160 rows (40) 28.8 and 30.1, 333 (88) 36.9 and 31.5.
        const long long blocks = (long long)grid.x * grid.y * grid.z, sms = ctx->sms;
        const bool full = (blocks <= 2 * sms && 20 * blocks > (kper >= 1024 ? 21 : 30) * sms) || (blocks <= 4 * sms && 5 * blocks > 17 * sms) ||
                          (3 * blocks <= sms && kper >= 4096);
        const bool whole = ((uintptr_t)x & 15) == 0 && !(full && (long long)n * K <= 6 << 20);  // (K and kper are multiples of 16)
#define QB_WIDE(T)                                                                                                                    \
    return whole ? launch(ctx, gemm_f16_staged_kernel<T>, grid, dim3(128), StagedCfg<T>::SMEM, st, w, x, xrows, K, ntiles, n, kper, Y, ldy) \
                 : launch(ctx, gemm_f16_wide_kernel<T>, grid, dim3(128), 0, st, w, x, xrows, K, ntiles, n, kper, Y, ldy)
        if (per == 6) QB_WIDE(6);
        if (per == 4) QB_WIDE(4);
        QB_WIDE(2);
#undef QB_WIDE
    }
    return launch(ctx, gemm_f16_plain_kernel<4>, grid, dim3(128), 0, st, w, x, xrows, K, ntiles, n, kper, Y, ldy);
}
