// What the tcgen05 kernels share (the W4A16 products and the prompt attention; one block or a pair of blocks per tile):
// descriptors, the product / commit / tensor-memory wrappers, arrivals across a pair, and the dealing of (tile, k block) lists.
#pragma once
#include <cuda.h>
#include "common.cuh"

namespace qb {
namespace tc {

// instruction descriptor of tcgen05.mma kind::f16, M = 256 (a pair of blocks), N = n: D f32 (bits 4-5 = 1), A and B f16
// (0), both K-major (0), N >> 3 at bits 17-22, M >> 4 at bits 24-28
__device__ __forceinline__ uint32_t idesc_pair(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24); }

// shared-memory matrix descriptor of a K-major operand with the 128-byte swizzle: start address >> 4, leading byte
// offset 1 (unused with a swizzle), stride byte offset 1024 >> 4 (between 8-row groups), descriptor version 1
// (bit 46), layout type 2 = SWIZZLE_128B (bits 61-63)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
            "r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::
            "r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];\n" ::"l"(map), "r"(x), "r"(y), "r"(smem_u32(src))
                 : "memory");
}
// ---- The products and their commits are issued by WHOLE WARPS: every lane walks the loop and elect.sync picks the one that issues.
// A tcgen05.mma takes its addresses and descriptors from uniform registers; in a branch that one lane takes the compiler moves
// them there one by one, and the issue, 70 to 270 cycles a product, hid what the tensor core takes: a product of M = 128 takes 34
// cycles (N = 64) or 66 (N = 128) with A from tensor memory, 50 or 66 with A from shared memory, issued so (the 40-row MLP: 87.0 ->
// 84.7 us).
#define QB_ELECT ".reg .pred q;\nelect.sync _|q, 0xffffffff;\n"
template <int CTAS>
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t id, uint32_t accumulate) {
    if (CTAS == 1)
        asm volatile("{\n.reg .pred p;\n" QB_ELECT "setp.ne.b32 p, %4, 0;\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
                     "r"(a_tmem), "l"(bdesc), "r"(id), "r"(accumulate)
                     : "memory");
    else
        asm volatile("{\n.reg .pred p;\n" QB_ELECT "setp.ne.b32 p, %4, 0;\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d_tmem),
                     "r"(a_tmem), "l"(bdesc), "r"(id), "r"(accumulate)
                     : "memory");
}
template <int CTAS>
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t id, uint32_t accumulate) {
    if (CTAS == 1)
        asm volatile("{\n.reg .pred p;\n" QB_ELECT "setp.ne.b32 p, %4, 0;\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
                     "l"(adesc), "l"(bdesc), "r"(id), "r"(accumulate)
                     : "memory");
    else
        asm volatile("{\n.reg .pred p;\n" QB_ELECT "setp.ne.b32 p, %4, 0;\n@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
                     "l"(adesc), "l"(bdesc), "r"(id), "r"(accumulate)
                     : "memory");
}
// a value that all lanes share, in a uniform register (the compiler does not know it of what comes from shared memory or from a
// loop over a block's share, and would move it there product by product)
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
// four products over consecutive 16-wide steps of k: A 8 tensor-memory columns (or 32 bytes of its 128-byte rows), B 32 bytes of
// its 128-byte rows further each time; the first overwrites the accumulator where `accumulate` is 0
template <int CTAS>
__device__ __forceinline__ void umma_ts4(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t id, uint32_t accumulate) {
#pragma unroll
    for (int i = 0; i < 4; i++) umma_ts<CTAS>(d_tmem, a_tmem + 8 * i, bdesc + 2 * i, id, i ? 1u : accumulate);
}
template <int CTAS>
__device__ __forceinline__ void umma_ss4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t id, uint32_t accumulate) {
#pragma unroll
    for (int i = 0; i < 4; i++) umma_ss<CTAS>(d_tmem, adesc + 2 * i, bdesc + 2 * i, id, i ? 1u : accumulate);
}
// one block (M = 128): instruction descriptor
__device__ __forceinline__ constexpr uint32_t idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24); }
// arrives on the barrier once the products issued so far have completed; over a pair, on the barrier at this offset in both blocks
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("{\n" QB_ELECT "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void umma2_commit(uint64_t* bar) {
    asm volatile("{\n" QB_ELECT
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}\n" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}
// a bounded wait of a whole warp: one answer in all lanes
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); }
// arrive on the first block's barrier. The scopes are the default ones: what is handed over lives in tensor memory
// (tcgen05.wait::st and fence::before_thread_sync come first) or was written for the tensor core's async proxy (a TMA copy, or
// stores behind fence.proxy.async); a release at cluster scope here costs a memory barrier of about a microsecond per
// stage and warp, which made the product 1.7 times slower.
__device__ __forceinline__ void mbar_arrive_at(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(addr) : "memory");
}
// a 16 x 16 block of halves per k16 step, four steps: lane (g, t) holds rows g and g + 8 of column pairs t and t + 4 of each
__device__ __forceinline__ void tmem_st_16x128_x8(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(taddr), "r"(r[0]),
        "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// A list of `iters` (tile, k block) pairs dealt to g blocks (or pairs of blocks) in equal contiguous shares: share b is [start(b),
// start(b + 1)), start(b) = floor(iters b / g). In 32 bits: the divisions are on every role's way to its first stage and to a cut
// tile's ticket, and a 64-bit one is a subroutine of hundreds of cycles (40 rows of 5120 x 6144
// 15.9 -> 15.0 us, 333 rows with zero points 36.8 -> 36.2).
struct Shares {
    int q, r, g, iters;  // iters = q g + r
    __device__ Shares(int iters_, int g_) : q(iters_ / g_), r(iters_ % g_), g(g_), iters(iters_) {}
    __device__ int start(int b) const { return q * b + r * b / g; }  // (r and b are below g, the number of SMs)
    __device__ int of(int it) const {  // the share that holds it: an estimate, then to the place
        int b = min((int)(((float)it + 0.5f) * (float)g / (float)iters), g - 1);
        while (b + 1 < g && start(b + 1) <= it) b++;
        while (b > 0 && start(b) > it) b--;
        return b;
    }
};

// A pair's work as a list of segments (tile, k blocks [kb0, kb1)); every role of both blocks walks the same list.
// SHARES: equal contiguous shares of the (tile, k block) list, cut between units of `unit` k blocks (1, or nkb: whole tiles); otherwise
// pair b takes the whole tiles b, b + grid, ...
template <bool SHARES>
struct Walk {
    int tiles, nkb, G, b, j = 0;
    int it, it1;
    __device__ Walk(int iters, int tiles_, int nkb_, int G_, int b_, int unit = 1) : tiles(tiles_), nkb(nkb_), G(G_), b(b_) {
        const Shares s(iters / unit, G);
        it = SHARES ? s.start(b) * unit : 0;
        it1 = SHARES ? s.start(b + 1) * unit : 0;
    }
    __device__ bool next(int& tile, int& kb0, int& kb1) {
        if (!SHARES) {
            tile = j * G + b; kb0 = 0; kb1 = nkb; j++;
            return tile < tiles;
        }
        if (it >= it1) return false;
        tile = it / nkb; kb0 = it - tile * nkb; kb1 = min(nkb, kb0 + (it1 - it));
        it += kb1 - kb0;
        return true;
    }
    // the pairs that hold the parts of a tile cut by this walk: the first one and how many
    __device__ void parts_of(int tile, int& first, int& parts) const {
        const Shares s(tiles * nkb, G);
        first = s.of(tile * nkb);
        parts = s.of((tile + 1) * nkb - 1) - first + 1;
    }
};

}  // namespace tc
}  // namespace qb
