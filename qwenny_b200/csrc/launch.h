// One launch helper for every kernel: cudaLaunchKernelEx with the programmatic-dependent-launch attribute when the
// context asks for it. Every grid of the library calls pdl_wait() before it ends and before it touches anything that an earlier kernel
// of the stream may still write, so a grid's end means the end of all before it, whichever launches carry the attribute.
//
// What a kernel reads BEFORE its wait is therefore weights, and the step's token lists, which no kernel writes. A kernel that lets
// its dependents start at its first line says nothing about the kernels before it: several small ones in a row can all be resident
// at once, so "written by an earlier step" is not enough for an early read. It is enough behind a kernel that waits first and lets
// its dependents start only then (mark_seen and embed, the first of a step): whatever starts after that one starts after the
// end of everything before it. The model runner reads the slots of its one-launch mixers and the older cache entries early on that
// ground (qb_delta_mixer_as, qb_attn_decode_as: ahead = 1).
#pragma once
#include "ctx.h"

namespace qb {

template <typename... KArgs, typename... Args>
static inline int launch(const qb_ctx* ctx, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t st, Args... args) {
    if (int rc = prepare_kernel(ctx->device, (const void*)kern, (int)smem)) return rc;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = grid;
    lc.blockDim = block;
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = ctx->pdl ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&lc, kern, static_cast<KArgs>(args)...);
    return e == cudaSuccess ? QB_OK : (int)e;
}

}  // namespace qb
