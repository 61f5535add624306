/* Measurement-only entry points of libqwenny_b200.so: exported for the timing and profiling drivers, not part of the
 * public ABI (include/qwenny_b200.h) and not for a serving host. */
#pragma once
#include "ctx.h"
#ifdef __cplusplus
extern "C" {
#endif
/* Fixes the tile shape (cg x kg consumer warps), ring depth and blocks per SM of the next qb_marlin_gemm calls on the
 * context; zeros restore the built-in choice. ctas < 0: as -ctas, and stream-K only; nstages < 0: as -nstages, and no
 * tensor-core path for more than 16 rows. */
int qb_marlin_tune(qb_ctx* ctx, int cg, int kg, int nstages, int ctas_per_sm);
/* The following qb_marlin_gemm calls write per-block timestamps (ns of the global timer: start, first stage landed,
 * last stage consumed, end; 4 x 1024 int64 per call) into consecutive slices of `buf`; NULL switches it off. */
int qb_marlin_trace(qb_ctx* ctx, long long* buf);
/* mode 1 makes the products' consumers release every stage unread, so a launch times the copy pipeline alone (its
 * results are meaningless); mode 2 (tests) makes the copy warp leave out its second stage and cuts the consumers' wait
 * to 1024 polls: their wait runs out, they record error 2 and walk on, the kernel ends; 0 restores the product. */
int qb_marlin_probe(qb_ctx* ctx, int mode);
/* Tests: the next n graph captures of the model report out of memory without touching the GPU. */
struct qb_model;
int qb_model_fail_captures(struct qb_model* m, int n);
/* Host-only checks of the step-graph cache policy (with fakes behind its hooks) and of the per-device
 * kernel-attribute bookkeeping; 0 when they hold. */
int qb_graph_cache_selftest(void);
int qb_attr_cache_selftest(void);
/* The 16-row tiles that a block of qb_gemm_f16_plain multiplies its 32 rows by, on a part with `sms` SMs. */
int qb_gemm_f16_block_tiles(int ntiles, int splits, int kper, int n, int sms);
/* Host only (host pointers): whether a prompt attention of more than 1664 keys and one key split runs on pairs of blocks (1) or as a
 * block per two tiles (0) on a part with `sms` SMs. qb_marlin_tune with ctas_per_sm 1002 / 1003 forces blocks / pairs. */
int qb_attn_tiles_on_pairs(const int* h_ptile, int ntile, const int* h_tok_slot, const int* h_tok_pos, int sms);
/* Host only: whether qb_attn_decode deals a step's splits out to a block per SM (1) or gives each a block (0), and all that the attention
 * launches of a step are chosen by beside its counts (ndseg or ntile 0: none of that kind), for the key of a captured step. */
int qb_attn_dec_dealt(int ndseg, int max_keys, int sms);
int qb_attn_step_form(int ndseg, int dec_keys, int ntile, int tile_keys, int sms);
/* Tests: the context goes on as one that was created where the prompt-sized kernels' scratch did not fit. */
int qb_scratch_forget(qb_ctx* ctx);
/* .. as one where the delta rule's tiles of only so many chunks fit (0: none). */
int qb_scratch_chunks(qb_ctx* ctx, int chunks);
/* Tests: one block waits on an mbarrier that nothing arrives on, with the library's bounded wait cut to `limit` polls
 * (at most 2^20); the wait runs out and the context's error word reads 99 (qb_device_error). */
int qb_wait_probe(qb_ctx* ctx, void* stream, unsigned limit);
#ifdef __cplusplus
}
#endif
