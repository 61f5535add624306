// The library context: what the reference's Gemm::load allocates once per model (src/cuda/core.rs:437-464) — the SM
// count and the scratch its blocks reduce through — plus the device error word of the bounded waits.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/qwenny_b200.h"

struct qb_ctx {
    int device = 0;
    int sms = 0;
    // split-K partial sums of the skinny int4 products (L2 resident) and the per-64-output arrival tickets
    float* scratch = nullptr;
    size_t scratch_bytes = 0;
    int* counters = nullptr;
    size_t ncounters = 0;
    int* err = nullptr;  // device word
    int* form = nullptr; // two device words: the form of the prompt attention that the step under way takes, a counter of its work
    // The prompt-sized kernels' scratch, in one area with `scratch` (calls use it in turn) and one allocation with the rest
    // (`block`). A device with less room gets a context with fewer chunks, or without either part, whose calls take the
    // forms that need none.
    void* block = nullptr;
    float* tc_part = nullptr;   // partial tiles of the tensor-core W4A16 products' shares (sms x 256 KB)
    int* tc_tickets = nullptr;  // their tickets, two per tile (QB_TC_TICKETS, zero between launches)
    void* delta_tp = nullptr;   // the chunked delta rule's tiles per chunk, key head and value head (4.4 MB a chunk)
    int delta_chunks = 0;       // .. of so many chunks
    // measurement override of the GEMV plan (0: built-in choice)
    int tune_cg = 0, tune_kg = 0, tune_nstages = 0, tune_ctas = 0;
    bool no_cluster = false, no_tc = false;
    // programmatic dependent launch on the launches that support it
    bool pdl = false;
    int probe = 0;               // measurement: see qb_marlin_probe
    int early = 1;               // stages of weights the next skinny product requests before it waits for the kernel
                                 // before it (set by the caller that knows what that kernel is; see model.cu)
    long long* trace = nullptr;  // measurement: per-block timestamps of the next products
};

constexpr int QB_DELTA_CHUNKS = 50;     // the most chunks of a step of 2048 tokens (25 segments of 81)
constexpr int QB_TC_TICKETS = 1 << 17;  // two per tile of a tensor-core W4A16 product (256 outputs x 256 tokens each)
#define QB_CUDA(x)                         \
    do {                                   \
        cudaError_t e_ = (x);              \
        if (e_ != cudaSuccess) return (int)e_; \
    } while (0)

namespace qb {

// cuTensorMapEncodeTiled, resolved through the runtime (the library does not link the driver); null when unavailable
typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled();

// Kernel attributes (the opt-in to more than 48 KB of dynamic shared memory, the shared-memory carve-out) belong to the
// device that is current when cudaFuncSetAttribute runs, so what has been set is remembered per (device, kernel), not
// per process: a process that drives several GPUs opts every kernel in on each of them. AttrCache is the bookkeeping
// alone (no CUDA call), shared by all host threads behind one mutex.
class AttrCache {
  public:
    // true when `kern` on `device` has not yet been given at least `smem` bytes (or, smem == 0, has not been seen at
    // all); the new value is recorded, so the caller must then set the attribute
    bool need(int device, const void* kern, int smem);
    // the resident-cluster counts the driver reported for (device, kernel, shared memory), filled by the caller
    int* clusters(int device, const void* kern, int smem);
};
AttrCache& attr_cache();
// sets what `kern` needs on `device` (which must be current) before a launch with `smem` bytes of dynamic shared memory
int prepare_kernel(int device, const void* kern, int smem);

}  // namespace qb

// the many-tile prompt attention on tcgen05 (attn_prefill_tc.cu); reached through qb_attn_prefill
int qb_attn_prefill_tc_launch(qb_ctx* ctx, cudaStream_t st, const float* q, const void* kc, const void* vc, const float* ks,
                              const float* vs, const int* ptile, int ntile, const int* tok_slot, const int* tok_pos,
                              int cap, float* out, void* mix_f16, const int* on_pairs);
int qb_attn_prefill_short_launch(qb_ctx* ctx, cudaStream_t st, const float* q, const void* kc, const void* vc, const float* ks,
                                 const float* vs, const int* ptile, int ntile, const int* tok_slot, const int* tok_pos,
                                 int cap, float* out, void* mix_f16, int* on_pairs);  // short contexts, short runs (attn_prefill_short.cu)
// qb_attn_prefill for a caller that knows qb_attn_tiles_on_pairs of its tiles (as: 0 or 1; -1: not known), and its launches
int qb_attn_prefill_as(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks, const float* vs,
                       const int* ptile, const int* tok_slot, const int* tok_pos, int cap, int ntile, int max_keys, float* part_ml,
                       float* part_acc, float* out, void* mix_f16, int as);
int qb_attn_prefill_launches(const qb_ctx* ctx, int ntile, int max_keys, int as);
// qb_delta_mixer for a caller that vouches (ahead = 1) for the slots: between this call and the last kernel that wrote
// them lies one whose blocks all wait for the kernels before it before they let the next one start. The slots' metadata, state
// and bank are then read ahead of the kernel before; the public entry point (ahead = 0) reads them behind it.
int qb_delta_mixer_as(qb_ctx* ctx, void* stream, const float* p, int splits, int n, const float* ba, int ba_splits, const float* cw,
                      const float* a_log, const float* dt_bias, const float* nw, float* mem, long long sst, int* meta, float* out, void* y,
                      const int* seg_start, const int* seg_len, const int* seg_slot, const int* seg_pos0, int segs, int ahead);
// the kernels that qb_delta_rule launches for a step of n tokens
int qb_delta_rule_launches(const qb_ctx* ctx, int n, int segs);
// qb_attn_decode for a caller that vouches in the same way (ahead = 1) for the cache entries of earlier steps
int qb_attn_decode_as(qb_ctx* ctx, void* stream, const float* q, const void* kc, const void* vc, const float* ks, const float* vs,
                      const int* dseg, const int* dtok, const int* dkeys, const int* tok_slot, const int* tok_pos, int cap, int ndseg,
                      int ndec, int dmax, int max_keys, float* part_ml, float* part_acc, float* out, void* mix_f16, int ahead);
// the prompt-sized W4A16 product on tcgen05 (w4a16_gemm_tc.cu); reached through qb_marlin_gemm for more than 64 rows and
// qb_marlin_gemm_z (zp: S carries the offsets' table after the scales) for more than 16
int qb_gemm_tc_launch(qb_ctx* ctx, cudaStream_t st, const void* X, const void* B, void* Y, const void* S, int m, int n,
                      int k, int row0, int epi, int zp);
// bytes of the prompt-sized kernels' scratch: tc_part on a part with `sms` SMs, delta_tp
size_t qb_tc_part_bytes(int sms);
size_t qb_delta_tp_bytes(int chunks);
// the product for 17 .. 64 rows (w4a16_gemm_mid.cu), symmetric matrices; reached through qb_marlin_gemm
int qb_gemm_mid_launch(qb_ctx* ctx, cudaStream_t st, const void* X, const void* B, void* Y, const void* S, int m, int n, int k,
                       int row0, int epi, const int* xrows, unsigned long long* keys, int n_valid);
int qb_gemm_mid_gathers(const qb_ctx* ctx, int m, int k);  // whether it can take gathered rows: they are copied together first
// the kernels that qb_marlin_gemm launches for m gathered rows
int qb_marlin_gathered_launches(const qb_ctx* ctx, int m, int k);
