// Context creation and the error word.
#include "ctx.h"
#include "common.cuh"
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <tuple>

namespace qb {

namespace {
std::mutex g_attr_mutex;
std::map<std::pair<int, const void*>, int> g_attr_smem;
std::map<std::tuple<int, const void*, int>, std::array<int, 9>> g_attr_clusters;
}  // namespace

bool AttrCache::need(int device, const void* kern, int smem) {
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    auto it = g_attr_smem.find({device, kern});
    if (it == g_attr_smem.end()) {
        g_attr_smem[{device, kern}] = smem;
        return true;
    }
    if (it->second >= smem) return false;
    it->second = smem;
    return true;
}

int* AttrCache::clusters(int device, const void* kern, int smem) {
    std::lock_guard<std::mutex> lock(g_attr_mutex);
    return g_attr_clusters.try_emplace(std::make_tuple(device, kern, smem), std::array<int, 9>{}).first->second.data();
}

AttrCache& attr_cache() {
    static AttrCache c;
    return c;
}

int prepare_kernel(int device, const void* kern, int smem) {
    if (!attr_cache().need(device, kern, smem)) return QB_OK;
    // Every kernel asks for the same L1 / shared-memory split (all shared): the big streaming kernels need it, and an
    // SM whose split has to change between two kernels drains first, which would undo the overlap of neighbours.
    QB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    if (smem > 48 * 1024) QB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return QB_OK;
}

// Clears words of a new allocation before anything can use them: on a stream that waits for no other (a context's stream need not
// wait for the default one, and creation need not wait for what runs there). One stream per device, kept: creating
// one each time took a third of a context's creation (500 us, 390 without).
static cudaError_t zero_now(int device, void* p, size_t bytes) {
    static std::mutex m;
    static std::map<int, cudaStream_t> streams;
    std::lock_guard<std::mutex> lock(m);
    cudaStream_t& st = streams[device];
    for (int fresh = st == nullptr;; fresh = 1) {
        cudaError_t e = fresh ? cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) : cudaSuccess;
        if (e == cudaSuccess) e = cudaMemsetAsync(p, 0, bytes, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e == cudaSuccess) return e;
        (void)cudaGetLastError();
        st = nullptr;
        if (fresh) return e;  // (a kept stream may have gone with a reset of its device: once more with a new one)
    }
}

}  // namespace qb

extern "C" {

// Host-only check of the per-device attribute bookkeeping (no CUDA call): 0 when two devices each get their own
// opt-in for the same kernel, a larger request on one device asks again there only, and repeats ask for nothing.
int qb_attr_cache_selftest(void) {
    static int k1, k2;  // stand-ins for two kernels
    qb::AttrCache& c = qb::attr_cache();
    const int d0 = 1000, d1 = 1001;  // device numbers no real GPU has
    if (!c.need(d0, &k1, 100000)) return 1;
    if (c.need(d0, &k1, 100000)) return 2;
    if (c.need(d0, &k1, 50000)) return 3;
    if (!c.need(d1, &k1, 100000)) return 4;   // the second device has not been opted in by the first one's call
    if (!c.need(d0, &k2, 0)) return 5;
    if (c.need(d0, &k2, 0)) return 6;
    if (!c.need(d0, &k1, 200000)) return 7;
    if (c.need(d1, &k1, 100000)) return 8;
    int* a = c.clusters(d0, &k1, 4096);
    a[3] = 17;
    if (c.clusters(d1, &k1, 4096)[3] != 0 || c.clusters(d0, &k1, 4096)[3] != 17) return 9;
    return 0;
}

const char* qb_version(void) { return "qwenny_b200 0.1 (sm_100a)"; }

int qb_create(int device, qb_ctx** out) {
    if (!out) return QB_ERR_ARG;
    QB_CUDA(cudaSetDevice(device));
    int sms = 0;
    QB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    // One allocation: the words that must be zero (counters, error word, tickets) and one area that the skinny products, the
    // prompt-sized ones and the delta rule use in turn (none leaves anything there for a later call, and every kernel waits
    // for the one before it before it writes there). Calls allocate nothing, so that they can be captured and a host may give all
    // other memory away; where only a part fits, the context does without the rest.
    // The split-K partials' largest user is a 16-row product, [n/64][nsplit][2][4][32] float4; 32 MiB covers
    // n * nsplit up to 2^17 * 8 (the 27B shapes need under 6 MiB).
    const size_t ncounters = 1 << 14, err_at = ncounters * sizeof(int), tickets_at = err_at + 256;
    // The area starts on a 2 MiB page of its own (behind the tickets on the same page the 17 to 64-row products took 1 to 3 %
    // longer: 5120 x 17408, 40 rows 33.0 and 33.7 us).
    const size_t zeroed = tickets_at + QB_TC_TICKETS * sizeof(int), scratch_at = 2u << 20, scratch_bytes = 32u << 20;
    static_assert((1 << 14) * sizeof(int) + 256 + QB_TC_TICKETS * sizeof(int) <= (2u << 20), "the words come before the area");
    char* b = nullptr;
    // The delta rule's chunks: those of any step (219 MB), those of 2048 tokens of one sequence (140 MB), of 784 (52 MB); no chunks (39 MB); without
    // the prompt-sized products' part as well.
    const int chunks[4] = {QB_DELTA_CHUNKS, 32, 12, 0};
    int got = 0;
    auto bytes = [&](int i) {
        return scratch_at + (i == 4 ? scratch_bytes : std::max({scratch_bytes, qb_tc_part_bytes(sms), qb_delta_tp_bytes(chunks[i])}));
    };
    for (; got < 4 && cudaMalloc(&b, bytes(got)) != cudaSuccess; got++) (void)cudaGetLastError();
    if (got == 4) QB_CUDA(cudaMalloc(&b, bytes(4)));
    const cudaError_t e = qb::zero_now(device, b, zeroed);
    if (e != cudaSuccess) {
        cudaFree(b);
        return (int)e;
    }
    qb_ctx* c = new qb_ctx();
    c->device = device;
    c->sms = sms;
    c->block = b;
    c->counters = (int*)b;
    c->ncounters = ncounters;
    c->err = (int*)(b + err_at);
    c->form = c->err + 16;
    c->scratch = (float*)(b + scratch_at);
    c->scratch_bytes = scratch_bytes;
    if (got < 4) {
        c->tc_tickets = (int*)(b + tickets_at);
        c->tc_part = c->scratch;
        c->delta_tp = c->scratch;
        c->delta_chunks = chunks[got];
    }
    *out = c;
    return QB_OK;
}

void qb_destroy(qb_ctx* c) {
    if (!c) return;
    cudaFree(c->block);
    delete c;
}

int qb_scratch_forget(qb_ctx* c) {
    if (!c) return QB_ERR_ARG;
    c->tc_part = nullptr; c->tc_tickets = nullptr; c->delta_tp = nullptr;
    c->delta_chunks = 0;
    return QB_OK;
}

int qb_scratch_chunks(qb_ctx* c, int chunks) {
    if (!c || chunks < 0 || chunks > c->delta_chunks) return QB_ERR_ARG;
    c->delta_chunks = chunks;
    return QB_OK;
}

int qb_device_error(qb_ctx* c) {
    if (!c) return QB_ERR_ARG;
    int v = 0;
    QB_CUDA(cudaDeviceSynchronize());
    QB_CUDA(cudaMemcpy(&v, c->err, sizeof(int), cudaMemcpyDeviceToHost));
    if (v) QB_CUDA(cudaMemset(c->err, 0, sizeof(int)));
    return v;
}

int qb_sm_count(const qb_ctx* c) { return c ? c->sms : 0; }

int qb_set_pdl(qb_ctx* c, int on) {
    if (!c) return QB_ERR_ARG;
    c->pdl = on != 0;
    return QB_OK;
}

}  // extern "C"


namespace qb {
EncodeTiled encode_tiled() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) == cudaSuccess &&
            qr == cudaDriverEntryPointSuccess)
            fn = (EncodeTiled)p;
    }
    return fn;
}
}  // namespace qb

// ---------------------------------------------------------------------------------------------------------------
// Test of the waits' way out: a block waits (with the library's bounded wait, here with a short poll limit) on an
// mbarrier that nothing ever arrives on; the wait runs out, the block records code 99 in the context's error word and
// returns. The host reads it with qb_device_error and the context stays usable.
namespace qb {
__global__ void wait_probe_kernel(int* err, uint32_t limit) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) ok = mbar_wait(&bar, 0, limit);
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok && threadIdx.x == 0) atomicExch(err, 99);
}
}  // namespace qb

extern "C" int qb_wait_probe(qb_ctx* ctx, void* stream, unsigned limit) {
    if (!ctx || limit == 0 || limit > (1u << 20)) return QB_ERR_ARG;
    qb::wait_probe_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(ctx->err, limit);
    return (int)cudaGetLastError();
}
