// fa_api.cu — context lifecycle, argument validation and the C entry points of
// libfa_sm120.so (the ABI of goml's libs/fa_sm120/src/fa_ctx.cu:55-235).
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <new>

#include "../../include/fa_sm120.h"
#include "fa_fwd_sm100.h"

namespace {

// While it lives, a stream capture that another thread has begun does not forbid this thread's allocations and frees (they are
// on streams that are not being captured).
struct BesideCaptures {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// What all contexts of one GPU share: the stream-ordered pool their scratch is drawn from (freed blocks stay cached in it,
// so steady-state calls do not reach the driver allocator) and, per stream, scratch kept between calls.  Work on one
// stream is ordered, so consecutive calls there can use the same buffers and a call costs no allocation.  Kept: small
// buffers only (a large one is drawn from the pool per call, where the 2 us do not show), for a fixed number of streams;
// a stream that has not called for KEPT_AGE calls of others, or is gone, gives its place and buffers up to a new one.
// Streams are told apart by their id, which the driver never reuses.  Calls that are being captured into a graph do not
// use it: a graph may be replayed on any stream.  Created with the first context of the GPU, released with the last.
struct Kept {
    unsigned long long stream_id = 0;
    uint8_t* scratch = nullptr;    // whatever the call writes before it reads it
    size_t scratch_bytes = 0;
    uint32_t* flags = nullptr;     // zero when allocated, afterwards values of earlier epochs
    size_t flag_words = 0;
    uint32_t epoch = 0;
    uint32_t* zeros = nullptr;     // words that every call finds zero and leaves zero
    size_t zero_words = 0;
    bool used = false;
    int users = 0;                 // calls that hold the slot or wait for it
    unsigned long long last = 0;   // number of the slot's last call
    std::mutex busy;               // held from the look-up until the kernels that use the buffers are on the stream: calls on one
                                   // stream take turns, calls on others do not wait for them
    cudaEvent_t done = nullptr;    // recorded behind every call: the stream itself may be gone when the buffers are given back

    // gives the buffers back behind the slot's last call, without waiting for it here; `s` is a stream of the library's own
    void give_back(cudaStream_t s) {
        BesideCaptures relaxed;
        if (done) {
            cudaStreamWaitEvent(s, done, 0);
            cudaEventDestroy(done);
        }
        if (scratch) cudaFreeAsync(scratch, s);
        if (flags) cudaFreeAsync(flags, s);
        if (zeros) cudaFreeAsync(zeros, s);
        scratch = nullptr; flags = zeros = nullptr; done = nullptr;
        scratch_bytes = flag_words = zero_words = 0;
        used = false;
    }
};
constexpr int MAX_DEVICES = 64;
constexpr int KEPT_STREAMS = 8;
// well above KEPT_STREAMS: more streams than places that call in turn do not chase each other's buffers
constexpr unsigned long long KEPT_AGE = 64;
constexpr size_t KEPT_SCRATCH_MAX = (size_t)64 << 20;
constexpr size_t KEPT_WORDS_MAX = (size_t)1 << 20;
struct DeviceScratch {
    std::mutex lock;               // of the members here and of which slot belongs to which stream; never held over a launch
    int contexts = 0;
    cudaMemPool_t pool = nullptr;
    cudaStream_t reaper = nullptr; // where kept buffers are given back
    unsigned long long calls = 0;
    Kept kept[KEPT_STREAMS];

    cudaError_t acquire(int dev) {
        std::lock_guard<std::mutex> g(lock);
        if (contexts == 0) {
            BesideCaptures relaxed;
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.handleTypes = cudaMemHandleTypeNone;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaError_t e = cudaMemPoolCreate(&pool, &props);
            if (e == cudaSuccess && (e = cudaStreamCreateWithFlags(&reaper, cudaStreamNonBlocking)) != cudaSuccess) cudaMemPoolDestroy(pool);
            if (e != cudaSuccess) return e;
            unsigned long long keep = ~0ull;  // keep freed scratch cached in the pool
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        }
        contexts++;
        return cudaSuccess;
    }
    void release(int dev) {
        std::lock_guard<std::mutex> g(lock);
        if (--contexts > 0) return;
        // All of it is ordered behind the work that uses it and waits for nothing: kernels may still run, and a synchronising
        // call would break a capture that some other thread has begun.
        BesideCaptures relaxed;
        int cur = -1;
        cudaGetDevice(&cur);
        if (cur != dev) cudaSetDevice(dev);
        for (Kept& k : kept) k.give_back(reaper);
        cudaMemPoolDestroy(pool);      // pending frees complete first (stream-ordered)
        cudaStreamDestroy(reaper);     // likewise
        if (cur >= 0 && cur != dev) cudaSetDevice(cur);
        pool = nullptr;
        reaper = nullptr;
    }
    // the slot of a stream, or nullptr when all belong to streams that still call; leave() follows
    Kept* enter(unsigned long long stream_id) {
        std::lock_guard<std::mutex> g(lock);
        calls++;
        Kept* mine = nullptr;
        Kept* oldest = nullptr;    // a vacant slot, or the one unused for longest
        for (Kept& k : kept) {
            if (k.used && k.stream_id == stream_id) { mine = &k; break; }
            if (k.users == 0 && (!oldest || (oldest->used && (!k.used || k.last < oldest->last)))) oldest = &k;
        }
        if (!mine && oldest && (!oldest->used || calls - oldest->last > KEPT_AGE)) {
            if (oldest->used) oldest->give_back(reaper);
            mine = oldest;
            mine->used = true;
            mine->stream_id = stream_id;
        }
        if (mine) {
            mine->users++;
            mine->last = calls;
        }
        return mine;
    }
    void leave(Kept* k) {
        std::lock_guard<std::mutex> g(lock);
        k->users--;
    }
};
DeviceScratch g_scratch[MAX_DEVICES];

}  // namespace

struct fa_ctx {
    int device;
    int cc_major, cc_minor;
    bool arch_ok;
    DeviceScratch* shared;   // nullptr on an unsupported GPU
    char last_err[256];
};

namespace {

void set_err(fa_ctx_t* c, const char* fmt, const char* a = "", const char* b = "") {
    if (c) snprintf(c->last_err, sizeof(c->last_err), fmt, a, b);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Checks shared by every forward entry.  `who` prefixes messages.
fa_status_t validate(fa_ctx_t* c, const char* who, const void* q, const void* k, const void* v, const void* o,
                     int bh, int sl, int hd, int causal, int window, const void* l_out = nullptr) {
    if (!c->arch_ok || !c->shared) { set_err(c, "%s: context was created on an unsupported GPU", who); return FA_ERR_UNSUPPORTED_ARCH; }
    if (!q || !k || !v || !o) { set_err(c, "%s: null pointer in q/k/v/o", who); return FA_ERR_INVALID_ARG; }
    if (bh <= 0 || sl <= 0) { set_err(c, "%s: bh/sl must be > 0", who); return FA_ERR_INVALID_ARG; }
    if (hd != 64 && hd != 128) { set_err(c, "%s: head_dim must be 64 or 128", who); return FA_ERR_UNSUPPORTED_HD; }
    if (window < 0 || window > sl) { set_err(c, "%s: window must be in [0, seq_len]", who); return FA_ERR_INVALID_ARG; }
    if (causal != 0 && causal != 1) { set_err(c, "%s: causal must be 0 or 1", who); return FA_ERR_INVALID_ARG; }
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) {
        set_err(c, "%s: q/k/v/o must be 16-byte aligned", who);
        return FA_ERR_INVALID_ARG;
    }
    if (reinterpret_cast<uintptr_t>(l_out) & 3) { set_err(c, "%s: l_out must be 4-byte aligned", who); return FA_ERR_INVALID_ARG; }
    if (fa_dispatch_select(bh, sl, hd, causal, window) == FA_KERNEL_NONE) {
        set_err(c, "%s: no kernel matches this configuration", who);
        return FA_ERR_UNSUPPORTED_SHAPE;
    }
    return FA_OK;
}

// One call's scratch: the stream's kept buffers where they serve, else blocks drawn from the pool for this call.
struct Scratch {
    void* ptr = nullptr;
    uint32_t* flags = nullptr;   // nullptr: none kept for this stream (a capture, more streams than slots)
    uint32_t epoch = 0;
    uint32_t* zeros = nullptr;
    void* pooled[2] = {nullptr, nullptr};
    cudaStream_t stream = nullptr;
    DeviceScratch* owner = nullptr;
    Kept* slot = nullptr;
    std::unique_lock<std::mutex> lock;

    ~Scratch() {
        if (!slot) return;
        lock.unlock();
        owner->leave(slot);
    }

    // grows one kept buffer of a stream; a block that is replaced is released behind the kernels that use it
    template <typename T>
    static cudaError_t grow(cudaMemPool_t pool, T*& buf, size_t& have, size_t want, size_t least, bool zero, cudaStream_t s) {
        if (have >= want) return cudaSuccess;
        size_t n = least;
        while (n < want) n *= 2;
        if (buf) { cudaFreeAsync(buf, s); buf = nullptr; have = 0; }
        const size_t bytes = n * sizeof(T);
        void* p = nullptr;
        cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, pool, s);
        if (e != cudaSuccess) return e;
        if (zero && (e = cudaMemsetAsync(p, 0, bytes, s)) != cudaSuccess) { cudaFreeAsync(p, s); return e; }
        buf = static_cast<T*>(p);
        have = n;
        return cudaSuccess;
    }

    cudaError_t take(fa_ctx_t* c, cudaStream_t s, size_t bytes, size_t flag_words, size_t zero_words) {
        const cudaError_t e = take_from(c, s, bytes, flag_words, zero_words);
        if (e != cudaSuccess) give_back();
        return e;
    }
    cudaError_t take_from(fa_ctx_t* c, cudaStream_t s, size_t bytes, size_t flag_words, size_t zero_words) {
        stream = s;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        cudaError_t e = cudaStreamIsCapturing(s, &cap);
        if (e != cudaSuccess) return e;
        unsigned long long id = 0;
        if (cap == cudaStreamCaptureStatusNone && cudaStreamGetId(s, &id) == cudaSuccess) {
            Kept* k = c->shared->enter(id);
            if (k) {
                lock = std::unique_lock<std::mutex>(k->busy);
                owner = c->shared;
                slot = k;
                if (!k->done && (e = cudaEventCreateWithFlags(&k->done, cudaEventDisableTiming)) != cudaSuccess) return e;
                if (flag_words && flag_words <= KEPT_WORDS_MAX) {
                    const uint32_t* before = k->flags;
                    if ((e = grow(c->shared->pool, k->flags, k->flag_words, flag_words, 4096, true, s)) != cudaSuccess) return e;
                    if (k->flags != before) k->epoch = 0;
                    if (++k->epoch == 0) {   // 2^32 calls later the words hold every value again
                        if ((e = cudaMemsetAsync(k->flags, 0, k->flag_words * 4, s)) != cudaSuccess) return e;
                        k->epoch = 1;
                    }
                    flags = k->flags;
                    epoch = k->epoch;
                }
                if (zero_words && zero_words <= KEPT_WORDS_MAX) {
                    if ((e = grow(c->shared->pool, k->zeros, k->zero_words, zero_words, 4096, true, s)) != cudaSuccess) return e;
                    zeros = k->zeros;
                }
                if (bytes && bytes <= KEPT_SCRATCH_MAX) {
                    if ((e = grow(c->shared->pool, k->scratch, k->scratch_bytes, bytes, (size_t)1 << 20, false, s)) != cudaSuccess) return e;
                    ptr = k->scratch;
                }
            }
        }
        if (bytes && !ptr) {
            if ((e = cudaMallocFromPoolAsync(&pooled[0], bytes, c->shared->pool, s)) != cudaSuccess) return e;
            ptr = pooled[0];
        }
        if (zero_words && !zeros) {
            if ((e = cudaMallocFromPoolAsync(&pooled[1], zero_words * 4, c->shared->pool, s)) != cudaSuccess) return e;
            if ((e = fa_sm100::launch_clear_words(static_cast<uint32_t*>(pooled[1]), zero_words, s)) != cudaSuccess) return e;
            zeros = static_cast<uint32_t*>(pooled[1]);
        }
        return cudaSuccess;
    }
    // behind the call's kernels, or behind what a failed call has queued
    cudaError_t give_back() {
        cudaError_t r = slot && slot->done ? cudaEventRecord(slot->done, stream) : cudaSuccess;
        for (void*& p : pooled)
            if (p) {
                const cudaError_t e = cudaFreeAsync(p, stream);
                if (e != cudaSuccess) r = e;
                p = nullptr;
            }
        return r;
    }
};

fa_status_t run(fa_ctx_t* c, const char* who, const fa_sm100::LaunchArgs& a) {
    int cur = -1;
    cudaError_t e = cudaGetDevice(&cur);
    if (e != cudaSuccess) { set_err(c, "%s: cudaGetDevice: %s", who, cudaGetErrorString(e)); return FA_ERR_CUDA; }
    if (cur != c->device) {
        // one context serves the device it was created on; the caller keeps that device current
        set_err(c, "%s: the calling thread's current device differs from the context's device", who);
        return FA_ERR_INVALID_ARG;
    }
    if (fa_sm100::needs_no_scratch(a)) {
        e = fa_sm100::launch(a);
        if (e != cudaSuccess) { set_err(c, "%s: launch: %s", who, cudaGetErrorString(e)); return FA_ERR_CUDA; }
        return FA_OK;
    }
    fa_sm100::LaunchArgs b = a;
    Scratch ws;
    e = ws.take(c, a.stream, fa_sm100::workspace_bytes(a.bh, a.sl, a.hd), fa_sm100::v_flag_count(a.bh, a.sl), 0);
    if (e != cudaSuccess) {
        set_err(c, "%s: workspace allocation: %s", who, cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? FA_ERR_OOM : FA_ERR_CUDA;
    }
    b.v16_workspace = ws.ptr;
    b.v_flags = ws.flags;
    b.v_epoch = ws.epoch;
    e = fa_sm100::launch(b);
    const cudaError_t fe = ws.give_back();  // stream-ordered: released after the kernel
    if (e != cudaSuccess) { set_err(c, "%s: launch: %s", who, cudaGetErrorString(e)); return FA_ERR_CUDA; }
    if (fe != cudaSuccess) { set_err(c, "%s: workspace release: %s", who, cudaGetErrorString(fe)); return FA_ERR_CUDA; }
    return FA_OK;
}

}  // namespace

extern "C" {

fa_status_t fa_create(fa_ctx_t** ctx_out) {
    if (!ctx_out) return FA_ERR_INVALID_ARG;
    *ctx_out = nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return FA_ERR_CUDA;
    fa_ctx_t* c = new (std::nothrow) fa_ctx_t();
    if (!c) return FA_ERR_OOM;
    c->device = dev;
    c->last_err[0] = '\0';
    if (cudaDeviceGetAttribute(&c->cc_major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&c->cc_minor, cudaDevAttrComputeCapabilityMinor, dev) != cudaSuccess) {
        delete c;
        return FA_ERR_CUDA;
    }
    c->arch_ok = (c->cc_major == 10);
    c->shared = nullptr;
    if (c->arch_ok) {
        const cudaError_t pe = dev < MAX_DEVICES ? g_scratch[dev].acquire(dev) : cudaErrorInvalidDevice;
        if (pe != cudaSuccess) {
            snprintf(c->last_err, sizeof(c->last_err), "fa_create: cudaMemPoolCreate: %s", cudaGetErrorString(pe));
            *ctx_out = c;
            return FA_ERR_CUDA;
        }
        c->shared = &g_scratch[dev];
    }
    *ctx_out = c;  // returned even on an unsupported GPU so the caller can read the reason
    if (!c->arch_ok) {
        snprintf(c->last_err, sizeof(c->last_err),
                 "GPU compute capability %d.%d is not sm_100a (need 10.x).", c->cc_major, c->cc_minor);
        return FA_ERR_UNSUPPORTED_ARCH;
    }
    return FA_OK;
}

fa_status_t fa_destroy(fa_ctx_t* ctx) {
    if (ctx && ctx->shared) ctx->shared->release(ctx->device);
    delete ctx;
    return FA_OK;
}

const char* fa_version(void) { return "1.0.0+tcgen05-sm100a"; }

const char* fa_status_str(fa_status_t s) {
    switch (s) {
        case FA_OK: return "OK";
        case FA_ERR_INVALID_ARG: return "invalid argument";
        case FA_ERR_UNSUPPORTED_ARCH: return "unsupported GPU arch (need sm_100a)";
        case FA_ERR_UNSUPPORTED_HD: return "unsupported head_dim (need 64 or 128)";
        case FA_ERR_UNSUPPORTED_SHAPE: return "unsupported shape";
        case FA_ERR_CUDA: return "CUDA runtime error";
        case FA_ERR_OOM: return "out of memory";
        case FA_ERR_INTERNAL: return "internal error";
    }
    return "unknown";
}

const char* fa_last_cuda_error(fa_ctx_t* ctx) { return ctx ? ctx->last_err : ""; }

fa_status_t fa_forward_train(fa_ctx_t* ctx, const void* q, const void* k, const void* v, void* o, void* l_out,
                             int bh, int sl, int hd, int causal, int window, float scale, fa_stream_t stream) {
    if (!ctx) return FA_ERR_INVALID_ARG;
    fa_status_t s = validate(ctx, "fa_forward_train", q, k, v, o, bh, sl, hd, causal, window, l_out);
    if (s != FA_OK) return s;
    fa_sm100::LaunchArgs a{};
    a.q = q; a.k = k; a.v = v; a.o = o; a.lse = static_cast<float*>(l_out);
    a.bh = bh; a.sl = sl; a.hd = hd; a.causal = causal; a.window = window;
    a.scale = scale; a.v_descale = 1.0f;
    a.stream = reinterpret_cast<cudaStream_t>(stream);
    return run(ctx, "fa_forward_train", a);
}

fa_status_t fa_forward(fa_ctx_t* ctx, const void* q, const void* k, const void* v, void* o, int bh, int sl, int hd,
                       int causal, int window, float scale, fa_stream_t stream) {
    if (!ctx) return FA_ERR_INVALID_ARG;
    fa_status_t s = validate(ctx, "fa_forward", q, k, v, o, bh, sl, hd, causal, window);
    if (s != FA_OK) return s;
    fa_sm100::LaunchArgs a{};
    a.q = q; a.k = k; a.v = v; a.o = o; a.lse = nullptr;
    a.bh = bh; a.sl = sl; a.hd = hd; a.causal = causal; a.window = window;
    a.scale = scale; a.v_descale = 1.0f;
    a.stream = reinterpret_cast<cudaStream_t>(stream);
    return run(ctx, "fa_forward", a);
}

static fa_status_t forward_ex(fa_ctx_t* ctx, const fa_forward_args_t* g, float* o_amax, const char* who) {
    if (!ctx) return FA_ERR_INVALID_ARG;
    if (!g) { set_err(ctx, "%s: null argument block", who); return FA_ERR_INVALID_ARG; }
    fa_status_t s = validate(ctx, who, g->q, g->k, g->v, g->o, g->batch_heads, g->seq_len, g->head_dim,
                             g->causal, g->window, g->l_out);
    if (s != FA_OK) return s;
    fa_sm100::LaunchArgs a{};
    a.q = g->q; a.k = g->k; a.v = g->v; a.o = g->o; a.lse = static_cast<float*>(g->l_out);
    a.bh = g->batch_heads; a.sl = g->seq_len; a.hd = g->head_dim; a.causal = g->causal; a.window = g->window;
    a.scale = g->scale; a.v_descale = (g->v_descale == 0.0f) ? 1.0f : g->v_descale;
    a.scale_q_dev = g->scale_q_dev; a.scale_k_dev = g->scale_k_dev; a.scale_v_dev = g->scale_v_dev;
    a.stream = reinterpret_cast<cudaStream_t>(g->stream);
    a.o_amax = o_amax;
    return run(ctx, who, a);
}

fa_status_t fa_forward_ex(fa_ctx_t* ctx, const fa_forward_args_t* g) { return forward_ex(ctx, g, nullptr, "fa_forward_ex"); }

fa_status_t fa_forward_raise(fa_ctx_t* ctx, const fa_forward_args_t* g, float* o_amax) {
    if (ctx && (!o_amax || (reinterpret_cast<uintptr_t>(o_amax) & 3))) {
        set_err(ctx, "%s: o_amax must be a 4-byte aligned device pointer", "fa_forward_raise");
        return FA_ERR_INVALID_ARG;
    }
    return forward_ex(ctx, g, o_amax, "fa_forward_raise");
}

fa_status_t fa_decode(fa_ctx_t* ctx, const fa_decode_args_t* g) {
    const char* who = "fa_decode";
    if (!ctx) return FA_ERR_INVALID_ARG;
    if (!g) { set_err(ctx, "%s: null argument block", who); return FA_ERR_INVALID_ARG; }
    if (!ctx->arch_ok || !ctx->shared) { set_err(ctx, "%s: context was created on an unsupported GPU", who); return FA_ERR_UNSUPPORTED_ARCH; }
    if (!g->q || !g->k_cache || !g->v_cache || !g->o) { set_err(ctx, "%s: null pointer in q/k_cache/v_cache/o", who); return FA_ERR_INVALID_ARG; }
    const bool paged = g->block_table != nullptr;
    if (paged && (g->page_size <= 0 || g->page_size % 64 != 0 || g->max_pages_per_seq <= 0 || g->num_pages <= 0 ||
                  (long long)g->page_size * g->max_pages_per_seq > 0x7fffffffLL)) {
        set_err(ctx, "%s: paged cache needs page_size a positive multiple of 64, max_pages_per_seq > 0 and num_pages > 0", who);
        return FA_ERR_INVALID_ARG;
    }
    const int s_max = paged ? g->page_size * g->max_pages_per_seq : g->s_max;
    if (g->batch <= 0 || g->q_heads <= 0 || g->kv_heads <= 0 || s_max <= 0) { set_err(ctx, "%s: batch/heads/s_max must be > 0", who); return FA_ERR_INVALID_ARG; }
    if (g->head_dim != 64 && g->head_dim != 128) { set_err(ctx, "%s: head_dim must be 64 or 128", who); return FA_ERR_UNSUPPORTED_HD; }
    if (g->q_heads % g->kv_heads != 0 || g->q_heads / g->kv_heads > 16) {
        set_err(ctx, "%s: q_heads must be a multiple of kv_heads with at most 16 query heads per kv head", who);
        return FA_ERR_UNSUPPORTED_SHAPE;
    }
    if (!g->seq_lens && (g->seq_len < 0 || g->seq_len > s_max)) { set_err(ctx, "%s: seq_len must be in [0, s_max]", who); return FA_ERR_INVALID_ARG; }
    if ((reinterpret_cast<uintptr_t>(g->q) & 3) || !aligned16(g->k_cache) || !aligned16(g->v_cache) || (reinterpret_cast<uintptr_t>(g->o) & 1)) {
        set_err(ctx, "%s: k_cache/v_cache must be 16-byte aligned, q 4-byte aligned", who);
        return FA_ERR_INVALID_ARG;
    }
    int cur = -1;
    cudaError_t e = cudaGetDevice(&cur);
    if (e != cudaSuccess) { set_err(ctx, "%s: cudaGetDevice: %s", who, cudaGetErrorString(e)); return FA_ERR_CUDA; }
    if (cur != ctx->device) { set_err(ctx, "%s: the calling thread's current device differs from the context's device", who); return FA_ERR_INVALID_ARG; }
    fa_sm100::DecodeArgs a{};
    a.q = g->q; a.k_cache = g->k_cache; a.v_cache = g->v_cache; a.o = g->o; a.lse = static_cast<float*>(g->l_out);
    a.seq_lens = g->seq_lens;
    a.batch = g->batch; a.q_heads = g->q_heads; a.kv_heads = g->kv_heads; a.hd = g->head_dim;
    a.s_max = s_max; a.seq_len = g->seq_len;
    a.block_table = g->block_table; a.page_size = g->page_size; a.max_pages = g->max_pages_per_seq; a.num_pages = g->num_pages;
    a.scale = g->scale; a.v_descale = (g->v_descale == 0.0f) ? 1.0f : g->v_descale;
    a.scale_q_dev = g->scale_q_dev; a.scale_k_dev = g->scale_k_dev; a.scale_v_dev = g->scale_v_dev;
    a.stream = reinterpret_cast<cudaStream_t>(g->stream);
    Scratch ws;
    const int span = fa_sm100::decode_span(a);
    e = ws.take(ctx, a.stream, fa_sm100::decode_workspace_bytes(a.batch, a.q_heads, a.kv_heads, a.hd, span), 0,
                fa_sm100::decode_arrival_count(a.batch, a.q_heads, a.kv_heads, a.hd, span));
    if (e != cudaSuccess) { set_err(ctx, "%s: workspace allocation: %s", who, cudaGetErrorString(e)); return e == cudaErrorMemoryAllocation ? FA_ERR_OOM : FA_ERR_CUDA; }
    a.workspace = ws.ptr;
    a.arrivals = ws.zeros;
    a.behind_clear = ws.pooled[1] != nullptr;
    e = fa_sm100::launch_decode(a);
    const cudaError_t fe = ws.give_back();  // stream-ordered: released after the kernels
    if (e != cudaSuccess) { set_err(ctx, "%s: launch: %s", who, cudaGetErrorString(e)); return FA_ERR_CUDA; }
    if (fe != cudaSuccess) { set_err(ctx, "%s: workspace release: %s", who, cudaGetErrorString(fe)); return FA_ERR_CUDA; }
    return FA_OK;
}

fa_status_t fa_selftest_wait_expiry(fa_ctx_t* ctx, fa_stream_t stream) {
    if (!ctx) return FA_ERR_INVALID_ARG;
    if (!ctx->arch_ok) { set_err(ctx, "%s: context was created on an unsupported GPU", "fa_selftest_wait_expiry"); return FA_ERR_UNSUPPORTED_ARCH; }
    const cudaError_t e = fa_sm100::launch_wait_expiry_selftest(reinterpret_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) { set_err(ctx, "%s: launch: %s", "fa_selftest_wait_expiry", cudaGetErrorString(e)); return FA_ERR_CUDA; }
    return FA_OK;
}

fa_status_t fa_device_status(fa_ctx_t* ctx) {
    if (!ctx) return FA_ERR_INVALID_ARG;
    const int code = fa_sm100::device_status();
    if (code == 0) return FA_OK;
    if (code < 0) {
        set_err(ctx, "%s: %s", "fa_device_status", cudaGetErrorString(static_cast<cudaError_t>(-code)));
        return FA_ERR_CUDA;
    }
    snprintf(ctx->last_err, sizeof(ctx->last_err), "a kernel wait ran out (device status 0x%x)", code);
    return FA_ERR_INTERNAL;
}

}  // extern "C"
