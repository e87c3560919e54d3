// Device context, staging of host buffers, launch bookkeeping.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <utility>
#include <vector>

#include "host_stage.cuh"
#include "status.hpp"

namespace zb { struct UploadLane; }

struct zant_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = true;
    char* arena = nullptr;        // staging arena for host-pointer calls and op workspaces
    size_t arena_bytes = 0;
    size_t arena_used = 0;
    size_t arena_limit = 0;       // 0 = the staging arena may grow on demand; else its hard cap in bytes
    uint64_t launches = 0;
    int sm_count = 148;
    int* status_word = nullptr;   // device int: kernels with bounded waits report here
    zb::HostStage* stage = nullptr;   // page-locked ring for pageable host buffers, created on first use
    zb::UploadLane* lane = nullptr;   // uploads of a call's large weights beside the kernels of the call before, created on first use
    int give_up_cta = -1;         // self test: this CTA of the next irb_band_kernel gives up its first wait (-1: none)
    bool in_plan = false;         // the launches are a plan's: weights and constants were written before the run
    int tf32 = 0;                 // float contractions: 0 = the exact FP32 kernels, 1 = tensor cores (kind::tf32, single pass), 2 = tensor cores, split operands (3 x TF32)
};

namespace zb {

#define ZB_CUDA(expr)                                                                         \
    do {                                                                                      \
        cudaError_t _e = (expr);                                                              \
        if (_e != cudaSuccess)                                                                \
            return zb::fail(ZANT_E_CUDA, "%s -> %s", #expr, cudaGetErrorString(_e));          \
    } while (0)

// Opt-in to more than 48 KiB of dynamic shared memory.  The attribute belongs to the function ON ONE DEVICE, so it is
// set once per device (a process may drive several: one worker thread per device, each with its own context).
#define ZB_SMEM_ATTR(ctx, kernel, bytes)                                                      \
    do {                                                                                      \
        static std::atomic<unsigned long long> zb_done_{0ull};                                \
        const unsigned long long zb_bit_ = 1ull << ((ctx)->device & 63);                      \
        if (!(zb_done_.load(std::memory_order_acquire) & zb_bit_)) {                          \
            ZB_CUDA(cudaFuncSetAttribute((kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))); \
            zb_done_.fetch_or(zb_bit_, std::memory_order_release);                            \
        }                                                                                     \
    } while (0)

// Device allocations: an out-of-memory answer is the reference's MemError (src/Utils/errorHandler.zig:36-52).
#define ZB_ALLOC(ptr, bytes)                                                                  \
    do {                                                                                      \
        cudaError_t _e = zb::dev_malloc((void**)&(ptr), (bytes));                             \
        if (_e == cudaErrorMemoryAllocation) { cudaGetLastError(); return zb::fail(ZANT_E_MEM_ERROR, "device allocation of %zu bytes failed", (size_t)(bytes)); } \
        if (_e != cudaSuccess) return zb::fail(ZANT_E_CUDA, "cudaMalloc(%zu) -> %s", (size_t)(bytes), cudaGetErrorString(_e)); \
    } while (0)

#ifndef ZB_TRY
#define ZB_TRY(expr) do { int32_t _s = (expr); if (_s != ZANT_OK) return _s; } while (0)
#endif

// Launches behind the stream's previous kernel with programmatic dependent launch: a network is a chain of launches of a few
// microseconds each, and the next kernel's scheduling, barrier and TMEM set-up then overlap the previous one's tail.  Every
// kernel launched this way calls ptx::grid_wait before it touches what another kernel wrote (ptx_sm100.cuh).
template <typename... P, typename... A>
inline void launch(zant_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);      // an error is picked up by check_launch
}

// The same for kernels that read their weights and per-filter constants before grid_wait: in a plan these were written long ago;
// in a single-operator call the launch before may have written them, so the kernel starts when everything before it is done.
template <typename... P, typename... A>
inline void launch_const(zant_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, A&&... args) {
    if (ctx->in_plan) launch(ctx, kernel, grid, block, smem, std::forward<A>(args)...);
    else kernel<<<grid, block, smem, ctx->stream>>>(std::forward<A>(args)...);
}

// The same in clusters of `n` CTAs (1: none).
template <typename... P, typename... A>
inline void launch_cluster(zant_ctx* ctx, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, unsigned n, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension; attr[1].val.clusterDim.x = n; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = n > 1 ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

inline int32_t check_launch(zant_ctx* ctx, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(ZANT_E_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(e));
    ctx->launches++;
    return ZANT_OK;
}

// Where a host-visible copy of the status word lands: the context's page-locked ring where there is one.
inline HostStage* host_stage(zant_ctx* ctx) {
    if (!ctx->stage) ctx->stage = HostStage::create();
    return ctx->stage;
}

// Work enqueued now becomes part of a CUDA graph that the caller is capturing on the context's stream.
inline bool stream_capturing(zant_ctx* ctx) {
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &s) != cudaSuccess) { cudaGetLastError(); return true; }
    return s != cudaStreamCaptureStatusNone;
}

inline int32_t refuse_capture(zant_ctx* ctx) {
    return stream_capturing(ctx) ? fail(ZANT_E_CUDA, "the context's stream is being captured: it cannot be waited for") : ZANT_OK;
}

// Host buffer -> device, ordered on the context's stream; `src` may be changed as soon as this returns.  Not in a capture: the copy would
// become a node that reads the ring's slot at every replay, which holds something else by then.
inline cudaError_t copy_to_device(zant_ctx* ctx, void* dst, const void* src, size_t bytes) {
    if (bytes == 0) return cudaSuccess;
    if (HostStage* st = host_stage(ctx)) return st->to_device(dst, src, bytes, ctx->stream);
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream);      // no page-locked memory to be had
}

// Drains the stream and reads the device status word that kernels with bounded waits write when
// they give up; a non-zero value is reported once and cleared.  With `host_dst` the same wait also brings a result back
// (`bytes` from device memory): one synchronisation for both.  A small one for pageable memory lands in the ring first; page-locked
// memory (`dst_pinned`) takes it directly.  The stream must not be in a capture (refuse_capture).
inline int32_t drain_and_check_status(zant_ctx* ctx, void* host_dst = nullptr, const void* dev_src = nullptr, size_t bytes = 0, bool dst_pinned = false) {
    int h = 0;
    char* slot = nullptr;
    const bool ring = host_dst && bytes && !dst_pinned && bytes + 256 <= HostStage::kSlot;
    if (ctx->stage || ring) {
        if (HostStage* st = host_stage(ctx)) slot = (char*)st->result_slot(256 + (ring ? bytes : 0), ctx->stream);
    }
    const bool via_slot = slot && ring;
    if (host_dst && bytes) ZB_CUDA(cudaMemcpyAsync(via_slot ? (void*)(slot + 256) : host_dst, dev_src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    ZB_CUDA(cudaMemcpyAsync(slot ? (void*)slot : (void*)&h, ctx->status_word, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    ZB_CUDA(cudaStreamSynchronize(ctx->stream));
    if (ctx->stage) ctx->stage->drained();
    if (slot) h = *reinterpret_cast<volatile int*>(slot);
    if (via_slot) std::memcpy(host_dst, slot + 256, bytes);
    if (h != 0) {
        ZB_CUDA(cudaMemsetAsync(ctx->status_word, 0, sizeof(int), ctx->stream));
        return fail(ZANT_E_DEVICE_TIMEOUT, "a kernel gave up a bounded wait (device error %d)", h);
    }
    return ZANT_OK;
}

// What a caller's pointer is: everything the library asks about it, in one driver query.
struct PtrKind { bool device = false, foreign = false, pinned = false; };
inline PtrKind ptr_kind(const void* p, int device) {
    PtrKind k;
    if (!p) return k;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return k;
    }
    k.device = a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
    // Device memory that belongs to another GPU than `device`: a kernel of this context must not be handed such a pointer
    // (without peer access it would take an illegal-address fault, which is sticky for the whole CUDA context).  Managed
    // memory migrates and is accepted on every device.
    k.foreign = a.type == cudaMemoryTypeDevice && a.device != device;
    // Page-locked host memory (cudaHostAlloc / cudaHostRegister): copies to and from it are truly asynchronous, so calls
    // that are handed such buffers need not wait for the stream.
    k.pinned = a.type == cudaMemoryTypeHost;
    return k;
}
inline bool is_device_ptr(const void* p) { return ptr_kind(p, 0).device; }

// Every device allocation of the library goes through here.  `alloc_failures_armed()` is the test
// hook behind zant_b200_debug_fail_alloc: while it is positive it counts allocations down and the
// one that reaches zero reports cudaErrorMemoryAllocation without touching the driver.
inline std::atomic<int>& alloc_failures_armed() {
    static std::atomic<int> n{0};
    return n;
}
inline cudaError_t dev_malloc(void** p, size_t bytes) {
    int armed = alloc_failures_armed().load();
    while (armed > 0) {
        if (alloc_failures_armed().compare_exchange_weak(armed, armed - 1)) {
            if (armed == 1) { *p = nullptr; return cudaErrorMemoryAllocation; }
            break;
        }
    }
    return cudaMalloc(p, bytes);
}

constexpr size_t kArenaAlign = 256;
inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

inline int32_t arena_reserve(zant_ctx* ctx, size_t need_total) {
    if (need_total <= ctx->arena_bytes) return ZANT_OK;
    if (ctx->arena_used != 0) return fail(ZANT_E_ARENA_EXHAUSTED, "arena of %zu bytes exhausted (need %zu)", ctx->arena_bytes, need_total);
    if (ctx->arena_limit && need_total > ctx->arena_limit)
        return fail(ZANT_E_ARENA_EXHAUSTED, "call needs %zu bytes of staging arena, the context's limit is %zu", need_total, ctx->arena_limit);
    ZB_CUDA(cudaStreamSynchronize(ctx->stream));
    if (ctx->arena) ZB_CUDA(cudaFree(ctx->arena));
    ctx->arena = nullptr; ctx->arena_bytes = 0;
    size_t want = align_up(need_total + need_total / 4, 1 << 20);
    if (ctx->arena_limit && want > ctx->arena_limit) want = ctx->arena_limit;
    ZB_ALLOC(ctx->arena, want);
    ctx->arena_bytes = want;
    return ZANT_OK;
}

// Weights of a call on their way while the kernels of the call before still run (1.2 MB 93.6 -> 73 us a call, 3.9 MB 172 -> 109): a copy stream and two
// buffers that calls take in turn.
// The copy into a buffer waits for the last kernel that read it (`taken`), the context's stream for the copy (`ready`).
struct UploadLane {
    static constexpr size_t kMin = 256 << 10, kMax = 8 << 20;      // smaller ones share a copy with the call's other arrays
    cudaStream_t stream = nullptr;
    char* buf[2] = {nullptr, nullptr};
    size_t cap[2] = {0, 0};
    cudaEvent_t ready[2] = {nullptr, nullptr}, taken[2] = {nullptr, nullptr};
    int at = 0;
    static UploadLane* create() {
        UploadLane* l = new UploadLane();
        bool ok = cudaStreamCreateWithFlags(&l->stream, cudaStreamNonBlocking) == cudaSuccess;
        for (int i = 0; i < 2; ++i)
            ok = ok && cudaEventCreateWithFlags(&l->ready[i], cudaEventDisableTiming) == cudaSuccess && cudaEventCreateWithFlags(&l->taken[i], cudaEventDisableTiming) == cudaSuccess;
        if (ok) return l;
        cudaGetLastError();
        delete l;
        return nullptr;
    }
    ~UploadLane() {
        if (stream) { cudaStreamSynchronize(stream); cudaStreamDestroy(stream); }
        for (int i = 0; i < 2; ++i) {
            if (buf[i]) cudaFree(buf[i]);
            if (ready[i]) cudaEventDestroy(ready[i]);
            if (taken[i]) cudaEventDestroy(taken[i]);
        }
    }
    UploadLane() = default;
    UploadLane(const UploadLane&) = delete;
    UploadLane& operator=(const UploadLane&) = delete;
    // The current buffer holds `bytes`.
    bool reserve(size_t bytes) {
        if (cap[at] >= bytes) return true;
        if (buf[at]) { cudaEventSynchronize(taken[at]); cudaFree(buf[at]); }
        buf[at] = nullptr; cap[at] = 0;
        const size_t want = align_up(bytes, 1 << 20);
        if (dev_malloc((void**)&buf[at], want) != cudaSuccess) { cudaGetLastError(); return false; }
        cap[at] = want;
        return true;
    }
};

// Per-call staging: host inputs are copied into the arena, host outputs are copied back
// when the call finishes; device pointers pass through.  All buffers of one call must be
// declared (plan phase) before the first is materialised so the arena can grow once.
class Stager {
  public:
    explicit Stager(zant_ctx* c) : ctx_(c) {}
    ~Stager() {
        if (!ctx_) return;
        if (early_ == 2) end_early();
        ctx_->arena_used = 0;
    }

    struct Slot { const void* host_in; void* host_out; size_t bytes; size_t off; void* dev; bool staged; bool pinned = false; };

    int in(const void* p, size_t bytes) { return add(p, nullptr, bytes, true); }
    int out(void* p, size_t bytes) { return add(nullptr, p, bytes, false); }
    // Weights: large ones in pageable memory go by the context's upload lane, between start_early and end_early of this call, if it has one and may
    // allocate; everything else as with `in`.  One per call.
    int in_early(const void* p, size_t bytes) {
        if (early_ == 0 && bytes > UploadLane::kMin && bytes <= UploadLane::kMax && ctx_->arena_limit == 0 && p && !stream_capturing(ctx_)) {
            const PtrKind k = ptr_kind(p, ctx_->device);
            if (!k.device && !k.pinned) {
                if (!ctx_->lane) ctx_->lane = UploadLane::create();
                if (ctx_->lane && ctx_->lane->reserve(bytes)) {
                    Slot s{p, nullptr, bytes, 0, ctx_->lane->buf[ctx_->lane->at], false};
                    slots_.push_back(s);
                    early_ = 1; early_slot_ = (int)slots_.size() - 1;
                    return early_slot_;
                }
            }
        }
        return in(p, bytes);
    }
    bool early() const { return early_ != 0; }
    // The upload, and the context's stream behind it: what may run beside it is launched before.
    int32_t start_early() {
        if (early_ != 1) return ZANT_OK;
        UploadLane* l = ctx_->lane;
        Slot& s = slots_[early_slot_];
        ZB_CUDA(cudaStreamWaitEvent(l->stream, l->taken[l->at], 0));
        HostStage* st = host_stage(ctx_);
        const cudaError_t e = st ? st->to_device(s.dev, s.host_in, s.bytes, l->stream) : cudaMemcpyAsync(s.dev, s.host_in, s.bytes, cudaMemcpyHostToDevice, l->stream);
        if (e != cudaSuccess) { cudaStreamSynchronize(l->stream); ZB_CUDA(e); }
        ZB_CUDA(cudaEventRecord(l->ready[l->at], l->stream));
        ZB_CUDA(cudaStreamWaitEvent(ctx_->stream, l->ready[l->at], 0));
        early_ = 2;
        return ZANT_OK;
    }
    // The kernels that read the uploaded weights have been launched.
    void end_early() {
        if (early_ != 2) return;
        UploadLane* l = ctx_->lane;
        if (cudaEventRecord(l->taken[l->at], ctx_->stream) != cudaSuccess) { cudaGetLastError(); cudaStreamSynchronize(ctx_->stream); }
        l->at ^= 1;
        early_ = 3;
    }
    int scratch(size_t bytes) {
        Slot s{nullptr, nullptr, bytes, 0, nullptr, true};
        slots_.push_back(s);
        return (int)slots_.size() - 1;
    }

    // Arena space for every staged slot.  False when the arena may not or cannot grow that far: a kernel that wants less workspace is
    // tried then.  (Anything else that is wrong with the buffers is left to commit.)
    bool room() {
        if (foreign_ || stream_capturing(ctx_)) return true;
        const int32_t st = arena_reserve(ctx_, layout());
        return st != ZANT_E_ARENA_EXHAUSTED && st != ZANT_E_MEM_ERROR;
    }

    // Allocates arena space for every staged slot and issues the H2D copies.
    int32_t commit() {
        if (foreign_) return fail(ZANT_E_INVALID_INPUT, "a device buffer belongs to another GPU than the context's device %d", ctx_->device);
        const size_t total = layout();
        if (total) {
            // the arena is the next call's as soon as this one returns: a replay would find that call's data there
            if (stream_capturing(ctx_)) return fail(ZANT_E_CUDA, "a call with host buffers or a workspace cannot be captured into a CUDA graph");
            int32_t st = arena_reserve(ctx_, total);
            if (st != ZANT_OK) return st;
            ctx_->arena_used = total;
        }
        // the small arrays lie together (layout): one copy
        std::vector<HostStage::Part> parts;
        size_t span = 0;
        for (auto& s : slots_)
            if (gathered(s)) { parts.push_back(HostStage::Part{s.host_in, s.bytes, s.off}); span = std::max(span, s.off + s.bytes); }
        HostStage* st = parts.size() > 1 && span <= HostStage::kSlot / 4 ? host_stage(ctx_) : nullptr;
        if (st) ZB_CUDA(st->to_device(ctx_->arena, parts.data(), parts.size(), span, ctx_->stream));
        for (auto& s : slots_) {
            if (!s.staged) continue;
            s.dev = ctx_->arena + s.off;
            if (!s.host_in || !s.bytes || (st && gathered(s))) continue;
            if (s.pinned) { ZB_CUDA(cudaMemcpyAsync(s.dev, s.host_in, s.bytes, cudaMemcpyHostToDevice, ctx_->stream)); wait_ = true; }
            else ZB_CUDA(copy_to_device(ctx_, s.dev, s.host_in, s.bytes));
        }
        return ZANT_OK;
    }

    template <typename T> T* ptr(int i) { return reinterpret_cast<T*>(slots_[i].dev); }

    // Copies staged outputs back and waits for the stream when there is one, or when the device still reads the caller's
    // page-locked input.  (Pageable inputs left through the context's ring: nothing to wait for.)
    int32_t finish() {
        Slot* last = nullptr;
        for (auto& s : slots_) {
            if (!s.staged || !s.host_out || !s.bytes) continue;
            if (last) ZB_CUDA(cudaMemcpyAsync(last->host_out, last->dev, last->bytes, cudaMemcpyDeviceToHost, ctx_->stream));
            last = &s;
        }
        ctx_->arena_used = 0;
        if (!last && !wait_) return ZANT_OK;
        // the call waits anyway: also pick up the status word that a bounded device-side wait writes
        // when it gives up, so that the time-out is reported by the call that suffered it
        return last ? drain_and_check_status(ctx_, last->host_out, last->dev, last->bytes, last->pinned) : drain_and_check_status(ctx_);
    }

  private:
    size_t layout() {
        size_t total = 0;
        for (int rest = 0; rest < 2; ++rest)
            for (auto& s : slots_) if (s.staged && gathered(s) == (rest == 0)) { s.off = total; total += align_up(s.bytes ? s.bytes : 1, kArenaAlign); }
        return total;
    }
    // Pageable inputs that may leave as one copy: weights, multipliers and biases of a call were three, each a few microseconds on the host and the
    // stream (33 x 45 x 27 x 27 -> 85 filters 32.6 -> 25.5 us a call).
    static bool gathered(const Slot& s) { return s.staged && s.host_in && s.bytes && !s.pinned && s.bytes <= HostStage::kSlot / 4; }
    int add(const void* pin, void* pout, size_t bytes, bool is_in) {
        const void* p = is_in ? pin : pout;
        Slot s{nullptr, nullptr, bytes, 0, nullptr, false};
        if (p == nullptr) { s.dev = nullptr; }
        else {
            const PtrKind k = ptr_kind(p, ctx_->device);
            if (k.device) { s.dev = const_cast<void*>(p); foreign_ = foreign_ || k.foreign; }
            else { s.staged = true; s.pinned = k.pinned; s.host_in = pin; s.host_out = pout; }
        }
        slots_.push_back(s);
        return (int)slots_.size() - 1;
    }
    zant_ctx* ctx_;
    std::vector<Slot> slots_;
    bool foreign_ = false, wait_ = false;
    int early_ = 0, early_slot_ = -1;      // 0 none, 1 declared, 2 on its way, 3 read
};

inline int grid_for(size_t work_items, int block, int sm_count, int waves = 8) {
    size_t blocks = (work_items + block - 1) / block;
    const size_t cap = (size_t)sm_count * waves;
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    return (int)blocks;
}

}  // namespace zb
