// Plan: the run-time form of a generated predict() — graph tensors at fixed offsets of one
// cudaMalloc'd arena, constants uploaded once, nodes launched in insertion order.
// (src/codeGen/predict.zig:23-70 emits the straight-line op calls this replays;
//  :110-142, :265-272 is the one-static-array-per-tensor memory plan mirrored here.)
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <algorithm>
#include <climits>
#include <cmath>
#include <functional>
#include <memory>
#include <string>
#include <vector>

#include "../../include/zant_b200.h"
#include "context.cuh"
#include "geometry.hpp"
#include "ops.cuh"
#include "fused_cnn.cuh"
#include "tc_gemm.cuh"
#include "tc_conv_generic.cuh"
#include "tc_conv_nchw.cuh"
#include "tc_pw_nchw.cuh"
#include "dwconv_q8.cuh"
#include "smallc_conv_q8.cuh"
#include "tc_conv_nhwc.cuh"
#include "tc_gemm_tf32.cuh"
#include "small_gemm_q8.cuh"
#include "tc_nhwc_net.cuh"
#include "first_layer_q8.cuh"
#include "fused_cnn_few.cuh"
#include "irb_band.cuh"
#include "irb_q8.cuh"
#include "status.hpp"

using namespace zb;

struct PlanTensor {
    int32_t dtype = ZANT_F32;
    std::vector<size_t> shape;
    size_t bytes = 0;
    bool is_const = false;
    std::vector<char> host;     // initializer bytes (kept until finalize)
    size_t offset = 0;          // arena offset
    void* arena_ptr = nullptr;  // address inside the plan's arena
    void* bound = nullptr;      // caller's device buffer bound for the current run (input/output)
    int alias = -1;             // Reshape output: shares the buffer of this tensor
    bool elided = false;        // interior of a fused chain: never materialised, no arena space
    // Kept channels-last between convolutions (tc_nhwc_net.cuh): pixels `nh_pix` bytes apart, channel 0 of pixel (0,0) `nh_off` bytes
    // into the buffer of tensor `nh_root` (a Concat's operands live in its result; else the tensor itself).
    bool nh = false;
    int nh_root = -1;
    size_t nh_off = 0, nh_pix = 0;
    int nh_lo = 0;              // split TF32: channels from a hi half to its lo half
};

struct PlanNode {
    int32_t op = 0;
    std::vector<int> in, out;
    zant_node_attrs a{};
};

// A convolution with what follows it, as one channels-last step.
struct NhGroup {
    size_t first = 0, count = 0;
    int x = -1, y = -1;                  // tensors read and written
    std::vector<int> interior;
    int qact = -1;                       // int8: activation flag that a Relu node became (-1: the node's own)
    int lut_node = -1;                   // int8: activation node that becomes a table
    int fact = 0; float slope = 0.0f;    // TF32
    bool pool = false, up2 = false;
    int dequant = -1;                    // DequantizeLinear node
    int quant = -1;                      // QuantizeLinear node in front of it that the same kernel takes (first_layer_q8.cuh)
    bool on = false;                     // the layout pass took it
};

struct zant_plan {
    zant_ctx* ctx = nullptr;
    std::vector<PlanTensor> t;
    std::vector<PlanNode> nodes;
    std::vector<std::vector<char>> aux_host;   // derived constants (multipliers, tables)
    std::vector<size_t> aux_off;
    std::vector<size_t> scratch_bytes;         // internal buffers of fused steps (private layouts)
    std::vector<size_t> scratch_off;
    int input = -1, output = -1;
    bool finalized = false;
    char* arena = nullptr;
    size_t arena_bytes = 0;
    std::vector<std::function<int32_t()>> steps;
    std::vector<std::function<int32_t()>> init_steps;   // run once when the constants are in the arena: weights into a kernel's layout
    std::vector<std::string> step_names;
    std::vector<double> step_macs, step_bytes;   // algorithmic work of each step: multiply-accumulates, bytes crossing the step's boundary
    int launches_per_run = 0;
    bool profiling = false;
    cudaGraphExec_t graph_exec = nullptr;   // replay of all steps on arena buffers
    std::vector<cudaEvent_t> prof_events;   // pool, reused between reads
    size_t prof_used = 0;                   // events recorded since the last read

    // additions inside a convolution's step, with the proof of their short form (once for equal parameters)
    std::vector<QAddTail> proved_adds;
    QAddTail prove(QAddTail t) {
        for (const QAddTail& p : proved_adds) {
            QAddTail q = p;
            q.proved = 0;
            if (std::memcmp(&q, &t, sizeof q) == 0) return p;
        }
        QAddTail p = t;
        qadd_prove(p);
        proved_adds.push_back(p);
        return p;
    }
    std::vector<NhGroup> nh_groups;   // channels-last convolution groups found by the layout pass, by first node
    std::vector<std::pair<int, char*>> nchw_copies;   // channels-last tensors whose address was asked for, and buffers that hold them in the graph's order after each run
    void* ptr(int id) const {
        int r = id;
        while (t[r].alias >= 0) r = t[r].alias;
        return t[r].bound ? t[r].bound : t[r].arena_ptr;
    }
    template <typename T> T* p(int id) const { return id < 0 ? nullptr : reinterpret_cast<T*>(ptr(id)); }
    void* aux(int id) const { return arena + aux_off[id]; }
    void* scratch(int id) const { return arena + scratch_off[id]; }
    int add_scratch(size_t bytes) { scratch_bytes.push_back(bytes); return (int)scratch_bytes.size() - 1; }
    // One buffer for the im2col matrices of all tensor-core steps: steps run one after another on
    // one stream, so they can share it; it is as large as the largest request.
    // float activation that the fusion pass asks the next Conv step to apply, and the tensor that step writes instead of its own
    int pending_fact = 0; float pending_slope = 0.0f; int pending_y = -1; bool pending_used = false;
    int pending_pool = -1;      // exact path: the 2x2 / 2 MaxPool behind that activation, as the tensor it writes
    int im2col_scratch = -1;
    int shared_im2col_scratch(size_t bytes) {
        if (im2col_scratch < 0) im2col_scratch = add_scratch(bytes);
        else scratch_bytes[im2col_scratch] = std::max(scratch_bytes[im2col_scratch], bytes);
        return im2col_scratch;
    }
    int add_aux(const void* data, size_t bytes) {
        aux_host.emplace_back((const char*)data, (const char*)data + bytes);
        return (int)aux_host.size() - 1;
    }
    // Takes back what an earlier finalize that failed has derived: tensors, nodes and initializers stay as they were declared.
    void reset_build() {
        if (arena) { cudaStreamSynchronize(ctx->stream); cudaFree(arena); arena = nullptr; arena_bytes = 0; }
        steps.clear(); init_steps.clear(); step_names.clear(); step_macs.clear(); step_bytes.clear();
        aux_host.clear(); aux_off.clear(); scratch_bytes.clear(); scratch_off.clear(); nh_groups.clear();
        im2col_scratch = -1;
        pending_fact = 0; pending_slope = 0.0f; pending_y = -1; pending_used = false; pending_pool = -1;
        for (PlanTensor& x : t) {
            x.alias = -1; x.elided = false; x.arena_ptr = nullptr; x.bound = nullptr;
            x.nh = false; x.nh_root = -1; x.nh_off = x.nh_pix = 0; x.nh_lo = 0;
        }
    }
};

namespace {

struct InPlan {
    explicit InPlan(zant_ctx* c) : ctx(c) { ctx->in_plan = true; }
    ~InPlan() { ctx->in_plan = false; }
    zant_ctx* ctx;
};

const char* kAutoPadNames[] = {"NOTSET", "SAME_UPPER", "SAME_LOWER", "VALID"};

int32_t need_inputs(const PlanNode& n, size_t lo, size_t hi, const char* name) {
    if (n.in.size() < lo || n.in.size() > hi) return fail(ZANT_E_INVALID_INPUT, "%s takes %zu..%zu inputs, got %zu", name, lo, hi, n.in.size());
    if (n.out.size() != 1) return fail(ZANT_E_INVALID_INPUT, "%s produces one output", name);
    return ZANT_OK;
}

int opt_in(const PlanNode& n, size_t i) { return i < n.in.size() ? n.in[i] : -1; }

int32_t want_dtype(const zant_plan* pl, int id, int32_t dt, const char* what) {
    if (id >= 0 && pl->t[id].dtype != dt) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "%s: tensor %d has dtype %d, expected %d", what, id, pl->t[id].dtype, dt);
    return ZANT_OK;
}

// Table for a unary function between two quantized tensors:
//   lut[code] = sat(rne(f(float(q - zp_in) * s_in) / s_out) + zp_out)
template <typename F>
void build_unary_lut(int32_t dtype, float s_in, int zp_in, float s_out, int zp_out, F f, uint8_t lut[256]) {
    for (int code = 0; code < 256; ++code) {
        const int q = dtype == ZANT_U8 ? code : (int)(int8_t)(uint8_t)code;
        volatile float x = (float)(q - zp_in) * s_in;
        volatile float a = f((float)x);
        volatile float v = a / s_out;
        float c = std::fmin(std::fmax((float)v, -512.0f), 511.0f);
        int t = (int)std::nearbyintf(c) + zp_out;
        const int lo = dtype == ZANT_U8 ? 0 : -128, hi = dtype == ZANT_U8 ? 255 : 127;
        t = std::min(std::max(t, lo), hi);
        lut[code] = (uint8_t)t;
    }
}

// Table of a Relu / LeakyRelu / Clip node between two quantized tensors of type `dt`.
void activation_lut(const PlanNode& n, int32_t dt, uint8_t lut[256]) {
    const zant_node_attrs& a = n.a;
    const float p0 = a.alpha, p1 = a.beta;
    if (n.op == ZANT_OP_RELU) build_unary_lut(dt, a.x_scale, a.x_zp, a.y_scale, a.y_zp, [](float v) { return v > 0.0f ? v : 0.0f; }, lut);
    else if (n.op == ZANT_OP_LEAKY_RELU) build_unary_lut(dt, a.x_scale, a.x_zp, a.y_scale, a.y_zp, [p0](float v) { volatile float s = p0 * v; return v <= 0.0f ? (float)s : v; }, lut);
    else build_unary_lut(dt, a.x_scale, a.x_zp, a.y_scale, a.y_zp, [p0, p1](float v) { return std::fmin(std::fmax(v, p0), p1); }, lut);
}

}  // namespace

extern "C" {

int32_t zant_b200_plan_create(zant_ctx* ctx, zant_plan** out) {
    if (!out) return fail(ZANT_E_NULL_POINTER, "out is NULL");
    *out = nullptr;
    if (!ctx) return fail(ZANT_E_CUDA_UNAVAILABLE, "no context; there is no CPU fallback");
    zant_plan* p = new zant_plan();
    p->ctx = ctx;
    *out = p;
    return ZANT_OK;
}

int32_t zant_b200_plan_destroy(zant_plan* plan) {
    if (!plan) return ZANT_OK;
    cudaSetDevice(plan->ctx->device);
    cudaStreamSynchronize(plan->ctx->stream);
    if (plan->graph_exec) cudaGraphExecDestroy(plan->graph_exec);
    if (plan->arena) cudaFree(plan->arena);
    for (auto& c : plan->nchw_copies) cudaFree(c.second);
    for (cudaEvent_t e : plan->prof_events) cudaEventDestroy(e);
    cudaGetLastError();
    delete plan;
    return ZANT_OK;
}

int32_t zant_b200_plan_tensor(zant_plan* plan, int32_t dtype, const size_t* shape, size_t rank, const void* const_data, int32_t* id) {
    if (!plan) return fail(ZANT_E_BAD_HANDLE, "plan is NULL");
    if (plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan already finalized");
    if (!id || (rank && !shape)) return fail(ZANT_E_NULL_POINTER, "id/shape is NULL");
    if (!dtype_valid(dtype)) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "dtype %d", dtype);
    if (rank > 8) return fail(ZANT_E_UNSUPPORTED_DIMENSION, "rank %zu", rank);
    PlanTensor t;
    t.dtype = dtype;
    t.shape.assign(shape, shape + rank);
    t.bytes = numel(shape, rank) * dtype_size(dtype);
    if (const_data) {
        t.is_const = true;
        t.host.assign((const char*)const_data, (const char*)const_data + t.bytes);
    }
    plan->t.push_back(std::move(t));
    *id = (int32_t)plan->t.size() - 1;
    return ZANT_OK;
}

int32_t zant_b200_plan_node(zant_plan* plan, int32_t op, const int32_t* inputs, size_t n_inputs,
                            const int32_t* outputs, size_t n_outputs, const zant_node_attrs* attrs) {
    if (!plan) return fail(ZANT_E_BAD_HANDLE, "plan is NULL");
    if (plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan already finalized");
    if ((n_inputs && !inputs) || (n_outputs && !outputs)) return fail(ZANT_E_NULL_POINTER, "inputs/outputs is NULL");
    PlanNode n;
    n.op = op;
    const int nt = (int)plan->t.size();
    for (size_t i = 0; i < n_inputs; ++i) {
        if (inputs[i] < -1 || inputs[i] >= nt) return fail(ZANT_E_INVALID_INPUT, "input %zu: unknown tensor id %d", i, inputs[i]);
        n.in.push_back(inputs[i]);
    }
    for (size_t i = 0; i < n_outputs; ++i) {
        if (outputs[i] < 0 || outputs[i] >= nt) return fail(ZANT_E_INVALID_INPUT, "output %zu: unknown tensor id %d", i, outputs[i]);
        if (plan->t[outputs[i]].is_const) return fail(ZANT_E_INVALID_INPUT, "output %zu is an initializer", i);
        n.out.push_back(outputs[i]);
    }
    if (attrs) n.a = *attrs;
    plan->nodes.push_back(std::move(n));
    return ZANT_OK;
}

static int32_t build_node(zant_plan* pl, size_t node_index, int32_t fuse);
static int32_t build_node_impl(zant_plan* pl, size_t node_index, int32_t fuse);
static int32_t try_fuse(zant_plan* pl, size_t node_index, size_t& consumed);
static int32_t try_fuse_small_cnn(zant_plan* pl, size_t node_index, size_t& consumed, bool probe = false);
static int32_t try_fuse_qconv_group(zant_plan* pl, size_t node_index, size_t& consumed);
static int32_t try_fuse_fconv_group(zant_plan* pl, size_t node_index, size_t& consumed);
static int32_t try_fuse_irb(zant_plan* pl, size_t node_index, size_t& consumed);
static void nh_layout(zant_plan* pl);
static int32_t build_nh(zant_plan* pl, size_t node_index, size_t& consumed);
static int32_t refresh_nchw_copy(zant_plan* pl, int id, char* y);

// Multiply-accumulates of one node (contractions only; everything else counts as 0).
static double node_macs(const zant_plan* pl, const PlanNode& n) {
    auto shape = [&](int id) -> const std::vector<size_t>& { return pl->t[id].shape; };
    auto count = [&](int id) { double c = 1; for (size_t d : shape(id)) c *= (double)d; return c; };
    switch (n.op) {
        case ZANT_OP_CONV:
        case ZANT_OP_QLINEAR_CONV: {
            if (n.in.size() < 2 || n.out.empty() || shape(n.in[1]).size() != 4) return 0;
            const auto& w = shape(n.in[1]);
            return count(n.out[0]) * (double)w[1] * (double)w[2] * (double)w[3];
        }
        case ZANT_OP_MATMUL:
        case ZANT_OP_QLINEAR_MATMUL:
        case ZANT_OP_GEMM: {
            if (n.in.size() < 2 || n.out.empty() || shape(n.in[0]).size() < 2) return 0;
            const auto& a = shape(n.in[0]);
            const size_t k = (n.op == ZANT_OP_GEMM && n.a.trans_a) ? a[a.size() - 2] : a[a.size() - 1];
            return count(n.out[0]) * (double)k;
        }
        default: return 0;
    }
}

// Cost of the steps that cover nodes [first, first + count): MACs of the nodes; bytes = every tensor that is read
// from outside the group (initializers included) or written by it and still materialised, each counted once.
static void record_step_cost(zant_plan* pl, size_t first_step, size_t first, size_t count) {
    double macs = 0, bytes = 0;
    std::vector<char> produced(pl->t.size(), 0), seen(pl->t.size(), 0);
    auto root = [&](int id) { while (pl->t[id].alias >= 0) id = pl->t[id].alias; return id; };
    for (size_t i = first; i < first + count; ++i) for (int o : pl->nodes[i].out) produced[root(o)] = 1;
    for (size_t i = first; i < first + count; ++i) {
        const PlanNode& n = pl->nodes[i];
        macs += node_macs(pl, n);
        if (n.op == ZANT_OP_RESHAPE) continue;
        for (int id : n.in) {
            if (id < 0) continue;
            const int r = root(id);
            if (!produced[r] && !seen[r]) { seen[r] = 1; bytes += (double)pl->t[id].bytes; }
        }
        for (int o : n.out) {
            const int r = root(o);
            if (!pl->t[r].elided && !seen[r]) { seen[r] = 1; bytes += (double)pl->t[o].bytes; }
        }
    }
    pl->step_macs.resize(pl->steps.size(), 0.0);
    pl->step_bytes.resize(pl->steps.size(), 0.0);
    if (pl->steps.size() > first_step) {       // a group may emit several steps: the work is booked on its last one
        pl->step_macs.back() = macs;
        pl->step_bytes.back() = bytes;
    }
}

int32_t zant_b200_plan_finalize(zant_plan* plan, int32_t input_id, int32_t output_id, int32_t fuse) {
    if (!plan) return fail(ZANT_E_BAD_HANDLE, "plan is NULL");
    if (plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan already finalized");
    const int nt = (int)plan->t.size();
    if (input_id < 0 || input_id >= nt || output_id < 0 || output_id >= nt) return fail(ZANT_E_INVALID_INPUT, "input/output id out of range");
    plan->input = input_id; plan->output = output_id;
    zant_ctx* ctx = plan->ctx;
    ZB_CUDA(cudaSetDevice(ctx->device));

    // 1. validate nodes, derive constants, record launch closures
    plan->reset_build();
    size_t i = 0;
    if (fuse) nh_layout(plan);
    while (i < plan->nodes.size()) {
        size_t consumed = 0;
        if (fuse) {
            int32_t st = build_nh(plan, i, consumed);
            if (st != ZANT_OK) return st;
        }
        if (fuse && consumed == 0) {
            int32_t st = try_fuse(plan, i, consumed);
            if (st != ZANT_OK) return st;
        }
        if (consumed == 0) {
            int32_t st = build_node(plan, i, fuse);
            if (st != ZANT_OK) return st;
            consumed = 1;
        }
        i += consumed;
    }

    // 2. arena layout: every non-aliased tensor and every derived constant at a fixed offset
    size_t off = 0;
    for (size_t id = 0; id < plan->t.size(); ++id) {
        PlanTensor& t = plan->t[id];
        if (t.alias >= 0 || t.elided || (t.nh && t.nh_root != (int)id)) continue;
        t.offset = off;
        const size_t bytes = t.nh ? t.shape[0] * t.shape[2] * t.shape[3] * t.nh_pix : t.bytes;
        off += align_up(bytes ? bytes : 1, kArenaAlign);
    }
    plan->aux_off.resize(plan->aux_host.size());
    for (size_t a = 0; a < plan->aux_host.size(); ++a) {
        plan->aux_off[a] = off;
        off += align_up(plan->aux_host[a].size() ? plan->aux_host[a].size() : 1, kArenaAlign);
    }
    plan->scratch_off.resize(plan->scratch_bytes.size());
    for (size_t a = 0; a < plan->scratch_bytes.size(); ++a) {
        plan->scratch_off[a] = off;
        off += align_up(plan->scratch_bytes[a] ? plan->scratch_bytes[a] : 1, kArenaAlign);
    }
    plan->arena_bytes = off;
    ZB_ALLOC(plan->arena, off);
    for (auto& t : plan->t) {
        if (t.alias >= 0 || t.elided) continue;
        t.arena_ptr = t.nh ? plan->arena + plan->t[t.nh_root].offset + t.nh_off : plan->arena + t.offset;
        if (t.is_const && t.bytes) ZB_CUDA(cudaMemcpyAsync(t.arena_ptr, t.host.data(), t.bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    for (size_t a = 0; a < plan->aux_host.size(); ++a)
        if (!plan->aux_host[a].empty())
            ZB_CUDA(cudaMemcpyAsync(plan->arena + plan->aux_off[a], plan->aux_host[a].data(), plan->aux_host[a].size(), cudaMemcpyHostToDevice, ctx->stream));
    const uint64_t launched = ctx->launches;
    for (auto& s : plan->init_steps) { int32_t st = s(); if (st != ZANT_OK) return st; }
    plan->init_steps.clear();
    ctx->launches = launched;
    ZB_CUDA(cudaStreamSynchronize(ctx->stream));

    // 3. one dry count of launches
    plan->finalized = true;
    const uint64_t before = ctx->launches;
    InPlan scope(ctx);
    for (auto& s : plan->steps) { int32_t st = s(); if (st != ZANT_OK) { plan->finalized = false; return st; } }
    ZB_CUDA(cudaStreamSynchronize(ctx->stream));
    plan->launches_per_run = (int)(ctx->launches - before);
    ctx->launches = before;
    for (auto& t : plan->t) { t.host.clear(); t.host.shrink_to_fit(); }
    log_line("zant_b200 plan: %zu tensors, %zu nodes, %zu steps, %d launches, arena %zu bytes", plan->t.size(), plan->nodes.size(), plan->steps.size(), plan->launches_per_run, plan->arena_bytes);
    return ZANT_OK;
}

int32_t zant_b200_plan_run(zant_plan* plan, const void* input, void* output) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    if (!input || !output) return fail(ZANT_E_NULL_POINTER, "input/output is NULL");
    zant_ctx* ctx = plan->ctx;
    ZB_CUDA(cudaSetDevice(ctx->device));
    PlanTensor& ti = plan->t[plan->input];
    PlanTensor& to = plan->t[plan->output];
    int out_root = plan->output;
    while (plan->t[out_root].alias >= 0) out_root = plan->t[out_root].alias;
    PlanTensor& tor = plan->t[out_root];
    const PtrKind ki = ptr_kind(input, ctx->device), ko = ptr_kind(output, ctx->device);
    const bool in_dev = ki.device, out_dev = ko.device;
    // Pinned host buffers on both sides: the whole run stays asynchronous on the stream (the caller overlaps it with other
    // contexts and calls zant_b200_ctx_synchronize).  Pageable buffers: wait, so that the result is in place when the call
    // returns.
    const bool async = out_dev || (ko.pinned && (in_dev || ki.pinned));
    auto copy_in = [&]() -> cudaError_t {
        if (in_dev || ki.pinned) return cudaMemcpyAsync(ti.arena_ptr, input, ti.bytes, in_dev ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, ctx->stream);
        // (captured by the caller: a plain copy, which reads `input` at every replay)
        if (stream_capturing(ctx)) return cudaMemcpyAsync(ti.arena_ptr, input, ti.bytes, cudaMemcpyHostToDevice, ctx->stream);
        return copy_to_device(ctx, ti.arena_ptr, input, ti.bytes);
    };
    // copies the result out; a call that has to wait reads the status word with the same synchronisation
    auto copy_out = [&]() -> int32_t {
        if (!async) return drain_and_check_status(ctx, output, tor.arena_ptr, to.bytes, ko.pinned);
        ZB_CUDA(cudaMemcpyAsync(output, tor.arena_ptr, to.bytes, out_dev ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, ctx->stream));
        return ZANT_OK;
    };
    if (ki.foreign || ko.foreign)
        return fail(ZANT_E_INVALID_INPUT, "input/output is device memory of another GPU than the plan's device %d", ctx->device);
    if (!async) ZB_TRY(refuse_capture(ctx));
    if (plan->graph_exec && !plan->profiling) {
        // replay: everything runs on the arena's own buffers
        ZB_CUDA(copy_in());
        ZB_CUDA(cudaGraphLaunch(plan->graph_exec, ctx->stream));
        ctx->launches += (uint64_t)plan->launches_per_run;
        for (auto& c : plan->nchw_copies) ZB_TRY(refresh_nchw_copy(plan, c.first, c.second));
        return copy_out();
    }
    ti.bound = in_dev ? const_cast<void*>(input) : nullptr;
    tor.bound = out_dev ? output : nullptr;
    if (!in_dev) ZB_CUDA(copy_in());
    auto mark = [&]() -> int32_t {
        if (plan->prof_used == plan->prof_events.size()) {
            cudaEvent_t e;
            ZB_CUDA(cudaEventCreate(&e));
            plan->prof_events.push_back(e);
        }
        ZB_CUDA(cudaEventRecord(plan->prof_events[plan->prof_used++], ctx->stream));
        return ZANT_OK;
    };
    InPlan scope(ctx);
    for (size_t s = 0; s < plan->steps.size(); ++s) {
        if (plan->profiling) { int32_t st = mark(); if (st != ZANT_OK) return st; }
        int32_t st = plan->steps[s]();
        if (st != ZANT_OK) { ti.bound = nullptr; tor.bound = nullptr; return st; }
    }
    if (plan->profiling) { int32_t st = mark(); if (st != ZANT_OK) return st; }
    ti.bound = nullptr; tor.bound = nullptr;
    for (auto& c : plan->nchw_copies) ZB_TRY(refresh_nchw_copy(plan, c.first, c.second));
    return out_dev ? ZANT_OK : copy_out();
}

int32_t zant_b200_plan_use_graph(zant_plan* plan, int32_t enable) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    zant_ctx* ctx = plan->ctx;
    ZB_CUDA(cudaSetDevice(ctx->device));
    ZB_CUDA(cudaStreamSynchronize(ctx->stream));
    if (plan->graph_exec) { cudaGraphExecDestroy(plan->graph_exec); plan->graph_exec = nullptr; }
    if (!enable) return ZANT_OK;
    // every step has run at least once (the dry run of finalize), so one-time function attributes are set
    plan->t[plan->input].bound = nullptr;
    {
        int r = plan->output;
        while (plan->t[r].alias >= 0) r = plan->t[r].alias;
        plan->t[r].bound = nullptr;
    }
    const uint64_t before = ctx->launches;
    InPlan scope(ctx);
    ZB_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    int32_t st = ZANT_OK;
    for (auto& step : plan->steps) { st = step(); if (st != ZANT_OK) break; }
    cudaGraph_t graph = nullptr;
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    ctx->launches = before;
    if (st != ZANT_OK) { if (graph) cudaGraphDestroy(graph); return st; }
    if (e != cudaSuccess || !graph) { cudaGetLastError(); return fail(ZANT_E_CUDA, "stream capture failed: %s", cudaGetErrorString(e)); }
    const cudaError_t ei = cudaGraphInstantiate(&plan->graph_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) { plan->graph_exec = nullptr; cudaGetLastError(); return fail(ZANT_E_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(ei)); }
    return ZANT_OK;
}

size_t zant_b200_plan_arena_bytes(zant_plan* plan) { return plan ? plan->arena_bytes : 0; }
int32_t zant_b200_plan_launches_per_run(zant_plan* plan) { return plan ? plan->launches_per_run : 0; }
void* zant_b200_plan_tensor_ptr(zant_plan* plan, int32_t id) {
    if (!plan || !plan->finalized || id < 0 || id >= (int)plan->t.size()) return nullptr;
    int r = id;
    while (plan->t[r].alias >= 0) r = plan->t[r].alias;
    if (plan->t[r].nh) {
        // kept in another layout: the address of a copy in the graph's order, which every run from now on brings up to date
        for (auto& c : plan->nchw_copies) if (c.first == r) return c.second;
        char* y = nullptr;
        if (cudaSetDevice(plan->ctx->device) != cudaSuccess || dev_malloc((void**)&y, plan->t[r].bytes) != cudaSuccess) { cudaGetLastError(); return nullptr; }
        if (refresh_nchw_copy(plan, r, y) != ZANT_OK) { cudaFree(y); return nullptr; }
        plan->nchw_copies.emplace_back(r, y);
        return y;
    }
    return plan->ptr(id);
}

int32_t zant_b200_plan_step_count(zant_plan* plan) { return (plan && plan->finalized) ? (int32_t)plan->steps.size() : 0; }
const char* zant_b200_plan_step_name(zant_plan* plan, int32_t step) {
    if (!plan || step < 0 || step >= (int32_t)plan->step_names.size()) return "";
    return plan->step_names[step].c_str();
}

int32_t zant_b200_plan_step_cost(zant_plan* plan, int32_t step, double* macs, double* bytes) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    if (step < 0 || step >= (int32_t)plan->steps.size()) return fail(ZANT_E_INVALID_INPUT, "step %d of %zu", step, plan->steps.size());
    if (macs) *macs = step < (int32_t)plan->step_macs.size() ? plan->step_macs[step] : 0.0;
    if (bytes) *bytes = step < (int32_t)plan->step_bytes.size() ? plan->step_bytes[step] : 0.0;
    return ZANT_OK;
}

int32_t zant_b200_plan_profile(zant_plan* plan, int32_t enable) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    plan->profiling = enable != 0;
    plan->prof_used = 0;
    return ZANT_OK;
}

int32_t zant_b200_plan_profile_read(zant_plan* plan, float* sum_ms, int32_t* runs) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    if (!sum_ms || !runs) return fail(ZANT_E_NULL_POINTER, "sum_ms/runs is NULL");
    ZB_CUDA(cudaSetDevice(plan->ctx->device));
    ZB_CUDA(cudaStreamSynchronize(plan->ctx->stream));
    const size_t per_run = plan->steps.size() + 1;
    const size_t n_runs = plan->prof_used / per_run;
    for (size_t r = 0; r < n_runs; ++r)
        for (size_t s = 0; s + 1 < per_run; ++s) {
            float ms = 0.0f;
            ZB_CUDA(cudaEventElapsedTime(&ms, plan->prof_events[r * per_run + s], plan->prof_events[r * per_run + s + 1]));
            sum_ms[s] += ms;
        }
    *runs = (int32_t)n_runs;
    plan->prof_used = 0;
    return ZANT_OK;
}

int32_t zant_b200_plan_read_tensor(zant_plan* plan, int32_t id, void* host_dst) {
    if (!plan || !plan->finalized) return fail(ZANT_E_BAD_HANDLE, "plan is NULL or not finalized");
    if (id < 0 || id >= (int)plan->t.size()) return fail(ZANT_E_INVALID_INPUT, "tensor id %d", id);
    if (!host_dst) return fail(ZANT_E_NULL_POINTER, "host_dst is NULL");
    {
        int r = id;
        while (plan->t[r].alias >= 0) r = plan->t[r].alias;
        if (plan->t[r].elided) return fail(ZANT_E_UNSUPPORTED, "tensor %d is interior to a fused chain and is not materialised", id);
    }
    ZB_CUDA(cudaSetDevice(plan->ctx->device));
    ZB_CUDA(cudaStreamSynchronize(plan->ctx->stream));
    int r = id;
    while (plan->t[r].alias >= 0) r = plan->t[r].alias;
    const PlanTensor& t = plan->t[r];
    if (t.nh) {
        const size_t N = t.shape[0], C = t.shape[1], hw = t.shape[2] * t.shape[3], esz = dtype_size(t.dtype);
        const PlanTensor& root = plan->t[t.nh_root];
        std::vector<char> raw(N * hw * t.nh_pix);
        ZB_CUDA(cudaMemcpy(raw.data(), root.arena_ptr, raw.size(), cudaMemcpyDeviceToHost));
        for (size_t n = 0; n < N; ++n)
            for (size_t c = 0; c < C; ++c)
                for (size_t p = 0; p < hw; ++p) {
                    const char* src = raw.data() + (n * hw + p) * t.nh_pix + t.nh_off + c * esz;
                    char* dst = (char*)host_dst + ((n * C + c) * hw + p) * esz;
                    std::memcpy(dst, src, esz);
                    if (t.nh_lo) {
                        float hi, lo;
                        std::memcpy(&hi, src, 4); std::memcpy(&lo, src + (size_t)t.nh_lo * 4, 4);
                        hi += lo;
                        std::memcpy(dst, &hi, 4);
                    }
                }
        return ZANT_OK;
    }
    ZB_CUDA(cudaMemcpy(host_dst, plan->ptr(id), plan->t[id].bytes, cudaMemcpyDeviceToHost));
    return ZANT_OK;
}

}  // extern "C"

// --------------------------------------------------------------------------------------------
// QLinearConv, alone or as the head of a fused group.  `fz` carries what the fusion pass found behind the node:
// an activation override (a Relu that keeps scale and zero point), a 256-entry table (LeakyRelu, Clip, a Relu
// that changes scale) applied to the finished codes, the tensor the step writes instead of the node's own
// output, and a 2x2 / stride-2 MaxPool that the implicit-GEMM kernel can apply in its epilogue.
// --------------------------------------------------------------------------------------------
struct QConvFusion {
    int activation = -1;     // >= 0: replaces the node's own activation attribute
    int lut_aux = -1;        // aux id of the table, -1 = none
    int y_act = -1;          // tensor written when the pool is not fused (-1: the node's output)
    int y_pool = -1;         // pooled tensor; >= 0 asks for the fused pool
    bool pool_done = false;  // out: the step writes y_pool
    int add_node = -1;       // QLinearAdd behind the convolution (and its activation); its other operand
    int add_res = -1;
    bool add_done = false;   // out: the step writes the sum
};

static int32_t build_qconv(zant_plan* pl, const PlanNode& n, QConvFusion& fz) {
    const zant_node_attrs& a = n.a;
    zant_ctx* ctx = pl->ctx;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    ZB_TRY(need_inputs(n, 3, 5, "QLinearConv"));
    const int x = n.in[0], w = n.in[1], ws = n.in[2], wz = opt_in(n, 3), b = opt_in(n, 4), y0 = n.out[0];
    if (x < 0 || w < 0 || ws < 0) return fail(ZANT_E_INVALID_INPUT, "QLinearConv needs x, w, w_scale");
    ZB_TRY(want_dtype(pl, w, ZANT_I8, "QLinearConv w")); ZB_TRY(want_dtype(pl, ws, ZANT_F32, "QLinearConv w_scale"));
    ZB_TRY(want_dtype(pl, wz, ZANT_I32, "QLinearConv w_zp")); ZB_TRY(want_dtype(pl, b, ZANT_I32, "QLinearConv bias"));
    const int32_t xd = T(x).dtype, yd = T(y0).dtype;
    if ((xd != ZANT_I8 && xd != ZANT_U8) || (yd != ZANT_I8 && yd != ZANT_U8)) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QLinearConv x/y dtype");
    ZB_TRY(check_zero_point(xd, a.x_zp, "QLinearConv x"));
    if (!T(w).is_const || !T(ws).is_const || (wz >= 0 && !T(wz).is_const)) return fail(ZANT_E_UNSUPPORTED, "QLinearConv weights and scales must be initializers");
    ConvGeom g;
    if (a.channels_last) {
        // the geometry is that of the NCHW operator on the permuted shapes
        if (T(x).shape.size() != 4 || T(y0).shape.size() != 4) return fail(ZANT_E_INVALID_DIMENSIONS, "channels-last QLinearConv takes rank-4 tensors");
        const size_t xs[4] = {T(x).shape[0], T(x).shape[3], T(x).shape[1], T(x).shape[2]}, ys[4] = {T(y0).shape[0], T(y0).shape[3], T(y0).shape[1], T(y0).shape[2]};
        ZB_TRY(conv_resolve_onnx(xs, 4, T(w).shape.data(), T(w).shape.size(), ys, 4,
                                 a.strides, a.n_strides, a.pads, a.n_pads, a.dilations, a.n_dilations, a.group, a.auto_pad < 0 ? 0 : a.auto_pad, g));
    } else {
        ZB_TRY(conv_resolve_onnx(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(), T(y0).shape.data(), T(y0).shape.size(),
                                 a.strides, a.n_strides, a.pads, a.n_pads, a.dilations, a.n_dilations, a.group, a.auto_pad < 0 ? 0 : a.auto_pad, g));
    }
    const size_t nws = numel(T(ws).shape.data(), T(ws).shape.size());
    if (nws != 1 && nws != (size_t)g.M) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearConv w_scale size");
    if (b >= 0 && numel(T(b).shape.data(), T(b).shape.size()) != (size_t)g.M) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearConv bias size");
    std::vector<float> mult;
    requant_multipliers(a.x_scale, (const float*)T(ws).host.data(), nws, a.y_scale, (size_t)g.M, mult);
    std::vector<int32_t> wzv((size_t)g.M, 0);
    if (wz >= 0) {
        const size_t nwz = numel(T(wz).shape.data(), T(wz).shape.size());
        if (nwz != 1 && nwz != (size_t)g.M) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearConv w_zp size");
        for (int m = 0; m < g.M; ++m) wzv[m] = ((const int32_t*)T(wz).host.data())[nwz == 1 ? 0 : m];
    }
    const int xzp = a.x_zp;
    const Requant rq0{a.y_scale, a.y_zp, fz.activation >= 0 ? fz.activation : a.activation};
    const int lut_aux = fz.lut_aux;
    // the requantisation parameters with the table's device address, resolved at launch time (the arena exists by then)
    auto rq_of = [pl, rq0, lut_aux]() { Requant r = rq0; r.lut = lut_aux >= 0 ? (const uint8_t*)pl->aux(lut_aux) : nullptr; return r; };
    bool wz_zero = true;
    for (int32_t v : wzv) wz_zero = wz_zero && v == 0;
    const bool const_bias = b < 0 || T(b).is_const;
    const int y = fz.y_act >= 0 ? fz.y_act : y0;          // written unless the pool is fused too
    const std::string tail = std::string(fz.activation >= 0 ? "+Relu" : "") + (lut_aux >= 0 ? "+ActivationLut" : "");
    auto push = [&](const std::string& name, std::function<int32_t()> fn) { pl->steps.push_back(std::move(fn)); pl->step_names.push_back(name); };
    fz.pool_done = false;
    // a QLinearAdd behind the convolution, for the kernels that take it: the sum's tensor, and the operation with its operand's address
    const int add_res = fz.add_res, y_sum = fz.add_node >= 0 ? pl->nodes[fz.add_node].out[0] : -1;
    QAddTail add0{};
    if (fz.add_node >= 0) {
        const PlanNode& an = pl->nodes[fz.add_node];
        const bool first = an.in[0] == add_res;
        add0 = pl->prove(qadd_tail<false>(first ? an.a.x_scale : an.a.b_scale, first ? an.a.x_zp : an.a.b_zp, first ? an.a.b_scale : an.a.x_scale, first ? an.a.b_zp : an.a.x_zp, an.a.y_scale, an.a.y_zp, an.a.activation));
    }
    auto add_of = [pl, add0, add_res]() { QAddTail t = add0; t.res = (const uint8_t*)pl->ptr(add_res); return t; };

    if (a.channels_last) {
        TcConvPlan ncp;
        if (!const_bias || !tc_conv_nhwc_plan(g, wz_zero, xzp, ncp)) return fail(ZANT_E_UNSUPPORTED, "shape not taken by the channels-last QLinearConv kernel");
        std::vector<int8_t> w_blk; std::vector<float> mp; std::vector<int32_t> bp;
        tc_conv_nhwc_prepare(ncp, (const int8_t*)T(w).host.data(), mult.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, w_blk, mp, bp);
        const int aw = pl->add_aux(w_blk.data(), w_blk.size()), am = pl->add_aux(mp.data(), mp.size() * 4), ab = pl->add_aux(bp.data(), bp.size() * 4);
        const double max_product = tc_conv_max_product(mp, bp, (long long)g.Cg * g.KH * g.KW);
        push("QLinearConv(tc-nhwc)" + tail, [=]() {
            if (!tc_conv_ptr_ok(pl->ptr(x)) || !tc_conv_ptr_ok(pl->ptr(y))) return fail(ZANT_E_INVALID_INPUT, "channels-last QLinearConv buffers must be 16-byte aligned");
            return tc_conv_nhwc_run(ctx, ncp, pl->ptr(x), xd == ZANT_U8, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am),
                                    (const int32_t*)pl->aux(ab), pl->ptr(y), yd == ZANT_U8, rq_of(), max_product);
        });
        return ZANT_OK;
    }
    PwConvPlan pwp;
    const bool stem = const_bias && pw_stem_plan(g, wz_zero, xzp, ctx->sm_count, pwp);
    if (stem || (const_bias && pw_conv_plan(g, wz_zero, ctx->sm_count, pwp))) {
        // 1x1: filters on the accumulator lanes, activations straight from NCHW as the MN-major operand; 3x3 stems: the same
        // kernel on patches written in shared memory
        std::vector<int8_t> w_blk; std::vector<int32_t> bf;
        pw_conv_prepare(pwp, (const int8_t*)T(w).host.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, w_blk, bf);
        bool finite = true;
        for (float f : mult) finite = finite && std::isfinite(f);
        const int aw = pl->add_aux(w_blk.data(), w_blk.size()), am = pl->add_aux(mult.data(), mult.size() * 4), ab = pl->add_aux(bf.data(), bf.size() * 4);
        std::vector<int32_t> caps;
        const bool capped = finite && yd == ZANT_I8 && rq0.y_zp == 0 && requant_relu_caps(mult.data(), mult.size(), rq0.act, lean_six(rq0.y_scale), caps);
        const int ac = capped ? pl->add_aux(caps.data(), caps.size() * 4) : -1;
        // In the short form (proved) from 384 KB of output on with at most 64 filters, from 1 MB with more, where a CTA has enough pixels for the
        // longer epilogue to cost less than a launch (us, in it / as a step of its own: 24 filters at 56 x 56 294 KB 22.1 / 21.9, 882 KB 23.5 / 24.3, 9.4 MB
        // 59 / 59, 107 MB 491 / 497; 96 at 20 x 20 225 KB 23.2 / 20.4, 900 KB 25.8 / 25.3, 37 MB 240 / 249; 256 at 28 x 28 392 KB 23.1 / 20.5, 1.6 MB 23.5 /
        // 23.0, 98 MB 251 / 264).  The long form from 8 MB (its 15 instructions a value cost more than the launch at every size: 24 filters at
        // 56 x 56 9.4 MB 88 / 71, 107 MB 793 / 648; below 8 MB it is a step of its own).
        const long long add_from = add0.proved ? (g.M <= 64 ? 384LL << 10 : 1LL << 20) : 8LL << 20;
        if (!stem && fz.add_node >= 0 && (long long)g.N * g.M * g.OH * g.OW >= add_from && xd == ZANT_I8 && yd == ZANT_I8 && rq0.y_zp == 0 && finite) {
            fz.add_done = true;
            push("QLinearConv(tc-pointwise)" + tail + "+QLinearAdd", [=]() {
                if (!pw_conv_ptr_ok(pl->ptr(x), pl->ptr(y_sum))) return fail(ZANT_E_INVALID_INPUT, "pointwise QLinearConv buffers must be 16-byte (input) and 32-byte (output) aligned");
                const QAddTail add = add_of();
                return pw_conv_run(ctx, pwp, pl->ptr(x), false, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am), (const int32_t*)pl->aux(ab), pl->ptr(y_sum), false, rq_of(), true,
                                   ac >= 0 ? (const int32_t*)pl->aux(ac) : nullptr, &add);
            });
            return ZANT_OK;
        }
        const std::vector<PwConvPlan> parts = stem ? std::vector<PwConvPlan>{} : pw_conv_parts(g, wz_zero, ctx->sm_count, pwp);
        if (!parts.empty()) {
            std::vector<int> aws, abs;
            int m0 = 0;
            for (const PwConvPlan& part : parts) {
                pw_conv_prepare(part, (const int8_t*)T(w).host.data() + (size_t)m0 * g.C, b >= 0 ? (const int32_t*)T(b).host.data() + m0 : nullptr, xzp, w_blk, bf);
                aws.push_back(pl->add_aux(w_blk.data(), w_blk.size())); abs.push_back(pl->add_aux(bf.data(), bf.size() * 4));
                m0 += part.a.M;
            }
            push("QLinearConv(tc-pointwise)" + tail, [=]() {
                if (!pw_conv_ptr_ok(pl->ptr(x), pl->ptr(y))) return fail(ZANT_E_INVALID_INPUT, "pointwise QLinearConv buffers must be 16-byte (input) and 32-byte (output) aligned");
                int at = 0;
                for (size_t i = 0; i < parts.size(); ++i) {
                    ZB_TRY(pw_conv_run(ctx, parts[i], pl->ptr(x), xd == ZANT_U8, (const int8_t*)pl->aux(aws[i]), (const float*)pl->aux(am) + at, (const int32_t*)pl->aux(abs[i]),
                                       (uint8_t*)pl->ptr(y) + (size_t)at * g.H * g.W, yd == ZANT_U8, rq_of(), finite, ac >= 0 ? (const int32_t*)pl->aux(ac) + at : nullptr));
                    at += parts[i].a.M;
                }
                return (int32_t)ZANT_OK;
            });
            return ZANT_OK;
        }
        push(std::string(stem ? "QLinearConv(tc-stem)" : "QLinearConv(tc-pointwise)") + tail, [=]() {
            if (!pw_conv_ptr_ok(pl->ptr(x), pl->ptr(y))) return fail(ZANT_E_INVALID_INPUT, "pointwise QLinearConv buffers must be 16-byte (input) and 32-byte (output) aligned");
            return pw_conv_run(ctx, pwp, pl->ptr(x), xd == ZANT_U8, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am),
                               (const int32_t*)pl->aux(ab), pl->ptr(y), yd == ZANT_U8, rq_of(), finite, ac >= 0 ? (const int32_t*)pl->aux(ac) : nullptr);
        });
        return ZANT_OK;
    }
    if (const_bias && qconv_smallc_eligible(g, wz_zero)) {
        // 3x3 on at most four input channels (network stems); arena tensors are 256-byte aligned
        std::vector<uint32_t> wfrag; std::vector<int32_t> bf;
        qconv_smallc_prepare(g, (const int8_t*)T(w).host.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, wfrag, bf);
        const int aw = pl->add_aux(wfrag.data(), wfrag.size() * 4), am = pl->add_aux(mult.data(), mult.size() * 4), ab = pl->add_aux(bf.data(), bf.size() * 4);
        const double max_product = tc_conv_max_product(mult, bf, (long long)g.C * 9);
        push("QLinearConv(small-c)" + tail, [=]() {
            if (!qconv_smallc_ptr_ok(pl->ptr(x))) return fail(ZANT_E_INVALID_INPUT, "QLinearConv input buffer must be 4-byte aligned");
            return run_qconv_smallc(ctx, g, pl->ptr(x), xd == ZANT_U8, xzp, (const uint32_t*)pl->aux(aw), (const float*)pl->aux(am),
                                    (const int32_t*)pl->aux(ab), pl->ptr(y), yd == ZANT_U8, rq_of(), max_product);
        });
        return ZANT_OK;
    }
    TcConvPlan tcp;
    if (const_bias && (long long)g.N * g.OH * g.OW >= 256) {
        // implicit GEMM from NCHW (stride 1): weights blocked once here, one launch per run; with a fused pool the
        // epilogue writes the pooled tensor only.  Arena tensors are 256-byte aligned; a caller-bound input that is
        // not 16-byte aligned is refused at run time.
        const bool pooled = fz.y_pool >= 0 && tc_conv_plan(g, wz_zero, tcp, true);
        if (pooled || tc_conv_plan(g, wz_zero, tcp, false)) {
            std::vector<int8_t> w_blk; std::vector<float> mp; std::vector<int32_t> bp;
            tc_conv_prepare(tcp, (const int8_t*)T(w).host.data(), mult.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, w_blk, mp, bp);
            const int aw = pl->add_aux(w_blk.data(), w_blk.size()), am = pl->add_aux(mp.data(), mp.size() * 4), ab = pl->add_aux(bp.data(), bp.size() * 4);
            const double max_product = tc_conv_max_product(mp, bp, (long long)g.Cg * g.KH * g.KW);
            const int yw = pooled ? fz.y_pool : y;
            fz.pool_done = pooled;
            push("QLinearConv(tc-implicit)" + tail + (pooled ? "+MaxPool" : ""), [=]() {
                if (!tc_conv_ptr_ok(pl->ptr(x))) return fail(ZANT_E_INVALID_INPUT, "QLinearConv input buffer must be 16-byte aligned");
                return tc_conv_run(ctx, tcp, pl->ptr(x), xd == ZANT_U8, xzp, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am),
                                   (const int32_t*)pl->aux(ab), pl->ptr(yw), yd == ZANT_U8, rq_of(), max_product);
            });
            return ZANT_OK;
        }
    }
    if (const_bias && qdwconv_eligible(g, wz_zero)) {
        // depthwise 3x3: one HBM-bound pass; arena tensors are 256-byte aligned
        std::vector<uint32_t> wrow; std::vector<int32_t> bf;
        qdwconv_prepare(g, (const int8_t*)T(w).host.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, wrow, bf);
        bool finite = true;
        for (float f : mult) finite = finite && std::isfinite(f);
        const int aw = pl->add_aux(wrow.data(), wrow.size() * 4), am = pl->add_aux(mult.data(), mult.size() * 4), ab = pl->add_aux(bf.data(), bf.size() * 4);
        std::vector<int32_t> caps;
        const bool capped = finite && yd == ZANT_I8 && rq0.y_zp == 0 && requant_relu_caps(mult.data(), mult.size(), rq0.act, lean_six(rq0.y_scale), caps);
        const int ac = capped ? pl->add_aux(caps.data(), caps.size() * 4) : -1;
        push("QLinearConv(depthwise)" + tail, [=]() {
            if (!qdwconv_ptr_ok(pl->ptr(x)) || !qdwconv_ptr_ok(pl->ptr(y))) return fail(ZANT_E_INVALID_INPUT, "depthwise QLinearConv buffers must be 4-byte aligned");
            return run_qdwconv(ctx, g, pl->ptr(x), xd == ZANT_U8, xzp, (const uint32_t*)pl->aux(aw), (const float*)pl->aux(am),
                               (const int32_t*)pl->aux(ab), pl->ptr(y), yd == ZANT_U8, rq_of(), finite, ac >= 0 ? (const int32_t*)pl->aux(ac) : nullptr);
        });
        return ZANT_OK;
    }
    if (qconv_tc_eligible(g, wz_zero) && const_bias) {
        // tensor-core path: weights re-blocked once here, im2col + tcgen05 GEMM per run
        auto prep = std::make_shared<QGemmPrep>();
        qconv_gemm_prepare(g, (const int8_t*)T(w).host.data(), mult.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, *prep, ctx->sm_count);
        const int aw = pl->add_aux(prep->w_blk.data(), prep->w_blk.size()), am = pl->add_aux(prep->mult.data(), prep->mult.size() * 4);
        const int ab = pl->add_aux(prep->bias.data(), prep->bias.size() * 4);
        const int sa = pl->shared_im2col_scratch(qgemm_a_bytes((size_t)g.N * g.OH * g.OW, *prep));
        prep->w_blk.clear(); prep->w_blk.shrink_to_fit();
        push("QLinearConv(tc)" + tail, [=]() {
            return run_qconv_tc(ctx, g, pl->ptr(x), xd == ZANT_U8, xzp, *prep, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am),
                                (const int32_t*)pl->aux(ab), (uint8_t*)pl->scratch(sa), pl->ptr(y), yd == ZANT_U8, rq_of());
        });
        return ZANT_OK;
    }
    if (const_bias && small_gemm_eligible(g, wz_zero)) {
        // few output positions: warp-level MMAs, K split over the warps of many small CTAs
        const SmallGemmPlan sg = small_gemm_plan(g, ctx->sm_count);
        const int aw = pl->add_scratch(sg.w_bytes), am = pl->add_aux(mult.data(), mult.size() * 4), ab = xzp != 0 ? pl->add_scratch((size_t)g.M * 4) : -1;
        auto bias_of = [=]() { return ab >= 0 ? (int32_t*)pl->scratch(ab) : pl->p<int32_t>(b); };
        pl->init_steps.push_back([=]() { return run_small_gemm_weights(ctx, g, sg, false, pl->p<int8_t>(w), pl->p<int32_t>(b), xzp, pl->scratch(aw), bias_of()); });
        if (fz.add_node >= 0 && yd == ZANT_I8) {
            fz.add_done = true;
            push("QLinearConv" + tail + "+QLinearAdd", [=]() {
                const QAddTail add = add_of();
                return run_small_gemm(ctx, g, sg, pl->ptr(x), xd == ZANT_U8, xzp, pl->scratch(aw), (const float*)pl->aux(am), bias_of(), pl->ptr(y_sum), false, rq_of(), &add);
            });
            return ZANT_OK;
        }
        push("QLinearConv" + tail, [=]() {
            return run_small_gemm(ctx, g, sg, pl->ptr(x), xd == ZANT_U8, xzp, pl->scratch(aw), (const float*)pl->aux(am), bias_of(), pl->ptr(y), yd == ZANT_U8, rq_of());
        });
        return ZANT_OK;
    }
    const int am = pl->add_aux(mult.data(), mult.size() * 4), az = pl->add_aux(wzv.data(), wzv.size() * 4);
    push("QLinearConv" + tail, [=]() {
        QConvArgs q{};
        q.x = pl->ptr(x); q.w = pl->p<int8_t>(w); q.y = pl->ptr(y);
        q.mult = (const float*)pl->aux(am); q.w_zp = (const int32_t*)pl->aux(az); q.bias = pl->p<int32_t>(b);
        q.x_zp = xzp; q.rq = rq_of(); q.g = g;
        return run_qconv_generic(ctx, q, xd, yd);
    });
    return ZANT_OK;
}

// --------------------------------------------------------------------------------------------
// One node -> one (or a few) kernel launches, using the same resolvers as the single-op ABI.
// --------------------------------------------------------------------------------------------
static int32_t build_node(zant_plan* pl, size_t node_index, int32_t fuse) {
    const size_t first_step = pl->steps.size();
    ZB_TRY(build_node_impl(pl, node_index, fuse));
    record_step_cost(pl, first_step, node_index, 1);
    return ZANT_OK;
}

static int32_t build_node_impl(zant_plan* pl, size_t node_index, int32_t /*fuse*/) {
    const PlanNode& n = pl->nodes[node_index];
    const zant_node_attrs& a = n.a;
    zant_ctx* ctx = pl->ctx;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    auto push = [&](const char* name, std::function<int32_t()> fn) { pl->steps.push_back(std::move(fn)); pl->step_names.push_back(name); };

    switch (n.op) {
        case ZANT_OP_CONV: {
            ZB_TRY(need_inputs(n, 2, 3, "Conv"));
            const int x = n.in[0], w = n.in[1], b = opt_in(n, 2), y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "Conv")); ZB_TRY(want_dtype(pl, w, ZANT_F32, "Conv")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "Conv"));
            ConvGeom g;
            const char* ap = (a.auto_pad >= 0 && a.auto_pad <= 3) ? kAutoPadNames[a.auto_pad] : nullptr;
            ZB_TRY(conv_resolve_ref(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(),
                                    T(y).shape.data(), T(y).shape.size(), a.strides, a.n_strides,
                                    a.n_pads ? a.pads : nullptr, a.n_pads, a.n_dilations ? a.dilations : nullptr, a.n_dilations,
                                    a.group, ap, ap ? std::strlen(ap) : 0, g));
            if (b >= 0 && numel(T(b).shape.data(), T(b).shape.size()) != (size_t)g.M) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "Conv bias size");
            if (ctx->tf32 && T(w).is_const && (b < 0 || T(b).is_const) && g.M <= 2048 && (long long)g.N * g.OH * g.OW >= 128) {
                // tensor-core float path: weights blocked once here; im2col gather + tcgen05 kind::tf32 GEMM per run, with the
                // activation the fusion pass found behind the node in the epilogue
                auto prep = std::make_shared<TfGemmPrep>();
                const int K = g.C * g.KH * g.KW;
                tf_gemm_prepare((const float*)T(w).host.data(), g.M, K, K, 1, b >= 0 ? (const float*)T(b).host.data() : nullptr, *prep, (long long)g.N * g.OH * g.OW, ctx->tf32 == 2);
                tf_conv_table(g, *prep);
                const int aw = pl->add_aux(prep->w_blk.data(), prep->w_blk.size() * 4), ab = pl->add_aux(prep->bias.data(), prep->bias.size() * 4);
                const int at = pl->add_aux(prep->ktab.data(), prep->ktab.size() * 4);
                const int sa = pl->shared_im2col_scratch(tf_gemm_a_bytes((size_t)g.N * g.OH * g.OW, *prep));
                prep->w_blk.clear(); prep->w_blk.shrink_to_fit();
                const int fact = pl->pending_fact; const float fslope = pl->pending_slope;
                const int yw = pl->pending_y >= 0 ? pl->pending_y : y;
                push(fact == FACT_NONE ? "Conv(tf32)" : (fact == FACT_RELU ? "Conv(tf32)+Relu" : "Conv(tf32)+LeakyRelu"), [=]() {
                    return run_conv_tf32(ctx, g, pl->p<float>(x), *prep, (const float*)pl->aux(aw), (const float*)pl->aux(ab), (const int32_t*)pl->aux(at), (float*)pl->scratch(sa), fact, fslope, pl->p<float>(yw));
                });
                pl->pending_used = true;
                return ZANT_OK;
            }
            // exact path; constant weights are transposed once to [K][filters], the order the kernel's slabs have
            const int K = g.C * g.KH * g.KW, N4 = (g.M + 3) / 4 * 4;
            int at = -1;
            if (T(w).is_const && (long long)K * N4 <= (1LL << 28) && K <= 65535 * 32) {
                at = pl->add_scratch((size_t)K * N4 * 4);
                pl->init_steps.push_back([=]() { return run_transpose_pad_f32(ctx, pl->p<float>(w), (float*)pl->scratch(at), g.M, K, N4); });
            }
            const int fact = pl->pending_fact; const float fslope = pl->pending_slope;
            const bool pool = pl->pending_pool >= 0;
            const int yw = pool ? pl->pending_pool : (pl->pending_y >= 0 ? pl->pending_y : y);
            pl->pending_used = pool || pl->pending_y >= 0;
            const std::string name = std::string("Conv") + (fact == FACT_RELU ? "+Relu" : (fact == FACT_LEAKY ? "+LeakyRelu" : "")) + (pool ? "+MaxPool" : "");
            push(name.c_str(), [=]() {
                ContractFusion fu;
                fu.act = fact == FACT_RELU ? CT_ACT_RELU : (fact == FACT_LEAKY ? CT_ACT_LEAKY : CT_ACT_NONE); fu.slope = fslope; fu.pool = pool;
                return run_conv_f32(ctx, g, pl->p<float>(x), pl->p<float>(w), pl->p<float>(b), pl->p<float>(yw), fu, at >= 0 ? (const float*)pl->scratch(at) : nullptr);
            });
            return ZANT_OK;
        }
        case ZANT_OP_MATMUL: {
            ZB_TRY(need_inputs(n, 2, 2, "MatMul"));
            const int x = n.in[0], w = n.in[1], y = n.out[0];
            MatGeom g;
            ZB_TRY(matmul_check(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(), T(y).shape.data(), T(y).shape.size(), g));
            if (ctx->tf32 && T(w).is_const && T(w).dtype == ZANT_F32 && g.N <= 2048 && g.M >= 128 && g.K <= 0x7fffffffULL && g.M <= 0x7fffffffULL) {
                auto prep = std::make_shared<TfGemmPrep>();
                tf_gemm_prepare((const float*)T(w).host.data(), (int)g.N, (int)g.K, 1, (long long)g.N, nullptr, *prep, (long long)g.M, ctx->tf32 == 2);
                const int aw = pl->add_aux(prep->w_blk.data(), prep->w_blk.size() * 4), ab = pl->add_aux(prep->bias.data(), prep->bias.size() * 4);
                const int sa = pl->shared_im2col_scratch(tf_gemm_a_bytes(g.M, *prep));
                prep->w_blk.clear(); prep->w_blk.shrink_to_fit();
                const MatGeom gg = g;
                push("MatMul(tf32)", [=]() {
                    return run_matmul_tf32(ctx, pl->p<float>(x), (long long)gg.M, (int)gg.K, (long long)gg.K, 1, *prep, (const float*)pl->aux(aw), (const float*)pl->aux(ab),
                                           (float*)pl->scratch(sa), FACT_NONE, 0.0f, pl->p<float>(y));
                });
                return ZANT_OK;
            }
            push("MatMul", [=]() { return run_matmul_f32(ctx, g, pl->p<float>(x), pl->p<float>(w), pl->p<float>(y)); });
            return ZANT_OK;
        }
        case ZANT_OP_GEMM: {
            ZB_TRY(need_inputs(n, 2, 3, "Gemm"));
            const int x = n.in[0], w = n.in[1], c = opt_in(n, 2), y = n.out[0];
            GemmGeom g;
            ZB_TRY(gemm_check_lean(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(),
                              c >= 0 ? T(c).shape.data() : nullptr, c >= 0 ? T(c).shape.size() : 0, c >= 0,
                              a.trans_a != 0, a.trans_b != 0, a.beta, T(y).shape.data(), T(y).shape.size(), g));
            const float alpha = a.alpha, beta = a.beta; const bool ta = a.trans_a != 0, tb = a.trans_b != 0;
            {
                // tensor-core float path for the fully-connected form: Y = A B' + row vector C (alpha = beta = 1)
                const bool c_row = c < 0 || (T(c).is_const && beta == 1.0f && g.c_mode != 0 && g.c_rows == 1 && g.c_cols == g.cols && numel(T(c).shape.data(), T(c).shape.size()) == g.cols);
                if (ctx->tf32 && !ta && alpha == 1.0f && T(w).is_const && c_row && g.batch == 1 && g.cols <= 2048 && g.rows >= 128 && g.K <= 0x7fffffffULL && g.rows <= 0x7fffffffULL) {
                    auto prep = std::make_shared<TfGemmPrep>();
                    tf_gemm_prepare((const float*)T(w).host.data(), (int)g.cols, (int)g.K, tb ? (long long)g.K : 1, tb ? 1 : (long long)g.cols,
                                    c >= 0 ? (const float*)T(c).host.data() : nullptr, *prep, (long long)g.rows, ctx->tf32 == 2);
                    const int aw = pl->add_aux(prep->w_blk.data(), prep->w_blk.size() * 4), ab = pl->add_aux(prep->bias.data(), prep->bias.size() * 4);
                    const int sa = pl->shared_im2col_scratch(tf_gemm_a_bytes(g.rows, *prep));
                    prep->w_blk.clear(); prep->w_blk.shrink_to_fit();
                    const GemmGeom gg = g;
                    push("Gemm(tf32)", [=]() {
                        return run_matmul_tf32(ctx, pl->p<float>(x), (long long)gg.rows, (int)gg.K, (long long)gg.K, 1, *prep, (const float*)pl->aux(aw), (const float*)pl->aux(ab),
                                               (float*)pl->scratch(sa), FACT_NONE, 0.0f, pl->p<float>(y));
                    });
                    return ZANT_OK;
                }
            }
            push("Gemm", [=]() { return run_gemm_f32(ctx, g, pl->p<float>(x), pl->p<float>(w), pl->p<float>(c), alpha, beta, ta, tb, pl->p<float>(y)); });
            return ZANT_OK;
        }
        case ZANT_OP_MAXPOOL: {
            ZB_TRY(need_inputs(n, 1, 1, "MaxPool"));
            const int x = n.in[0], y = n.out[0];
            PoolGeom g;
            const size_t ones[2] = {1, 1};
            ZB_TRY(pool_resolve(T(x).shape.data(), T(x).shape.size(), T(y).shape.data(), T(y).shape.size(), a.kernel_shape, 2,
                                a.n_strides ? a.strides : ones, 2, a.n_dilations ? a.dilations : ones, 2, a.pads, a.n_pads, a.auto_pad < 0 ? 0 : a.auto_pad, g));
            const int32_t dt = T(x).dtype;
            if (dt != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "MaxPool dtype mismatch");
            if (dt == ZANT_F32) push("MaxPool", [=]() { return run_maxpool<float>(ctx, g, pl->p<float>(x), pl->p<float>(y)); });
            else if (dt == ZANT_I8) push("MaxPool", [=]() { return run_maxpool<int8_t>(ctx, g, pl->p<int8_t>(x), pl->p<int8_t>(y)); });
            else if (dt == ZANT_U8) push("MaxPool", [=]() { return run_maxpool<uint8_t>(ctx, g, pl->p<uint8_t>(x), pl->p<uint8_t>(y)); });
            else return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "MaxPool on int32");
            return ZANT_OK;
        }
        case ZANT_OP_TRANSPOSE:
        case ZANT_OP_SLICE: {
            ZB_TRY(need_inputs(n, 1, 1, "Transpose/Slice"));
            const int x = n.in[0], y = n.out[0];
            if (T(x).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Transpose/Slice dtype mismatch");
            StridedMap m;
            const std::vector<size_t>& xs = T(x).shape; const std::vector<size_t>& ys = T(y).shape;
            if (n.op == ZANT_OP_TRANSPOSE) {
                size_t perm[8];
                if (a.n_perm > 8) return fail(ZANT_E_INVALID_PERMUTATION, "perm holds %zu entries", a.n_perm);
                for (size_t i = 0; i < a.n_perm; ++i) perm[i] = a.perm[i] < 0 ? (size_t)-1 : (size_t)a.perm[i];
                ZB_TRY(transpose_resolve(xs.data(), xs.size(), a.n_perm ? perm : nullptr, a.n_perm, ys.data(), ys.size(), m));
            } else {
                if (a.n_slice > 8) return fail(ZANT_E_INVALID_SLICE_INDICES, "%zu slice entries", a.n_slice);
                size_t od[8];
                ZB_TRY(slice_resolve(xs.data(), xs.size(), a.slice_starts, a.slice_ends, a.n_slice, a.slice_has_axes ? a.slice_axes : nullptr,
                                     a.slice_has_steps ? a.slice_steps : nullptr, od, &m));
                if (ys.size() != xs.size()) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "Slice output rank");
                for (size_t d = 0; d < xs.size(); ++d) if (ys[d] != od[d]) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "Slice output dim %zu", d);
            }
            const size_t esz = dtype_size(T(x).dtype);
            push(n.op == ZANT_OP_TRANSPOSE ? "Transpose" : "Slice", [=]() { return run_strided_copy(ctx, esz, pl->ptr(x), pl->ptr(y), m); });
            return ZANT_OK;
        }
        case ZANT_OP_GATHER: {
            ZB_TRY(need_inputs(n, 2, 2, "Gather"));
            const int x = n.in[0], ind = n.in[1], y = n.out[0];
            if (T(x).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Gather dtype mismatch");
            ZB_TRY(want_dtype(pl, ind, ZANT_I32, "Gather indices"));
            if (!T(ind).is_const) return fail(ZANT_E_UNSUPPORTED, "Gather indices must be an initializer");
            const size_t ni = numel(T(ind).shape.data(), T(ind).shape.size());
            std::vector<size_t> idx(ni);
            for (size_t i = 0; i < ni; ++i) {
                const int32_t v = ((const int32_t*)T(ind).host.data())[i];
                idx[i] = v < 0 ? (size_t)-1 : (size_t)v;      // a negative index is out of bounds, as for the reference's usize
            }
            GatherGeom g;
            ZB_TRY(gather_resolve(T(x).shape.data(), T(x).shape.size(), idx.data(), T(ind).shape.data(), T(ind).shape.size(), a.axis,
                                  T(y).shape.data(), T(y).shape.size(), g));
            const size_t esz = dtype_size(T(x).dtype);
            push("Gather", [=]() { return run_gather(ctx, esz, pl->ptr(x), pl->p<int32_t>(ind), pl->ptr(y), g); });
            return ZANT_OK;
        }
        case ZANT_OP_SIGMOID:
        case ZANT_OP_TANH:
        case ZANT_OP_CEIL: {
            ZB_TRY(need_inputs(n, 1, 1, "unary"));
            const int x = n.in[0], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "unary")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "unary"));
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(y).shape.data(), T(y).shape.size())) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "unary sizes differ");
            if (n.op == ZANT_OP_SIGMOID) push("Sigmoid", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, SigmoidOp{}, "sigmoid_f32"); });
            else if (n.op == ZANT_OP_TANH) push("Tanh", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, TanhOp{}, "tanh_f32"); });
            else push("Ceil", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, CeilOp{}, "ceil_f32"); });
            return ZANT_OK;
        }
        case ZANT_OP_SOFTMAX: {
            ZB_TRY(need_inputs(n, 1, 1, "Softmax"));
            const int x = n.in[0], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "Softmax")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "Softmax"));
            if (T(x).shape.size() != 2) return fail(ZANT_E_INVALID_DIMENSIONS, "Softmax takes a 2-D tensor");
            if (T(y).shape != T(x).shape) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "Softmax shapes differ");
            const size_t rows = T(x).shape[0], cols = T(x).shape[1];
            push("Softmax", [=]() { return run_softmax_f32(ctx, pl->p<float>(x), pl->p<float>(y), rows, cols); });
            return ZANT_OK;
        }
        case ZANT_OP_MUL:
        case ZANT_OP_DIV: {
            ZB_TRY(need_inputs(n, 2, 2, "Mul/Div"));
            const int x = n.in[0], w = n.in[1], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "Mul/Div")); ZB_TRY(want_dtype(pl, w, ZANT_F32, "Mul/Div")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "Mul/Div"));
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(w).shape.data(), T(w).shape.size())) return fail(ZANT_E_MISMATCHED_SHAPE, "Mul/Div operands differ in size");
            if (cnt != numel(T(y).shape.data(), T(y).shape.size())) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "Mul/Div output size");
            const bool divide = n.op == ZANT_OP_DIV;
            push(divide ? "Div" : "Mul", [=]() { return run_binary_same_f32(ctx, pl->p<float>(x), pl->p<float>(w), pl->p<float>(y), cnt, divide); });
            return ZANT_OK;
        }
        case ZANT_OP_RELU:
        case ZANT_OP_LEAKY_RELU:
        case ZANT_OP_CLIP: {
            ZB_TRY(need_inputs(n, 1, 1, "activation"));
            const int x = n.in[0], y = n.out[0];
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(y).shape.data(), T(y).shape.size())) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "activation sizes differ");
            const int32_t dt = T(x).dtype;
            if (dt != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "activation dtype mismatch");
            const float p0 = a.alpha, p1 = a.beta;
            if (dt == ZANT_F32) {
                if (n.op == ZANT_OP_RELU) push("Relu", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, ReluOp{}, "relu_f32"); });
                else if (n.op == ZANT_OP_LEAKY_RELU) push("LeakyRelu", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, LeakyOp{p0}, "leaky_relu_f32"); });
                else push("Clip", [=]() { return run_unary_f32(ctx, pl->p<float>(x), pl->p<float>(y), cnt, ClipOp{p0, p1}, "clip_f32"); });
                return ZANT_OK;
            }
            if (dt == ZANT_I32) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "activation on int32");
            // Quantized tensors: dequantise, activate, requantise through a 256-entry table.
            uint8_t lut[256];
            activation_lut(n, dt, lut);
            const int aux = pl->add_aux(lut, 256);
            push("ActivationLut", [=]() { return run_lut(ctx, pl->p<char>(x), pl->p<char>(y), cnt, (const uint8_t*)pl->aux(aux)); });
            return ZANT_OK;
        }
        case ZANT_OP_ADD: {
            ZB_TRY(need_inputs(n, 2, 2, "Add"));
            const int x = n.in[0], w = n.in[1], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "Add")); ZB_TRY(want_dtype(pl, w, ZANT_F32, "Add")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "Add"));
            BcastGeom g;
            ZB_TRY(bcast_resolve(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(), T(y).shape.data(), T(y).shape.size(), g));
            push("Add", [=]() { return run_add_f32(ctx, g, pl->p<float>(x), pl->p<float>(w), pl->p<float>(y)); });
            return ZANT_OK;
        }
        case ZANT_OP_CONCAT: {
            if (n.in.empty() || n.out.size() != 1) return fail(ZANT_E_EMPTY_TENSOR_LIST, "Concat needs inputs and one output");
            const int y = n.out[0];
            std::vector<const size_t*> shapes; std::vector<size_t> ranks;
            for (int id : n.in) {
                if (id < 0) return fail(ZANT_E_INVALID_INPUT, "Concat input missing");
                if (T(id).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Concat dtype mismatch");
                shapes.push_back(T(id).shape.data()); ranks.push_back(T(id).shape.size());
            }
            ConcatGeom g; size_t os[8];
            ZB_TRY(concat_resolve(shapes.data(), ranks.data(), n.in.size(), a.axis, os, g));
            if (T(y).shape.size() != g.rank) return fail(ZANT_E_MISMATCHED_RANK, "Concat output rank");
            for (size_t d = 0; d < g.rank; ++d) if (T(y).shape[d] != os[d]) return fail(ZANT_E_MISMATCHED_SHAPE, "Concat output dim %zu", d);
            const size_t esz = dtype_size(T(y).dtype);
            const std::vector<int> ins = n.in;
            push("Concat", [=]() {
                std::vector<const void*> ptrs(ins.size());
                for (size_t i = 0; i < ins.size(); ++i) ptrs[i] = pl->ptr(ins[i]);
                return run_concat(ctx, g, esz, ptrs.data(), pl->ptr(y));
            });
            return ZANT_OK;
        }
        case ZANT_OP_RESIZE: {
            ZB_TRY(need_inputs(n, 1, 1, "Resize"));
            const int x = n.in[0], y = n.out[0];
            const size_t r = T(x).shape.size();
            if (r == 0 || r > 4 || a.n_scales != r) return fail(ZANT_E_INVALID_INPUT, "Resize scales length != rank");
            if (T(x).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Resize dtype mismatch");
            std::vector<size_t> os(r);
            ZB_TRY(resize_output_shape(T(x).shape.data(), r, a.scales, a.n_scales, nullptr, 0, os.data()));
            if (T(y).shape != os) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "Resize output shape");
            std::vector<int32_t> table, axis_offset;
            resize_index_table(T(x).shape.data(), os.data(), r, a.coord_mode, table, axis_offset);
            const int aux = pl->add_aux(table.data(), table.size() * 4);
            const std::vector<size_t> xs = T(x).shape;
            const size_t esz = dtype_size(T(x).dtype);
            push("Resize", [=]() { return run_resize(ctx, esz, pl->ptr(x), pl->ptr(y), (const int32_t*)pl->aux(aux), xs.data(), os.data(), r, axis_offset); });
            return ZANT_OK;
        }
        case ZANT_OP_REDUCE_MEAN: {
            ZB_TRY(need_inputs(n, 1, 1, "ReduceMean"));
            const int x = n.in[0], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "ReduceMean")); ZB_TRY(want_dtype(pl, y, ZANT_F32, "ReduceMean"));
            ReduceGeom g;
            ZB_TRY(reduce_resolve(T(x).shape.data(), T(x).shape.size(), T(y).shape.data(), T(y).shape.size(), a.n_axes ? a.axes : nullptr, a.n_axes, a.noop_with_empty_axes != 0, g));
            push("ReduceMean", [=]() { return run_reduce_mean_f32(ctx, g, pl->p<float>(x), pl->p<float>(y)); });
            return ZANT_OK;
        }
        case ZANT_OP_RESHAPE: {
            ZB_TRY(need_inputs(n, 1, 1, "Reshape"));
            const int x = n.in[0], y = n.out[0];
            if (T(x).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Reshape dtype mismatch");
            if (numel(T(x).shape.data(), T(x).shape.size()) != numel(T(y).shape.data(), T(y).shape.size()))
                return fail(ZANT_E_INPUT_ARRAY_WRONG_SIZE, "Reshape changes the element count");
            // Row-major order is preserved, so the output is a view: no kernel, no copy.
            pl->t[y].alias = x;
            return ZANT_OK;
        }
        case ZANT_OP_QUANTIZE_LINEAR: {
            ZB_TRY(need_inputs(n, 1, 1, "QuantizeLinear"));
            const int x = n.in[0], y = n.out[0];
            ZB_TRY(want_dtype(pl, x, ZANT_F32, "QuantizeLinear"));
            const int32_t dt = T(y).dtype;
            if (dt != ZANT_I8 && dt != ZANT_U8) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QuantizeLinear output dtype");
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(y).shape.data(), T(y).shape.size())) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "QuantizeLinear sizes differ");
            const float sc = a.y_scale; const int zp = a.y_zp;
            push("QuantizeLinear", [=]() { return run_quantize(ctx, pl->p<float>(x), pl->ptr(y), cnt, sc, zp, dt); });
            return ZANT_OK;
        }
        case ZANT_OP_DEQUANTIZE_LINEAR: {
            ZB_TRY(need_inputs(n, 1, 1, "DequantizeLinear"));
            const int x = n.in[0], y = n.out[0];
            ZB_TRY(want_dtype(pl, y, ZANT_F32, "DequantizeLinear"));
            const int32_t dt = T(x).dtype;
            if (dt == ZANT_F32) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "DequantizeLinear input dtype");
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(y).shape.data(), T(y).shape.size())) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "DequantizeLinear sizes differ");
            const float sc = a.x_scale; const int zp = a.x_zp;
            push("DequantizeLinear", [=]() { return run_dequantize(ctx, dt, pl->ptr(x), pl->p<float>(y), cnt, sc, zp); });
            return ZANT_OK;
        }
        case ZANT_OP_QLINEAR_CONV: {
            QConvFusion none;
            return build_qconv(pl, n, none);
        }
        case ZANT_OP_QLINEAR_MATMUL: {
            ZB_TRY(need_inputs(n, 3, 5, "QLinearMatMul"));
            const int x = n.in[0], w = n.in[1], ws = n.in[2], wz = opt_in(n, 3), b = opt_in(n, 4), y = n.out[0];
            if (x < 0 || w < 0 || ws < 0) return fail(ZANT_E_INVALID_INPUT, "QLinearMatMul needs a, b, b_scale");
            ZB_TRY(want_dtype(pl, w, ZANT_I8, "QLinearMatMul b")); ZB_TRY(want_dtype(pl, ws, ZANT_F32, "QLinearMatMul b_scale"));
            ZB_TRY(want_dtype(pl, wz, ZANT_I32, "QLinearMatMul b_zp")); ZB_TRY(want_dtype(pl, b, ZANT_I32, "QLinearMatMul bias"));
            const int32_t xd = T(x).dtype, yd = T(y).dtype;
            if (xd != ZANT_I8 && xd != ZANT_U8) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QLinearMatMul a dtype");
            ZB_TRY(check_zero_point(xd, a.x_zp, "QLinearMatMul a"));
            if (yd == ZANT_F32) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QLinearMatMul y dtype");
            if (!T(w).is_const || !T(ws).is_const || (wz >= 0 && !T(wz).is_const)) return fail(ZANT_E_UNSUPPORTED, "QLinearMatMul weights and scales must be initializers");
            if (T(x).shape.size() != 2 || T(w).shape.size() != 2 || T(y).shape.size() != 2) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearMatMul takes 2-D operands");
            const size_t M = T(x).shape[0], K = T(x).shape[1], N = T(w).shape[1];
            if (T(w).shape[0] != K || M * N == 0 || K == 0) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearMatMul inner dims");
            if (T(y).shape[0] != M || T(y).shape[1] != N) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "QLinearMatMul output shape");
            const size_t nws = numel(T(ws).shape.data(), T(ws).shape.size());
            if (nws != 1 && nws != N) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearMatMul b_scale size");
            if (b >= 0 && numel(T(b).shape.data(), T(b).shape.size()) != N) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearMatMul bias size");
            std::vector<float> mult;
            requant_multipliers(a.x_scale, (const float*)T(ws).host.data(), nws, a.y_scale, N, mult);
            std::vector<int32_t> bz(N, 0);
            if (wz >= 0) {
                const size_t nwz = numel(T(wz).shape.data(), T(wz).shape.size());
                if (nwz != 1 && nwz != N) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "QLinearMatMul b_zp size");
                for (size_t j = 0; j < N; ++j) bz[j] = ((const int32_t*)T(wz).host.data())[nwz == 1 ? 0 : j];
            }
            const int xzp = a.x_zp; const Requant rq{a.y_scale, a.y_zp, a.activation};
            bool bz_zero = true;
            for (int32_t v : bz) bz_zero = bz_zero && v == 0;
            if (M <= 0x7fffffffULL && N <= 0x7fffffffULL && K <= 0x7fffffffULL) {
                ConvGeom g{};   // a matrix product is a 1x1 convolution over M "images" of one pixel
                g.N = (int)M; g.C = (int)K; g.H = g.W = 1; g.M = (int)N; g.Cg = (int)K; g.KH = g.KW = 1;
                g.sh = g.sw = g.dh = g.dw = 1; g.OH = g.OW = 1; g.G = 1;
                if (yd != ZANT_I32 && qconv_tc_eligible(g, bz_zero) && (b < 0 || T(b).is_const)) {
                    std::vector<int8_t> bt(K * N);
                    const int8_t* bw = (const int8_t*)T(w).host.data();
                    for (size_t k = 0; k < K; ++k) for (size_t j = 0; j < N; ++j) bt[j * K + k] = bw[k * N + j];
                    auto prep = std::make_shared<QGemmPrep>();
                    qgemm_prepare(bt.data(), (int)N, (int)K, mult.data(), b >= 0 ? (const int32_t*)T(b).host.data() : nullptr, xzp, *prep, (long long)M, ctx->sm_count);
                    const int aw = pl->add_aux(prep->w_blk.data(), prep->w_blk.size()), am = pl->add_aux(prep->mult.data(), prep->mult.size() * 4);
                    const int ab = pl->add_aux(prep->bias.data(), prep->bias.size() * 4);
                    const int sa = pl->shared_im2col_scratch(qgemm_a_bytes(M, *prep));
                    prep->w_blk.clear(); prep->w_blk.shrink_to_fit();
                    push("QLinearMatMul(tc)", [=]() {
                        return run_qconv_tc(ctx, g, pl->ptr(x), xd == ZANT_U8, xzp, *prep, (const int8_t*)pl->aux(aw), (const float*)pl->aux(am),
                                            (const int32_t*)pl->aux(ab), (uint8_t*)pl->scratch(sa), pl->ptr(y), yd == ZANT_U8, rq);
                    });
                    return ZANT_OK;
                }
            }
            if (M < 256 && N <= (1u << 20) && K <= (1u << 20) && yd != ZANT_I32 && (b < 0 || T(b).is_const)) {
                ConvGeom g{};
                g.N = (int)M; g.C = (int)K; g.H = g.W = 1; g.M = (int)N; g.Cg = (int)K; g.KH = g.KW = 1;
                g.sh = g.sw = g.dh = g.dw = 1; g.OH = g.OW = 1; g.G = 1;
                if (small_gemm_eligible(g, bz_zero)) {
                    const SmallGemmPlan sg = small_gemm_plan(g, ctx->sm_count);
                    const int aw = pl->add_scratch(sg.w_bytes), am = pl->add_aux(mult.data(), mult.size() * 4), ab = xzp != 0 ? pl->add_scratch(N * 4) : -1;
                    auto bias_of = [=]() { return ab >= 0 ? (int32_t*)pl->scratch(ab) : pl->p<int32_t>(b); };
                    pl->init_steps.push_back([=]() { return run_small_gemm_weights(ctx, g, sg, true, pl->p<int8_t>(w), pl->p<int32_t>(b), xzp, pl->scratch(aw), bias_of()); });
                    push("QLinearMatMul", [=]() {
                        return run_small_gemm(ctx, g, sg, pl->ptr(x), xd == ZANT_U8, xzp, pl->scratch(aw), (const float*)pl->aux(am), bias_of(), pl->ptr(y), yd == ZANT_U8, rq);
                    });
                    return ZANT_OK;
                }
            }
            const int am = pl->add_aux(mult.data(), mult.size() * 4), az = pl->add_aux(bz.data(), bz.size() * 4);
            push("QLinearMatMul", [=]() {
                QMatArgs q{};
                q.a = pl->ptr(x); q.b = pl->p<int8_t>(w); q.y = pl->ptr(y);
                q.mult = (const float*)pl->aux(am); q.b_zp = (const int32_t*)pl->aux(az); q.bias = pl->p<int32_t>(b);
                q.a_zp = xzp; q.rq = rq; q.M = (int)M; q.N = (int)N; q.K = (int)K; q.y_i32 = yd == ZANT_I32;
                return run_qmatmul_generic(ctx, q, xd, yd);
            });
            return ZANT_OK;
        }
        case ZANT_OP_QLINEAR_ADD: {
            ZB_TRY(need_inputs(n, 2, 2, "QLinearAdd"));
            const int x = n.in[0], w = n.in[1], y = n.out[0];
            const int32_t dt = T(x).dtype;
            if ((dt != ZANT_I8 && dt != ZANT_U8) || T(w).dtype != dt || T(y).dtype != dt) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QLinearAdd dtypes");
            const size_t cnt = numel(T(x).shape.data(), T(x).shape.size());
            if (cnt != numel(T(w).shape.data(), T(w).shape.size()) || cnt != numel(T(y).shape.data(), T(y).shape.size()))
                return fail(ZANT_E_INPUT_TENSOR_DIFFERENT_SIZE, "QLinearAdd sizes differ");
            const zant_node_attrs aa = a;
            push("QLinearAdd", [=]() { return run_qadd(ctx, dt, pl->ptr(x), aa.x_scale, aa.x_zp, pl->ptr(w), aa.b_scale, aa.b_zp, aa.y_scale, aa.y_zp, aa.activation, pl->ptr(y), cnt); });
            return ZANT_OK;
        }
        case ZANT_OP_QLINEAR_GLOBAL_AVGPOOL: {
            ZB_TRY(need_inputs(n, 1, 1, "QLinearGlobalAveragePool"));
            const int x = n.in[0], y = n.out[0];
            const int32_t dt = T(x).dtype;
            if ((dt != ZANT_I8 && dt != ZANT_U8) || T(y).dtype != dt) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "QLinearGlobalAveragePool dtypes");
            if (T(x).shape.size() != 4) return fail(ZANT_E_INVALID_DIMENSIONS, "QLinearGlobalAveragePool needs a 4-D input");
            const size_t planes = T(x).shape[0] * T(x).shape[1], hw = T(x).shape[2] * T(x).shape[3];
            if (numel(T(y).shape.data(), T(y).shape.size()) != planes || hw == 0) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "QLinearGlobalAveragePool output size");
            const zant_node_attrs aa = a;
            push("QLinearGlobalAveragePool", [=]() { return run_qgap(ctx, dt, pl->ptr(x), pl->ptr(y), planes, (int)hw, aa.x_scale, aa.x_zp, aa.y_scale, aa.y_zp); });
            return ZANT_OK;
        }
        case ZANT_OP_LUT_Q8: {
            ZB_TRY(need_inputs(n, 2, 2, "LutQ8"));
            const int x = n.in[0], l = n.in[1], y = n.out[0];
            if (T(l).bytes != 256) return fail(ZANT_E_INPUT_TENSORS_WRONG_SHAPE, "table must hold 256 bytes");
            const size_t cnt = T(x).bytes;
            if (dtype_size(T(x).dtype) != 1 || T(y).bytes != cnt) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "LutQ8 works on 8-bit tensors of equal size");
            push("LutQ8", [=]() { return run_lut(ctx, pl->ptr(x), pl->ptr(y), cnt, pl->p<uint8_t>(l)); });
            return ZANT_OK;
        }
        default:
            return fail(ZANT_E_UNSUPPORTED, "operator %d is not supported", n.op);
    }
}

// --------------------------------------------------------------------------------------------
// Fusion.  `try_fuse` looks for a known chain starting at `node_index` and, if every shape,
// attribute and data-flow condition holds, emits fused steps and reports how many nodes they
// cover (0 = nothing matched; the caller builds the node on its own).
//
// Chain recognised today (the reference's example CNN in QLinear form):
//   QuantizeLinear(u8) -> QLinearConv(1->32,3x3) -> Relu -> MaxPool 2x2/2
//                      -> QLinearConv(32->64,3x3) -> Relu -> MaxPool 2x2/2 -> Reshape
//                      -> QLinearMatMul -> Relu -> QLinearMatMul -> DequantizeLinear
// on [N,1,28,28] inputs.  Intermediate tensors of a fused chain are not materialised in their
// graph layout: they live in private scratch buffers (C16-planar / GEMM-ordered).
// --------------------------------------------------------------------------------------------
namespace {

struct ChainCtx {
    zant_plan* pl;
    std::vector<int> consumers;   // per tensor: number of nodes reading it
};

bool only_feeds_next(const ChainCtx& c, int tensor) {
    return c.consumers[tensor] == 1 && tensor != c.pl->output && !c.pl->t[tensor].is_const;
}

// The graph's output, or a tensor whose memory a Reshape hands on as the output's: in a run the caller's buffer, of whatever alignment.
bool holds_output(const zant_plan* pl, int id) {
    std::vector<int> same{id};
    auto has = [&](int k) { return std::find(same.begin(), same.end(), k) != same.end(); };
    for (const PlanNode& n : pl->nodes) if (n.op == ZANT_OP_RESHAPE && n.in.size() == 1 && n.out.size() == 1 && has(n.in[0])) same.push_back(n.out[0]);
    return has(pl->output);
}

bool shape_is(const PlanTensor& t, std::initializer_list<size_t> s) { return t.shape == std::vector<size_t>(s); }

bool plain_conv3x3(const zant_node_attrs& a) {
    auto one = [](const size_t* v, size_t n) { for (size_t i = 0; i < n; ++i) if (v[i] != 1) return false; return true; };
    bool nopad = true;
    for (size_t i = 0; i < a.n_pads; ++i) nopad = nopad && a.pads[i] == 0;
    return one(a.strides, a.n_strides) && one(a.dilations, a.n_dilations) && nopad && (a.group == 0 || a.group == 1) &&
           (a.auto_pad < 0 || a.auto_pad == ZANT_PAD_NOTSET || a.auto_pad == ZANT_PAD_VALID);
}

bool pool2x2(const zant_node_attrs& a) {
    bool nopad = true;
    for (size_t i = 0; i < a.n_pads; ++i) nopad = nopad && a.pads[i] == 0;
    const bool d1 = a.n_dilations == 0 || (a.dilations[0] == 1 && a.dilations[1] == 1);
    return a.kernel_shape[0] == 2 && a.kernel_shape[1] == 2 && a.n_strides == 2 && a.strides[0] == 2 && a.strides[1] == 2 && nopad && d1 &&
           (a.auto_pad < 0 || a.auto_pad == ZANT_PAD_NOTSET || a.auto_pad == ZANT_PAD_VALID);
}

// A quantized Relu node that keeps scale and zero point is max(q, zp): foldable into the producer.
bool identity_scale_relu(const PlanNode& n) {
    return n.op == ZANT_OP_RELU && n.a.x_scale == n.a.y_scale && n.a.x_zp == n.a.y_zp;
}

bool all_zero_i32(const PlanTensor& t) {
    const int32_t* v = (const int32_t*)t.host.data();
    for (size_t i = 0; i < t.bytes / 4; ++i) if (v[i] != 0) return false;
    return true;
}

bool positive_finite(const std::vector<float>& m) {
    for (float v : m) if (!(v > 0.0f) || !std::isfinite(v)) return false;
    return true;
}

}  // namespace

static int32_t try_fuse(zant_plan* pl, size_t i0, size_t& consumed) {
    consumed = 0;
    ZB_TRY(try_fuse_small_cnn(pl, i0, consumed));
    if (consumed) return ZANT_OK;
    ZB_TRY(try_fuse_irb(pl, i0, consumed));
    if (consumed) return ZANT_OK;
    ZB_TRY(try_fuse_qconv_group(pl, i0, consumed));
    if (consumed) return ZANT_OK;
    return try_fuse_fconv_group(pl, i0, consumed);
}

// QLinearConv 1x1 -> QLinearConv depthwise 3x3 -> QLinearConv 1x1 [-> QLinearAdd with the group's input] as one step (irb_q8.cuh for
// many images on small planes, irb_band.cuh for few).  Both activations are ReLU or a ReLU6 whose bound is the type's own, all tensors int8, zero points 0 between the convolutions,
// interior tensors read by the next node only.  Whatever does not qualify is left to the steps of its own.
static int32_t try_fuse_irb(zant_plan* pl, size_t i0, size_t& consumed) {
    consumed = 0;
    if (i0 + 3 > pl->nodes.size()) return ZANT_OK;
    const PlanNode *e = &pl->nodes[i0], *d = e + 1, *p = e + 2;
    for (const PlanNode* n : {e, d, p})
        if (n->op != ZANT_OP_QLINEAR_CONV || n->in.size() < 3 || n->in.size() > 5 || n->out.size() != 1 || n->a.channels_last) return ZANT_OK;
    ChainCtx c{pl, std::vector<int>(pl->t.size(), 0)};
    for (const PlanNode& n : pl->nodes) for (int id : n.in) if (id >= 0) c.consumers[id]++;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    const int x = e->in[0], t1 = e->out[0], t2 = d->out[0], y0 = p->out[0];
    if (x < 0 || d->in[0] != t1 || p->in[0] != t2 || !only_feeds_next(c, t1) || !only_feeds_next(c, t2)) return ZANT_OK;
    auto plain = [&](int id) { return T(id).dtype == ZANT_I8 && T(id).shape.size() == 4 && !T(id).nh && T(id).alias < 0 && !T(id).elided && !T(id).is_const; };
    if (!plain(x) || !plain(t1) || !plain(t2) || !plain(y0) || x == pl->input || holds_output(pl, x) || holds_output(pl, y0)) return ZANT_OK;
    // parameters of the three convolutions
    ConvGeom g[3];
    std::vector<float> mult[3]; std::vector<int32_t> bias[3];
    const PlanNode* conv[3] = {e, d, p};
    for (int i = 0; i < 3; ++i) {
        const PlanNode& n = *conv[i];
        const int w = n.in[1], ws = n.in[2], wz = opt_in(n, 3), b = opt_in(n, 4);
        if (w < 0 || ws < 0 || !T(w).is_const || T(w).dtype != ZANT_I8 || !T(ws).is_const || T(ws).dtype != ZANT_F32 || T(w).shape.size() != 4) return ZANT_OK;
        if (b >= 0 && (!T(b).is_const || T(b).dtype != ZANT_I32)) return ZANT_OK;
        if (wz >= 0 && (!T(wz).is_const || T(wz).dtype != ZANT_I32 || !all_zero_i32(T(wz)))) return ZANT_OK;
        if (check_zero_point(ZANT_I8, n.a.x_zp, "x") != ZANT_OK || n.a.y_zp != 0 || (i > 0 && n.a.x_zp != 0)) return ZANT_OK;
        if (conv_resolve_onnx(T(n.in[0]).shape.data(), 4, T(w).shape.data(), 4, T(n.out[0]).shape.data(), 4, n.a.strides, n.a.n_strides, n.a.pads, n.a.n_pads,
                              n.a.dilations, n.a.n_dilations, n.a.group, n.a.auto_pad < 0 ? 0 : n.a.auto_pad, g[i]) != ZANT_OK) return ZANT_OK;
        const size_t M = (size_t)g[i].M, nws = T(ws).bytes / 4;
        if ((nws != 1 && nws != M) || (b >= 0 && T(b).bytes != M * 4)) return ZANT_OK;
        if (wz >= 0 && T(wz).bytes != 4 && T(wz).bytes != M * 4) return ZANT_OK;
        requant_multipliers(n.a.x_scale, (const float*)T(ws).host.data(), nws, n.a.y_scale, M, mult[i]);
        if (!positive_finite(mult[i])) return ZANT_OK;
        bias[i].assign(M, 0);
        if (b >= 0) std::memcpy(bias[i].data(), T(b).host.data(), M * 4);
        if (i < 2) {
            std::vector<int32_t> caps;
            if (!requant_relu_caps(mult[i].data(), M, n.a.activation, lean_six(n.a.y_scale), caps)) return ZANT_OK;
            for (int32_t v : caps) if (v != 0x7fffffff) return ZANT_OK;
        } else if (n.a.activation != ZANT_QACT_NONE) return ZANT_OK;
    }
    if (e->a.x_zp != 0) {
        const int8_t* w = (const int8_t*)T(e->in[1]).host.data();
        for (int m = 0; m < g[0].M; ++m) {
            int sum = 0;
            for (int k = 0; k < g[0].C; ++k) sum += w[(size_t)m * g[0].C + k];
            bias[0][m] -= e->a.x_zp * sum;
        }
    }
    // the residual addition: its other operand is the group's input
    int y = y0;
    consumed = 3;
    QAddTail add{};
    bool with_add = false;
    if (i0 + 3 < pl->nodes.size() && only_feeds_next(c, y0)) {
        const PlanNode& n = pl->nodes[i0 + 3];
        if (n.op == ZANT_OP_QLINEAR_ADD && n.in.size() == 2 && n.out.size() == 1 && ((n.in[0] == x && n.in[1] == y0) || (n.in[0] == y0 && n.in[1] == x)) &&
            plain(n.out[0]) && !holds_output(pl, n.out[0]) && T(n.out[0]).bytes == T(x).bytes && T(x).bytes == T(y0).bytes && g[0].C == g[2].M &&
            check_zero_point(ZANT_I8, n.a.y_zp, "QLinearAdd y") == ZANT_OK) {
            const bool first = n.in[0] == x;
            add = pl->prove(qadd_tail<false>(first ? n.a.x_scale : n.a.b_scale, first ? n.a.x_zp : n.a.b_zp, first ? n.a.b_scale : n.a.x_scale, first ? n.a.b_zp : n.a.x_zp, n.a.y_scale, n.a.y_zp, n.a.activation));
            with_add = true;
            y = n.out[0];
            consumed = 4;
        }
    }
    zant_ctx* ctx = pl->ctx;
    auto host = [&](int id) { return (const int8_t*)T(id).host.data(); };
    IrbPlan q;
    IrbBandPlan qb;
    const bool can_one = irb_plan(g[0], g[1], g[2], with_add, q), can_band = irb_band_plan(g[0], g[1], g[2], with_add, ctx->sm_count, qb);
    const IrbForm form = irb_form(can_one ? &q : nullptr, can_band ? &qb : nullptr, g[1], with_add, with_add && !add.proved, ctx->sm_count);
    std::vector<uint8_t> stages;
    if (form == IrbForm::kSeparate ||
        !(form == IrbForm::kBand ? irb_band_prepare(qb, host(e->in[1]), mult[0].data(), bias[0].data(), host(d->in[1]), mult[1].data(), bias[1].data(), host(p->in[1]), mult[2].data(), bias[2].data(), stages)
                                 : irb_prepare(q, host(e->in[1]), mult[0].data(), bias[0].data(), host(d->in[1]), mult[1].data(), bias[1].data(), host(p->in[1]), stages))) {
        consumed = 0;
        return ZANT_OK;
    }
    const int aw = pl->add_aux(stages.data(), stages.size());
    const size_t first_step = pl->steps.size();
    pl->step_names.push_back(with_add ? "QLinearConv(expand+depthwise+project)+QLinearAdd" : "QLinearConv(expand+depthwise+project)");
    if (form == IrbForm::kBand) {
        pl->steps.push_back([=]() { return irb_band_run(ctx, qb, pl->ptr(x), (const uint8_t*)pl->aux(aw), pl->ptr(y), with_add ? &add : nullptr); });
    } else {
        const int am = pl->add_aux(mult[2].data(), mult[2].size() * 4), ab = pl->add_aux(bias[2].data(), bias[2].size() * 4);
        pl->steps.push_back([=]() { return irb_run(ctx, q, pl->ptr(x), (const uint8_t*)pl->aux(aw), (const float*)pl->aux(am), (const int32_t*)pl->aux(ab), pl->ptr(y), with_add ? &add : nullptr); });
    }
    pl->t[t1].elided = pl->t[t2].elided = true;
    if (with_add) pl->t[y0].elided = true;
    record_step_cost(pl, first_step, i0, consumed);
    return ZANT_OK;
}

// Float Conv -> [Relu | LeakyRelu] -> [MaxPool 2x2 / 2] and MatMul -> Add(row vector) -> [Relu | LeakyRelu] as one step: what
// lies behind the contraction runs on its finished sums, in the nodes' own order and with their own roundings, so the exact
// path stays bit-identical to the node-by-node plan.  (Tensor-core path: the activation behind a Conv only.)
static int32_t try_fuse_fconv_group(zant_plan* pl, size_t i0, size_t& consumed) {
    consumed = 0;
    const PlanNode& head = pl->nodes[i0];
    const bool conv = head.op == ZANT_OP_CONV, mat = head.op == ZANT_OP_MATMUL && !pl->ctx->tf32;
    if ((!conv && !mat) || head.out.size() != 1 || head.in.size() < 2 || i0 + 1 >= pl->nodes.size()) return ZANT_OK;
    ChainCtx c{pl, std::vector<int>(pl->t.size(), 0)};
    for (const PlanNode& n : pl->nodes) for (int id : n.in) if (id >= 0) c.consumers[id]++;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    size_t j = i0 + 1;
    int cur = head.out[0], bias = -1;
    std::vector<int> interior;
    if (mat) {
        const PlanNode& add = pl->nodes[j];
        if (add.op != ZANT_OP_ADD || add.in.size() != 2 || add.out.size() != 1 || add.in[0] != cur || !only_feeds_next(c, cur)) return ZANT_OK;
        bias = add.in[1];
        const auto& ys = T(cur).shape;
        if (bias < 0 || T(bias).dtype != ZANT_F32 || T(cur).dtype != ZANT_F32 || T(add.out[0]).shape != ys || ys.empty()) return ZANT_OK;
        // a row vector of the product's columns: the last dimension and nothing else
        if (T(bias).shape.empty() || T(bias).shape.back() != ys.back() || numel(T(bias).shape.data(), T(bias).shape.size()) != ys.back() || T(bias).shape.size() > ys.size()) return ZANT_OK;
        BcastGeom bg;
        if (bcast_resolve(ys.data(), ys.size(), T(bias).shape.data(), T(bias).shape.size(), ys.data(), ys.size(), bg) != ZANT_OK) return ZANT_OK;
        interior.push_back(cur);
        cur = add.out[0];
        ++j;
    }
    int fact = FACT_NONE; float slope = 0.0f;
    if (j < pl->nodes.size() && only_feeds_next(c, cur)) {
        const PlanNode& act = pl->nodes[j];
        if ((act.op == ZANT_OP_RELU || act.op == ZANT_OP_LEAKY_RELU) && act.in.size() == 1 && act.out.size() == 1 && act.in[0] == cur &&
            T(act.out[0]).dtype == ZANT_F32 && T(cur).dtype == ZANT_F32 && T(act.out[0]).bytes == T(cur).bytes) {
            fact = act.op == ZANT_OP_RELU ? FACT_RELU : FACT_LEAKY; slope = act.a.alpha;
            interior.push_back(cur);
            cur = act.out[0];
            ++j;
        }
    }
    const size_t first_step = pl->steps.size();
    if (mat) {
        const int x = head.in[0], w = head.in[1];
        ZB_TRY(need_inputs(head, 2, 2, "MatMul"));
        MatGeom g;
        ZB_TRY(matmul_check(T(x).shape.data(), T(x).shape.size(), T(w).shape.data(), T(w).shape.size(), T(head.out[0]).shape.data(), T(head.out[0]).shape.size(), g));
        if (numel(T(head.out[0]).shape.data(), T(head.out[0]).shape.size()) != g.M * g.N) return ZANT_OK;      // (a batched product: only its first matrix is computed)
        zant_ctx* ctx = pl->ctx;
        const int yw = cur;
        pl->steps.push_back([=]() {
            ContractFusion fu;
            fu.bias = pl->p<float>(bias); fu.act = fact == FACT_RELU ? CT_ACT_RELU : (fact == FACT_LEAKY ? CT_ACT_LEAKY : CT_ACT_NONE); fu.slope = slope;
            return run_matmul_f32(ctx, g, pl->p<float>(x), pl->p<float>(w), pl->p<float>(yw), fu);
        });
        pl->step_names.push_back(std::string("MatMul+Add") + (fact == FACT_RELU ? "+Relu" : (fact == FACT_LEAKY ? "+LeakyRelu" : "")));
    } else {
        int pool_y = -1;
        if (!pl->ctx->tf32 && j < pl->nodes.size() && only_feeds_next(c, cur)) {
            const PlanNode& pool = pl->nodes[j];
            if (pool.op == ZANT_OP_MAXPOOL && pool.in.size() == 1 && pool.out.size() == 1 && pool.in[0] == cur && pool2x2(pool.a) &&
                T(pool.out[0]).dtype == ZANT_F32 && T(cur).dtype == ZANT_F32 && T(cur).shape.size() == 4 && T(pool.out[0]).shape.size() == 4) {
                const auto& si = T(cur).shape; const auto& so = T(pool.out[0]).shape;
                if (so[0] == si[0] && so[1] == si[1] && so[2] == si[2] / 2 && so[3] == si[3] / 2 && so[2] > 0 && so[3] > 0) {
                    pool_y = pool.out[0];
                    interior.push_back(cur);
                    ++j;
                }
            }
        }
        if (interior.empty()) return ZANT_OK;
        pl->pending_fact = fact; pl->pending_slope = slope; pl->pending_y = fact == FACT_NONE ? -1 : cur; pl->pending_pool = pool_y;
        pl->pending_used = false;
        const int32_t st = build_node_impl(pl, i0, 1);
        const bool used = pl->pending_used;
        pl->pending_fact = FACT_NONE; pl->pending_slope = 0.0f; pl->pending_y = -1; pl->pending_pool = -1; pl->pending_used = false;
        if (st != ZANT_OK) return st;
        if (!used) { interior.clear(); j = i0 + 1; }
    }
    for (int id : interior) pl->t[id].elided = true;
    consumed = j - i0;
    record_step_cost(pl, first_step, i0, consumed);
    return ZANT_OK;
}

// --------------------------------------------------------------------------------------------
// Generic epilogue fusion: QLinearConv -> [Relu | LeakyRelu | Clip] -> [MaxPool 2x2 / stride 2].
// The generator emits one call per node (src/codeGen/predict.zig:73-92, src/codeGen/math_handler.zig:45-105), so
// between a convolution and the pool behind it two full-size int8 tensors are written and read back.  Here the
// activation becomes part of the producer's epilogue (an activation flag when it keeps scale and zero point, else
// a 256-entry table applied to the finished code), and the pool is applied in the epilogue of the implicit-GEMM
// kernel where its tiling allows; the tensors in between are never materialised.  Every step is the composition of
// the exact per-node functions on the same integer codes, so results stay bit-identical to the node-by-node plan.
// Conditions: each interior tensor has exactly one consumer and is not the graph output; the pool has a 2x2
// window, stride 2, no padding, no dilation (MaxPool rule: src/Core/Tensor/TensorMath/op_pooling.zig:570-659).
// --------------------------------------------------------------------------------------------
static int32_t try_fuse_qconv_group(zant_plan* pl, size_t i0, size_t& consumed) {
    consumed = 0;
    const PlanNode& conv = pl->nodes[i0];
    if (conv.op != ZANT_OP_QLINEAR_CONV || conv.out.size() != 1 || conv.in.size() < 3) return ZANT_OK;
    ChainCtx c{pl, std::vector<int>(pl->t.size(), 0)};
    for (const PlanNode& n : pl->nodes) for (int id : n.in) if (id >= 0) c.consumers[id]++;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    auto q8 = [&](int id) { return T(id).dtype == ZANT_I8 || T(id).dtype == ZANT_U8; };
    QConvFusion fz;
    size_t j = i0 + 1;
    int cur = conv.out[0];
    if (!q8(cur)) return ZANT_OK;
    std::vector<int> interior;
    // activation behind the convolution
    if (j < pl->nodes.size() && only_feeds_next(c, cur)) {
        const PlanNode& act = pl->nodes[j];
        const bool is_act = act.op == ZANT_OP_RELU || act.op == ZANT_OP_LEAKY_RELU || act.op == ZANT_OP_CLIP;
        if (is_act && act.in.size() == 1 && act.out.size() == 1 && act.in[0] == cur && T(act.out[0]).dtype == T(cur).dtype &&
            T(act.out[0]).bytes == T(cur).bytes && act.a.x_scale == conv.a.y_scale && act.a.x_zp == conv.a.y_zp) {
            if (identity_scale_relu(act)) {
                fz.activation = conv.a.activation == ZANT_QACT_NONE ? ZANT_QACT_RELU : conv.a.activation;
            } else {
                uint8_t lut[256];
                activation_lut(act, T(cur).dtype, lut);
                fz.lut_aux = pl->add_aux(lut, 256);
            }
            interior.push_back(cur);
            cur = act.out[0];
            ++j;
        }
    }
    // pool behind that
    bool want_pool = false;
    if (!conv.a.channels_last && j < pl->nodes.size() && only_feeds_next(c, cur)) {
        const PlanNode& pool = pl->nodes[j];
        if (pool.op == ZANT_OP_MAXPOOL && pool.in.size() == 1 && pool.out.size() == 1 && pool.in[0] == cur && pool2x2(pool.a) &&
            T(pool.out[0]).dtype == T(cur).dtype && T(cur).shape.size() == 4 && T(pool.out[0]).shape.size() == 4) {
            const auto& si = T(cur).shape; const auto& so = T(pool.out[0]).shape;
            if (so[0] == si[0] && so[1] == si[1] && so[2] == si[2] / 2 && so[3] == si[3] / 2 && so[2] > 0 && so[3] > 0) {
                want_pool = true;
                fz.y_pool = pool.out[0];
            }
        }
    }
    // residual addition behind that: the other operand is a tensor that an earlier node left in the arena
    if (!want_pool && !conv.a.channels_last && j < pl->nodes.size() && only_feeds_next(c, cur)) {
        const PlanNode& add = pl->nodes[j];
        if (add.op == ZANT_OP_QLINEAR_ADD && add.in.size() == 2 && add.out.size() == 1 && (add.in[0] == cur) != (add.in[1] == cur)) {
            const int r = add.in[0] == cur ? add.in[1] : add.in[0], y = add.out[0];
            bool there = false;
            for (size_t k = 0; k < i0; ++k) for (int id : pl->nodes[k].out) there = there || id == r;
            if (r >= 0 && there && !T(r).elided && !T(r).nh && T(r).alias < 0 && r != pl->input && !holds_output(pl, r) && y != pl->output && T(cur).dtype == ZANT_I8 &&
                T(r).dtype == ZANT_I8 && T(y).dtype == ZANT_I8 && T(r).bytes == T(cur).bytes && T(y).bytes == T(cur).bytes && check_zero_point(ZANT_I8, add.a.y_zp, "QLinearAdd y") == ZANT_OK) {
                fz.add_node = (int)j;
                fz.add_res = r;
            }
        }
    }
    if (interior.empty() && !want_pool && fz.add_node < 0) return ZANT_OK;        // nothing behind the node: the plain path builds it
    fz.y_act = cur;
    const size_t first_step = pl->steps.size();
    ZB_TRY(build_qconv(pl, conv, fz));
    if (fz.pool_done || fz.add_done) { interior.push_back(cur); ++j; }
    if (interior.empty()) {
        // the pool or the addition was asked for but the chosen kernel cannot take it: nothing was fused after all
        record_step_cost(pl, first_step, i0, 1);
        consumed = 1;
        return ZANT_OK;
    }
    for (int id : interior) pl->t[id].elided = true;
    consumed = j - i0;
    record_step_cost(pl, first_step, i0, consumed);
    return ZANT_OK;
}

static int32_t try_fuse_small_cnn(zant_plan* pl, size_t i0, size_t& consumed, bool probe) {
    consumed = 0;
    if (i0 + 12 > pl->nodes.size()) return ZANT_OK;
    const int kOps[12] = {ZANT_OP_QUANTIZE_LINEAR, ZANT_OP_QLINEAR_CONV, ZANT_OP_RELU, ZANT_OP_MAXPOOL, ZANT_OP_QLINEAR_CONV, ZANT_OP_RELU,
                          ZANT_OP_MAXPOOL, ZANT_OP_RESHAPE, ZANT_OP_QLINEAR_MATMUL, ZANT_OP_RELU, ZANT_OP_QLINEAR_MATMUL, ZANT_OP_DEQUANTIZE_LINEAR};
    for (int k = 0; k < 12; ++k) if (pl->nodes[i0 + k].op != kOps[k]) return ZANT_OK;
    ChainCtx c{pl, std::vector<int>(pl->t.size(), 0)};
    for (const PlanNode& n : pl->nodes) for (int id : n.in) if (id >= 0) c.consumers[id]++;
    const PlanNode* N = &pl->nodes[i0];
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    // data flow: each node's first input is the previous node's only output, used nowhere else
    for (int k = 1; k < 12; ++k) {
        if (N[k].in.empty() || N[k - 1].out.size() != 1 || N[k].in[0] != N[k - 1].out[0]) return ZANT_OK;
        if (!only_feeds_next(c, N[k - 1].out[0])) return ZANT_OK;
    }
    const int x = N[0].in[0], y = N[11].out[0];
    if (T(x).dtype != ZANT_F32 || T(x).shape.size() != 4) return ZANT_OK;
    const size_t B = T(x).shape[0];
    if (B == 0 || B > 0x3fffffffULL) return ZANT_OK;
    if (!shape_is(T(x), {B, 1, 28, 28}) || T(N[0].out[0]).dtype != ZANT_U8) return ZANT_OK;
    // conv1
    const PlanNode& c1 = N[1];
    if (c1.in.size() < 3 || !plain_conv3x3(c1.a) || !shape_is(T(c1.in[1]), {32, 1, 3, 3}) || !shape_is(T(c1.out[0]), {B, 32, 26, 26})) return ZANT_OK;
    if (T(c1.out[0]).dtype != ZANT_I8 || c1.a.activation == ZANT_QACT_RELU6 || c1.a.y_zp != 0) return ZANT_OK;
    if (c1.a.x_scale != N[0].a.y_scale || c1.a.x_zp != N[0].a.y_zp) return ZANT_OK;
    if (opt_in(c1, 3) >= 0 && !all_zero_i32(T(c1.in[3]))) return ZANT_OK;
    if (!identity_scale_relu(N[2]) || N[2].a.x_scale != c1.a.y_scale || N[2].a.x_zp != c1.a.y_zp) return ZANT_OK;
    if (!pool2x2(N[3].a) || !shape_is(T(N[3].out[0]), {B, 32, 13, 13})) return ZANT_OK;
    // conv2
    const PlanNode& c2 = N[4];
    if (c2.in.size() < 3 || !plain_conv3x3(c2.a) || !shape_is(T(c2.in[1]), {64, 32, 3, 3}) || !shape_is(T(c2.out[0]), {B, 64, 11, 11})) return ZANT_OK;
    if (T(c2.out[0]).dtype != ZANT_I8 || c2.a.activation == ZANT_QACT_RELU6 || c2.a.y_zp != 0) return ZANT_OK;
    if (c2.a.x_scale != c1.a.y_scale || c2.a.x_zp != c1.a.y_zp) return ZANT_OK;
    if (opt_in(c2, 3) >= 0 && !all_zero_i32(T(c2.in[3]))) return ZANT_OK;
    if (!identity_scale_relu(N[5]) || N[5].a.x_scale != c2.a.y_scale || N[5].a.x_zp != c2.a.y_zp) return ZANT_OK;
    if (!pool2x2(N[6].a) || !shape_is(T(N[6].out[0]), {B, 64, 5, 5})) return ZANT_OK;
    if (!shape_is(T(N[7].out[0]), {B, 1600})) return ZANT_OK;
    // fc1, fc2
    const PlanNode& f1 = N[8];
    const PlanNode& f2 = N[10];
    if (f1.in.size() < 3 || f2.in.size() < 3) return ZANT_OK;
    if (!shape_is(T(f1.in[1]), {1600, 512}) || !shape_is(T(f1.out[0]), {B, 512}) || T(f1.out[0]).dtype != ZANT_I8) return ZANT_OK;
    if (f1.a.x_scale != c2.a.y_scale || f1.a.x_zp != c2.a.y_zp || f1.a.activation == ZANT_QACT_RELU6 || f1.a.y_zp != 0) return ZANT_OK;
    if (opt_in(f1, 3) >= 0 && !all_zero_i32(T(f1.in[3]))) return ZANT_OK;
    if (!identity_scale_relu(N[9]) || N[9].a.x_scale != f1.a.y_scale || N[9].a.x_zp != f1.a.y_zp) return ZANT_OK;
    if (T(f2.in[1]).shape.size() != 2 || T(f2.in[1]).shape[0] != 512 || T(f2.out[0]).dtype != ZANT_I8) return ZANT_OK;
    const size_t NCLS = T(f2.in[1]).shape[1];
    if (NCLS == 0 || NCLS > 64 || !shape_is(T(f2.out[0]), {B, NCLS}) || !shape_is(T(y), {B, NCLS})) return ZANT_OK;
    if (f2.a.x_scale != f1.a.y_scale || f2.a.x_zp != f1.a.y_zp || f2.a.activation != ZANT_QACT_NONE) return ZANT_OK;
    if (opt_in(f2, 3) >= 0 && !all_zero_i32(T(f2.in[3]))) return ZANT_OK;
    if (N[11].a.x_scale != f2.a.y_scale || N[11].a.x_zp != f2.a.y_zp || T(y).dtype != ZANT_F32) return ZANT_OK;
    for (const PlanNode* q : {&c1, &c2, &f1, &f2})
        for (size_t k = 1; k < q->in.size(); ++k)
            if (q->in[k] >= 0 && !T(q->in[k]).is_const) return ZANT_OK;

    if (NCLS > 16 || B > (1u << 20)) return ZANT_OK;         // two column blocks of classes; counts of images, tiles and windows far inside 32 bits
    if (probe) { consumed = 12; return ZANT_OK; }
    zant_ctx* ctx = pl->ctx;
    auto push = [&](const char* name, std::function<int32_t()> fn) { pl->steps.push_back(std::move(fn)); pl->step_names.push_back(name); };
    auto scales_of = [&](const PlanNode& q, size_t M, std::vector<float>& mult) {
        const PlanTensor& ws = T(q.in[2]);
        const size_t nws = ws.bytes / 4;
        if (ws.dtype != ZANT_F32 || (nws != 1 && nws != M)) return false;
        requant_multipliers(q.a.x_scale, (const float*)ws.host.data(), nws, q.a.y_scale, M, mult);
        return positive_finite(mult);
    };
    auto bias_of = [&](const PlanNode& q, size_t M, std::vector<int32_t>& bias) {
        bias.assign(M, 0);
        const int b = opt_in(q, 4);
        if (b < 0) return true;
        if (T(b).dtype != ZANT_I32 || T(b).bytes != M * 4) return false;
        std::memcpy(bias.data(), T(b).host.data(), M * 4);
        return true;
    };

    // ---- stage 1 parameters (weights travel as kernel parameters)
    std::vector<float> m1; std::vector<int32_t> b1;
    if (!scales_of(c1, 32, m1) || !bias_of(c1, 32, b1)) return ZANT_OK;
    Conv1Args a1{};
    {
        const int8_t* w = (const int8_t*)T(c1.in[1]).host.data();
        for (int m = 0; m < 32; ++m) {
            int sum = 0;
            for (int kh = 0; kh < 3; ++kh) {
                const uint32_t w0 = (uint8_t)w[m * 9 + kh * 3 + 0], w1 = (uint8_t)w[m * 9 + kh * 3 + 1], w2 = (uint8_t)w[m * 9 + kh * 3 + 2];
                a1.wpack[m][kh][0] = w0 | (w1 << 8) | (w2 << 16);
                a1.wpack[m][kh][1] = (w0 << 8) | (w1 << 16) | (w2 << 24);
                sum += w[m * 9 + kh * 3] + w[m * 9 + kh * 3 + 1] + w[m * 9 + kh * 3 + 2];
            }
            a1.mult[m] = m1[m];
            a1.bias[m] = b1[m] - c1.a.x_zp * sum;
        }
        a1.n_images = (int)B; a1.x_scale = N[0].a.y_scale; a1.x_zp = N[0].a.y_zp;
        a1.y_scale = c1.a.y_scale; a1.y_zp = c1.a.y_zp; a1.act = ZANT_QACT_RELU;
    }
    // ---- stage 2 parameters
    std::vector<float> m2; std::vector<int32_t> b2;
    if (!scales_of(c2, 64, m2) || !bias_of(c2, 64, b2)) return ZANT_OK;
    std::vector<int8_t> w2arr(TcConvPoolCfg::W_BYTES);
    bool acc_base2 = true;                                          // accumulators and biases small enough for kAccBase
    {
        const int8_t* w = (const int8_t*)T(c2.in[1]).host.data();   // [64][32][3][3]
        for (int m = 0; m < 64; ++m) {
            int sum = 0;
            long long abs_sum = 0;
            for (int i = 0; i < 288; ++i) { sum += w[m * 288 + i]; abs_sum += std::abs((int)w[m * 288 + i]); }
            b2[m] -= c2.a.x_zp * sum;
            acc_base2 = acc_base2 && acc_base_ok(b2[m]) && std::abs((long long)b2[m]) + 128 * abs_sum < (1 << 22);
        }
        tc_conv_pool_weights(w, w2arr.data());
    }
    bool acc_base = true;
    for (int m = 0; m < 32; ++m) acc_base = acc_base && acc_base_ok(a1.bias[m]);
    // Few images: one kernel, a cluster for as few of them as fill the clusters that run at once, up to two rounds of sixteen a cluster (480 images 20.3
    // us in four kernels, 19.8 in one; 512, three rounds, 20.3 and 27.3).
    const int few_clusters = irb_band_resident(1, CnnFewCfg::CTAS, pl->ctx->sm_count);
    int few_imgs = 1;
    while (few_imgs < CnnFewCfg::IMGS && (size_t)few_imgs * few_clusters < B) few_imgs *= 2;
    const bool few = acc_base && acc_base2 && B <= (size_t)2 * CnnFewCfg::IMGS * few_clusters;
    // ---- fc1: rows re-ordered from the graph's (c,h,w) flatten order to the (h,w,c) order stage 2 writes
    std::vector<float> m3; std::vector<int32_t> b3;
    if (!scales_of(f1, 512, m3) || !bias_of(f1, 512, b3)) return ZANT_OK;
    // images per block of stages 1 and 2, blocks; windows per item of stage 2.  Five windows of a row share their column pairs; single windows
    // fill the SMs better while there are few of them.  A single window is counted as 1.2 of a shared one.  (Whole network, fives -> singles: 512
    // images 24.7 -> 20.3 us, 1024 28.4 -> 22.4, 2048 32.7 -> 27.4.)
    const int ib = (int)std::min<size_t>(B, 128), blocks128 = (int)((B + 127) / 128);
    const long long sms = pl->ctx->sm_count, singles = (blocks128 * 25 + sms - 1) / sms * 6, fives = (blocks128 * 5 + sms - 1) / sms * 25;
    const int c2_wins = singles <= fives ? 1 : 5, c2_items = blocks128 * 25 / c2_wins;
    // The narrowest column tile whose grid fits the SMs: a CTA streams all of K for its columns (batch 1: 12.6 us with two CTAs of 256).  Its CTAs
    // start on the SMs that stage 2 leaves free, two to an SM; where that takes all of them in, but not one to an SM, those that share one
    // finish last and a wider tile is faster (385 to 512 images, 64 CTAs for 48 SMs: 23.3 us, 20.3 with 32 CTAs).
    constexpr int FC_KC = 4, FC_STAGES = 8;
    int FC_NT = 32;
    const int free_sms = std::max(0, (int)sms - c2_items);
    auto fc_ctas = [&](int nt) { return blocks128 * (512 / nt); };
    while (FC_NT < 256 && (fc_ctas(FC_NT) > sms || (fc_ctas(FC_NT) > free_sms && fc_ctas(FC_NT) <= 2 * free_sms))) FC_NT *= 2;
    std::vector<int8_t> w3blk(1600 * 512);      // [512/NT][100 chunks][NT][16], K in (h,w,c) order
    {
        const int8_t* w = (const int8_t*)T(f1.in[1]).host.data();   // [1600][512], row = c*25 + h*5 + w
        std::vector<int> colsum(512, 0);
        // (16-bit sums of 200 rows, at most 25600: the host adds twice as many at a time)
        for (int k0 = 0; k0 < 1600; k0 += 200) {
            int16_t part[512] = {};
            for (int k = k0; k < k0 + 200; ++k)
                for (int n = 0; n < 512; ++n) part[n] = (int16_t)(part[n] + w[(size_t)k * 512 + n]);
            for (int n = 0; n < 512; ++n) colsum[n] += part[n];
        }
        // 16 channels of a position are a K chunk: 16 rows of the matrix, transposed
        for (int hw = 0; hw < 25 && !few; ++hw)
            for (int c16 = 0; c16 < 4; ++c16) {
                const int8_t* src = &w[(size_t)(c16 * 16 * 25 + hw) * 512];
                for (int n = 0; n < 512; ++n) {
                    int8_t* dst = &w3blk[((size_t)(n / FC_NT) * 100 * FC_NT + (size_t)(hw * 4 + c16) * FC_NT + n % FC_NT) * 16];
                    for (int c = 0; c < 16; ++c) dst[c] = src[(size_t)c * 25 * 512 + n];
                }
            }
        for (int n = 0; n < 512; ++n) b3[n] -= f1.a.x_zp * colsum[n];
    }
    std::vector<float> m4; std::vector<int32_t> b4;
    if (!scales_of(f2, NCLS, m4) || !bias_of(f2, NCLS, b4)) return ZANT_OK;
    {
        const int8_t* w = (const int8_t*)T(f2.in[1]).host.data();   // [512][NCLS]
        for (size_t n = 0; n < NCLS; ++n) {
            int sum = 0;
            for (int k = 0; k < 512; ++k) sum += w[(size_t)k * NCLS + n];
            b4[n] -= f2.a.x_zp * sum;
        }
    }

    const int a_m3 = pl->add_aux(m3.data(), m3.size() * 4), a_b3 = pl->add_aux(b3.data(), b3.size() * 4);
    const int a_m4 = pl->add_aux(m4.data(), m4.size() * 4), a_b4 = pl->add_aux(b4.data(), b4.size() * 4);
    const int w4 = f2.in[1];

    // B-fragment words, bias and multipliers in the per-lane order of the warp-level MMA
    std::vector<uint32_t> wfrag(4 * 4 * 32);
    std::vector<float> floorfrag(4 * 32 * 2), multfrag(4 * 32 * 2);
    {
        const int8_t* w = (const int8_t*)T(c1.in[1]).host.data();   // [32][1][3][3]
        for (int lane = 0; lane < 32; ++lane) {
            const int g = lane >> 2, t = lane & 3;
            for (int j = 0; j < 4; ++j) {
                const int ch = 8 * (g / 2) + 2 * j + (g % 2);        // column g of channel group j
                for (int m = 0; m < 4; ++m) {
                    const int dy = m >> 1, dx = m & 1, kh = t - dy;
                    uint32_t word = 0;
                    for (int sx = 0; sx < 4; ++sx) {
                        const int kw = sx - dx;
                        if (kh >= 0 && kh < 3 && kw >= 0 && kw < 3) word |= (uint32_t)(uint8_t)w[ch * 9 + kh * 3 + kw] << (8 * sx);
                    }
                    wfrag[(m * 4 + j) * 32 + lane] = word;
                }
                for (int b = 0; b < 2; ++b) {
                    const int cc = 8 * t + 2 * j + b;                // the lane's accumulator columns 2t, 2t+1
                    floorfrag[(j * 32 + lane) * 2 + b] = acc_base ? kAccBase - (float)a1.bias[cc] : int_bits_as_float(a1.bias[cc]);
                    multfrag[(j * 32 + lane) * 2 + b] = a1.mult[cc];
                }
            }
        }
    }
    QuantSteps steps{};
    if (a1.x_zp < 0 || a1.x_zp > 255 || !quant_steps(a1.x_scale, -a1.x_zp, 255 - a1.x_zp, steps)) steps = QuantSteps{0.0f, 0.0f};
    const int a_wf = pl->add_aux(wfrag.data(), wfrag.size() * 4);
    const int a_bf = pl->add_aux(floorfrag.data(), floorfrag.size() * 4);
    const int a_mf = pl->add_aux(multfrag.data(), multfrag.size() * 4);
    for (int k = 0; k < 11; ++k) pl->t[N[k].out[0]].elided = true;   // interior tensors live only inside the fused kernels
    consumed = 12;
    // algorithmic work of the fused steps: tensors that cross a kernel boundary once at their storage type,
    // weights included; of the 13 x 13 pooled pixels of stage 1 only the 12 x 12 that stage 2's pool reads exist
    const double Bd = (double)B, nc = (double)NCLS;
    auto costs = [&](std::initializer_list<double> macs, std::initializer_list<double> bytes) {
        pl->step_macs.resize(pl->steps.size() - macs.size(), 0.0); pl->step_bytes.resize(pl->steps.size() - bytes.size(), 0.0);
        pl->step_macs.insert(pl->step_macs.end(), macs); pl->step_bytes.insert(pl->step_bytes.end(), bytes);
    };
    if (few) {
        std::vector<uint8_t> blob;
        cnn_few_weights((const int8_t*)T(c2.in[1]).host.data(), (const int8_t*)T(f1.in[1]).host.data(), (const int8_t*)T(f2.in[1]).host.data(), (int)NCLS, blob);
        std::vector<float> floor2(64);
        for (int m = 0; m < 64; ++m) floor2[m] = kAccBase - (float)b2[m];
        const int a_blob = pl->add_aux(blob.data(), blob.size()), a_f2 = pl->add_aux(floor2.data(), 256), a_m2 = pl->add_aux(m2.data(), 256);
        CnnFewArgs k{};
        k.n_images = (int)B; k.imgs = few_imgs;
        k.x_scale = a1.x_scale; k.x_zp = a1.x_zp; k.q_rh = steps.rh; k.q_rl = steps.rl;
        k.ncls = (int)NCLS; k.y_scale = f2.a.y_scale; k.y_zp = f2.a.y_zp; k.dq_scale = N[11].a.x_scale; k.dq_zp = N[11].a.x_zp;
        push("Fused[QuantizeLinear+(QLinearConv+Relu+MaxPool)x2+QLinearMatMul+Relu+QLinearMatMul+DequantizeLinear] mma", [=]() {
            using Cfg = CnnFewCfg;
            CnnFewArgs a = k;
            a.x = pl->p<float>(x); a.y = pl->p<float>(y); a.status = ctx->status_word;
            if (!aligned16(a.x)) return fail(ZANT_E_INVALID_INPUT, "QuantizeLinear input buffer must be 16-byte aligned");
            a.wfrag = (const uint32_t*)pl->aux(a_wf); a.floor1 = (const float*)pl->aux(a_bf); a.mult1 = (const float*)pl->aux(a_mf);
            a.w = (const uint8_t*)pl->aux(a_blob); a.floor2 = (const float*)pl->aux(a_f2); a.mult2 = (const float*)pl->aux(a_m2);
            a.mult3 = (const float*)pl->aux(a_m3); a.bias3 = (const int32_t*)pl->aux(a_b3); a.mult4 = (const float*)pl->aux(a_m4); a.bias4 = (const int32_t*)pl->aux(a_b4);
            const unsigned grid = (unsigned)((k.n_images + k.imgs - 1) / k.imgs * Cfg::CTAS);
            auto go = [&](auto two) -> int32_t {
                ZB_SMEM_ATTR(ctx, (cnn_few_kernel<decltype(two)::value>), Cfg::SMEM_BYTES);
                launch_cluster(ctx, cnn_few_kernel<decltype(two)::value>, grid, Cfg::THREADS, Cfg::SMEM_BYTES, Cfg::CTAS, a);
                return ZANT_OK;
            };
            ZB_TRY(k.imgs > Cfg::CTAS ? go(std::true_type{}) : go(std::false_type{}));
            return check_launch(ctx, "cnn_few_kernel");
        });
        costs({Bd * (194688.0 + 2230272.0 + 819200.0 + 512.0 * nc)}, {Bd * (784.0 * 4 + 4.0 * nc) + 288.0 + 64.0 * 288 + 1600.0 * 512 + 512.0 * nc});
        return ZANT_OK;
    }
    // stage 1 -> stage 2 hand-over: image blocks
    const int s_pool1 = pl->add_scratch(blocks128 * (size_t)c2_block_bytes(ib));
    const int s_pool2 = pl->add_scratch((size_t)blocks128 * ib * 1600);
    const int s_fc1 = pl->add_scratch(B * 512);
    const int a_w2 = pl->add_aux(w2arr.data(), w2arr.size());
    const int a_w3 = pl->add_aux(w3blk.data(), w3blk.size());
    push("Fused[QuantizeLinear+QLinearConv+Relu+MaxPool] mma", [=]() {
        Conv1MmaArgs k{};
        k.x = pl->p<float>(x); k.y = (int8_t*)pl->scratch(s_pool1); k.n_images = (int)B; k.ib = ib;
        if (!aligned16(k.x)) return fail(ZANT_E_INVALID_INPUT, "QuantizeLinear input buffer must be 16-byte aligned");
        k.x_scale = a1.x_scale; k.x_zp = a1.x_zp; k.q_rh = steps.rh; k.q_rl = steps.rl;
        k.wfrag = (const uint32_t*)pl->aux(a_wf); k.floorfrag = (const float*)pl->aux(a_bf); k.multfrag = (const float*)pl->aux(a_mf); k.status = ctx->status_word;
        const int blocks = std::min<int>((int)((B + C1M_G - 1) / C1M_G), ctx->sm_count * 2);
        launch(ctx, acc_base ? conv1_mma_relu_pool_kernel<true> : conv1_mma_relu_pool_kernel<false>, blocks, C1M_THREADS, 0, k);
        return check_launch(ctx, "conv1_mma_relu_pool_kernel");
    });
    push("Fused[QLinearConv+Relu+MaxPool] tcgen05", [=]() {
        using Cfg = TcConvPoolCfg;
        TcConvPoolArgs k{};
        k.x = (const int8_t*)pl->scratch(s_pool1); k.w = (const int8_t*)pl->aux(a_w2);
        for (int m = 0; m < 64; ++m) { k.mult[m] = m2[m]; k.bias[m] = acc_base2 ? kAccBase - (float)b2[m] : int_bits_as_float(b2[m]); }
        k.y = (int8_t*)pl->scratch(s_pool2); k.n_images = (int)B; k.ib = ib; k.status = ctx->status_word;
        k.wins = c2_wins; k.items = c2_items;
        const int blocks = std::min<int>(k.items, ctx->sm_count);
        auto with = [&](auto base) -> int32_t {
            ZB_SMEM_ATTR(ctx, (tc_conv3x3_pool_kernel<decltype(base)::value>), Cfg::SMEM_BYTES);
            launch_const(ctx, tc_conv3x3_pool_kernel<decltype(base)::value>, blocks, Cfg::THREADS, Cfg::SMEM_BYTES, k);
            return check_launch(ctx, "tc_conv3x3_pool_kernel");
        };
        return acc_base2 ? with(std::true_type{}) : with(std::false_type{});
    });
    const zant_node_attrs f1a = f1.a, f2a = f2.a, dqa = N[11].a;
    push("Fused[Reshape+QLinearMatMul+Relu] tcgen05", [=]() {
        TcGemmArgs k{};
        k.a = (const int8_t*)pl->scratch(s_pool2); k.w = (const int8_t*)pl->aux(a_w3); k.a_rows = ib;
        k.mult = (const float*)pl->aux(a_m3); k.bias = (const int32_t*)pl->aux(a_b3);
        k.y = (int8_t*)pl->scratch(s_fc1); k.M = (int)B; k.N = 512; k.K16 = 100;
        k.y_scale = f1a.y_scale; k.y_zp = f1a.y_zp; k.act = ZANT_QACT_RELU; k.status = ctx->status_word;
        auto with = [&](auto nt) -> int32_t {
            constexpr int NT = decltype(nt)::value;
            using Cfg = TcGemmCfg<NT, FC_KC, FC_STAGES>;
            ZB_SMEM_ATTR(ctx, (tc_gemm_i8_kernel<NT, FC_KC, FC_STAGES>), Cfg::SMEM_BYTES);
            launch_const(ctx, tc_gemm_i8_kernel<NT, FC_KC, FC_STAGES>, std::min(blocks128 * (512 / NT), ctx->sm_count), Cfg::THREADS, Cfg::SMEM_BYTES, k);
            return check_launch(ctx, "tc_gemm_i8_kernel");
        };
        switch (FC_NT) {
            case 32: return with(std::integral_constant<int, 32>{});
            case 64: return with(std::integral_constant<int, 64>{});
            case 128: return with(std::integral_constant<int, 128>{});
            default: return with(std::integral_constant<int, 256>{});
        }
    });
    push("Fused[QLinearMatMul+DequantizeLinear]", [=]() {
        FcOutArgs k{};
        k.a = (const int8_t*)pl->scratch(s_fc1); k.w = pl->p<int8_t>(w4);
        k.mult = (const float*)pl->aux(a_m4); k.bias = (const int32_t*)pl->aux(a_b4);
        k.y = pl->p<float>(y); k.M = (int)B; k.K = 512; k.NCLS = (int)NCLS;
        k.y_scale = f2a.y_scale; k.y_zp = f2a.y_zp; k.dq_scale = dqa.x_scale; k.dq_zp = dqa.x_zp;
        // one or two column blocks of 8 classes
        auto with = [&](auto nc) -> int32_t {
            constexpr int NC = decltype(nc)::value;
            constexpr int smem = fcout_smem_bytes<NC, 512>();
            ZB_SMEM_ATTR(ctx, (fc_out_dequant_kernel<NC, 512>), smem);
            const int blocks = std::min<int>((int)((B + 127) / 128), ctx->sm_count * 3);
            launch(ctx, fc_out_dequant_kernel<NC, 512>, blocks, FCOUT_THREADS, smem, k);
            return check_launch(ctx, "fc_out_dequant_kernel");
        };
        return NCLS <= 8 ? with(std::integral_constant<int, 8>{}) : with(std::integral_constant<int, 16>{});
    });
    costs({Bd * 194688.0, Bd * 2230272.0, Bd * 819200.0, Bd * 512.0 * nc},
          {Bd * (784.0 * 4 + 144.0 * 32) + 288.0, Bd * (144.0 * 32 + 1600.0) + 64.0 * 288, Bd * (1600.0 + 512.0) + 1600.0 * 512, Bd * (512.0 + 4.0 * nc) + 512.0 * nc});
    return ZANT_OK;
}

// --------------------------------------------------------------------------------------------
// Layout pass: activations between convolutions stay channels-last (tc_nhwc_net.cuh) where their producer can write and every
// reader can read that form.  Producers: convolution groups, MaxPool, Concat over channels (its operands are written in place),
// and, for at most four channels, QuantizeLinear; readers: convolution groups, MaxPool, Concat.  Everything else - graph
// input and output, and whatever this pass does not know - keeps NCHW.  int8 contexts and, in TF32 mode, float ones alike.
// --------------------------------------------------------------------------------------------
static int nh_kind(const zant_plan* pl, int32_t dtype) {
    if (dtype == ZANT_I8) return NH_I8;
    if (dtype == ZANT_U8) return NH_U8;
    if (dtype == ZANT_F32 && pl->ctx->tf32) return pl->ctx->tf32 == 2 ? NH_TF32X3 : NH_TF32;
    return -1;
}

static bool nh_conv_geom(const zant_plan* pl, const PlanNode& n, ConvGeom& g) {
    const PlanTensor &x = pl->t[n.in[0]], &w = pl->t[n.in[1]], &y = pl->t[n.out[0]];
    const zant_node_attrs& a = n.a;
    if (n.op == ZANT_OP_QLINEAR_CONV)
        return conv_resolve_onnx(x.shape.data(), x.shape.size(), w.shape.data(), w.shape.size(), y.shape.data(), y.shape.size(), a.strides, a.n_strides, a.pads, a.n_pads,
                                 a.dilations, a.n_dilations, a.group, a.auto_pad < 0 ? 0 : a.auto_pad, g) == ZANT_OK;
    const char* ap = (a.auto_pad >= 0 && a.auto_pad <= 3) ? kAutoPadNames[a.auto_pad] : nullptr;
    return conv_resolve_ref(x.shape.data(), x.shape.size(), w.shape.data(), w.shape.size(), y.shape.data(), y.shape.size(), a.strides, a.n_strides, a.n_pads ? a.pads : nullptr,
                            a.n_pads, a.n_dilations ? a.dilations : nullptr, a.n_dilations, a.group, ap, ap ? std::strlen(ap) : 0, g) == ZANT_OK;
}

// Reads the convolution at node `i` with the activation, pool, upsampling and dequantisation behind it; false when the
// channels-last kernel cannot run it.
static bool nh_parse(const zant_plan* pl, const ChainCtx& c, size_t i, NhGroup& q) {
    const PlanNode& n = pl->nodes[i];
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    const bool i8 = n.op == ZANT_OP_QLINEAR_CONV;
    if ((!i8 && n.op != ZANT_OP_CONV) || n.a.channels_last || n.out.size() != 1 || n.in.size() < (i8 ? 3u : 2u) || n.in.size() > (i8 ? 5u : 3u)) return false;
    for (size_t k = 1; k < n.in.size(); ++k) if (n.in[k] >= 0 && !T(n.in[k]).is_const) return false;
    const int x = n.in[0], w = n.in[1];
    if (x < 0 || w < 0 || T(x).is_const || T(x).shape.size() != 4 || T(w).shape.size() != 4 || T(n.out[0]).shape.size() != 4 || (i8 && n.in[2] < 0)) return false;
    const int kind = nh_kind(pl, T(x).dtype);
    if (kind < 0 || (kind <= NH_U8) != i8 || (!i8 && T(x).dtype != ZANT_F32)) return false;
    ConvGeom g;
    if (!nh_conv_geom(pl, n, g)) return false;
    bool monotone = true;
    if (i8) {
        if (T(n.out[0]).dtype != ZANT_I8 || n.a.y_zp != 0 || T(w).dtype != ZANT_I8 || T(n.in[2]).dtype != ZANT_F32) return false;
        if (check_zero_point(T(x).dtype, n.a.x_zp, "QLinearConv x") != ZANT_OK) return false;
        if ((g.pt || g.pl || g.pb || g.pr) && n.a.x_zp != 0) return false;            // the halo is zero fill
        const int wz = opt_in(n, 3), b = opt_in(n, 4);
        if (wz >= 0 && (T(wz).dtype != ZANT_I32 || (T(wz).bytes != 4 && T(wz).bytes != (size_t)g.M * 4) || !all_zero_i32(T(wz)))) return false;
        if (b >= 0 && (T(b).dtype != ZANT_I32 || T(b).bytes != (size_t)g.M * 4)) return false;
        const size_t nws = T(n.in[2]).bytes / 4;
        if (nws != 1 && nws != (size_t)g.M) return false;
        std::vector<float> mult;
        requant_multipliers(n.a.x_scale, (const float*)T(n.in[2]).host.data(), nws, n.a.y_scale, (size_t)g.M, mult);
        if (!positive_finite(mult)) return false;
    } else {
        // (fewer than 128 positions stay with the exact kernels, as without this pass)
        if (T(w).dtype != ZANT_F32 || T(n.out[0]).dtype != ZANT_F32 || g.M > 2048 || (long long)g.N * g.OH * g.OW < 128) return false;
        const int b = opt_in(n, 2);
        if (b >= 0 && (T(b).dtype != ZANT_F32 || T(b).bytes != (size_t)g.M * 4)) return false;
    }
    // the input has to come channels-last from somewhere, or be a first layer's (no search for a tiling otherwise)
    if (T(x).shape[1] > 4) {
        bool from = false;
        for (size_t k = 0; k < i; ++k) {
            const PlanNode& p = pl->nodes[k];
            bool makes = false;
            for (int id : p.out) makes = makes || id == x;
            if (!makes) continue;
            const bool conv = p.op == ZANT_OP_QLINEAR_CONV || p.op == ZANT_OP_CONV;
            from = (conv && p.a.group <= 1) || p.op == ZANT_OP_RELU || p.op == ZANT_OP_LEAKY_RELU || p.op == ZANT_OP_CLIP || p.op == ZANT_OP_MAXPOOL || p.op == ZANT_OP_RESIZE || p.op == ZANT_OP_CONCAT;
        }
        if (!from) return false;
    }
    q = NhGroup{};
    q.first = i; q.x = x;
    size_t j = i + 1;
    int cur = n.out[0];
    auto next = [&](int32_t op) { return j < pl->nodes.size() && only_feeds_next(c, cur) && pl->nodes[j].op == op && !pl->nodes[j].in.empty() && pl->nodes[j].in[0] == cur && pl->nodes[j].out.size() == 1; };
    auto take = [&]() { q.interior.push_back(cur); cur = pl->nodes[j].out[0]; ++j; };
    if (i8 && (next(ZANT_OP_RELU) || next(ZANT_OP_LEAKY_RELU) || next(ZANT_OP_CLIP))) {
        const PlanNode& act = pl->nodes[j];
        if (act.in.size() == 1 && T(act.out[0]).dtype == ZANT_I8 && T(act.out[0]).shape == T(cur).shape && act.a.x_scale == n.a.y_scale && act.a.x_zp == n.a.y_zp) {
            if (identity_scale_relu(act)) q.qact = n.a.activation == ZANT_QACT_NONE ? ZANT_QACT_RELU : n.a.activation;
            else {
                q.lut_node = (int)j;
                uint8_t lut[256];
                activation_lut(act, ZANT_I8, lut);
                for (int v = -127; v < 128; ++v) monotone = monotone && (int8_t)lut[v & 255] >= (int8_t)lut[(v - 1) & 255];
            }
            take();
        }
    } else if (!i8 && (next(ZANT_OP_RELU) || next(ZANT_OP_LEAKY_RELU))) {
        const PlanNode& act = pl->nodes[j];
        if (act.in.size() == 1 && T(act.out[0]).dtype == ZANT_F32 && T(act.out[0]).shape == T(cur).shape) {
            q.fact = act.op == ZANT_OP_RELU ? FACT_RELU : FACT_LEAKY; q.slope = act.a.alpha;
            take();
        }
    }
    NhConvPlan np;
    if (monotone && next(ZANT_OP_MAXPOOL)) {
        const PlanNode& pool = pl->nodes[j];
        const auto& so = T(pool.out[0]).shape;
        if (pool.in.size() == 1 && pool2x2(pool.a) && T(pool.out[0]).dtype == T(cur).dtype && so.size() == 4 && so[0] == (size_t)g.N && so[1] == (size_t)g.M &&
            so[2] == (size_t)g.OH / 2 && so[3] == (size_t)g.OW / 2 && nh_conv_plan(g, kind, true, pl->ctx->sm_count, np)) {
            q.pool = true;
            take();
        }
    }
    if (!q.pool && !nh_conv_plan(g, kind, false, pl->ctx->sm_count, np)) return false;
    if (next(ZANT_OP_RESIZE)) {
        // nearest neighbour by two, as the index table says: every pixel goes to a 2 x 2 block
        const PlanNode& rs = pl->nodes[j];
        const auto &si = T(cur).shape, &so = T(rs.out[0]).shape;
        if (rs.in.size() == 1 && T(rs.out[0]).dtype == T(cur).dtype && rs.a.n_scales == 4 && so.size() == 4 && so[0] == si[0] && so[1] == si[1] && so[2] == 2 * si[2] && so[3] == 2 * si[3]) {
            std::vector<int32_t> table, off;
            resize_index_table(si.data(), so.data(), 4, rs.a.coord_mode, table, off);
            size_t os[4];
            bool ok = resize_output_shape(si.data(), 4, rs.a.scales, rs.a.n_scales, nullptr, 0, os) == ZANT_OK && std::equal(so.begin(), so.end(), os);
            for (int d = 0; d < 4; ++d) for (size_t o = 0; o < so[d]; ++o) ok = ok && table[off[d] + o] == (int32_t)(d < 2 ? o : o / 2);
            if (ok) { q.up2 = true; take(); }
        }
    } else if (i8 && next(ZANT_OP_DEQUANTIZE_LINEAR) && pl->nodes[j].in.size() == 1 && T(pl->nodes[j].out[0]).dtype == ZANT_F32 && T(pl->nodes[j].out[0]).shape == T(cur).shape) {
        q.dequant = (int)j;
        take();
    }
    q.y = cur;
    q.count = j - i;
    return true;
}

static void nh_layout(zant_plan* pl) {
    pl->nh_groups.clear();
    ChainCtx c{pl, std::vector<int>(pl->t.size(), 0)};
    for (const PlanNode& n : pl->nodes) for (int id : n.in) if (id >= 0) c.consumers[id]++;
    auto T = [&](int id) -> PlanTensor& { return pl->t[id]; };
    const size_t nn = pl->nodes.size();
    std::vector<int> group_of(nn, -1);
    std::vector<char> own(nn, 0);                            // nodes of the small CNN's own chain
    for (size_t i = 0; i < nn; ++i) {
        size_t took = 0;
        if (pl->nodes[i].op == ZANT_OP_QUANTIZE_LINEAR) try_fuse_small_cnn(pl, i, took, true);
        for (size_t k = i; k < i + took; ++k) own[k] = 1;
    }
    for (size_t i = 0; i < nn; ++i) {
        NhGroup q;
        if (own[i] || group_of[i] >= 0 || !nh_parse(pl, c, i, q)) continue;
        q.on = true;
        for (size_t k = i; k < i + q.count; ++k) group_of[k] = (int)pl->nh_groups.size();
        pl->nh_groups.push_back(q);
    }
    if (pl->nh_groups.empty()) return;
    std::vector<char> lay(pl->t.size(), 0);
    for (size_t id = 0; id < pl->t.size(); ++id) {
        const PlanTensor& t = T((int)id);
        lay[id] = !t.is_const && t.shape.size() == 4 && (int)id != pl->input && (int)id != pl->output && nh_kind(pl, t.dtype) >= 0 && t.bytes != 0;
    }
    std::vector<int> concat_of(pl->t.size(), -1);            // Concat node that a tensor is an operand of
    std::vector<char> operand_twice(pl->t.size(), 0);
    for (size_t i = 0; i < nn; ++i)
        if (pl->nodes[i].op == ZANT_OP_CONCAT) for (int id : pl->nodes[i].in) if (id >= 0) { operand_twice[id] = operand_twice[id] || concat_of[id] >= 0; concat_of[id] = (int)i; }
    auto first_layer = [&](int id) { return T(id).shape.size() == 4 && T(id).shape[1] <= 4; };
    bool changed = true;
    while (changed) {
        changed = false;
        auto off = [&](int id) { if (id >= 0 && lay[id]) { lay[id] = 0; changed = true; } };
        for (size_t i = 0; i < nn; ++i) {
            const PlanNode& n = pl->nodes[i];
            const int gi = group_of[i];
            if (gi >= 0 && pl->nh_groups[gi].on) {
                NhGroup& q = pl->nh_groups[gi];
                if (i != q.first) continue;
                for (int id : q.interior) lay[id] = 0;                             // interior: no layout of its own
                // the epilogue stores 16 channels at a time, and dequantised values as NCHW only
                if (T(q.y).shape[1] % 16 != 0 || q.dequant >= 0) off(q.y);
                const bool in_ok = lay[q.x] || (first_layer(q.x) && lay[q.y]);
                // an NCHW result cannot be upsampled in place, and a first layer pays for its conversion only in front of more such layers
                if (!in_ok || (!lay[q.y] && q.up2)) { q.on = false; changed = true; off(q.x); off(q.y); }
                continue;
            }
            switch (n.op) {
                case ZANT_OP_MAXPOOL:
                    if (n.in.size() == 1 && n.out.size() == 1 && lay[n.in[0]] && lay[n.out[0]] && T(n.in[0]).shape[1] % 16 == 0) break;
                    for (int id : n.in) off(id);
                    for (int id : n.out) off(id);
                    break;
                case ZANT_OP_CONCAT: {
                    const int64_t ax = n.a.axis < 0 ? n.a.axis + 4 : n.a.axis;
                    bool ok = ax == 1 && n.out.size() == 1 && lay[n.out[0]] && concat_of[n.out[0]] < 0;
                    for (int id : n.in) ok = ok && id >= 0 && lay[id] && T(id).shape[1] % 16 == 0 && !operand_twice[id];
                    if (ok) break;
                    for (int id : n.in) off(id);
                    for (int id : n.out) off(id);
                    break;
                }
                case ZANT_OP_QUANTIZE_LINEAR:
                    for (int id : n.in) off(id);
                    for (int id : n.out)
                        if (own[i] || n.out.size() != 1 || !lay[id] || !first_layer(id) || check_zero_point(T(id).dtype, n.a.y_zp, "QuantizeLinear y") != ZANT_OK) off(id);
                    break;
                default:
                    for (int id : n.in) off(id);
                    for (int id : n.out) off(id);
            }
        }
    }
    // storage
    const int parts = pl->ctx->tf32 == 2 ? 2 : 1;
    for (size_t id = 0; id < pl->t.size(); ++id) {
        PlanTensor& t = T((int)id);
        if (!lay[id]) continue;
        const size_t esz = dtype_size(t.dtype), chans = t.shape[1] <= 4 ? (esz == 1 ? 16 : (parts == 2 ? 8 : 4)) : t.shape[1];
        t.nh = true;
        t.nh_root = concat_of[id] >= 0 ? pl->nodes[concat_of[id]].out[0] : (int)id;
        if (t.nh_root == (int)id) { t.nh_pix = chans * esz * (esz == 4 ? parts : 1); t.nh_lo = esz == 4 && parts == 2 ? (int)chans : 0; }
    }
    for (size_t i = 0; i < nn; ++i) {
        const PlanNode& n = pl->nodes[i];
        if (n.op != ZANT_OP_CONCAT || !T(n.out[0]).nh) continue;
        size_t o = 0;
        for (int id : n.in) {
            PlanTensor& t = T(id);
            t.nh_off = o; t.nh_pix = T(n.out[0]).nh_pix; t.nh_lo = T(n.out[0]).nh_lo;
            o += t.shape[1] * dtype_size(t.dtype);
        }
    }
    for (NhGroup& q : pl->nh_groups) {
        if (!q.on) continue;
        for (int id : q.interior) T(id).elided = true;
        // a first layer that a QuantizeLinear feeds alone quantises its own input
        const PlanNode& n = pl->nodes[q.first];
        ConvGeom g;
        if (q.first == 0 || !q.pool || q.up2 || !T(q.y).nh || !T(q.x).nh || !only_feeds_next(c, q.x) || !nh_conv_geom(pl, n, g) || !first_q8_takes(g, pl->ctx->sm_count)) continue;
        const PlanNode& ql = pl->nodes[q.first - 1];
        if (ql.op != ZANT_OP_QUANTIZE_LINEAR || ql.in.size() != 1 || ql.out.size() != 1 || ql.out[0] != q.x) continue;
        q.quant = (int)q.first - 1;
        T(q.x).nh = false; T(q.x).elided = true;
    }
}

static NhView nh_view(zant_plan* pl, int id) {
    const PlanTensor& t = pl->t[id];
    return NhView{t.arena_ptr, (long long)t.nh_pix, (int)t.shape[2], (int)t.shape[3], t.nh_lo};
}

static int32_t refresh_nchw_copy(zant_plan* pl, int id, char* y) {
    const PlanTensor& t = pl->t[id];
    const uint64_t launched = pl->ctx->launches;
    const int32_t st = run_from_nhwc(pl->ctx, nh_view(pl, id), y, t.shape[0], t.shape[1], dtype_size(t.dtype));
    pl->ctx->launches = launched;                    // (not an operator launch)
    return st;
}

// Multipliers and biases (-x_zp * sum of the filter folded in) of `pad` filters: their numbers in the plan.
static void nh_int8_constants(zant_plan* pl, const NhGroup& q, const ConvGeom& g, size_t pad, int& am, int& ab) {
    const PlanNode& n = pl->nodes[q.first];
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    std::vector<float> mp; std::vector<int32_t> bp(pad, 0);
    const PlanTensor& ws = T(n.in[2]);
    const int b = opt_in(n, 4);
    requant_multipliers(n.a.x_scale, (const float*)ws.host.data(), ws.bytes / 4, n.a.y_scale, (size_t)g.M, mp);
    mp.resize(pad, 1.0f);
    const int K = g.Cg * g.KH * g.KW;
    for (int m = 0; m < g.M; ++m) {
        int sum = 0;
        if (n.a.x_zp != 0) for (int k = 0; k < K; ++k) sum += ((const int8_t*)T(n.in[1]).host.data())[(size_t)m * K + k];
        bp[m] = (b >= 0 ? ((const int32_t*)T(b).host.data())[m] : 0) - n.a.x_zp * sum;
    }
    am = pl->add_aux(mp.data(), mp.size() * 4); ab = pl->add_aux(bp.data(), bp.size() * 4);
}

// A group with its QuantizeLinear, whose nodes the caller has checked.
static int32_t build_first_layer(zant_plan* pl, const NhGroup& q, size_t& consumed) {
    const PlanNode &ql = pl->nodes[q.quant], &n = pl->nodes[q.first];
    zant_ctx* ctx = pl->ctx;
    const size_t first_step = pl->steps.size();
    ConvGeom g;
    if (!nh_conv_geom(pl, n, g)) return fail(ZANT_E_INVALID_DIMENSIONS, "convolution geometry");
    FirstQ8Args base{};
    const int x = ql.in[0], y = q.y;
    const bool u8 = pl->t[q.x].dtype == ZANT_U8;
    base.zp = ql.a.y_zp;
    base.qf = quant_fast(ql.a.y_scale, (float)((u8 ? 0 : -128) - base.zp), (float)((u8 ? 255 : 127) - base.zp));
    if (!quant_steps(ql.a.y_scale, (u8 ? 0 : -128) - base.zp, (u8 ? 255 : 127) - base.zp, base.qs)) base.qs = QuantSteps{0.0f, 0.0f};
    const int act = q.qact >= 0 ? q.qact : n.a.activation;
    base.floor = act == ZANT_QACT_NONE ? INT_MIN : 0;
    std::vector<uint8_t> table;                              // behind the ReLU: the bound of a ReLU6, the activation's table
    const int six = lean_six(n.a.y_scale);
    if (act == ZANT_QACT_RELU6 || q.lut_node >= 0) {
        table.resize(256);
        uint8_t lut[256];
        if (q.lut_node >= 0) activation_lut(pl->nodes[q.lut_node], ZANT_I8, lut);
        for (int v = 0; v < 256; ++v) {
            const uint8_t code = (uint8_t)(act == ZANT_QACT_RELU6 ? std::min(v, six & 255) : v);
            table[v] = q.lut_node >= 0 ? lut[code] : code;
        }
    }
    const int alut = table.empty() ? -1 : pl->add_aux(table.data(), table.size());
    std::vector<uint32_t> wfrag;
    first_q8_weights(g, (const int8_t*)pl->t[n.in[1]].host.data(), wfrag);
    const int aw = pl->add_aux(wfrag.data(), wfrag.size() * 4);
    int am, ab;
    nh_int8_constants(pl, q, g, (size_t)g.M, am, ab);
    pl->steps.push_back([=]() {
        FirstQ8Args a = base;
        const NhView v = nh_view(pl, y);
        a.x = pl->p<float>(x); a.wfrag = (const uint32_t*)pl->aux(aw); a.mult = (const float*)pl->aux(am); a.bias = (const int32_t*)pl->aux(ab);
        a.lut = alut >= 0 ? (const uint8_t*)pl->aux(alut) : nullptr;
        a.y = (uint8_t*)v.ptr; a.y_pix = v.pix; a.y_row = v.pix * v.W; a.y_img = a.y_row * v.H;
        return first_q8_run(ctx, g, u8, a);
    });
    pl->step_names.push_back(std::string("Fused[QuantizeLinear+QLinearConv") + (q.qact >= 0 ? "+Relu" : "") + (q.lut_node >= 0 ? "+ActivationLut" : "") + "+MaxPool]");
    record_step_cost(pl, first_step, (size_t)q.quant, q.count + 1);
    consumed = q.count + 1;
    return ZANT_OK;
}

static int32_t build_nh(zant_plan* pl, size_t i, size_t& consumed) {
    consumed = 0;
    const PlanNode& n = pl->nodes[i];
    zant_ctx* ctx = pl->ctx;
    auto T = [&](int id) -> const PlanTensor& { return pl->t[id]; };
    auto push = [&](const std::string& name, std::function<int32_t()> fn) { pl->steps.push_back(std::move(fn)); pl->step_names.push_back(name); };
    const size_t first_step = pl->steps.size();
    if (n.op == ZANT_OP_CONCAT && n.out.size() == 1 && T(n.out[0]).nh) {      // its operands are in place
        std::vector<const size_t*> shapes; std::vector<size_t> ranks;
        for (int id : n.in) { shapes.push_back(T(id).shape.data()); ranks.push_back(T(id).shape.size()); }
        ConcatGeom g; size_t os[8];
        ZB_TRY(concat_resolve(shapes.data(), ranks.data(), n.in.size(), n.a.axis, os, g));
        for (int id : n.in) if (T(id).dtype != T(n.out[0]).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "Concat dtype mismatch");
        for (size_t d = 0; d < 4; ++d) if (T(n.out[0]).shape[d] != os[d]) return fail(ZANT_E_MISMATCHED_SHAPE, "Concat output dim %zu", d);
        consumed = 1;
        return ZANT_OK;
    }
    const NhGroup* found = nullptr;
    for (const NhGroup& q : pl->nh_groups) if (q.on && (q.quant >= 0 ? (size_t)q.quant : q.first) == i) found = &q;
    if (n.op == ZANT_OP_QUANTIZE_LINEAR && n.out.size() == 1 && (T(n.out[0]).nh || found)) {
        ZB_TRY(need_inputs(n, 1, 1, "QuantizeLinear"));
        const int x = n.in[0], y = n.out[0];
        ZB_TRY(want_dtype(pl, x, ZANT_F32, "QuantizeLinear"));
        if (T(x).bytes != T(y).bytes * 4) return fail(ZANT_E_OUTPUT_TENSOR_DIFFERENT_SIZE, "QuantizeLinear sizes differ");
        if (found) return build_first_layer(pl, *found, consumed);
        const int N = (int)T(y).shape[0], C = (int)T(y).shape[1];
        const long long hw = (long long)(T(y).shape[2] * T(y).shape[3]);
        const float sc = n.a.y_scale; const int zp = n.a.y_zp; const bool u8 = T(y).dtype == ZANT_U8;
        QuantSteps steps{};
        if (!quant_steps(sc, (u8 ? 0 : -128) - zp, (u8 ? 255 : 127) - zp, steps)) steps = QuantSteps{0.0f, 0.0f};
        push("QuantizeLinear", [=]() { return run_to_nhwc(ctx, 0, pl->ptr(x), pl->t[y].arena_ptr, N, C, hw, sc, zp, u8, steps); });
        record_step_cost(pl, first_step, i, 1);
        consumed = 1;
        return ZANT_OK;
    }
    if (n.op == ZANT_OP_MAXPOOL && n.out.size() == 1 && T(n.out[0]).nh) {
        const zant_node_attrs& a = n.a;
        const int x = n.in[0], y = n.out[0];
        PoolGeom g;
        const size_t ones[2] = {1, 1};
        ZB_TRY(pool_resolve(T(x).shape.data(), T(x).shape.size(), T(y).shape.data(), T(y).shape.size(), a.kernel_shape, 2, a.n_strides ? a.strides : ones, 2,
                            a.n_dilations ? a.dilations : ones, 2, a.pads, a.n_pads, a.auto_pad < 0 ? 0 : a.auto_pad, g));
        if (T(x).dtype != T(y).dtype) return fail(ZANT_E_INPUT_ARRAY_WRONG_TYPE, "MaxPool dtype mismatch");
        const int kind = nh_kind(pl, T(x).dtype), N = (int)T(x).shape[0], C = (int)T(x).shape[1];
        push("MaxPool", [=]() { return run_nh_maxpool(ctx, kind, g, N, C, nh_view(pl, x), nh_view(pl, y)); });
        record_step_cost(pl, first_step, i, 1);
        consumed = 1;
        return ZANT_OK;
    }
    if (!found) return ZANT_OK;
    const NhGroup q = *found;
    ConvGeom g;
    if (!nh_conv_geom(pl, n, g)) return fail(ZANT_E_INVALID_DIMENSIONS, "convolution geometry");
    const int kind = nh_kind(pl, T(q.x).dtype);
    auto np = std::make_shared<NhConvPlan>();
    if (!nh_conv_plan(g, kind, q.pool, ctx->sm_count, *np)) return fail(ZANT_E_UNSUPPORTED, "shape not taken by the channels-last kernel");
    const bool i8 = kind <= NH_U8, split = kind == NH_TF32X3;
    const int x = q.x, y = q.y;
    int xbuf = -1;                                            // scratch of a first layer's converted input
    if (!T(x).nh) {
        const size_t px = (size_t)g.N * g.H * g.W;
        xbuf = pl->add_scratch(px * (split ? 64 : 16));
        const int mode = i8 ? 1 : (split ? 3 : 2), C = g.C; const long long hw = (long long)g.H * g.W;
        push(i8 ? "ToChannelsLast" : "ToChannelsLast(tf32)", [=]() { return run_to_nhwc(ctx, mode, pl->ptr(x), pl->scratch(xbuf), g.N, C, hw, 1.0f, 0, false); });
    }
    NhConvArgs base = np->a;
    int am = -1, ab = -1, alut = -1;
    std::string name;
    if (i8) {
        nh_int8_constants(pl, q, g, (size_t)base.const_n, am, ab);
        base.act = q.qact >= 0 ? q.qact : n.a.activation;
        base.six = lean_six(n.a.y_scale);
        name = "QLinearConv(tc-implicit)";
        if (q.qact >= 0) name += "+Relu";
        if (q.lut_node >= 0) {
            uint8_t lut[256];
            activation_lut(pl->nodes[q.lut_node], ZANT_I8, lut);
            alut = pl->add_aux(lut, 256);
            name += "+ActivationLut";
        }
        if (q.pool) name += "+MaxPool";
        if (q.dequant >= 0) { base.dq_scale = pl->nodes[q.dequant].a.x_scale; base.dq_zp = pl->nodes[q.dequant].a.x_zp; }
    } else {
        std::vector<float> bp((size_t)base.const_n, 0.0f);
        const int b = opt_in(n, 2);
        if (b >= 0) std::memcpy(bp.data(), T(b).host.data(), (size_t)g.M * 4);
        ab = pl->add_aux(bp.data(), bp.size() * 4);
        base.act = q.fact; base.slope = q.slope;
        name = std::string("Conv(tf32)") + (q.fact == FACT_RELU ? "+Relu" : (q.fact == FACT_LEAKY ? "+LeakyRelu" : ""));
    }
    if (q.up2) name += "+Resize";
    if (q.dequant >= 0) name += "+DequantizeLinear";
    const int aw = pl->add_scratch(np->w_bytes), w = n.in[1];
    pl->init_steps.push_back([=]() { return run_nh_weights(ctx, *np, pl->ptr(w), pl->scratch(aw)); });
    base.up2 = q.up2 ? 1 : 0;
    push(name, [=]() {
        NhConvArgs a = base;
        const PlanTensor& yt = pl->t[y];
        a.w = (const uint8_t*)pl->scratch(aw);
        if (i8) { a.mult = (const float*)pl->aux(am); a.bias = (const int32_t*)pl->aux(ab); a.lut = alut >= 0 ? (const uint8_t*)pl->aux(alut) : nullptr; }
        else a.fbias = (const float*)pl->aux(ab);
        if (yt.nh) {
            const NhView v = nh_view(pl, y);
            a.y = (uint8_t*)v.ptr; a.y_pix = v.pix; a.y_row = v.pix * v.W; a.y_img = a.y_row * v.H; a.lo_out = v.lo; a.round_out = 1;
        } else {
            a.y = (uint8_t*)pl->ptr(y); a.nchw = q.dequant >= 0 ? 2 : 1;
        }
        const NhView xv = xbuf >= 0 ? NhView{pl->scratch(xbuf), split ? 64 : 16, g.H, g.W, split ? 8 : 0} : nh_view(pl, x);
        return nh_conv_run(ctx, *np, a, xv);
    });
    record_step_cost(pl, first_step, i, q.count);
    consumed = q.count;
    return ZANT_OK;
}
