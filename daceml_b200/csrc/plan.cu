// Launch plans: the calls of a compiled graph as one native object.
//
// A graph is compiled once and run many times with other tensors.  Run from Python, every call of the graph costs the
// wrapper's share of interpreter time (views, strides, parameter blocks, a foreign-function call): 12-17 us per launch,
// several times the kernels' own time for small batches.  A plan keeps the parameter blocks of all its calls in one
// blob, with a list of the places that hold addresses of the graph's inputs and outputs; a run copies the blob, writes
// the tensors' addresses into those places and makes the calls.  Everything an entry point decides from its arguments
// (alignment, kernel choice, tensor maps) is still decided at each run, on the addresses of that run.
//
// Measured on one B200 (us per pass, passes enqueued back to back, before -> with the plan): one convolution 26.4 -> 12.2,
// an MLP of four launches at batch 4096 67.7 -> 44.1 (then bound by its kernels), a four-layer encoder of 37 launches
// 545 -> 390.
#include "common.cuh"

#include <string.h>
#include <new>
#include <vector>

namespace {

enum PlanOp : int32_t {
    P_GEMM = 0, P_SOFTMAX, P_LAYERNORM, P_REDUCE, P_UNARY, P_BINARY, P_BIAS_ACT, P_TRANSPOSE, P_CAST, P_CONV2D, P_SE_GATE,
    P_ATTENTION, P_STRIDED_COPY, P_STRIDED_COPY_PARTS, P_GATHER, P_WHERE, P_COMPARE, P_MAXPOOL2D, P_COUNT
};
// Words of each call: its arguments between the context and the stream, in order.  A structure or an array is stored in
// the blob itself and its word holds its offset.
constexpr int kWords[P_COUNT] = {2, 9, 10, 7, 7, 9, 8, 6, 5, 1, 10, 1, 7, 8, 8, 10, 9, 14};

struct Patch {
    int64_t at;      // byte offset of the pointer in the blob
    int32_t slot;    // which of the run's tensors
    int64_t offset;  // bytes past that tensor's first element
};

struct Words {
    char* base;
    int64_t* w;
    int32_t i32(int i) const { return static_cast<int32_t>(w[i]); }
    int64_t i64(int i) const { return w[i]; }
    float f(int i) const {
        double d;
        memcpy(&d, &w[i], sizeof(d));
        return static_cast<float>(d);
    }
    void* p(int i) const { return reinterpret_cast<void*>(w[i]); }
    template <typename T>
    T* at(int i) const {
        return reinterpret_cast<T*>(base + w[i]);
    }
};

}  // namespace

struct b200ml_plan {
    std::vector<int32_t> ops;
    std::vector<int64_t> offsets;
    std::vector<char> blob;
    std::vector<Patch> patches;
    int32_t n_slots = 0;
};

using namespace b200ml;

static int plan_call(b200ml_ctx* ctx, int32_t op, const Words& a, b200ml_stream s) {
    switch (op) {
        case P_GEMM: return b200ml_gemm_packed(ctx, a.at<b200ml_gemm_params>(0), a.p(1), s);
        case P_SOFTMAX:
            return b200ml_softmax(ctx, a.i32(0), a.p(1), a.p(2), a.p(3), a.i64(4), a.i64(5), a.i64(6), a.f(7), a.i32(8), s);
        case P_LAYERNORM:
            return b200ml_layernorm(ctx, a.i32(0), a.p(1), a.p(2), a.p(3), a.p(4), a.p(5), a.p(6), a.i64(7), a.i64(8), a.f(9), s);
        case P_REDUCE: return b200ml_reduce(ctx, a.i32(0), a.i32(1), a.p(2), a.p(3), a.i64(4), a.i64(5), a.i64(6), s);
        case P_UNARY: return b200ml_unary(ctx, a.i32(0), a.i32(1), a.p(2), a.p(3), a.i64(4), a.f(5), a.f(6), s);
        case P_BINARY:
            return b200ml_binary(ctx, a.i32(0), a.i32(1), a.p(2), a.p(3), a.p(4), a.i32(5), a.at<int64_t>(6), a.at<int64_t>(7),
                                 a.at<int64_t>(8), s);
        case P_BIAS_ACT:
            return b200ml_bias_act(ctx, a.i32(0), a.p(1), a.p(2), a.p(3), a.p(4), a.i64(5), a.i64(6), a.i32(7), s);
        case P_TRANSPOSE: return b200ml_transpose(ctx, a.i32(0), a.p(1), a.p(2), a.i32(3), a.at<int64_t>(4), a.at<int32_t>(5), s);
        case P_CAST: return b200ml_cast(ctx, a.i32(0), a.i32(1), a.p(2), a.p(3), a.i64(4), s);
        case P_CONV2D: return b200ml_conv2d(ctx, a.at<b200ml_conv_params>(0), s);
        case P_SE_GATE:
            return b200ml_se_gate(ctx, a.i32(0), a.p(1), a.p(2), a.p(3), a.p(4), a.p(5), a.p(6), a.i64(7), a.i64(8), a.i64(9), s);
        case P_ATTENTION: return b200ml_attention_f16(ctx, a.at<b200ml_attention_params>(0), s);
        case P_STRIDED_COPY:
            return b200ml_strided_copy(ctx, a.i32(0), a.p(1), a.p(2), a.i32(3), a.at<int64_t>(4), a.at<int64_t>(5), a.at<int64_t>(6), s);
        case P_STRIDED_COPY_PARTS:
            return b200ml_strided_copy_parts(ctx, a.i32(0), a.i32(1), a.at<const void*>(2), a.at<void*>(3), a.i32(4), a.at<int64_t>(5),
                                             a.at<int64_t>(6), a.at<int64_t>(7), s);
        case P_GATHER:
            return b200ml_gather(ctx, a.i32(0), a.p(1), static_cast<const int64_t*>(a.p(2)), a.p(3), a.i64(4), a.i64(5), a.i64(6), a.i64(7), s);
        case P_WHERE:
            return b200ml_where(ctx, a.i32(0), a.p(1), a.p(2), a.p(3), a.p(4), a.i32(5), a.at<int64_t>(6), a.at<int64_t>(7),
                                a.at<int64_t>(8), a.at<int64_t>(9), s);
        case P_COMPARE:
            return b200ml_compare(ctx, a.i32(0), a.i32(1), a.p(2), a.p(3), a.p(4), a.i32(5), a.at<int64_t>(6), a.at<int64_t>(7),
                                  a.at<int64_t>(8), s);
        case P_MAXPOOL2D:
            return b200ml_maxpool2d(ctx, a.i32(0), a.p(1), a.p(2), a.i64(3), a.i64(4), a.i64(5), a.i32(6), a.i32(7), a.i32(8), a.i32(9),
                                    a.i32(10), a.i32(11), a.i32(12), a.i32(13), s);
    }
    return fail(B200ML_ERR_INVALID, "plan_run: unknown operation %d", op);
}

extern "C" {

int b200ml_plan_create(int32_t n_calls, const int32_t* ops, const int64_t* offsets, const void* blob, int64_t blob_bytes,
                       int32_t n_patches, const int64_t* patches, int32_t n_slots, b200ml_plan** out) {
    B200ML_REQUIRE(out != nullptr, "plan_create: null output pointer");
    *out = nullptr;
    B200ML_REQUIRE(n_calls >= 0 && n_patches >= 0 && n_slots >= 0 && blob_bytes >= 0, "plan_create: negative count");
    B200ML_REQUIRE(n_calls == 0 || (ops && offsets && blob), "plan_create: null array");
    B200ML_REQUIRE(n_patches == 0 || patches, "plan_create: null patch list");
    for (int32_t i = 0; i < n_calls; ++i) {
        B200ML_REQUIRE(ops[i] >= 0 && ops[i] < P_COUNT, "plan_create: unknown operation %d", ops[i]);
        B200ML_REQUIRE(offsets[i] >= 0 && offsets[i] % 8 == 0 && offsets[i] + 8 * kWords[ops[i]] <= blob_bytes,
                       "plan_create: call %d lies outside the blob", i);
    }
    for (int32_t i = 0; i < n_patches; ++i) {
        B200ML_REQUIRE(patches[3 * i] >= 0 && patches[3 * i] % 8 == 0 && patches[3 * i] + 8 <= blob_bytes, "plan_create: patch %d lies outside the blob", i);
        B200ML_REQUIRE(patches[3 * i + 1] >= 0 && patches[3 * i + 1] < n_slots, "plan_create: patch %d names no tensor", i);
    }
    b200ml_plan* p = new (std::nothrow) b200ml_plan();
    if (!p) return fail(B200ML_ERR_CUDA, "plan_create: out of host memory");
    p->ops.assign(ops, ops + n_calls);
    p->offsets.assign(offsets, offsets + n_calls);
    p->blob.assign(static_cast<const char*>(blob), static_cast<const char*>(blob) + blob_bytes);
    for (int32_t i = 0; i < n_patches; ++i)
        p->patches.push_back(Patch{patches[3 * i], static_cast<int32_t>(patches[3 * i + 1]), patches[3 * i + 2]});
    p->n_slots = n_slots;
    *out = p;
    return B200ML_OK;
}

int b200ml_plan_destroy(b200ml_plan* plan) {
    delete plan;
    return B200ML_OK;
}

int b200ml_plan_run(const b200ml_plan* plan, b200ml_ctx* ctx, void* const* slots, int32_t n_slots, b200ml_stream stream) {
    B200ML_REQUIRE(plan != nullptr, "plan_run: null plan");
    B200ML_REQUIRE(ctx != nullptr, "plan_run: null context");
    B200ML_REQUIRE(n_slots == plan->n_slots && (n_slots == 0 || slots), "plan_run: %d tensors given, the plan has %d", n_slots, plan->n_slots);
    DeviceGuard guard(ctx->device);
    // a copy per thread: several threads may run one plan, each with tensors of its own
    static thread_local std::vector<int64_t> scratch;
    const size_t words = (plan->blob.size() + 7) / 8;
    if (scratch.size() < words) scratch.resize(words);
    char* blob = reinterpret_cast<char*>(scratch.data());
    memcpy(blob, plan->blob.data(), plan->blob.size());
    for (const Patch& q : plan->patches) {
        char* v = static_cast<char*>(slots[q.slot]) + q.offset;
        memcpy(blob + q.at, &v, sizeof(v));
    }
    for (size_t i = 0; i < plan->ops.size(); ++i) {
        const Words a{blob, reinterpret_cast<int64_t*>(blob + plan->offsets[i])};
        const int rc = plan_call(ctx, plan->ops[i], a, stream);
        if (rc) return rc;
    }
    return B200ML_OK;
}

}  // extern "C"
