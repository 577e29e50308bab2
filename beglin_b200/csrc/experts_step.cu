// Routed experts of a step as ONE call from the host: the launches of routing, layout, products, activations and the sum per token, one behind the
// other, on scratch that the caller allocates in one piece.  The kernels and their order are those of the single entries.  Outside a captured
// step these launches are what bounds a small one: eight tokens with identity experts and a shared one took 121 us as eight entries of some twelve
// arguments and seven tensors in all, for kernels of 42; as one call 47 (host 29).
#include "common.cuh"

// A layer's experts, bfloat16: what does not change from step to step.  The host side fills the fields by name.
struct ExpertsArgs {
    const float* router; const float* choice_bias; const float* logit_bias;    // [outputs][hidden], [outputs] or null
    const void* up; const void* down;                                           // [experts][intermediate (twice with a gate)][hidden], [experts][hidden][intermediate]
    const void* shared_up; const void* shared_down;                             // [shared_rows][hidden], [hidden][shared], or null
    unsigned* status;
    int hidden, intermediate, experts, outputs, top, mode, renorm, scale_input;
    int act;                    // of experts without a gate (gemm_grouped's)
    int gated;                  // 0: no gate branch; 1: the clamped form; 2: silu
    int extended;               // the sum per token with ids, identity experts and shared rows
    int shared, shared_rows, shared_block, shared_gated, few;                  // few: tokens up to which route_rows takes a step
    float route_scale, limit, shared_limit, alpha;
};

namespace {

struct Scratch {
    size_t ids, weights, offsets, row_of, src_of, counts, xp, gu, hp, yp, shared_gu, shared_act, shared_out, bytes;
    int n_counts;
    Scratch(const ExpertsArgs& a, int T, bool inside) {        // inside: the shared expert's products run in the call
        const size_t A = (size_t)T * a.top;
        size_t at = 0;
        auto take = [&](size_t n) { const size_t p = at; at += (n + 255) & ~(size_t)255; return p; };
        n_counts = bg_route_layout_wins(T, a.hidden, a.outputs, a.top);
        ids = take(A * 4); weights = take(A * 4); offsets = take((size_t)(a.outputs + 1) * 4); row_of = take(A * 4); src_of = take(A * 4);
        counts = take((size_t)n_counts * 4);
        xp = take(A * a.hidden * 2);
        gu = take(a.gated ? A * 2 * a.intermediate * 2 : 0);
        hp = take(A * a.intermediate * 2);
        yp = take(A * a.hidden * 4);
        const size_t own = inside && a.shared ? T : 0;
        shared_gu = take(own * a.shared_rows * 4); shared_act = take(own * a.shared * 2); shared_out = take(own * a.hidden * 4);
        bytes = at;
    }
};

// The sum per token, over the routed rows in scratch and the shared expert's.
int total(const ExpertsArgs& a, const Scratch& s, char* w, const void* h, int T, const float* shared, const void* sg, int sg_dtype, int sg_stride, float* out,
          cudaStream_t stream) {
    const float* weights = (const float*)(w + s.weights);
    const int* row_of = (const int*)(w + s.row_of);
    return a.extended ? bg_route_combine_ext(w + s.yp, BG_DTYPE_F32, weights, row_of, (const int*)(w + s.ids), a.experts, h, BG_DTYPE_BF16, a.hidden, shared, sg, sg_dtype,
                                             sg_stride, out, T, a.hidden, a.top, stream)
                      : bg_route_combine(w + s.yp, BG_DTYPE_F32, weights, row_of, out, T, a.hidden, a.top, a.scale_input ? 0 : 1, stream);
}

}  // namespace

using namespace bg;

// Bytes of what the host side mirrors field by field; it compares them when it loads the library.
extern "C" int bg_experts_bytes() { return (int)sizeof(ExpertsArgs); }

// -1 where bg_experts_step does not take a step of T tokens (on 16 bytes): to be asked before anything is made for it.  inside: whether the shared
// expert's products run in the call (with up_splits).
extern "C" long long bg_experts_scratch(const ExpertsArgs* a, int T, int inside) {
    if (T < 0 || a->hidden <= 0 || a->hidden % 8 || a->intermediate <= 0 || a->intermediate % 8 || (uintptr_t)a->router % 16) return -1;
    if (T == 0) return 0;
    if (T <= a->few ? !bg_route_rows_takes(T, a->hidden, a->outputs, a->top) : !bg_route_layout_counts(T, a->hidden, a->outputs, a->top)) return -1;
    return (long long)Scratch(*a, T, inside).bytes;
}

// out [T][hidden] float = the step's result for h [T][hidden] bfloat16.  A shared expert runs in the call as the two fused products of few tokens
// (up_splits and down_splits ranges of their inner sizes), behind the routed ones.  With up_splits nought the caller makes its rows in the same place,
// and bg_experts_sum ends the step (out is not written): in front of the routing its products have nothing to fetch their weights under (64 rows of
// 768 features, 16 experts and a shared one of 1,024, captured: 49.5 us in front, 46.8 behind; 2,048 rows of 4,096 features and 8 experts 212 and 206).
// `launched` counts the kernels.  BG_ERR_UNSUPPORTED, with nothing launched, where the routing does not take the sizes.
extern "C" int bg_experts_step(const ExpertsArgs* args, const void* h, int T, int pairs, int up_splits, int down_splits, void* scratch,
                               long long scratch_bytes, float* out, int* launched, cudaStream_t stream) {
    if (launched) *launched = 0;
    if (T <= 0) return BG_OK;
    const ExpertsArgs& a = *args;
    if (a.hidden <= 0 || a.hidden % 8 || a.intermediate <= 0 || a.intermediate % 8 || (uintptr_t)h % 16 || (uintptr_t)scratch % 16)
        return BG_ERR_UNSUPPORTED;
    const Scratch s(a, T, up_splits != 0);
    if (scratch_bytes < (long long)s.bytes) return BG_ERR_SHAPE;
    char* w = (char*)scratch;
    int* ids = (int*)(w + s.ids); float* weights = (float*)(w + s.weights); int* offsets = (int*)(w + s.offsets);
    int* row_of = (int*)(w + s.row_of); int* src_of = (int*)(w + s.src_of);
    const int A = T * a.top, F = BG_DTYPE_F32, B = BG_DTYPE_BF16;
    int rc, n = 0;
    rc = bg_route_place(h, B, a.hidden, a.router, T, a.hidden, a.outputs, a.top, a.mode, a.renorm, a.choice_bias, a.route_scale, a.logit_bias, ids, weights, offsets,
                        row_of, src_of, w + s.xp, a.scale_input, (int*)(w + s.counts), s.n_counts, &n, stream);
    if (rc != BG_OK) return rc;
    auto grouped = pairs ? bg_gemm_grouped_pair : bg_gemm_grouped_tc;
    auto gate = [&](const void* gu, int dtype, int ld, void* to, int rows, int cols, float limit, int block) {
        return a.gated == 1 ? bg_glu_clamped(gu, dtype, ld, to, B, rows, cols, limit, a.alpha, stream)
                            : bg_swiglu(gu, dtype, 1, 0, to, B, rows, cols, block, 0, 0.0f, stream);
    };
    // (rows of experts without weights stay empty: the products see the first `experts` offsets only)
    if (a.gated) {
        rc = grouped(a.up, a.experts, 2 * a.intermediate, a.hidden, a.hidden, w + s.xp, A, a.hidden, w + s.gu, B, 2 * a.intermediate, offsets, 0, a.status, stream);
        if (rc == BG_OK) rc = gate(w + s.gu, B, 2 * a.intermediate, w + s.hp, A, a.intermediate, a.limit, 0);
        n += 2;
    } else {
        rc = grouped(a.up, a.experts, a.intermediate, a.hidden, a.hidden, w + s.xp, A, a.hidden, w + s.hp, B, a.intermediate, offsets, a.act, a.status, stream);
        ++n;
    }
    if (rc == BG_OK) rc = grouped(a.down, a.experts, a.hidden, a.intermediate, a.intermediate, w + s.hp, A, a.intermediate, w + s.yp, F, a.hidden, offsets, 0, a.status, stream);
    ++n;
    const bool whole = !a.shared || up_splits;
    const float* shared = nullptr;
    const float* sg = nullptr;
    if (rc == BG_OK && a.shared && up_splits) {
        float* gu = (float*)(w + s.shared_gu);
        if (a.shared_block) {
            rc = bg_gemm_fused(a.shared_up, a.shared_rows, a.hidden, a.hidden, h, a.hidden, nullptr, 0, nullptr, 0, 0, nullptr, 0.0f, T, nullptr, 2, w + s.shared_act, B,
                               a.shared, nullptr, 0, up_splits, 0.0f, a.status, stream);
        } else {
            rc = bg_gemm_fused(a.shared_up, a.shared_rows, a.hidden, a.hidden, h, a.hidden, nullptr, 0, nullptr, 0, 0, nullptr, 0.0f, T, nullptr, 0, gu, F, a.shared_rows,
                               nullptr, 0, up_splits, 0.0f, a.status, stream);
            if (rc == BG_OK) rc = gate(gu, F, a.shared_rows, w + s.shared_act, T, a.shared, a.shared_limit, 0);
            ++n;
        }
        shared = (const float*)(w + s.shared_out);
        if (rc == BG_OK)
            rc = bg_gemm_fused(a.shared_down, a.hidden, a.shared, a.shared, w + s.shared_act, a.shared, nullptr, 0, nullptr, 0, 0, nullptr, 0.0f, T, nullptr, 0,
                               w + s.shared_out, F, a.hidden, nullptr, 0, down_splits, 0.0f, a.status, stream);
        n += 2;
        sg = a.shared_gated ? gu + 2 * a.shared : nullptr;
    }
    if (rc == BG_OK && whole) rc = total(a, s, w, h, T, shared, sg, F, a.shared_rows, out, stream);
    if (launched) *launched = n + (whole ? 1 : 0);
    return rc;
}

// The end of a step whose shared expert's rows the caller has made since: shared [T][hidden] float and, behind a gate, sg (its type and stride).
extern "C" int bg_experts_sum(const ExpertsArgs* args, const void* h, int T, const float* shared, const void* sg, int sg_dtype, int sg_stride, void* scratch,
                              long long scratch_bytes, float* out, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    const Scratch s(*args, T, false);
    if (!args->shared || !shared || (sg != nullptr) != (args->shared_gated != 0) || scratch_bytes < (long long)s.bytes) return BG_ERR_SHAPE;
    return total(*args, s, (char*)scratch, h, T, shared, sg, sg_dtype, sg_stride, out, stream);
}
