// Attention through a latent for a step of few rows as ONE call from the host: the launches from the mixer's normed rows to the gated heads, one behind
// the other, on scratch that the caller allocates in one piece.  The kernels and their order are those of the single entries, which cost the host
// 150 us a step (thirteen tensors, four views, nine entries with their checks) for kernels of 45 to 140.
#include "common.cuh"

// A layer's attention, bfloat16: what does not change from step to step.  The host side fills the fields by name.
struct LatentArgs {
    const void* down; const void* q_up; const void* k_up_t; const void* v_up;      // [n_down][hidden], [heads (dim + rot)][q_rank], [heads][kv_rank][dim], [heads][vdim][kv_rank]
    const void* q_norm; const void* kv_norm; const float* sink; unsigned* status;
    int hidden, n_down, q_rank, kv_rank, dim, rot, rot_dims, vdim, heads;
    int kv_col, gate_col, gated, per_feature, norm_dtype, window, hc, stages;      // hc, stages: the mma.sync kernel's
    float eps, scale;
};
// What a step brings.
struct LatentStep {
    const void* h; const float* cos_sin; const int* positions; const int* row_req; const int* block_table; void* pool; const int* qblk;
    void* scratch; long long scratch_bytes; void* out;                              // out [T][heads vdim]
    int T, ldh, max_pages, num_pages, page_size, n_qblk, bq;
    int tc, n_splits, split, ctas;                                                  // the attention's kernel and its ranges of keys
    int down_fused, down_splits, q_fused, q_splits;                                 // the products' kernels and their ranges
};

namespace {

struct Scratch {
    size_t down, cq, q, q_lat, o_lat, part_o, part_ml, bytes;
    Scratch(const LatentArgs& a, int T, int n_splits) {
        size_t at = 0;
        auto take = [&](size_t n) { const size_t p = at; at += (n + 255) & ~(size_t)255; return p; };
        const size_t rows = (size_t)T * a.heads;
        down = take((size_t)T * a.n_down * 4); cq = take((size_t)T * a.q_rank * 2); q = take(rows * (a.dim + a.rot) * 2);
        q_lat = take(rows * a.kv_rank * 4); o_lat = take(rows * a.kv_rank * 2);
        part_o = take(rows * n_splits * a.kv_rank * 4); part_ml = take(rows * n_splits * 2 * 4);
        bytes = at;
    }
};

int product(const void* W, int n_out, int K, const void* X, int ldx, int T, void* out, int dtype, int fused, int splits, unsigned* status, cudaStream_t stream) {
    if (fused) return bg_gemm_fused(W, n_out, K, K, X, ldx, nullptr, 0, nullptr, 0, 0, nullptr, 0.0f, T, nullptr, 0, out, dtype, n_out, nullptr, 0, splits, 0.0f, status, stream);
    return bg_gemm_bf16_tn(W, n_out, K, K, X, T, ldx, nullptr, out, dtype, n_out, 1, status, stream);
}

}  // namespace

using namespace bg;

// Bytes of what the host side mirrors field by field; it compares them when it loads the library.
extern "C" int bg_latent_bytes(int step) { return (int)(step ? sizeof(LatentStep) : sizeof(LatentArgs)); }

extern "C" long long bg_latent_step_scratch(const LatentArgs* a, int T, int n_splits) { return (long long)Scratch(*a, T, n_splits).bytes; }

extern "C" int bg_latent_step(const LatentArgs* args, const LatentStep* step, cudaStream_t stream) {
    const LatentArgs& a = *args;
    const LatentStep& s = *step;
    if (s.T <= 0) return BG_OK;
    if (a.hidden <= 0 || a.heads <= 0 || a.q_rank <= 0 || s.n_splits <= 0 || (uintptr_t)s.scratch % 16) return BG_ERR_SHAPE;
    const Scratch w(a, s.T, s.n_splits);
    if (s.scratch_bytes < (long long)w.bytes) return BG_ERR_SHAPE;
    char* b = (char*)s.scratch;
    const int T = s.T, H = a.heads, R = a.kv_rank, F = BG_DTYPE_F32, B = BG_DTYPE_BF16, qd = a.dim + a.rot;
    float* down = (float*)(b + w.down);
    float* q_lat = (float*)(b + w.q_lat);
    float* part_o = (float*)(b + w.part_o);
    float* part_ml = (float*)(b + w.part_ml);
    int rc = product(a.down, a.n_down, a.hidden, s.h, s.ldh, T, down, F, s.down_fused, s.down_splits, a.status, stream);
    if (rc == BG_OK)
        rc = bg_latent_append(down, F, a.n_down, a.kv_col, R, a.rot, a.rot_dims, a.kv_norm, a.norm_dtype, a.eps, s.cos_sin, s.positions, s.row_req, s.block_table,
                              s.max_pages, s.pool, B, s.num_pages, s.page_size, T, a.status, 0, a.q_rank, a.q_norm, b + w.cq, B, stream);
    if (rc == BG_OK) rc = product(a.q_up, H * qd, a.q_rank, b + w.cq, a.q_rank, T, b + w.q, B, s.q_fused, s.q_splits, a.status, stream);
    if (rc == BG_OK)
        rc = bg_gemm_heads(a.k_up_t, H, R, a.dim, b + w.q, T, H * qd, H * qd, 0, qd, T, q_lat, F, (long long)T * R, R, nullptr, F, 0, 0, 0, a.status, stream);
    if (rc == BG_OK)
        rc = s.tc ? bg_latent_attention_tc_partial(q_lat, (long long)T * R, R, b + w.q, H * qd, qd, a.dim, s.cos_sin, s.pool, s.num_pages, s.page_size, s.block_table,
                                                   s.max_pages, s.positions, s.qblk, s.n_qblk, part_o, part_ml, s.n_splits, H, R, a.rot, a.rot_dims, a.window, a.scale,
                                                   a.status, stream)
                  : bg_latent_attention_mma_partial(q_lat, (long long)T * R, R, b + w.q, H * qd, qd, a.dim, s.cos_sin, s.pool, s.num_pages, s.page_size, s.block_table,
                                                    s.max_pages, s.positions, s.qblk, s.n_qblk, part_o, part_ml, s.n_splits, s.n_splits, H, a.hc, R, a.rot, a.rot_dims,
                                                    s.split, s.bq, a.stages, a.window, a.scale, a.status, stream);
    if (rc == BG_OK)
        rc = bg_latent_attention_merge(part_o, part_ml, s.positions, b + w.o_lat, B, (long long)T * R, R, T, H, R, s.n_splits, s.split, a.window, a.sink, s.ctas, stream);
    if (rc == BG_OK)
        rc = bg_gemm_heads(a.v_up, H, a.vdim, R, b + w.o_lat, (long long)H * T, R, R, T, 0, T, s.out, B, a.vdim, H * a.vdim, a.gated ? down : nullptr, F, a.n_down,
                           a.gate_col, a.per_feature, a.status, stream);
    return rc;
}
