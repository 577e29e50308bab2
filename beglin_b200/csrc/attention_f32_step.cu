// Float attention of a step as ONE call from the host: q/k/v product, rotation and append, attention, merge and output product, one behind the
// other, on scratch that the caller allocates in one piece.  The kernels and their order are those of the single entries; outside a captured step those
// cost the host 80 to 90 us for kernels of 55 to 75.
#include "common.cuh"

// A layer's attention, float32, its plain form (heads of one size, no gates, no norms of queries and keys, a cache of its own in float32).  The host
// side fills the fields by name.
struct AttnF32Args {
    const float* qkv; const float* qkv_bias; const float* out; const float* out_bias;      // [(heads + 2 kv_heads) hd][hidden], [hidden][heads hd]; biases may be null
    const float* sink_w; unsigned* status;
    int hidden, heads, kv_heads, hd, rot, interleaved, window, keep, split, bq, tile, sink;
    float scale, softcap;
};
struct AttnF32Step {
    const float* h; const float* cos_sin; const int* positions; const int* row_req; const int* block_table; float* pool; const int* qblk; float* scratch; float* out;
    long long scratch_floats;
    int T, ldh, max_pages, num_pages, page_size, n_qblk, n_splits, pad;
};

namespace {

struct Scratch {
    long long qkv, q, rows, part_o, part_ml, rest, floats;
    Scratch(const AttnF32Args& a, int T, int n_splits) {
        long long at = 0;
        auto take = [&](long long n) { const long long p = at; at += (n + 63) & ~63LL; return p; };
        const long long qd = (long long)a.heads * a.hd, all = qd + 2LL * a.kv_heads * a.hd;
        qkv = take(T * all); q = take(T * qd); rows = take(T * qd);
        part_o = take((long long)T * a.heads * n_splits * a.hd); part_ml = take((long long)T * a.heads * n_splits * 2);
        const long long x = bg_gemm_f32_scratch(T, (int)all, a.hidden, 1), y = bg_gemm_f32_scratch(T, a.hidden, (int)qd, 1);
        rest = take(x > y ? x : y);
        floats = at;
    }
};

}  // namespace

using namespace bg;

// Bytes of what the host side mirrors field by field; it compares them when it loads the library.
extern "C" int bg_attention_f32_bytes(int step) { return (int)(step ? sizeof(AttnF32Step) : sizeof(AttnF32Args)); }

extern "C" long long bg_attention_f32_scratch(const AttnF32Args* a, int T, int n_splits) { return Scratch(*a, T, n_splits).floats; }

extern "C" int bg_attention_f32_step(const AttnF32Args* args, const AttnF32Step* step, cudaStream_t stream) {
    const AttnF32Args& a = *args;
    const AttnF32Step& s = *step;
    if (s.T <= 0) return BG_OK;
    if (a.hidden <= 0 || a.heads <= 0 || a.kv_heads <= 0 || a.hd <= 0 || s.n_splits <= 0 || (uintptr_t)s.scratch % 16) return BG_ERR_SHAPE;
    const Scratch w(a, s.T, s.n_splits);
    if (s.scratch_floats < w.floats) return BG_ERR_SHAPE;
    float* b = s.scratch;
    const int T = s.T, F = BG_DTYPE_F32, qd = a.heads * a.hd, all = qd + 2 * a.kv_heads * a.hd;
    int rc = bg_gemm_f32_nt(s.h, s.ldh, a.qkv, a.hidden, a.qkv_bias, b + w.qkv, all, T, all, a.hidden, 0, b + w.rest, a.status, stream);
    if (rc == BG_OK)
        rc = bg_rope_kv_append(b + w.qkv, F, all, 1, 0, b + w.q, F, qd, s.cos_sin, s.positions, s.row_req, s.block_table, s.max_pages, s.pool, F, s.num_pages,
                               s.page_size, T, a.heads, a.kv_heads, a.hd, a.rot, a.interleaved, a.status, stream);
    if (rc == BG_OK)
        rc = bg_attention_partial(b + w.q, F, qd, s.pool, F, s.num_pages, s.page_size, s.block_table, s.max_pages, s.positions, s.qblk, s.n_qblk, b + w.part_o,
                                  b + w.part_ml, s.n_splits, s.n_splits, a.heads, a.kv_heads, a.hd, a.hd, a.window, a.split, a.tile, a.bq, a.scale, a.softcap,
                                  a.keep, nullptr, 1, a.status, stream);
    if (rc == BG_OK)
        rc = bg_attention_merge(b + w.part_o, b + w.part_ml, s.positions, b + w.rows, F, qd, T, a.heads, a.hd, s.n_splits, a.split, a.window, a.sink, a.sink_w,
                                a.keep, stream);
    if (rc == BG_OK) rc = bg_gemm_f32_nt(b + w.rows, qd, a.out, qd, a.out_bias, s.out, a.hidden, T, a.hidden, qd, 0, b + w.rest, a.status, stream);
    return rc;
}
