// Mamba-2 between its two products as ONE call from the host: convolution, the walk of short portions, the chunks of long ones, norm and gate, one
// behind the other, on scratch that the caller allocates in one piece.  The kernels and their order are those of the single entries; outside a captured
// step those cost the host some 65 us beside the products' 28, for kernels of 30 to 40 in portions of a few hundred rows.
#include "common.cuh"

// What does not change from step to step; the host side fills the fields by name.
struct Mamba2Args {
    const void* conv_w; const void* conv_b; const void* dt_bias; const void* A_log; const void* D; const void* norm_w; unsigned* status;
    int w_dtype, norm_dtype, out_dtype, inner, channels, taps, H, P, N, G, norm_groups, tensor_cores, chunk;
    float eps;
};
struct Mamba2Step {
    const float* proj; float* state; const int* slots; const int* row_req; const int* requests; const int* reqs; const int* chunks; const int* longs;
    void* scratch; void* out;                  // out [T][inner]
    long long slot_stride, conv_off, scratch_bytes;
    int T, ldp, n_requests, n_req, n_chunks, n_long;      // requests: all of the step; reqs: those that are walked
};

namespace {

struct Scratch {
    size_t xbc, y, scores, work, decay, bytes;
    Scratch(const Mamba2Args& a, int T, int n_chunks) {
        size_t at = 0;
        auto take = [&](size_t n) { const size_t p = at; at += (n * 4 + 255) & ~(size_t)255; return p; };
        const size_t c = n_chunks;
        xbc = take((size_t)T * a.channels); y = take((size_t)T * a.inner);
        scores = take(c * a.G * a.chunk * a.chunk); work = take(c * a.H * a.N * a.P); decay = take(c * a.H);
        bytes = at;
    }
};

}  // namespace

using namespace bg;

// Bytes of what the host side mirrors field by field; it compares them when it loads the library.
extern "C" int bg_mamba2_bytes(int step) { return (int)(step ? sizeof(Mamba2Step) : sizeof(Mamba2Args)); }

extern "C" long long bg_mamba2_scratch(const Mamba2Args* a, int T, int n_chunks) { return (long long)Scratch(*a, T, n_chunks).bytes; }

// `launched` counts the kernels as the single entries do.
extern "C" int bg_mamba2_step(const Mamba2Args* args, const Mamba2Step* step, int* launched, cudaStream_t stream) {
    const Mamba2Args& a = *args;
    const Mamba2Step& s = *step;
    if (launched) *launched = 0;
    if (s.T <= 0) return BG_OK;
    if (a.inner <= 0 || a.channels <= 0 || a.H <= 0 || s.n_chunks < 0 || (uintptr_t)s.scratch % 16) return BG_ERR_SHAPE;
    const Scratch w(a, s.T, s.n_chunks);
    if (s.scratch_bytes < (long long)w.bytes) return BG_ERR_SHAPE;
    char* b = (char*)s.scratch;
    float* xbc = (float*)(b + w.xbc);
    float* y = (float*)(b + w.y);
    const int F = BG_DTYPE_F32, dt_col = a.inner + a.channels;
    int n = 0;
    int rc = bg_conv_silu(s.proj, F, s.ldp, a.inner, a.channels, a.taps, a.conv_w, a.conv_b, a.w_dtype, s.state, s.slot_stride, s.conv_off, s.slots, s.row_req,
                          s.requests, s.n_requests, xbc, s.T, 1, nullptr, &n, stream);
    if (rc == BG_OK && s.n_req) {
        rc = bg_ssm_scan(xbc, a.channels, s.proj, F, s.ldp, dt_col, a.dt_bias, a.A_log, a.D, a.w_dtype, s.state, s.slot_stride, s.slots, s.reqs, s.n_req, y, a.H, a.P,
                         a.N, a.G, stream);
        ++n;
    }
    if (rc == BG_OK && s.n_chunks) {
        rc = bg_ssm_chunked(xbc, a.channels, s.proj, F, s.ldp, dt_col, a.dt_bias, a.A_log, a.D, a.w_dtype, s.state, s.slot_stride, s.slots, s.chunks, s.n_chunks, s.longs,
                            s.n_long, (float*)(b + w.scores), (float*)(b + w.work), (float*)(b + w.decay), y, a.H, a.P, a.N, a.G, a.tensor_cores, a.status, stream);
        n += 4;
    }
    if (rc == BG_OK)
        rc = bg_gated_group_rmsnorm(y, s.proj, F, s.ldp, 0, a.norm_w, a.norm_dtype, a.eps, s.out, a.out_dtype, s.T, a.inner, a.norm_groups, 0, stream);
    if (launched) *launched = n + 1;
    return rc;
}
