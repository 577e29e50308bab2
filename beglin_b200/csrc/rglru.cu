// The real-gated linear recurrent unit: per channel c a state S_c that is carried from token to token,
//
//   r = sigmoid(gr + br),  i = sigmoid(gi + bi)        gr, gi: the gates' products of the convolved input u
//   log a = -C r softplus(lam_c),  a = e^(log a)
//   S <- a S + sqrt(1 - a^2) (i u),   out = S * gelu_tanh(y)      y: the other branch's product of the same token
//
// from S = 0 at a request's start (the first token is no special case).  Everything is float: the gates, the decay and
// its logarithm, the step and the state.  1 - a^2 = -e (2 + e) with e = expm1(log a), which does not cancel for a near one, and a = 1 + e
// down to a half; below, where 1 + e would keep fewer and fewer of a's own digits, a is an exponential of its own.
//
//   rglru_scan          one thread per (request, channel) walks the request's rows of the step in order from the state
//                       in the request's slot and leaves the new state there.  Steps of single tokens and short portions.
//   rglru_scan_chunked  long portions: the rows of a request are cut into chunks; S_end = P S_begin + Q with
//                       P = prod a, Q the chunk's walk from zero, so (1) every (chunk, channel) forms P and Q, (2) a
//                       thread per channel walks the chunks of a request to every chunk's starting state, (3) every
//                       (chunk, channel) walks its rows again from that state and writes the outputs, with the rows' (a, b)
//                       as the first walk left them.  The two walks differ from the plain one by rounding only.
//
// The gates' products come as [blocks][T][2 bs]: for channel c = b bs + o the recurrence gate at [b][t][o] and the
// input gate at [b][t][bs + o].
#include "common.cuh"

namespace bg {

constexpr int LRU_THREADS = 128;

struct LruParams {
    const float* gates;     // [blocks][T][2 bs]
    const float* u;         // [T][W] the convolved input
    const float* src;       // the input product's rows; y of channel c at src[t * src_stride + y_col + c]
    int src_stride, y_col;
    const float* by;        // [W] or null: added to y before its activation
    const float* br;        // [W] bias of the recurrence gate
    const float* bi;        // [W] bias of the input gate
    const float* sp;        // [W] C * softplus(lam), made once when the model is built
    float* state;           // [slots][slot_stride], S in the first W values of a slot
    long long slot_stride;
    const int* slots;       // [requests]
    const int* reqs;        // [n][3] = (request, first row, rows)
    void* out;              // [T][W]
    int T, W, bs;
};

__device__ __forceinline__ float sigmoid32(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float gelu_tanh32(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// The same for a result that leaves as TO.  Where it is rounded to bfloat16: (1 + tanh x) / 2 = sigmoid(2 x), an exponential and a division instead of a
// tanh, whose sum with 1 loses what is left of it for negative x (largest error over -3 .. -1 9.4e-7 of the value, with tanh 1.3e-5; over 1 .. 3
// 1.3e-7 and 1.2e-7).  2,048 rows of 4,096 channels, the whole mixer: 287 us, with tanh 293.
template <typename TO> __device__ __forceinline__ float branch_gelu(float z) {
    if constexpr (sizeof(TO) == 2) return z / (1.0f + expf(-1.5957691216057308f * (z + 0.044715f * z * z * z)));
    else return gelu_tanh32(z);
}

// (a, b) of S <- a S + b from the gates' arguments and the convolved input
__device__ __forceinline__ void lru_values(float gr, float gi, float u, float spc, float* a, float* b) {
    const float log_a = -sigmoid32(gr) * spc, e = expm1f(log_a);
    const float strong = expf(log_a);          // (always: under a branch it costs more than it takes)
    *a = e > -0.5f ? 1.0f + e : strong;
    *b = sqrtf(fmaf(-e, e, -2.0f * e)) * (sigmoid32(gi) * u);
}

// The same for row t of channel c.
__device__ __forceinline__ void lru_step(const LruParams& p, size_t gate_at, int t, int c, float brc, float bic, float spc, float* a,
                                         float* b) {
    lru_values(p.gates[gate_at] + brc, p.gates[gate_at + p.bs] + bic, p.u[(size_t)t * p.W + c], spc, a, b);
}

template <typename TO>
__global__ void __launch_bounds__(LRU_THREADS)
rglru_scan_kernel(LruParams p) {
    pdl_launch();
    pdl_wait();
    const int c = blockIdx.x * LRU_THREADS + threadIdx.x;
    if (c >= p.W) return;
    const int req = p.reqs[blockIdx.y * 3 + 0], row0 = p.reqs[blockIdx.y * 3 + 1], n = p.reqs[blockIdx.y * 3 + 2];
    if (n <= 0) return;
    const int blk = c / p.bs, o = c - blk * p.bs;
    const float brc = p.br[c], bic = p.bi[c], spc = p.sp[c];
    float* st = p.state + (size_t)p.slots[req] * p.slot_stride + c;
    float S = *st;
    TO* out = (TO*)p.out;
    const float yb = p.by ? p.by[c] : 0.0f;
    const size_t gbase = ((size_t)blk * p.T) * (2 * p.bs) + o;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
        const int t = row0 + j;
        float a, b;
        lru_step(p, gbase + (size_t)t * (2 * p.bs), t, c, brc, bic, spc, &a, &b);
        S = fmaf(a, S, b);
        out[(size_t)t * p.W + c] = from_float<TO>(S * branch_gelu<TO>(p.src[(size_t)t * p.src_stride + p.y_col + c] + yb));
    }
    *st = S;
}

// chunks: [n][4] = (request, first row, rows, 0); longs: [n][4] = (request, first row, rows, index of its first chunk).
// pq: [chunks][2][W] = (P, Q) of a chunk; after the walk, [chunk][0] is the state at the chunk's start.
__global__ void __launch_bounds__(LRU_THREADS)
rglru_chunk_sums_kernel(LruParams p, const int* __restrict__ chunks, float* __restrict__ pq, float2* __restrict__ ab) {
    pdl_launch();
    pdl_wait();
    const int c = blockIdx.x * LRU_THREADS + threadIdx.x;
    if (c >= p.W) return;
    const int ch = blockIdx.y;
    const int row0 = chunks[ch * 4 + 1], n = chunks[ch * 4 + 2];
    const int blk = c / p.bs, o = c - blk * p.bs;
    const float brc = p.br[c], bic = p.bi[c], spc = p.sp[c];
    const size_t gbase = ((size_t)blk * p.T) * (2 * p.bs) + o;
    float P = 1.0f, Q = 0.0f;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
        const int t = row0 + j;
        float a, b;
        lru_step(p, gbase + (size_t)t * (2 * p.bs), t, c, brc, bic, spc, &a, &b);
        ab[(size_t)t * p.W + c] = make_float2(a, b);
        P *= a;
        Q = fmaf(a, Q, b);
    }
    pq[((size_t)ch * 2 + 0) * p.W + c] = P;
    pq[((size_t)ch * 2 + 1) * p.W + c] = Q;
}

__global__ void __launch_bounds__(LRU_THREADS)
rglru_chunk_walk_kernel(LruParams p, const int* __restrict__ longs, int chunk_rows, float* __restrict__ pq) {
    pdl_launch();
    pdl_wait();
    const int c = blockIdx.x * LRU_THREADS + threadIdx.x;
    if (c >= p.W) return;
    const int req = longs[blockIdx.y * 4 + 0], n = longs[blockIdx.y * 4 + 2], first = longs[blockIdx.y * 4 + 3];
    const int n_chunks = (n + chunk_rows - 1) / chunk_rows;
    float* st = p.state + (size_t)p.slots[req] * p.slot_stride + c;
    float S = *st;
    // eight chunks' (P, Q) fetched at a time: the loads do not wait for the walk, only the eight products do
    for (int k0 = 0; k0 < n_chunks; k0 += 8) {
        float P[8], Q[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const size_t at = ((size_t)(first + min(k0 + j, n_chunks - 1)) * 2) * p.W + c;
            P[j] = pq[at];
            Q[j] = pq[at + p.W];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < n_chunks) {
                pq[((size_t)(first + k0 + j) * 2) * p.W + c] = S;
                S = fmaf(P[j], S, Q[j]);
            }
        }
    }
    *st = S;
}

template <typename TO>
__global__ void __launch_bounds__(LRU_THREADS)
rglru_chunk_out_kernel(LruParams p, const int* __restrict__ chunks, const float* __restrict__ pq, const float2* __restrict__ ab) {
    pdl_launch();
    pdl_wait();
    const int c = blockIdx.x * LRU_THREADS + threadIdx.x;
    if (c >= p.W) return;
    const int ch = blockIdx.y;
    const int row0 = chunks[ch * 4 + 1], n = chunks[ch * 4 + 2];
    TO* out = (TO*)p.out;
    const float yb = p.by ? p.by[c] : 0.0f;
    float S = pq[((size_t)ch * 2) * p.W + c];
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
        const int t = row0 + j;
        const float2 s = ab[(size_t)t * p.W + c];              // (a, b) of the row, as the first walk formed them
        S = fmaf(s.x, S, s.y);
        out[(size_t)t * p.W + c] = from_float<TO>(S * branch_gelu<TO>(p.src[(size_t)t * p.src_stride + p.y_col + c] + yb));
    }
}

// Both walks with two channels a thread, LRU_BATCH rows' values asked for before the first is used: 8-byte loads of gates, input and
// branch, 16 bytes of (a, b) for both channels.  For even sizes and rows on 8-byte boundaries.  The first is bound by its special
// functions, the second by bytes.  (The whole mixer of 4,096 channels over 2,048 rows: 333 us with a channel a thread, 301 so.)
constexpr int LRU_BATCH = 4;
__global__ void __launch_bounds__(LRU_THREADS)
rglru_chunk_sums_vec2_kernel(LruParams p, const int* __restrict__ chunks, float* __restrict__ pq, float4* __restrict__ ab, int folded) {
    if (!folded) pdl_launch();
    pdl_wait();
    const int c = (blockIdx.x * LRU_THREADS + threadIdx.x) * 2;
    if (c >= p.W) return;
    const int ch = blockIdx.y;
    const int row0 = chunks[ch * 4 + 1], n = chunks[ch * 4 + 2];
    const int blk = c / p.bs, o = c - blk * p.bs;
    const float2 br = *reinterpret_cast<const float2*>(p.br + c), bi = *reinterpret_cast<const float2*>(p.bi + c), sp = *reinterpret_cast<const float2*>(p.sp + c);
    const float* gates = p.gates + ((size_t)blk * p.T + row0) * (2 * p.bs) + o;
    const float* u = p.u + (size_t)row0 * p.W + c;
    float4* to = ab + ((size_t)row0 * p.W + c) / 2;
    float2 P = make_float2(1.0f, 1.0f), Q = make_float2(0.0f, 0.0f);
    for (int j0 = 0; j0 < n; j0 += LRU_BATCH) {
        float2 gr[LRU_BATCH], gi[LRU_BATCH], x[LRU_BATCH];
#pragma unroll
        for (int k = 0; k < LRU_BATCH; ++k) {
            const int j = min(j0 + k, n - 1);
            gr[k] = *reinterpret_cast<const float2*>(gates + (size_t)j * (2 * p.bs));
            gi[k] = *reinterpret_cast<const float2*>(gates + (size_t)j * (2 * p.bs) + p.bs);
            x[k] = *reinterpret_cast<const float2*>(u + (size_t)j * p.W);
        }
#pragma unroll
        for (int k = 0; k < LRU_BATCH; ++k) {
            if (j0 + k >= n) break;
            float4 v;
            lru_values(gr[k].x + br.x, gi[k].x + bi.x, x[k].x, sp.x, &v.x, &v.y);
            lru_values(gr[k].y + br.y, gi[k].y + bi.y, x[k].y, sp.y, &v.z, &v.w);
            to[(size_t)(j0 + k) * (p.W / 2)] = v;
            P.x *= v.x; P.y *= v.z;
            Q.x = fmaf(v.x, Q.x, v.y); Q.y = fmaf(v.z, Q.y, v.w);
        }
    }
    // (the kernel behind is the outputs', as many blocks as these: let in earlier, they crowd on the SMs that are free first.  2,560 channels, 64 chunks 61 us,
    // so 52)
    if (folded) pdl_launch();
    if (folded && (ch == 0 || chunks[(ch - 1) * 4] != chunks[ch * 4])) {       // a request's first chunk: its state, and the state behind the chunk
        const float* st = p.state + (size_t)p.slots[chunks[ch * 4]] * p.slot_stride + c;
        const float2 S = make_float2(st[0], st[1]);
        Q = make_float2(fmaf(P.x, S.x, Q.x), fmaf(P.y, S.y, Q.y));
        P = S;
    }
    *reinterpret_cast<float2*>(pq + ((size_t)ch * 2 + 0) * p.W + c) = P;
    *reinterpret_cast<float2*>(pq + ((size_t)ch * 2 + 1) * p.W + c) = Q;
}

// FOLDED: the walk over a request's chunks is made by every chunk for itself, up to its own start, and the last one leaves the state.  For steps of
// up to LRU_FOLDED chunks and few requests: a kernel less, for reads from the second-level cache that grow with the square of the chunks.  The recurrence's
// kernels, us, apart and folded: one request of 1,024 channels 64 chunks 36.4 and 31.7, 128 65.7 and 48.7; 2,560 channels 54.3 and 51.6, 96.6 and 98.5; 4,096 75.5
// and 69.4, 139 and 128; 8,192 131 and 122, 241 and 233; sixteen requests of eight chunks 52.3 and 43.6, 86.4 and 91.6, 125 and 119, 223 and 222.
constexpr int LRU_FOLDED = 128, LRU_FOLDED_LONGS = 16;
template <typename TO, bool FOLDED>
__global__ void __launch_bounds__(LRU_THREADS)
rglru_chunk_out_vec2_kernel(LruParams p, const int* __restrict__ chunks, const int* __restrict__ longs, int n_long, int chunk_rows,
                            const float* __restrict__ pq, const float4* __restrict__ ab) {
    pdl_launch();
    pdl_wait();
    const int c = (blockIdx.x * LRU_THREADS + threadIdx.x) * 2;
    if (c >= p.W) return;
    const int ch = blockIdx.y;
    const int row0 = chunks[ch * 4 + 1], n = chunks[ch * 4 + 2];
    const float2 yb = p.by ? *reinterpret_cast<const float2*>(p.by + c) : make_float2(0.0f, 0.0f);
    const float* y = p.src + (size_t)row0 * p.src_stride + p.y_col + c;
    const float4* from = ab + ((size_t)row0 * p.W + c) / 2;
    TO* out = (TO*)p.out + (size_t)row0 * p.W + c;
    float2 S;
    if constexpr (FOLDED) {
        bool last = false;
        int first = ch;
        for (int l = 0; l < n_long; ++l) {
            const int from_ch = longs[l * 4 + 3], count = (longs[l * 4 + 2] + chunk_rows - 1) / chunk_rows;
            if (ch >= from_ch && ch < from_ch + count) { first = from_ch; last = ch == from_ch + count - 1; }
        }
        const float* q = pq + (size_t)first * 2 * p.W + c;
        S = *reinterpret_cast<const float2*>(q + (ch == first ? 0 : p.W));
        for (int k0 = first + 1; k0 < ch; k0 += 8) {
            float2 P[8], Q[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float* at = pq + (size_t)min(k0 + k, ch) * 2 * p.W + c;
                P[k] = *reinterpret_cast<const float2*>(at);
                Q[k] = *reinterpret_cast<const float2*>(at + p.W);
            }
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (k0 + k < ch) S = make_float2(fmaf(P[k].x, S.x, Q[k].x), fmaf(P[k].y, S.y, Q[k].y));
        }
        if (last) {                                            // (nobody else looks at the slot any more)
            const float2 P = *reinterpret_cast<const float2*>(pq + (size_t)ch * 2 * p.W + c), Q = *reinterpret_cast<const float2*>(pq + ((size_t)ch * 2 + 1) * p.W + c);
            float* st = p.state + (size_t)p.slots[chunks[ch * 4]] * p.slot_stride + c;
            st[0] = ch == first ? Q.x : fmaf(P.x, S.x, Q.x);
            st[1] = ch == first ? Q.y : fmaf(P.y, S.y, Q.y);
        }
    } else {
        S = *reinterpret_cast<const float2*>(pq + ((size_t)ch * 2) * p.W + c);
    }
    for (int j0 = 0; j0 < n; j0 += LRU_BATCH) {
        float4 v[LRU_BATCH];
        float2 z[LRU_BATCH];
#pragma unroll
        for (int k = 0; k < LRU_BATCH; ++k) {
            const int j = min(j0 + k, n - 1);
            v[k] = from[(size_t)j * (p.W / 2)];
            z[k] = *reinterpret_cast<const float2*>(y + (size_t)j * p.src_stride);
        }
#pragma unroll
        for (int k = 0; k < LRU_BATCH; ++k) {
            if (j0 + k >= n) break;
            S.x = fmaf(v[k].x, S.x, v[k].y); S.y = fmaf(v[k].z, S.y, v[k].w);
            const float o0 = S.x * branch_gelu<TO>(z[k].x + yb.x), o1 = S.y * branch_gelu<TO>(z[k].y + yb.y);
            TO* d = out + (size_t)(j0 + k) * p.W;
            if constexpr (sizeof(TO) == 4) *reinterpret_cast<float2*>(d) = make_float2(o0, o1);
            else *reinterpret_cast<__nv_bfloat162*>(d) = __floats2bfloat162_rn(o0, o1);
        }
    }
}

// u [T][W] float -> x2 [blocks][T][2 bs] bfloat16: per part the rounding of u to bfloat16 followed by the rounding of what
// the first rounding left out.  A product of x2 with a part's matrix repeated twice along its inner size is then the
// product of u itself to sixteen bits, with float accumulation, on the tensor cores.
__global__ void rglru_split_kernel(const float* __restrict__ u, __nv_bfloat16* __restrict__ x2, int T, int W, int bs) {
    pdl_launch();
    pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)T * W) return;
    const int t = (int)(idx / W), c = (int)(idx - (size_t)t * W);
    const int blk = c / bs, o = c - blk * bs;
    const float v = u[idx];
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __nv_bfloat16 lo = __float2bfloat16_rn(v - __bfloat162float(hi));
    __nv_bfloat16* dst = x2 + ((size_t)blk * T + t) * (2 * bs);
    dst[o] = hi;
    dst[bs + o] = lo;
}

// The same, four channels a thread (parts of a multiple of 4 channels): 16 bytes in, two stores of 8 bytes out.
__global__ void rglru_split_vec4_kernel(const float* __restrict__ u, __nv_bfloat16* __restrict__ x2, int T, int W, int bs) {
    pdl_launch();
    pdl_wait();
    const size_t idx = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (idx >= (size_t)T * W) return;
    const int t = (int)(idx / W), c = (int)(idx - (size_t)t * W);
    const int blk = c / bs, o = c - blk * bs;
    const float4 v = *reinterpret_cast<const float4*>(u + idx);
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
    const float2 f0 = __bfloat1622float2(h0), f1 = __bfloat1622float2(h1);
    const __nv_bfloat162 l0 = __floats2bfloat162_rn(v.x - f0.x, v.y - f0.y), l1 = __floats2bfloat162_rn(v.z - f1.x, v.w - f1.y);
    __nv_bfloat16* dst = x2 + ((size_t)blk * T + t) * (2 * bs);
    uint2 hi, lo;
    hi.x = *reinterpret_cast<const unsigned*>(&h0); hi.y = *reinterpret_cast<const unsigned*>(&h1);
    lo.x = *reinterpret_cast<const unsigned*>(&l0); lo.y = *reinterpret_cast<const unsigned*>(&l1);
    *reinterpret_cast<uint2*>(dst + o) = hi;
    *reinterpret_cast<uint2*>(dst + bs + o) = lo;
}

// sp[c] = scale * softplus(lam[c]), float: log(1 + e^x), as x for large x.
template <typename TW>
__global__ void rglru_softplus_kernel(const TW* __restrict__ lam, float scale, float* __restrict__ sp, int W) {
    pdl_launch();
    pdl_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= W) return;
    const float x = to_float(lam[c]);
    sp[c] = scale * (x > 20.0f ? x : log1pf(expf(x)));
}

}  // namespace bg

using namespace bg;

static int lru_params(LruParams* p, const float* gates, const float* u, const float* src, int src_stride, int y_col, const float* by,
                      const float* br,
                      const float* bi, const float* sp, float* state, long long slot_stride, const int* slots, void* out, int T,
                      int W, int blocks) {
    if (W <= 0 || blocks <= 0 || W % blocks != 0 || T <= 0) return BG_ERR_SHAPE;
    p->gates = gates; p->u = u; p->src = src; p->src_stride = src_stride; p->y_col = y_col; p->by = by; p->br = br; p->bi = bi; p->sp = sp;
    p->state = state; p->slot_stride = slot_stride; p->slots = slots; p->reqs = nullptr; p->out = out; p->T = T; p->W = W;
    p->bs = W / blocks;
    return BG_OK;
}

// The requests `reqs` [n_req][3] of a step walked row by row.
extern "C" int bg_rglru_scan(const float* gates, const float* u, const float* src, int src_stride, int y_col, const float* by,
                             const float* br,
                             const float* bi, const float* sp, float* state, long long slot_stride, const int* slots,
                             const int* reqs, int n_req, void* out, int out_dtype, int T, int W, int blocks, cudaStream_t stream) {
    if (n_req <= 0 || T <= 0) return BG_OK;
    if (n_req > 65535) return BG_ERR_SHAPE;
    LruParams p;
    const int rc = lru_params(&p, gates, u, src, src_stride, y_col, by, br, bi, sp, state, slot_stride, slots, out, T, W, blocks);
    if (rc != BG_OK) return rc;
    p.reqs = reqs;
    const dim3 grid((W + LRU_THREADS - 1) / LRU_THREADS, n_req);
    BG_DISPATCH_DTYPE(out_dtype, TO, launch(rglru_scan_kernel<TO>, grid, dim3(LRU_THREADS), 0, stream, p));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// The long requests of a step in chunks of `chunk_rows` rows: chunks [n_chunks][4], longs [n_long][4], pq float
// [n_chunks][2][W] and ab float [T][W][2] of the caller's.
extern "C" int bg_rglru_scan_chunked(const float* gates, const float* u, const float* src, int src_stride, int y_col,
                                     const float* by, const float* br, const float* bi, const float* sp, float* state, long long slot_stride,
                                     const int* slots, const int* chunks, int n_chunks, const int* longs, int n_long,
                                     int chunk_rows, float* pq, float* ab, void* out, int out_dtype, int T, int W, int blocks,
                                     int* launched, cudaStream_t stream) {
    if (launched) *launched = 0;
    if (n_chunks <= 0 || n_long <= 0 || T <= 0) return BG_OK;
    if (n_chunks > 65535 || n_long > 65535 || chunk_rows <= 0) return BG_ERR_SHAPE;
    LruParams p;
    const int rc = lru_params(&p, gates, u, src, src_stride, y_col, by, br, bi, sp, state, slot_stride, slots, out, T, W, blocks);
    if (rc != BG_OK) return rc;
    const unsigned bx = (W + LRU_THREADS - 1) / LRU_THREADS, bx2 = (W / 2 + LRU_THREADS - 1) / LRU_THREADS;
    auto on = [](const void* q, unsigned bytes) { return (uintptr_t)q % bytes == 0; };
    const bool two = p.bs % 2 == 0 && src_stride % 2 == 0 && y_col % 2 == 0 && on(gates, 8) && on(u, 8) && on(src, 8) && on(br, 8) && on(bi, 8) &&
                     on(sp, 8) && on(pq, 8) && on(ab, 16) && on(out, 8) && (!by || on(by, 8));
    if (launched) *launched = 3;
    if (two) {
        const bool folded = n_chunks <= LRU_FOLDED && n_long <= LRU_FOLDED_LONGS;
        launch(rglru_chunk_sums_vec2_kernel, dim3(bx2, n_chunks), dim3(LRU_THREADS), 0, stream, p, chunks, pq, (float4*)ab, folded ? 1 : 0);
        BG_LAUNCH_CHECK();
        if (folded) {
            if (launched) *launched = 2;
            BG_DISPATCH_DTYPE(out_dtype, TO, launch(rglru_chunk_out_vec2_kernel<TO, true>, dim3(bx2, n_chunks), dim3(LRU_THREADS), 0, stream, p, chunks, longs,
                                                    n_long, chunk_rows, (const float*)pq, (const float4*)ab));
            BG_LAUNCH_CHECK();
            return BG_OK;
        }
    } else {
        launch(rglru_chunk_sums_kernel, dim3(bx, n_chunks), dim3(LRU_THREADS), 0, stream, p, chunks, pq, (float2*)ab);
        BG_LAUNCH_CHECK();
    }
    launch(rglru_chunk_walk_kernel, dim3(bx, n_long), dim3(LRU_THREADS), 0, stream, p, longs, chunk_rows, pq);
    BG_LAUNCH_CHECK();
    if (two)
        BG_DISPATCH_DTYPE(out_dtype, TO, launch(rglru_chunk_out_vec2_kernel<TO, false>, dim3(bx2, n_chunks), dim3(LRU_THREADS), 0, stream, p, chunks, longs, n_long,
                                                chunk_rows, (const float*)pq, (const float4*)ab));
    else
        BG_DISPATCH_DTYPE(out_dtype, TO, launch(rglru_chunk_out_kernel<TO>, dim3(bx, n_chunks), dim3(LRU_THREADS), 0, stream, p, chunks,
                                                (const float*)pq, (const float2*)ab));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_rglru_split(const float* u, void* x2, int T, int W, int blocks, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (W <= 0 || blocks <= 0 || W % blocks != 0) return BG_ERR_SHAPE;
    const size_t n = (size_t)T * W;
    if ((W / blocks) % 4 == 0 && (uintptr_t)u % 16 == 0 && (uintptr_t)x2 % 8 == 0) {
        launch(rglru_split_vec4_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, stream, u, (__nv_bfloat16*)x2, T, W,
               W / blocks);
        BG_LAUNCH_CHECK();
        return BG_OK;
    }
    launch(rglru_split_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, u, (__nv_bfloat16*)x2, T, W, W / blocks);
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_rglru_softplus(const void* lam, int lam_dtype, float scale, float* sp, int W, cudaStream_t stream) {
    if (W <= 0) return BG_OK;
    BG_DISPATCH_DTYPE(lam_dtype, TW, launch(rglru_softplus_kernel<TW>, dim3((W + 255) / 256), dim3(256), 0, stream, (const TW*)lam,
                                            scale, sp, W));
    BG_LAUNCH_CHECK();
    return BG_OK;
}
