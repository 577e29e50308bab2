// Linear attention with a decay per key channel.  Per head, with q, k, a (n features) and v (nv features) of a token:
//     S <- diag(a) S + k v^T        (S is n x nv, float, one per request and head, zero when the request starts)
//     o  = S^T q
// and the head's result o is RMS-normed by itself with a weight vector shared by the heads, and multiplied by silu of a
// further product of the token's row when there is a gate.  Two ways from the product's rows to q, k and a:
//   FORGET   a = l + (1 - l) sigmoid(f + b), k = 1 - a: the forget gate also decides what is written (l in [0, 1] per channel)
//   DECAY    k a product of its own, a = sigmoid(z)^(1/tau) with z = W r + b for a short row r of the token
// with q = silu(product) or product times a constant.  The state is carried from step to step in a slot of the cache
// manager's slab.  Everything behind the products is float: gates, decays, state, readout, norm.
//
//   gla_walk_kernel      a block per (head, request) walks the request's tokens in turn with the whole state in registers,
//                        and norms and gates the head's result itself.  Steps of single tokens and short portions.
//   gla_walk_mem_kernel  the same with the state in global memory: heads of any size.
//   gla_chunk_*          long portions in chunks of GC tokens: per chunk the gates, the decayed queries and keys and the scores
//                        of the chunk's own tokens; the chunks' decayed sums of k v^T; a pass over the chunks that turns them
//                        into the states at the chunks' starts; the chunks' outputs, normed and gated.
//
// A decay between two tokens is a PRODUCT of the a's between them; it is never formed as a quotient of products from a
// chunk's start (which underflow) nor from logarithms (a may be 0).  A chunk is cut into blocks of GB tokens, and a product
// over tokens of several blocks is split at the blocks' borders: (from the key's token to its block's end) x (whole blocks
// between) x (from the start of the query's block to its token), each a running product of numbers in [0, 1].
#include <type_traits>

#include "common.cuh"
#include "chunk_scan.cuh"
#include "chunk_tc.cuh"

namespace bg {

// (sigmoid(z), sigmoid(-z)) from one exponential of a number that is not positive
__device__ __forceinline__ float2 gla_sigmoids(float z) {
    const float e = expf(-fabsf(z)), big = __frcp_rn(1.0f + e), small = e * big;
    return z >= 0.0f ? make_float2(big, small) : make_float2(small, big);
}
__device__ __forceinline__ float gla_silu(float z) { return z * gla_sigmoids(z).x; }
// sigmoid(z)^p through the logarithm log sigmoid(z) = min(z, 0) - log1p(e^-|z|)
__device__ __forceinline__ float gla_root(float z, float p) { return expf(p * (fminf(z, 0.0f) - log1pf(expf(-fabsf(z))))); }

struct GlaParams {
    const float* src; int src_stride;           // rows of the product(s)
    int q_col, k_col, v_col, g_col;             // k_col: the forget gate's (FORGET) or the key's columns; g_col < 0: no gate
    int forget;                                 // FORGET or DECAY
    int q_silu; float q_scale;
    const float* bias;                          // [H n] b
    const float* lower;                         // FORGET: [H n] l
    int r_col, rank;                            // DECAY: the short row's columns
    const float* wa;                            // DECAY: [H n][rank]
    float power;                                // DECAY: 1 / tau
    const float* norm_w; float eps;             // [nv]
    float* state; size_t slot_stride;           // slab [slots][>= H n nv]
    const int* slots;
    const int* reqs;                            // [n_req][3] = (request, first row, rows)
    void* out; int out_float;                   // [T][H nv]
    int H, n, nv;
    // chunks
    const int* chunks;                          // [n_chunks][4] = (request, first row, rows, -)
    const int* longs;                           // [n_long][4]   = (request, first row, rows, first chunk)
    float* qd; float* kd;                       // [T][H np] queries times the decay from the chunk's start, keys times that to its end
    float* scores;                              // [n_chunks][H][GC (t)][GC (j)], j <= t (and noughts up to the end of t's block)
    float* work;                                // [n_chunks][H][np nvp]
    float* decay;                               // [n_chunks][H][n] the chunk's whole decay
    int np, nvp;                                // n, nv rounded up to multiples of 4
    int vec, vec_qk;                            // rows of values, and of q and k, lie on 16-byte boundaries
};

__device__ __forceinline__ float gla_query(const GlaParams& p, float raw) { return p.q_silu ? gla_silu(raw) * p.q_scale : raw * p.q_scale; }
// FORGET: (a, k) from the gate's product z of channel c
__device__ __forceinline__ void gla_forget(const GlaParams& p, int c, float raw, float* a, float* k) {
    const float l = p.lower[c];
    const float2 g = gla_sigmoids(raw + p.bias[c]);
    *a = fmaf(1.0f - l, g.x, l);
    *k = (1.0f - l) * g.y;
}
// DECAY: a of channel c from the token's row
__device__ __forceinline__ float gla_decay(const GlaParams& p, int c, const float* row) {
    float z = p.bias[c];
    const float* w = p.wa + (size_t)c * p.rank;
    for (int r = 0; r < p.rank; ++r) z = fmaf(w[r], row[p.r_col + r], z);
    return gla_root(z, p.power);
}
__device__ __forceinline__ void gla_store(const GlaParams& p, size_t at, float v) {
    if (p.out_float) ((float*)p.out)[at] = v; else ((__nv_bfloat16*)p.out)[at] = __float2bfloat16_rn(v);
}
__device__ __forceinline__ float gla_gate(const GlaParams& p, const float* row, int h, int c) {
    return p.g_col >= 0 ? gla_silu(row[p.g_col + h * p.nv + c]) : 1.0f;
}

// q, k, a (n values each) and v (nv) of a token's head into shared memory.
__device__ __forceinline__ void gla_load_token(const GlaParams& p, const float* row, int h, float* qs, float* ks, float* as, float* vs) {
    const int n = p.n, nv = p.nv, tid = threadIdx.x;
    for (int i = tid; i < n; i += blockDim.x) {
        const int c = h * n + i;
        qs[i] = gla_query(p, row[p.q_col + c]);
        if (p.forget) gla_forget(p, c, row[p.k_col + c], as + i, ks + i);
        else { ks[i] = row[p.k_col + c]; as[i] = gla_decay(p, c, row); }
    }
    for (int i = tid; i < nv; i += blockDim.x) vs[i] = row[p.v_col + h * nv + i];
}

// The state in registers: thread (slice, column) holds the R rows from slice R on of its column; `slices` threads share a
// column (blockDim.x / nv of them, whole columns only, slices R >= n).  q, k and a are padded with zeros up to slices R, so
// that a thread reads them four at a time and without a condition.
template <int R>
__global__ void __launch_bounds__(512) gla_walk_kernel(GlaParams p, int slices) {
    extern __shared__ __align__(16) float ga_s[];
    __shared__ float scratch[32];
    const int n = p.n, nv = p.nv, np = slices * R;
    float* qs = ga_s;                      // [np]
    float* ks = qs + np;                   // [np]
    float* as = ks + np;                   // [np]
    float* vs = as + np;                   // [nv]
    float* red = vs + nv;                  // [slices][nv]
    pdl_launch();
    const int h = blockIdx.x, r = blockIdx.y;
    const int req = p.reqs[r * 3 + 0], row0 = p.reqs[r * 3 + 1], rows = p.reqs[r * 3 + 2];
    const int tid = threadIdx.x;
    const int sl = tid / nv, c = tid - sl * nv, i0 = sl * R;
    const bool own = sl < slices && rows > 0;
    // the state was left by an earlier step: it is on its way while the product ahead still runs
    float* st = p.state + (size_t)p.slots[req] * p.slot_stride + (size_t)h * n * nv + (size_t)i0 * nv + c;
    float S[R];
#pragma unroll
    for (int k = 0; k < R; ++k) S[k] = (own && i0 + k < n) ? st[(size_t)k * nv] : 0.0f;
    for (int i = n + tid; i < np; i += blockDim.x) { qs[i] = 0.0f; ks[i] = 0.0f; as[i] = 0.0f; }
    pdl_wait();
    if (rows <= 0) return;
    for (int t = 0; t < rows; ++t) {
        const float* row = p.src + (size_t)(row0 + t) * p.src_stride;
        __syncthreads();
        gla_load_token(p, row, h, qs, ks, as, vs);
        __syncthreads();
        if (own) {
            const float v = vs[c];
            float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
            for (int k = 0; k < R; k += 4) {
                const float4 a = *reinterpret_cast<const float4*>(as + i0 + k), kk = *reinterpret_cast<const float4*>(ks + i0 + k);
                const float4 q = *reinterpret_cast<const float4*>(qs + i0 + k);
                S[k + 0] = fmaf(a.x, S[k + 0], kk.x * v); acc0 = fmaf(S[k + 0], q.x, acc0);
                S[k + 1] = fmaf(a.y, S[k + 1], kk.y * v); acc1 = fmaf(S[k + 1], q.y, acc1);
                S[k + 2] = fmaf(a.z, S[k + 2], kk.z * v); acc0 = fmaf(S[k + 2], q.z, acc0);
                S[k + 3] = fmaf(a.w, S[k + 3], kk.w * v); acc1 = fmaf(S[k + 3], q.w, acc1);
            }
            red[sl * nv + c] = acc0 + acc1;
        }
        __syncthreads();
        float o = 0.0f;
        if (tid < nv) for (int q = 0; q < slices; ++q) o += red[q * nv + tid];
        const float ss = block_sum(o * o, scratch);
        if (tid < nv)
            gla_store(p, (size_t)(row0 + t) * p.H * nv + (size_t)h * nv + tid,
                      o * (1.0f / sqrtf(ss / (float)nv + p.eps)) * p.norm_w[tid] * gla_gate(p, row, h, tid));
    }
    if (own) {
        int stride = nv;
        asm volatile("" : "+r"(stride));   // the addresses are worked out again here: kept from the loads, they would fill the registers
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (i0 + k < n) st[(size_t)k * stride] = S[k];
    }
}

// The same with the state in place: a thread walks whole columns.
__global__ void __launch_bounds__(256) gla_walk_mem_kernel(GlaParams p) {
    extern __shared__ float ga_s[];
    __shared__ float scratch[32];
    const int n = p.n, nv = p.nv;
    float* qs = ga_s; float* ks = qs + n; float* as = ks + n; float* vs = as + n; float* os = vs + nv;
    pdl_launch();
    pdl_wait();
    const int h = blockIdx.x, r = blockIdx.y, tid = threadIdx.x;
    const int req = p.reqs[r * 3 + 0], row0 = p.reqs[r * 3 + 1], rows = p.reqs[r * 3 + 2];
    if (rows <= 0) return;
    float* st = p.state + (size_t)p.slots[req] * p.slot_stride + (size_t)h * n * nv;
    for (int t = 0; t < rows; ++t) {
        const float* row = p.src + (size_t)(row0 + t) * p.src_stride;
        __syncthreads();
        gla_load_token(p, row, h, qs, ks, as, vs);
        __syncthreads();
        float ss = 0.0f;
        for (int c = tid; c < nv; c += blockDim.x) {
            const float v = vs[c];
            float acc = 0.0f;
            for (int i = 0; i < n; ++i) {
                const float s = fmaf(as[i], st[(size_t)i * nv + c], ks[i] * v);
                st[(size_t)i * nv + c] = s;
                acc = fmaf(s, qs[i], acc);
            }
            os[c] = acc;
            ss += acc * acc;
        }
        const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)nv + p.eps);
        for (int c = tid; c < nv; c += blockDim.x)
            gla_store(p, (size_t)(row0 + t) * p.H * nv + (size_t)h * nv + c, os[c] * inv * p.norm_w[c] * gla_gate(p, row, h, c));
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Chunks of GC tokens in blocks of GB.  Rows of a chunk beyond its last token have q = k = v = 0 and a = 1.
constexpr int GC = 64, GB = 16, GNB = GC / GB;
constexpr int GCP = GC + 4;               // row stride of the score tile
constexpr int GPT = 64;                   // value columns of a block
constexpr int GC_BATCH = 8;               // loads (of 16 bytes: half as many) a thread has on their way at a time
constexpr int GLA_RANK = 16;              // features of the short row taken at a time
constexpr int GLA_WS = GLA_RANK + 4;      // row stride of the decay's matrix in shared memory

// The (row, column) of element tid + k * blockDim.x of a [rows][w] tile, stepped without a division per element.
struct GlaWalk {
    int j, i, dj, di, w;
    __device__ __forceinline__ GlaWalk(int w_) : w(w_) {
        j = (int)threadIdx.x / w; i = (int)threadIdx.x - j * w;
        dj = (int)blockDim.x / w; di = (int)blockDim.x - dj * w;
    }
    __device__ __forceinline__ void next() { i += di; j += dj; if (i >= w) { i -= w; ++j; } }
};

__device__ __forceinline__ void gla_async16(float* dst, const float* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void gla_async_wait() { asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory"); }

// `n_rows` rows of `w` floats into a tile of row stride `ld` whose rows are `wp` wide (a multiple of 4); what lies beyond `rows`
// and `w` becomes nought.  16 bytes at a time when `vec` (rows on 16-byte boundaries, w a multiple of 4).
__device__ __forceinline__ void gla_rows(float* dst, int ld, const float* src, size_t stride, int n_rows, int rows, int w, int wp, int vec) {
    if (vec) {
        const int w4 = wp >> 2;
        for (int idx = threadIdx.x; idx < n_rows * w4; idx += blockDim.x) {
            const int r = idx / w4, c = (idx - r * w4) * 4;
            if (r < rows && c < w) gla_async16(dst + (size_t)r * ld + c, src + (size_t)r * stride + c);
            else *reinterpret_cast<float4*>(dst + (size_t)r * ld + c) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    } else {
        for (int idx = threadIdx.x; idx < n_rows * wp; idx += blockDim.x) {
            const int r = idx / wp, c = idx - r * wp;
            dst[(size_t)r * ld + c] = (r < rows && c < w) ? src[(size_t)r * stride + c] : 0.0f;
        }
    }
}

// Scores inside the blocks of a chunk: a warp takes four neighbouring keys of a block and walks the queries from the first of them to the
// block's end; a lane carries its channels of k_j times the decay from j to t along as t moves on, so that a score is one sum per query.
// L lanes share a key's channels, four neighbours at a time (M such groups a lane), and carry KEYS keys: the four keys read the same rows of
// queries and decays, once.
template <int L, int M>
__device__ __forceinline__ void gla_block_scores(const float* Qs, const float* Ks, const float* As, float* sc, int np, int ld) {
    constexpr int KEYS = L / 8;                      // of a lane's group; 32 / L groups a warp
    const int lane = threadIdx.x & 31, l = lane & (L - 1), warp = threadIdx.x >> 5;
    const int b0 = (warp >> 2) * GB, first = (warp & 3) * 4;                        // the warp's block and its first key in it
    const int key = (lane / L) * KEYS;                                              // the lane's first key of the four
    float w[KEYS][4 * M];
#pragma unroll
    for (int e = 0; e < KEYS; ++e)
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int i = 4 * (l + L * m);
            const float4 x = i < np ? *reinterpret_cast<const float4*>(Ks + (b0 + first + key + e) * ld + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            w[e][4 * m] = x.x; w[e][4 * m + 1] = x.y; w[e][4 * m + 2] = x.z; w[e][4 * m + 3] = x.w;
        }
    float* out = sc + b0 * GC + b0 + first;
    if (lane < 4)
        for (int t = 0; t < first; ++t) out[t * GC + lane] = 0.0f;                  // queries in front of the keys
    auto step = [&](int d, auto head) {                                             // query first + d; `head`: not all four keys are behind it
        const int row = (b0 + first + d) * ld;
        float acc[KEYS];
#pragma unroll
        for (int e = 0; e < KEYS; ++e) acc[e] = 0.0f;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const int i = 4 * (l + L * m);                                          // (a lane beyond the channels carries noughts)
            const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float4 a4 = i < np ? *reinterpret_cast<const float4*>(As + row + i) : none;
            const float4 q4 = i < np ? *reinterpret_cast<const float4*>(Qs + row + i) : none;
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int e = 0; e < KEYS; ++e) {
                const bool on = !decltype(head)::value || d > key + e;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    w[e][4 * m + c] *= on ? a[c] : 1.0f;
                    acc[e] = fmaf(w[e][4 * m + c], q[c], acc[e]);
                }
            }
        }
        // KEYS sums over L lanes: the lanes halve the keys between them first, so that each carries one, then add up the rest
        float v;
        if constexpr (KEYS == 4) {
            const bool hi = lane & 16;
            float x = (hi ? acc[2] : acc[0]) + __shfl_xor_sync(0xffffffffu, hi ? acc[0] : acc[2], 16);
            float y = (hi ? acc[3] : acc[1]) + __shfl_xor_sync(0xffffffffu, hi ? acc[1] : acc[3], 16);
            const bool odd = lane & 8;
            v = (odd ? y : x) + __shfl_xor_sync(0xffffffffu, odd ? x : y, 8);
        } else if constexpr (KEYS == 2) {
            const bool odd = lane & 8;
            v = (odd ? acc[1] : acc[0]) + __shfl_xor_sync(0xffffffffu, odd ? acc[0] : acc[1], 8);
        } else {
            v = acc[0];
        }
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        const int mine = lane >> 3;                                                 // (every eight lanes end with one key's)
        if ((lane & 7) == 0) out[(first + d) * GC + mine] = !decltype(head)::value || d >= mine ? v : 0.0f;
    };
#pragma unroll
    for (int d = 0; d < 4; ++d) step(d, std::true_type{});
#pragma unroll 2
    for (int d = 4; d < GB - first; ++d) step(d, std::false_type{});
}

// Gates, decayed queries and keys and scores of a chunk's head.  Bound by instructions (4,200 a warp, issued in 65 % of the cycles), which the
// scores inside the blocks, those across, the decays' small product and roots, and the loads share about evenly; two blocks an SM by the three
// tiles of 64 rows.  Sixteen warps each (with eight, 46 %); the raw rows by asynchronous copies, the decay's matrix through shared memory
// (read by a thread per channel it took 16 x 32 sectors a warp), scores of four keys a warp at once: 135 -> 105 us for 2,048 rows of 32
// heads of 128 features, rank 16 (32 -> 20 us of that the decays).  Storing the results in front of the last products lost 6 us (64 registers).
constexpr int GP_THREADS = 512;           // a warp per four keys of the chunk

__global__ void __launch_bounds__(GP_THREADS, 2) gla_chunk_prep_kernel(GlaParams p) {
    extern __shared__ __align__(16) float gc_s[];
    const int n = p.n, np = p.np, ld = np + 8;
    float* Qs = gc_s;                          // [GC][ld]
    float* Ks = Qs + (size_t)GC * ld;          // [GC][ld]
    float* As = Ks + (size_t)GC * ld;          // [GC][ld]
    float* F = As + (size_t)GC * ld;           // [GNB][np] a block's whole decay
    const int h = blockIdx.x, ch = blockIdx.y, tid = threadIdx.x;
    float* Rs = F;                             // [GC][GLA_RANK] the short rows, a few features at a time
    float* Ws = As;                            // [np][GLA_WS] the head's rows of the decay's matrix, its first features
    if (!p.forget) {
        const bool vec = p.rank % 4 == 0 && (uintptr_t)p.wa % 16 == 0;
        for (int idx = tid; idx < np * (GLA_RANK / 4); idx += GP_THREADS) {
            const int i = idx / (GLA_RANK / 4), r = idx % (GLA_RANK / 4) * 4;
            const float* w = p.wa + (size_t)(h * n + (i < n ? i : 0)) * p.rank + r;
            float* dst = Ws + i * GLA_WS + r;
            if (vec && i < n && r < p.rank) gla_async16(dst, w);
            else
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[e] = i < n && r + e < p.rank ? w[e] : 0.0f;
        }
    }
    pdl_launch();
    pdl_wait();
    const int row0 = p.chunks[ch * 4 + 1], rows = p.chunks[ch * 4 + 2];
    const float* src = p.src + (size_t)row0 * p.src_stride;
    // the raw rows into the tiles, all on their way at once; then a thread makes queries, keys and decays of what it asked for itself
    const int n4 = np >> 2;
    for (GlaWalk w(n4); w.j < GC; w.next()) {
        const int i = 4 * w.i, at = w.j * ld + i;
        const float* r = src + (size_t)w.j * p.src_stride + h * n + i;
        if (p.vec_qk && w.j < rows) {
            gla_async16(Qs + at, r + p.q_col);
            gla_async16(Ks + at, r + p.k_col);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool on = w.j < rows && i + e < n;
                Qs[at + e] = on ? r[p.q_col + e] : 0.0f;
                Ks[at + e] = on ? r[p.k_col + e] : 0.0f;
            }
        }
    }
    if (!p.forget)
        for (int idx = tid; idx < GC * GLA_RANK; idx += GP_THREADS) {
            const int t = idx / GLA_RANK, r = idx % GLA_RANK;
            Rs[idx] = (t < rows && r < p.rank) ? src[(size_t)t * p.src_stride + p.r_col + r] : 0.0f;
        }
    gla_async_wait();
    if (p.forget || p.q_silu || p.q_scale != 1.0f)
        for (GlaWalk w(n4); w.j < rows; w.next()) {
            const int at = w.j * ld + 4 * w.i;
            float4 q = *reinterpret_cast<const float4*>(Qs + at);
            q = make_float4(gla_query(p, q.x), gla_query(p, q.y), gla_query(p, q.z), gla_query(p, q.w));
            *reinterpret_cast<float4*>(Qs + at) = q;
            if (p.forget) {
                const float4 y = *reinterpret_cast<const float4*>(Ks + at);
                const float ys[4] = {y.x, y.y, y.z, y.w};
                float a[4], k[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    a[e] = 1.0f; k[e] = 0.0f;
                    if (4 * w.i + e < n) gla_forget(p, h * n + 4 * w.i + e, ys[e], &a[e], &k[e]);
                }
                *reinterpret_cast<float4*>(Ks + at) = make_float4(k[0], k[1], k[2], k[3]);
                *reinterpret_cast<float4*>(As + at) = make_float4(a[0], a[1], a[2], a[3]);
            }
        }
    if (p.forget) {
        for (int idx = tid; idx < (GC - rows) * n4; idx += GP_THREADS)
            *reinterpret_cast<float4*>(As + (rows + idx / n4) * ld + idx % n4 * 4) = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    } else {
        // z = W r + b, a thread per channel and every lanes-th token
        const int lanes = GP_THREADS / np;                                   // threads that share a channel (np is 256 at most)
        const int i = tid % np, part = tid / np;
        const int c = h * n + (i < n ? i : 0);
        const float b = i < n ? p.bias[c] : 0.0f;
        for (int r0 = 0; r0 < p.rank; r0 += GLA_RANK) {
            if (r0 > 0) {
                __syncthreads();
                for (int idx = tid; idx < GC * GLA_RANK; idx += GP_THREADS) {
                    const int t = idx / GLA_RANK, r = idx % GLA_RANK;
                    Rs[idx] = (t < rows && r0 + r < p.rank) ? src[(size_t)t * p.src_stride + p.r_col + r0 + r] : 0.0f;
                }
            }
            __syncthreads();
            float w[GLA_RANK];
            if (r0 == 0) {
#pragma unroll
                for (int r = 0; r < GLA_RANK; r += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(Ws + i * GLA_WS + r);
                    w[r] = v.x; w[r + 1] = v.y; w[r + 2] = v.z; w[r + 3] = v.w;
                }
                __syncthreads();                                             // (the decays take the matrix's place)
            } else {
#pragma unroll
                for (int r = 0; r < GLA_RANK; ++r) w[r] = (i < n && r0 + r < p.rank) ? p.wa[(size_t)c * p.rank + r0 + r] : 0.0f;
            }
            const bool last = r0 + GLA_RANK >= p.rank;
            for (int t = part < lanes ? part : GC; t < GC; t += lanes) {
                float z = r0 == 0 ? b : As[t * ld + i];
#pragma unroll
                for (int r = 0; r < GLA_RANK; r += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(Rs + t * GLA_RANK + r);
                    z = fmaf(w[r], v.x, z); z = fmaf(w[r + 1], v.y, z); z = fmaf(w[r + 2], v.z, z); z = fmaf(w[r + 3], v.w, z);
                }
                if (last) z = (t < rows && i < n) ? gla_root(z, p.power) : 1.0f;
                As[t * ld + i] = z;
            }
        }
    }
    __syncthreads();
    float* sc = p.scores + ((size_t)ch * p.H + h) * GC * GC;
    if (np <= 32) gla_block_scores<8, 1>(Qs, Ks, As, sc, np, ld);
    else if (np <= 64) gla_block_scores<16, 1>(Qs, Ks, As, sc, np, ld);
    else if (np <= 128) gla_block_scores<32, 1>(Qs, Ks, As, sc, np, ld);
    else gla_block_scores<32, 2>(Qs, Ks, As, sc, np, ld);
    __syncthreads();
    // q_t times the decay from its block's start up to t, k_j times the decay behind j to its block's end, the block's decay: a thread per
    // block and channel, whose values are read before any is written
    for (int e = tid; e < GNB * np; e += GP_THREADS) {
        const int b = e / np, i = e - b * np;
        const int at = b * GB * ld + i;
        float a[GB], x[GB], w = 1.0f;
#pragma unroll
        for (int t = 0; t < GB; ++t) { a[t] = As[at + t * ld]; x[t] = Qs[at + t * ld]; }
#pragma unroll
        for (int t = 0; t < GB; ++t) { w *= a[t]; Qs[at + t * ld] = x[t] * w; }
        F[e] = w;
#pragma unroll
        for (int t = 0; t < GB; ++t) x[t] = Ks[at + t * ld];
        w = 1.0f;
#pragma unroll
        for (int t = GB - 1; t >= 0; --t) { Ks[at + t * ld] = x[t] * w; w *= a[t]; }
    }
    __syncthreads();
    // scores across blocks: a tile of 4 x 4 (queries tq + 4 u, keys jq + 4 v of their blocks) per four threads, which share the
    // channels; a warp's tiles are those of one pair of blocks
    constexpr int PAIRS = GNB * (GNB - 1) / 2, PER_PAIR = (GB / 4) * (GB / 4);
    if (tid < PAIRS * PER_PAIR * 4) {
        const int part = tid & 3, tile = tid >> 2;
        const int pair = tile / PER_PAIR, in = tile % PER_PAIR;
        int I = 1, J = pair;                                                         // pairs (1,0) (2,0) (2,1) (3,0) ...
        while (J >= I) { J -= I; ++I; }
        const int t0 = I * GB + in / (GB / 4), j0 = J * GB + in % (GB / 4);
        float acc[4][4] = {};
        auto products = [&](auto apart) {                                            // `apart`: whole blocks lie between the two
            for (int i = 4 * part; i < np; i += 16) {
                float4 k[4], q[4];
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    k[v] = *reinterpret_cast<const float4*>(Ks + (j0 + 4 * v) * ld + i);
                    q[v] = *reinterpret_cast<const float4*>(Qs + (t0 + 4 * v) * ld + i);
                }
                if constexpr (decltype(apart)::value) {
                    for (int b = J + 1; b < I; ++b) {
                        const float4 f = *reinterpret_cast<const float4*>(F + b * np + i);
#pragma unroll
                        for (int v = 0; v < 4; ++v) { k[v].x *= f.x; k[v].y *= f.y; k[v].z *= f.z; k[v].w *= f.w; }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v)
                        acc[u][v] = fmaf(q[u].x, k[v].x, fmaf(q[u].y, k[v].y, fmaf(q[u].z, k[v].z, fmaf(q[u].w, k[v].w, acc[u][v]))));
            }
        };
        if (I - J > 1) products(std::true_type{}); else products(std::false_type{});
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                acc[u][v] += __shfl_xor_sync(0xffffffffu, acc[u][v], 1);
                acc[u][v] += __shfl_xor_sync(0xffffffffu, acc[u][v], 2);
                if (u == part) sc[(t0 + 4 * u) * GC + j0 + 4 * v] = acc[u][v];
            }
    }
    // the queries with the whole blocks in front of theirs, the keys with those behind
    for (int idx = tid; idx < rows * n4; idx += GP_THREADS) {
        const int t = idx / n4, i = (idx - t * n4) * 4, b = t / GB;
        float4 q = *reinterpret_cast<const float4*>(Qs + t * ld + i), k = *reinterpret_cast<const float4*>(Ks + t * ld + i);
#pragma unroll
        for (int m = 0; m < GNB; ++m) {
            const float4 f = *reinterpret_cast<const float4*>(F + m * np + i);
            if (m < b) { q.x *= f.x; q.y *= f.y; q.z *= f.z; q.w *= f.w; }
            if (m > b) { k.x *= f.x; k.y *= f.y; k.z *= f.z; k.w *= f.w; }
        }
        const size_t at = ((size_t)(row0 + t) * p.H + h) * np + i;
        *reinterpret_cast<float4*>(p.qd + at) = q;
        *reinterpret_cast<float4*>(p.kd + at) = k;
    }
    for (int i = tid; i < n; i += blockDim.x) {
        float w = F[i];
#pragma unroll
        for (int m = 1; m < GNB; ++m) w *= F[m * np + i];
        p.decay[((size_t)ch * p.H + h) * n + i] = w;
    }
}

__global__ void __launch_bounds__(256) gla_chunk_sum_kernel(GlaParams p) {
    extern __shared__ __align__(16) float gc_s[];
    const int np = p.np, nvp = p.nvp;
    float* Ks = gc_s;                          // [GC][np]
    float* Vs = Ks + (size_t)GC * np;          // [GC][GPT]
    pdl_launch();
    pdl_wait();
    const int h = blockIdx.x, ch = blockIdx.y, c_first = blockIdx.z * GPT, tid = threadIdx.x;
    const int wp = min(GPT, nvp - c_first), w = min(GPT, p.nv - c_first);
    const int row0 = p.chunks[ch * 4 + 1], rows = p.chunks[ch * 4 + 2];
    gla_rows(Ks, np, p.kd + ((size_t)row0 * p.H + h) * np, (size_t)p.H * np, GC, rows, np, np, 1);
    gla_rows(Vs, GPT, p.src + (size_t)row0 * p.src_stride + p.v_col + h * p.nv + c_first, p.src_stride, GC, rows, w, wp, p.vec);
    gla_async_wait();
    __syncthreads();
    float* A = p.work + ((size_t)ch * p.H + h) * np * nvp + c_first;
    const int tp = wp >> 2, tn = (np + 7) >> 3;
    for (int tile = tid; tile < tn * tp; tile += blockDim.x) {
        const int i0 = (tile / tp) * 8, c0 = (tile % tp) * 4;
        const bool two = i0 + 4 < np;
        float acc[8][4] = {};
#pragma unroll 4
        for (int j = 0; j < GC; ++j) {
            const float4 v = *reinterpret_cast<const float4*>(Vs + j * GPT + c0);
            const float4 k0 = *reinterpret_cast<const float4*>(Ks + (size_t)j * np + i0);
            const float4 k1 = two ? *reinterpret_cast<const float4*>(Ks + (size_t)j * np + i0 + 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float k[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                acc[u][0] = fmaf(k[u], v.x, acc[u][0]); acc[u][1] = fmaf(k[u], v.y, acc[u][1]);
                acc[u][2] = fmaf(k[u], v.z, acc[u][2]); acc[u][3] = fmaf(k[u], v.w, acc[u][3]);
            }
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u < np) *reinterpret_cast<float4*>(A + (size_t)(i0 + u) * nvp + c0) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
    }
}

// A thread per element of the state walks its request's chunks: the chunk's sum is replaced by the state at its start, the
// slot gets the state behind the last.  Eight chunks' sums and decays are fetched at a time.
__global__ void __launch_bounds__(256) gla_chunk_scan_kernel(GlaParams p) {
    pdl_launch();
    pdl_wait();
    const int e = blockIdx.x * blockDim.x + threadIdx.x, h = blockIdx.y, l = blockIdx.z;
    const int sz = p.n * p.nv;
    if (e >= sz) return;
    const int req = p.longs[l * 4 + 0], rows = p.longs[l * 4 + 2], c0 = p.longs[l * 4 + 3];
    const int n_chunks = (rows + GC - 1) / GC;
    const int i = e / p.nv, c_at = e - i * p.nv;
    float* st = p.state + (size_t)p.slots[req] * p.slot_stride + (size_t)h * sz + e;
    const size_t pad = (size_t)p.np * p.nvp;
    float* a0 = p.work + ((size_t)c0 * p.H + h) * pad + (size_t)i * p.nvp + c_at;
    const float* d0 = p.decay + ((size_t)c0 * p.H + h) * p.n + i;
    const size_t step = (size_t)p.H * pad, dstep = (size_t)p.H * p.n;
    float S = *st;
    for (int c = 0; c < n_chunks; c += GC_BATCH) {
        float A[GC_BATCH], D[GC_BATCH];
#pragma unroll
        for (int u = 0; u < GC_BATCH; ++u) {
            A[u] = c + u < n_chunks ? a0[(size_t)(c + u) * step] : 0.0f;
            D[u] = c + u < n_chunks ? d0[(size_t)(c + u) * dstep] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < GC_BATCH; ++u)
            if (c + u < n_chunks) {
                a0[(size_t)(c + u) * step] = S;
                S = fmaf(D[u], S, A[u]);
            }
    }
    *st = S;
}

// The same, four values a thread (heads of whole 16-byte pieces).
__global__ void __launch_bounds__(CS_THREADS) gla_chunk_scan4_kernel(GlaParams p) {
    pdl_launch();
    pdl_wait();
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) * 4, h = blockIdx.y, l = blockIdx.z, sz = p.n * p.nv;
    if (e >= sz) return;
    const int req = p.longs[l * 4 + 0], rows = p.longs[l * 4 + 2], c0 = p.longs[l * 4 + 3];
    const int i = e / p.nv;
    float4* st = reinterpret_cast<float4*>(p.state + (size_t)p.slots[req] * p.slot_stride + (size_t)h * sz + e);
    const size_t pad = (size_t)p.np * p.nvp, dstep = (size_t)p.H * p.n;
    const float* d0 = p.decay + ((size_t)c0 * p.H + h) * p.n + i;
    *st = chunk_walk4(p.work + ((size_t)c0 * p.H + h) * pad + (size_t)i * p.nvp + (e - i * p.nv), (size_t)p.H * pad, (rows + GC - 1) / GC,
                      [&](int c) { return d0[(size_t)c * dstep]; }, *st);
}
static void gla_scan(const GlaParams& p, int n_long, cudaStream_t stream) {
    const int sz = p.n * p.nv;
    if (p.nv % 4 == 0 && p.slot_stride % 4 == 0 && (uintptr_t)p.state % 16 == 0)          // (the scratch lies on 16 bytes)
        launch(gla_chunk_scan4_kernel, dim3((sz / 4 + CS_THREADS - 1) / CS_THREADS, p.H, n_long), dim3(CS_THREADS), 0, stream, p);
    else launch(gla_chunk_scan_kernel, dim3((sz + 255) / 256, p.H, n_long), dim3(256), 0, stream, p);
}

// The token that a thread's row u (of eight) stands for: a warp holds sixteen tokens, a half of it four neighbours and the four
// eight further on, so that the two halves' reads of a tile of rows fall on different banks.
__device__ __forceinline__ int gla_token(int u) {
    return ((int)threadIdx.x >> 5) * 16 + (((int)threadIdx.x >> 4) & 1) * 4 + (u & 3) + (u >> 2) * 8;
}

// acc[u][v] += sum over k of a[token of row u][k] b[k][v], k in steps of 4 up to `k_end`
__device__ __forceinline__ void gla_product(float (&acc)[8][4], const float* a, int lda, const float* b, int k_end) {
#pragma unroll 1
    for (int k = 0; k < k_end; k += 4) {
        float4 bb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) bb[i] = *reinterpret_cast<const float4*>(b + (size_t)(k + i) * GPT);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const float4 aa = *reinterpret_cast<const float4*>(a + gla_token(u) * lda + k);
            const float ak[4] = {aa.x, aa.y, aa.z, aa.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[u][0] = fmaf(ak[i], bb[i].x, acc[u][0]); acc[u][1] = fmaf(ak[i], bb[i].y, acc[u][1]);
                acc[u][2] = fmaf(ak[i], bb[i].z, acc[u][2]); acc[u][3] = fmaf(ak[i], bb[i].w, acc[u][3]);
            }
        }
    }
}

// o of GPT columns of a head in a chunk, its norm and gate.  The blocks of a head's columns form a cluster along z (of 1, 2, 4 or
// 8: those beyond the columns only take part in its barriers) and add up their rows' sums of squares in one another's shared
// memory.
__global__ void __launch_bounds__(128) gla_chunk_out_kernel(GlaParams p) {
    extern __shared__ __align__(16) float gc_s[];
    __shared__ float ssq[8][GC];               // [rank in the cluster][token]
    const int np = p.np, nvp = p.nvp, ldq = np + 4;
    float* Qs = gc_s;                          // [GC][np + 4]
    float* Ss = Qs + (size_t)GC * ldq;         // [np][GPT]
    float* Vs = Ss + (size_t)np * GPT;         // [GC][GPT]
    float* Ws = Vs + (size_t)GC * GPT;         // [GC (t)][GCP] scores
    const int h = blockIdx.x, ch = blockIdx.y, rank = blockIdx.z, n_rank = gridDim.z, c_first = rank * GPT, tid = threadIdx.x;
    const int wp = max(0, min(GPT, nvp - c_first)), w = max(0, min(GPT, p.nv - c_first));
    if (n_rank > 1) cluster_arrive_relaxed();  // waited for before the first store to a peer: every peer runs by then
    pdl_launch();
    pdl_wait();
    const int row0 = p.chunks[ch * 4 + 1], rows = p.chunks[ch * 4 + 2];
    const float* src = p.src + (size_t)row0 * p.src_stride;
    gla_rows(Qs, ldq, p.qd + ((size_t)row0 * p.H + h) * np, (size_t)p.H * np, GC, rows, np, np, 1);
    gla_rows(Ss, GPT, p.work + ((size_t)ch * p.H + h) * np * nvp + c_first, nvp, np, np, wp, wp, 1);
    gla_rows(Ws, GCP, p.scores + ((size_t)ch * p.H + h) * GC * GC, GC, GC, GC, GC, GC, 1);
    gla_rows(Vs, GPT, src + p.v_col + h * p.nv + c_first, p.src_stride, GC, rows, w, wp, p.vec);
    gla_async_wait();
    __syncthreads();
    const int t0 = (tid >> 5) * 16, c0 = (tid & 15) * 4;        // the warp's first token
    float acc[8][4] = {};
    if (t0 < rows && c0 < wp) {
        gla_product(acc, Qs, ldq, Ss + c0, np);
        gla_product(acc, Ws, GCP, Vs + c0, t0 + GB);            // (a warp's tokens are one block of GB)
    }
    if (n_rank > 1) { __syncwarp(); cluster_wait(); }
    // (columns beyond the head's own are noughts: the values and the state hold noughts there)
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        float s = acc[u][0] * acc[u][0] + acc[u][1] * acc[u][1] + acc[u][2] * acc[u][2] + acc[u][3] * acc[u][3];
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((tid & 15) == 0) {
            const int t = gla_token(u);
            if (n_rank == 1) ssq[0][t] = s;
            else for (int q = 0; q < n_rank; ++q) st_cluster(peer_addr((unsigned)__cvta_generic_to_shared(&ssq[rank][t]), (unsigned)q), s);
        }
    }
    __syncwarp();
    if (n_rank > 1) cluster_sync_all(); else __syncthreads();
    if (c0 >= w) return;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const int t = gla_token(u);
        if (t >= rows) continue;
        float total = 0.0f;
        for (int q = 0; q < n_rank; ++q) total += ssq[q][t];
        const float inv = 1.0f / sqrtf(total / (float)p.nv + p.eps);
        const float* row = src + (size_t)t * p.src_stride;
        const size_t at = (size_t)(row0 + t) * p.H * p.nv + (size_t)h * p.nv + c_first + c0;
#pragma unroll
        for (int v = 0; v < 4; ++v)
            if (c0 + v < w)
                gla_store(p, at + v, acc[u][v] * inv * p.norm_w[c_first + c0 + v] * gla_gate(p, row, h, c_first + c0 + v));
    }
}

// The chunks' outputs on the tensor cores, from operands in three bfloat16 parts (chunk_tc.cuh).  A CTA holds a whole head, so its norm
// needs no cluster.  2,048 tokens of 16 heads of 128 x 128, the whole chunked pass: 240 -> 158 us.  Left as floats for the
// measurement, the outputs are off by 2.04e-7 of 64 bits (2.07e-7 on the float units; 64 x 64 2.02e-7 and 2.06e-7, 96 x 96 3.46e-7 and 3.48e-7).
struct GlaTc {
    static constexpr bool SCORES = false;
    struct Shared { int unused; };
    GlaParams p;
    int n, nv, nv_ld;
    unsigned* status;
    int gate16;                                 // the gate's rows lie on 16-byte boundaries
    __device__ const float* state(int h, int ch) const { return p.work + ((size_t)ch * p.H + h) * n * nv; }
    struct Chunk {
        const GlaTc& r;
        int h, ch, row0, rows;
        __device__ Chunk(const GlaTc& r_, int h_, int ch_, Shared&) : r(r_), h(h_), ch(ch_) {
            row0 = r.p.chunks[ch * 4 + 1]; rows = r.p.chunks[ch * 4 + 2];
        }
        __device__ void begin() {}
        __device__ float4 made(const float* x, int t, int i) const {         // of the prepared queries or keys
            return t < rows ? *reinterpret_cast<const float4*>(x + ((size_t)(row0 + t) * r.p.H + h) * r.n + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __device__ float4 value_raw(int j, int v) const {
            return j < rows ? *reinterpret_cast<const float4*>(r.p.src + (size_t)(row0 + j) * r.p.src_stride + r.p.v_col + h * r.nv + v)
                            : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        __device__ float4 out_value(const float4& x, int, int) const { return x; }
        __device__ float4 query_raw(int t, int i) const { return made(r.p.qd, t, i); }
        __device__ float4 query(const float4& x, int, int) const { return x; }
        __device__ float factor(int) const { return 1.0f; }
        __device__ void weight_raw(float (&x)[CT_WEIGHTS]) const {
            const float* sc = r.p.scores + ((size_t)ch * r.p.H + h) * GC * GC;
#pragma unroll
            for (int u = 0; u < CT_WEIGHTS; ++u) {
                const int idx = u * CT_THREADS + threadIdx.x, t = idx / GC, j = idx % GC;
                x[u] = j <= t && t < rows ? sc[idx] : 0.0f;
            }
        }
        template <typename W> __device__ void weights(const float (&x)[CT_WEIGHTS], W put) const {
#pragma unroll
            for (int u = 0; u < CT_WEIGHTS; ++u) {
                const int idx = u * CT_THREADS + threadIdx.x;
                put(idx / GC, idx % GC, x[u]);
            }
        }
        // the head's norm and gate: the 2^SV lanes of a row add up its squares
        __device__ float4 finish_raw(int t, int v) const {
            if (r.p.g_col < 0 || t >= rows) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            const float* g = r.p.src + (size_t)(row0 + t) * r.p.src_stride + r.p.g_col + h * r.nv + v;
            return r.gate16 ? *reinterpret_cast<const float4*>(g) : make_float4(g[0], g[1], g[2], g[3]);
        }
        template <int SV> __device__ void finish(int t, int v, const float4& y, const float4& gate) const {
            float total = y.x * y.x + y.y * y.y + y.z * y.z + y.w * y.w;
#pragma unroll
            for (int o = (1 << SV) / 2; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
            if (v >= r.nv || t >= rows) return;
            const float inv = 1.0f / sqrtf(total / (float)r.nv + r.p.eps);
            const float4 w = make_float4(r.p.norm_w[v], r.p.norm_w[v + 1], r.p.norm_w[v + 2], r.p.norm_w[v + 3]);
            float4 o = make_float4(y.x * inv * w.x, y.y * inv * w.y, y.z * inv * w.z, y.w * inv * w.w);
            if (r.p.g_col >= 0) o = make_float4(o.x * gla_silu(gate.x), o.y * gla_silu(gate.y), o.z * gla_silu(gate.z), o.w * gla_silu(gate.w));
            const __nv_bfloat162 a = __floats2bfloat162_rn(o.x, o.y), b = __floats2bfloat162_rn(o.z, o.w);
            *reinterpret_cast<uint2*>((__nv_bfloat16*)r.p.out + (size_t)(row0 + t) * r.p.H * r.nv + (size_t)h * r.nv + v) =
                make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
        }
    };
};

static size_t gla_prep_smem(int np, int rank) {
    const size_t tail = (size_t)GNB * np > (size_t)GC * GLA_RANK || rank == 0 ? (size_t)GNB * np : (size_t)GC * GLA_RANK;
    return ((size_t)3 * GC * (np + 8) + tail) * sizeof(float);
}
static size_t gla_sum_smem(int np) { return ((size_t)GC * np + (size_t)GC * GPT) * sizeof(float); }
static size_t gla_out_smem(int np) { return ((size_t)GC * (np + 4) + (size_t)np * GPT + (size_t)GC * GPT + (size_t)GC * GCP) * sizeof(float); }
constexpr size_t GLA_SMEM_MAX = 222 * 1024;

}  // namespace bg

using namespace bg;

// What all entries share, as one struct of plain fields that the host side fills by name.
struct GlaArgs {
    const float* src; long long src_stride;
    int q_col, k_col, v_col, g_col, forget, q_silu, r_col, rank;
    float q_scale, power, eps, pad;
    const float* bias; const float* lower; const float* wa; const float* norm_w;
    float* state; long long slot_stride; const int* slots;
    void* out; int out_dtype, H, n, nv;
};

// Bytes of what the host side mirrors field by field; it compares them when it loads the library.
extern "C" int bg_gla_bytes() { return (int)sizeof(GlaArgs); }

static int gla_params(GlaParams& p, const GlaArgs* a) {
    if (a->H <= 0 || a->n <= 0 || a->nv <= 0 || a->H > 65535 || (a->forget ? !a->lower : (!a->wa || a->rank < 1)) || !a->bias || !a->norm_w) return BG_ERR_SHAPE;
    if (a->out_dtype != BG_DTYPE_F32 && a->out_dtype != BG_DTYPE_BF16) return BG_ERR_DTYPE;
    p.src = a->src; p.src_stride = (int)a->src_stride; p.q_col = a->q_col; p.k_col = a->k_col; p.v_col = a->v_col; p.g_col = a->g_col;
    p.forget = a->forget; p.q_silu = a->q_silu; p.q_scale = a->q_scale; p.bias = a->bias; p.lower = a->lower; p.r_col = a->r_col;
    p.rank = a->rank; p.wa = a->wa; p.power = a->power; p.norm_w = a->norm_w; p.eps = a->eps; p.state = a->state;
    p.slot_stride = (size_t)a->slot_stride; p.slots = a->slots; p.reqs = nullptr; p.out = a->out; p.out_float = a->out_dtype == BG_DTYPE_F32;
    p.H = a->H; p.n = a->n; p.nv = a->nv; p.chunks = nullptr; p.longs = nullptr; p.work = nullptr; p.decay = nullptr; p.qd = nullptr; p.kd = nullptr; p.scores = nullptr;
    const bool rows16 = a->src_stride % 4 == 0 && (uintptr_t)a->src % 16 == 0;
    p.vec = rows16 && a->nv % 4 == 0 && a->v_col % 4 == 0;
    p.vec_qk = rows16 && a->n % 4 == 0 && a->q_col % 4 == 0 && a->k_col % 4 == 0;
    p.np = (a->n + 3) / 4 * 4; p.nvp = (a->nv + 3) / 4 * 4;
    return BG_OK;
}

extern "C" int bg_gla_walk(const GlaArgs* args, const int* reqs, int n_req, cudaStream_t stream) {
    if (n_req <= 0) return BG_OK;
    GlaParams p;
    const int rc = gla_params(p, args);
    if (rc != BG_OK) return rc;
    if (n_req > 65535) return BG_ERR_SHAPE;
    p.reqs = reqs;
    const dim3 grid(p.H, n_req);
    // whole columns per block of up to 512 threads, four to 64 rows of its column a thread
    if (p.nv <= 512) {
        int slices = 512 / p.nv, R = 4;
        while (R < 64 && slices * R < p.n) R *= 2;
        slices = (p.n + R - 1) / R < slices ? (p.n + R - 1) / R : slices;
        const int threads = (slices * p.nv + 31) / 32 * 32;
        const size_t smem = ((size_t)3 * slices * R + p.nv + (size_t)slices * p.nv) * sizeof(float);
        if (slices * R >= p.n && smem <= BG_SMEM_OPT_IN) {
            switch (R) {
                case 4: launch(gla_walk_kernel<4>, grid, dim3(threads), smem, stream, p, slices); break;
                case 8: launch(gla_walk_kernel<8>, grid, dim3(threads), smem, stream, p, slices); break;
                case 16: launch(gla_walk_kernel<16>, grid, dim3(threads), smem, stream, p, slices); break;
                case 32: launch(gla_walk_kernel<32>, grid, dim3(threads), smem, stream, p, slices); break;
                default: launch(gla_walk_kernel<64>, grid, dim3(threads), smem, stream, p, slices); break;
            }
            BG_LAUNCH_CHECK();
            return BG_OK;
        }
    }
    const size_t smem = ((size_t)3 * p.n + 2 * p.nv) * sizeof(float);
    if (smem > 200 * 1024) return BG_ERR_UNSUPPORTED;
    if (smem > BG_SMEM_OPT_IN) {
        cudaError_t e = cudaFuncSetAttribute(gla_walk_mem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    launch(gla_walk_mem_kernel, grid, dim3(256), smem, stream, p);
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// 0 when the chunked kernels take heads of n x nv values (their tiles fit in shared memory), else BG_ERR_UNSUPPORTED.
extern "C" int bg_gla_chunk_plan(int n, int nv, int* chunk) {
    if (n <= 0 || nv <= 0) return BG_ERR_SHAPE;
    const int np = (n + 3) / 4 * 4, nvp = (nv + 3) / 4 * 4;
    if (chunk) *chunk = GC;
    // (the blocks of a head's columns are a cluster of at most eight)
    return np <= 256 && nvp <= 8 * GPT && gla_prep_smem(np, 1) <= GLA_SMEM_MAX && gla_out_smem(np) <= GLA_SMEM_MAX ? BG_OK : BG_ERR_UNSUPPORTED;
}

// Requests of many rows: chunks [n_chunks][4] and longs [n_long][4] as in decay_attention.cu.  Scratch, float, np and nvp being n
// and nv rounded up to multiples of 4: qd and kd [T][H np], scores [n_chunks][H][64 * 64], work [n_chunks][H][np nvp], decay
// [n_chunks][H][n].
extern "C" int bg_gla_chunked(const GlaArgs* args, const int* chunks, int n_chunks, const int* longs, int n_long, float* qd, float* kd,
                              float* scores, float* work, float* decay, unsigned* status, cudaStream_t stream) {
    if (n_chunks <= 0 || n_long <= 0) return BG_OK;
    GlaParams p;
    const int rc = gla_params(p, args);
    if (rc != BG_OK) return rc;
    if (n_chunks > 65535 || n_long > 65535) return BG_ERR_SHAPE;
    if (bg_gla_chunk_plan(p.n, p.nv, nullptr) != BG_OK) return BG_ERR_UNSUPPORTED;
    if ((uintptr_t)qd % 16 || (uintptr_t)kd % 16 || (uintptr_t)scores % 16 || (uintptr_t)work % 16) return BG_ERR_ALIGN;
    p.chunks = chunks; p.longs = longs; p.qd = qd; p.kd = kd; p.scores = scores; p.work = work; p.decay = decay;
    const size_t s_prep = gla_prep_smem(p.np, p.rank), s_sum = gla_sum_smem(p.np), s_out = gla_out_smem(p.np);
    const unsigned tiles = (unsigned)((p.nvp + GPT - 1) / GPT);
    cudaError_t e = cudaSuccess;
    if (s_prep > BG_SMEM_OPT_IN) e = cudaFuncSetAttribute(gla_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_prep);
    if (e == cudaSuccess && s_sum > BG_SMEM_OPT_IN) e = cudaFuncSetAttribute(gla_chunk_sum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_sum);
    if (e == cudaSuccess && s_out > BG_SMEM_OPT_IN) e = cudaFuncSetAttribute(gla_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s_out);
    if (e != cudaSuccess) return (int)e;
    launch(gla_chunk_prep_kernel, dim3(p.H, n_chunks), dim3(GP_THREADS), s_prep, stream, p);
    BG_LAUNCH_CHECK();
    // (the float32 path, whose results leave as floats, uses no tensor cores; the sums that become the state stay on the float units, whose
    // error against 64 bits is the smaller: 1.20e-7 against 1.25e-7 for 2,048 rows of 16 heads of 128 x 128)
    if (!p.out_float && ct_takes(p.n, p.nv) && p.vec && (uintptr_t)p.out % 8 == 0) {
        GlaTc r;
        r.p = p; r.n = p.n; r.nv = r.nv_ld = p.nv; r.status = status; r.gate16 = p.g_col % 4 == 0;
        launch(gla_chunk_sum_kernel, dim3(p.H, n_chunks, tiles), dim3(256), s_sum, stream, p);
        BG_LAUNCH_CHECK();
        gla_scan(p, n_long, stream);
        BG_LAUNCH_CHECK();
        const int trc = ct_out(r, p.H, n_chunks, stream);
        if (trc != BG_OK) return trc;
        BG_LAUNCH_CHECK();
        return BG_OK;
    }
    launch(gla_chunk_sum_kernel, dim3(p.H, n_chunks, tiles), dim3(256), s_sum, stream, p);
    BG_LAUNCH_CHECK();
    gla_scan(p, n_long, stream);
    BG_LAUNCH_CHECK();
    const unsigned cluster = tiles <= 2 ? tiles : tiles <= 4 ? 4 : 8;
    launch_cluster(gla_chunk_out_kernel, dim3(p.H, n_chunks, cluster), dim3(128), s_out, stream, (int)cluster, p);
    BG_LAUNCH_CHECK();
    return BG_OK;
}
