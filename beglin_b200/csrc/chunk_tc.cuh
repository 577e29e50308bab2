// The float products of recurrences that run in chunks of 64 tokens, on the tensor cores: per head and chunk, with keys k_j (n
// features), values v_j (nv), queries q_t, weights P[t][j] of the chunk's own tokens and the state S [n][nv] at the chunk's start,
//     chunk_sum_tc_kernel   A[i][v] = sum_j k_j[i] v_j[v]
//     chunk_out_tc_kernel   o_t[v]  = f_t sum_i q_t[i] S[i][v] + sum_j P[t][j] v_j[v]
// What k, v, q, P and f are is the recurrence's business (the policy `R`, a kernel parameter).
//
// No precision is given up for it: every float operand is cut into three bfloat16 numbers, x = h + m + l exactly but for 2^-25 of x
// (each the rounding of what is left), and a product of two floats is the six products of parts that are not below 2^-24 of it.  The
// small parts are added up before any h h, so that their sums are not rounded at the size of the large ones, and the h h products go
// half to an accumulator of their own; both are float in tensor memory and meet once, at the end.
//
// A number without three parts (infinite, not a number, or within a rounding of the largest float) makes whatever it is multiplied with not a
// number.  Where floats would do the same or make an infinity of it, that is left so: the sums, the state, a row's own query and scores.
// A value must not: the product multiplies it with the weights of nought of the queries in front of it, too.  Such values go into the
// tile as nought and are added afterwards, by floats, to the outputs of their own token and those behind it.
//
// The values' features are the M side of both products (an operand stored [token][feature] or [i][feature] is read M-major), so a lane
// of tensor memory is a feature and results leave in rows of 128 bytes.  A CTA of 256 threads converts what it fetches into swizzled
// tiles, the first warp issues the MMAs, all wait; two CTAs share an SM (96 KB, half of tensor memory each), so that one converts while the
// other multiplies.
#pragma once

#include "float_parts.cuh"

namespace bg {

constexpr int CT = 64;                       // tokens of a chunk
constexpr int CT_THREADS = 256;
constexpr unsigned CT_COLS = 256;            // tensor memory of a CTA
constexpr unsigned CT_BLOCK = CT * 128;      // 64 rows x 64 features of one part, bytes
constexpr unsigned CT_TILE = 3 * 2 * CT_BLOCK;       // 64 rows x 128 features, three parts

struct CtShared {
    unsigned long long done;
    unsigned tmem;
    int failed;
    int odd;                                 // a value of the chunk has no three parts
};

// x = h + m + l
__device__ __forceinline__ void ct_split(float x, __nv_bfloat16& h, __nv_bfloat16& m, __nv_bfloat16& l) {
    h = __float2bfloat16_rn(x);
    const float r = x - __bfloat162float(h);
    m = __float2bfloat16_rn(r);
    l = __float2bfloat16_rn(r - __bfloat162float(m));
}
__device__ __forceinline__ bool ct_splits(float x) { return fabsf(x) <= 3.3895313e38f; }       // (the largest bfloat16 number)
// the byte of element (row, col) in a part of a tile of 64 rows: blocks of 64 columns, rows of 128 bytes, 128-byte swizzle
__device__ __forceinline__ unsigned ct_at(int row, int col) {
    return (unsigned)(col >> 6) * CT_BLOCK + (unsigned)row * 128 + ((unsigned)(((col >> 3) ^ row) & 7) << 4) + (unsigned)(col & 7) * 2;
}
// four neighbouring columns (of a multiple of four) into the three parts, `part` bytes apart; two values a conversion
__device__ __forceinline__ void ct_put4(unsigned char* tile, unsigned part, int row, int col, const float4& x) {
    unsigned char* d = tile + ct_at(row, col);
    unsigned p[3], q[3];
    gt_split(pair2(x.x, x.y), p[0], p[1], p[2]);
    gt_split(pair2(x.z, x.w), q[0], q[1], q[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(d + i * part) = make_uint2(p[i], q[i]);
}
__device__ __forceinline__ void ct_put1(unsigned char* tile, unsigned part, int row, int col, float x) {
    __nv_bfloat16 h, m, l;
    ct_split(x, h, m, l);
    unsigned char* d = tile + ct_at(row, col);
    *reinterpret_cast<__nv_bfloat16*>(d) = h;
    *reinterpret_cast<__nv_bfloat16*>(d + part) = m;
    *reinterpret_cast<__nv_bfloat16*>(d + 2 * part) = l;
}
// A tile of 64 rows x `width` columns (a multiple of 4, at most 2^SH pieces of four), 2^SH threads a row: `fetch(row, col)` gives four raw
// values, `make(raw, row, col)` what is stored.  All fetches of a thread are on their way together, where it can be under the products
// before.  What a tile costs is mostly the instructions that make its values (the split, silu), so the columns are a constant of the
// kernel: with a row's length as an argument the decayed attention of 12 heads took 115 us instead of 89 for 2,048 tokens.
template <int SH> constexpr int CT_PASSES = CT * (1 << SH) / CT_THREADS;
template <int SH, typename F>
__device__ __forceinline__ void ct_fetch(float4 (&raw)[8], int width, F fetch) {
    const int col = (threadIdx.x & ((1 << SH) - 1)) * 4, row = threadIdx.x >> SH;
    if (col >= width) return;
#pragma unroll
    for (int u = 0; u < CT_PASSES<SH>; ++u) raw[u] = fetch(row + u * (CT_THREADS >> SH), col);
}
template <int SH, typename M>
__device__ __forceinline__ void ct_put(unsigned char* tile, unsigned part, const float4 (&raw)[8], int width, M make) {
    const int col = (threadIdx.x & ((1 << SH) - 1)) * 4, row = threadIdx.x >> SH;
    if (col >= width) return;
#pragma unroll
    for (int u = 0; u < CT_PASSES<SH>; ++u) ct_put4(tile, part, row + u * (CT_THREADS >> SH), col, make(raw[u], row + u * (CT_THREADS >> SH), col));
}

// One product of split operands over `steps` times 16 of the inner size: the five products of small parts into D2, then Ah Bh, the first
// `split` steps into D1 and the others on top of the small ones.  (An accumulator cuts off what does not fit it instead of rounding, and
// every MMA on a large sum is one such cut, always towards nought: two accumulators halve their number.)  A_M: the left operand is
// stored [inner][M] (else [M][inner]); B_N: the right one is stored [inner][N] (else [N][inner]).  One elected lane.
template <bool A_M, bool B_N>
__device__ __forceinline__ void ct_mma(unsigned d1, unsigned d2, unsigned a, unsigned a_part, unsigned b, unsigned b_part, int steps, int split,
                                       unsigned idesc, bool first) {
    auto da = [&](int p, int ks) {
        return A_M ? smem_desc_sw128_nmajor(a + p * a_part + ks * 2048, CT_BLOCK, 1024)
                   : smem_desc_sw128(a + p * a_part + (ks >> 2) * CT_BLOCK + (ks & 3) * 32);
    };
    auto db = [&](int p, int ks) {
        return B_N ? smem_desc_sw128_nmajor(b + p * b_part + ks * 2048, CT_BLOCK, 1024)
                   : smem_desc_sw128(b + p * b_part + (ks >> 2) * CT_BLOCK + (ks & 3) * 32);
    };
#pragma unroll 1
    for (int ks = 0; ks < steps; ++ks) {
        const unsigned long long ah = da(0, ks), am = da(1, ks), al = da(2, ks), bh = db(0, ks), bm = db(1, ks), bl = db(2, ks);
        tc_mma(d2, al, bh, idesc, first && ks == 0 ? 0u : 1u);
        tc_mma(d2, ah, bl, idesc, 1u);
        tc_mma(d2, am, bm, idesc, 1u);
        tc_mma(d2, am, bh, idesc, 1u);
        tc_mma(d2, ah, bm, idesc, 1u);
    }
#pragma unroll 1
    for (int ks = 0; ks < steps; ++ks) tc_mma(ks < split ? d1 : d2, da(0, ks), db(0, ks), idesc, first && ks == 0 && split > 0 ? 0u : 1u);
}
__host__ __device__ constexpr unsigned ct_idesc(int n, bool a_m, bool b_n) { return instr_desc_bf16(128, n, b_n ? 1 : 0) | (a_m ? 1u << 15 : 0u); }

// Barrier and tensor memory; the kernel behind this one may come only once the columns are held.
__device__ __forceinline__ void ct_begin(CtShared& s) {
    if (threadIdx.x == 0) { mbar_init(&s.done, 1); s.failed = 0; s.odd = 0; mbar_init_fence(); }
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s.tmem)), "r"(CT_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();
}
__device__ __forceinline__ void ct_end(CtShared& s, unsigned* status) {
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s.tmem), "r"(CT_COLS) : "memory");
    if (threadIdx.x == 0 && s.failed && status) atomicOr(status, BG_STATUS_TIMEOUT);
}
// What the threads wrote to shared memory is there for the MMAs that thread 0 issues; `phase` counts the CTA's products.  Between the two
// calls the tiles belong to the products; all threads wait.
template <typename I>
__device__ __forceinline__ void ct_issue(CtShared& s, I issue) {
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        if (elect_one()) {
            issue();
            tc_commit(&s.done);
        }
        __syncwarp();
    }
}
__device__ __forceinline__ void ct_wait(CtShared& s, unsigned& phase) {
    if (!mbar_wait(&s.done, phase & 1, &s.failed)) s.failed = 1;
    ++phase;
    tc_fence_after();
}

// R: the policy.  R::Chunk c(r, h, ch, shared): a CTA's head and chunk; c.begin(): what else it makes for them, while the first fetches are on their
// way (by all threads, ends with a barrier if it writes); c.rows; c.key_raw / c.key, c.value_raw / c.value; r.n, r.nv; r.sum_out(h, ch): A of
// the head and chunk, [n][r.nv_ld].
// (SN, SV: 4 for up to 64 features of keys, of values, 5 for up to 128)
template <typename R, int SN, int SV>
__global__ void __launch_bounds__(CT_THREADS, 2) chunk_sum_tc_kernel(R r) {
    extern __shared__ unsigned char ct_raw[];
    __shared__ __align__(8) CtShared s;
    __shared__ typename R::Shared rs;
    unsigned char* vt = (unsigned char*)(((uintptr_t)ct_raw + 1023) & ~(uintptr_t)1023);       // values, then keys
    unsigned char* kt = vt + CT_TILE;
    constexpr unsigned part = 2 * CT_BLOCK;
    ct_begin(s);
    pdl_wait();
    typename R::Chunk c(r, blockIdx.x, blockIdx.y, rs);
    float4 raw[8], vals[8];
    ct_fetch<SN>(raw, r.n, [&](int j, int i) { return c.key_raw(j, i); });
    ct_fetch<SV>(vals, r.nv, [&](int j, int v) { return c.value_raw(j, v); });
    c.begin();
    c.sum_begin();
    ct_put<SN>(kt, part, raw, r.n, [&](const float4& x, int j, int i) { return c.key(x, j, i); });
    ct_put<SV>(vt, part, vals, r.nv, [&](const float4& x, int j, int v) { return c.value(x, j, v); });
    unsigned phase = 0;
    const unsigned d1 = s.tmem, d2 = s.tmem + 128;
    ct_issue(s, [&] { ct_mma<true, true>(d1, d2, smem_u32(vt), part, smem_u32(kt), part, CT / 16, CT / 32, ct_idesc(r.n, true, true), true); });
    ct_wait(s, phase);
    if (!s.failed) {
        float* A = r.sum_out(blockIdx.x, blockIdx.y);
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, v = (warp & 3) * 32 + lane;
        const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
        for (int i0 = (warp >> 2) * 16; i0 < r.n; i0 += 32) {
            unsigned a[16], b[16];
            gt_ld16(d1 + lanes + i0, a);
            gt_ld16(d2 + lanes + i0, b);
            tc_wait_ld();
            if (v < r.nv) {
#pragma unroll
                for (int e = 0; e < 16; ++e) A[(size_t)(i0 + e) * r.nv_ld + v] = __uint_as_float(a[e]) + __uint_as_float(b[e]);
            }
            if (r.nv & 31) __syncwarp();     // (a load of tensor memory is the whole warp's: lanes without a column wait for the others)
        }
    }
    ct_end(s, r.status);
}

// Further members of R::Chunk: c.query_raw / c.query; with R::SCORES the weights are scores of this kernel's own: c.score_key_raw /
// c.score_key, and c.weight(score, t, j) for j <= t; else c.weight_raw(x) fetches a thread's CT_WEIGHTS scores and c.weights(x, put) calls put(t, j, P)
// for every t, j < CT, over all threads; r.state(h, ch): S; c.factor(t); c.finish_raw(t, v): what the results in columns v .. v + 3 need from
// memory besides, c.finish(t, v, y, raw): their end, from the products' float4 y (lanes whose columns are there; t may be behind the rows).
//
// What a CTA waits for is hidden by the other one on its SM, not within it, so each phase's loads leave before the wait ahead of it.  Read at the
// end (the values once more, the gate) or in a chain (the scores under their decays), they took a third to a half of a CTA's life: 33,600
// cycles for Mamba-2, of which weights 7,300 and end 4,900, and 49,600 for the decay per channel, of which 21,200 were its norm and gate (2,048 tokens:
// 59 -> 50 us for 24 heads of 128 x 128, 107 -> 88 for 32).  What is left is latency: without its MMAs the kernel takes 49 us of 58, without the
// splits 50; loops stay rolled, since a CTA runs its 60 to 100 KB of straight code once.
constexpr int CT_WEIGHTS = CT * CT / CT_THREADS;
constexpr int CT_OUT_LD = 132;
template <typename R, int SN, int SV>
__global__ void __launch_bounds__(CT_THREADS, 2) chunk_out_tc_kernel(R r) {
    extern __shared__ unsigned char ct_raw[];
    __shared__ __align__(8) CtShared s;
    __shared__ typename R::Shared rs;
    unsigned char* qt = (unsigned char*)(((uintptr_t)ct_raw + 1023) & ~(uintptr_t)1023);       // queries, later the weights
    unsigned char* xt = qt + CT_TILE;                                                            // keys, halves of the state, values
    constexpr unsigned part = 2 * CT_BLOCK;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lanes = (unsigned)((warp & 3) * 32) << 16;
    ct_begin(s);
    pdl_wait();
    typename R::Chunk c(r, blockIdx.x, blockIdx.y, rs);
    const unsigned d = s.tmem, q_a = smem_u32(qt), x_a = smem_u32(xt);
    unsigned phase = 0;
    float4 raw[8];
    const float* S = r.state(blockIdx.x, blockIdx.y);
    auto state_fetch = [&](int i0) {
        ct_fetch<SV>(raw, r.nv, [&](int i, int v) {
            return i0 + i < r.n ? *reinterpret_cast<const float4*>(S + (size_t)(i0 + i) * r.nv_ld + v) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        });
    };
    auto value_fetch = [&] { ct_fetch<SV>(raw, r.nv, [&](int j, int v) { return c.value_raw(j, v); }); };
    float weight_raw[R::SCORES ? 1 : CT_WEIGHTS];
    ct_fetch<SN>(raw, r.n, [&](int t, int i) { return c.query_raw(t, i); });
    c.begin();
    ct_put<SN>(qt, part, raw, r.n, [&](const float4& x, int t, int i) { return c.query(x, t, i); });
    if constexpr (R::SCORES) {
        // S^T [key][query]: rows 64 to 127 of the left operand are whatever follows its tile and their results are not read
        ct_fetch<SN>(raw, r.n, [&](int j, int i) { return c.score_key_raw(j, i); });
        ct_put<SN>(xt, part, raw, r.n, [&](const float4& x, int j, int i) { return c.score_key(x, j, i); });
        ct_issue(s, [&] { ct_mma<false, false>(d, d + 64, x_a, part, q_a, part, r.n / 16, r.n / 32, ct_idesc(CT, false, false), true); });
        state_fetch(0);
        ct_wait(s, phase);                   // (they stay in tensor memory until the queries' tile is free for the weights)
    } else {
        state_fetch(0);
    }
#pragma unroll 1
    for (int i0 = 0; i0 < r.n; i0 += 64) {
        const int w = min(64, r.n - i0);
        ct_put<SV>(xt, part, raw, r.nv, [&](const float4& x, int, int) { return x; });
        ct_issue(s, [&] {
            ct_mma<true, false>(d + 128, d + 192, x_a, part, q_a + (i0 >> 6) * CT_BLOCK, part, w / 16, i0 > 0 ? 0 : r.n > 64 ? w / 16 : w / 32,
                                ct_idesc(CT, true, false), i0 == 0);
        });
        if (i0 + 64 < r.n) state_fetch(i0 + 64);
        else {
            value_fetch();
            if constexpr (!R::SCORES) c.weight_raw(weight_raw);
        }
        ct_wait(s, phase);
    }
    if constexpr (R::SCORES) {
        if ((warp & 3) < 2) {                // lane: key (warp & 3) 32 + lane
            const int j = (warp & 3) * 32 + lane;
            for (int t0 = (warp >> 2) * 32; t0 < (warp >> 2) * 32 + 32; t0 += 16) {
                unsigned a[16], b[16];
                gt_ld16(d + lanes + t0, a);
                gt_ld16(d + 64 + lanes + t0, b);
                tc_wait_ld();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    ct_put1(qt, part, t0 + e, j, j <= t0 + e ? c.weight(__uint_as_float(a[e]) + __uint_as_float(b[e]), t0 + e, j) : 0.0f);
            }
        }
    } else {
        c.weights(weight_raw, [&](int t, int j, float w) { ct_put1(qt, part, t, j, w); });
    }
    bool split = true;
    ct_put<SV>(xt, part, raw, r.nv, [&](const float4& x, int j, int v) {
        const float4 y = c.out_value(x, j, v);
        split = split && ct_splits(y.x) && ct_splits(y.y) && ct_splits(y.z) && ct_splits(y.w);
        return y;
    });
    if (!split) {                            // (out of the way of the usual tile, and in few instructions: once more, with noughts)
        s.odd = 1;
        const int v = (threadIdx.x & ((1 << SV) - 1)) * 4;
#pragma unroll 1
        for (int j = threadIdx.x >> SV; j < CT; j += CT_THREADS >> SV) {
            const float4 y = c.out_value(c.value_raw(j, v), j, v);
            ct_put4(xt, part, j, v, make_float4(ct_splits(y.x) ? y.x : 0.0f, ct_splits(y.y) ? y.y : 0.0f, ct_splits(y.z) ? y.z : 0.0f, ct_splits(y.w) ? y.w : 0.0f));
        }
    }
    ct_issue(s, [&] { ct_mma<true, false>(d, d + 64, x_a, part, q_a, part, CT / 16, CT / 32, ct_idesc(CT, true, false), true); });
    ct_fetch<SV>(raw, r.nv, [&](int t, int v) { return c.finish_raw(t, v); });
    ct_wait(s, phase);
    float* out = reinterpret_cast<float*>(xt);               // [CT][CT_OUT_LD] (the weights stay where they are)
    {
        const int v = (warp & 3) * 32 + lane;
#pragma unroll 1
        for (int t0 = (warp >> 2) * 32; t0 < (warp >> 2) * 32 + 32; t0 += 8) {
            unsigned a[8], b[8], f[8], g[8];
            gt_ld8(d + 128 + lanes + t0, a);
            gt_ld8(d + 192 + lanes + t0, b);
            gt_ld8(d + lanes + t0, f);
            gt_ld8(d + 64 + lanes + t0, g);
            tc_wait_ld();
            if (v < r.nv) {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    out[(t0 + e) * CT_OUT_LD + v] = fmaf(c.factor(t0 + e), __uint_as_float(a[e]) + __uint_as_float(b[e]),
                                                         __uint_as_float(f[e]) + __uint_as_float(g[e]));
            }
            if (r.nv & 31) __syncwarp();     // (as in the sums)
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s.odd) {                             // values that the product left out: column v by two threads, every other query each
        const int v = threadIdx.x & 127;
        for (int j = 0; v < r.nv && j < c.rows; ++j) {
            const float4 x4 = c.out_value(c.value_raw(j, v & ~3), j, v & ~3);
            const float x = (v & 2) ? ((v & 1) ? x4.w : x4.z) : ((v & 1) ? x4.y : x4.x);
            if (ct_splits(x)) continue;
            for (int t = j + ((threadIdx.x >> 7) ^ (j & 1)); t < c.rows; t += 2) {
                const unsigned char* w = qt + ct_at(t, j);
                const float P = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(w)) + __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(w + part)) +
                                __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(w + 2 * part));
                out[t * CT_OUT_LD + v] = fmaf(P, x, out[t * CT_OUT_LD + v]);
            }
        }
        __syncthreads();
    }
    {                                        // the threads that fetched `raw`; a row's lanes all call, with or without columns
        const int v = (threadIdx.x & ((1 << SV) - 1)) * 4, row = threadIdx.x >> SV;
        if (!s.failed) {
#pragma unroll
            for (int u = 0; u < CT_PASSES<SV>; ++u) {
                const int t = row + u * (CT_THREADS >> SV);
                c.template finish<SV>(t, v, v < r.nv ? *reinterpret_cast<const float4*>(out + t * CT_OUT_LD + v) : make_float4(0.0f, 0.0f, 0.0f, 0.0f), raw[u]);
            }
        }
    }
    ct_end(s, r.status);
}

// (a block behind the tiles: the score product reads 128 rows from a tile of 64)
constexpr size_t CT_SMEM = 1024 + 2 * (size_t)CT_TILE + CT_BLOCK;
// Heads whose sizes fill whole MMA steps and most of a row's threads: n and nv multiples of 16 from 48 to 128.  (Four heads of 32 x 16: 23 us
// for 194 tokens on the float units, 23 to 33 here.)  Decayed attention of 12 heads, one chunk and 2,048 rows, all three kernels, float units and
// here: 48 x 48 30 and 20, 70 and 45 us; 64 x 64 53 and 21, 86 and 47; 96 x 96 66 and 34, 154 and 73; a chunk of 16 rows 27 and 20 (64 x 64), 39
// and 34 (128 x 128).  Per-channel decay of 16 heads: 48 x 48 46 and 39, 89 and 77; 64 x 64 50 and 39, 100 and 84.  Against 64 bits outputs and
// states are off by as much or less than on the float units at each of them.
__host__ inline bool ct_takes(int n, int nv) { return n >= 48 && n <= 128 && nv >= 48 && nv <= 128 && n % 16 == 0 && nv % 16 == 0; }

template <typename K, typename R>
inline int ct_launch(K kern, const R& r, int heads, int n_chunks, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CT_SMEM);
    if (e != cudaSuccess) return (int)e;
    e = launch(kern, dim3(heads, n_chunks), dim3(CT_THREADS), CT_SMEM, stream, r);
    return e == cudaSuccess ? BG_OK : (int)e;
}
template <typename R>
inline int ct_sum(const R& r, int heads, int n_chunks, cudaStream_t stream) {
    if (r.n <= 64) return r.nv <= 64 ? ct_launch(chunk_sum_tc_kernel<R, 4, 4>, r, heads, n_chunks, stream) : ct_launch(chunk_sum_tc_kernel<R, 4, 5>, r, heads, n_chunks, stream);
    return r.nv <= 64 ? ct_launch(chunk_sum_tc_kernel<R, 5, 4>, r, heads, n_chunks, stream) : ct_launch(chunk_sum_tc_kernel<R, 5, 5>, r, heads, n_chunks, stream);
}
template <typename R>
inline int ct_out(const R& r, int heads, int n_chunks, cudaStream_t stream) {
    if (r.n <= 64) return r.nv <= 64 ? ct_launch(chunk_out_tc_kernel<R, 4, 4>, r, heads, n_chunks, stream) : ct_launch(chunk_out_tc_kernel<R, 4, 5>, r, heads, n_chunks, stream);
    return r.nv <= 64 ? ct_launch(chunk_out_tc_kernel<R, 5, 4>, r, heads, n_chunks, stream) : ct_launch(chunk_out_tc_kernel<R, 5, 5>, r, heads, n_chunks, stream);
}

}  // namespace bg
