// The partial results of float queries over a float cache in blocks of registers: the float path's attention for head sizes that
// are multiples of 4 and that the tensor cores' kernel does not take (attention_f32_tc.cuh: 48 to 128 features in sixteens, one map;
// attention_partial_kernel in attention.cu runs the other sizes and types, and says what a partial result is).
//
// A CTA takes up to 64 rows (queries x query heads of a kv head) and one split of keys, 64 keys at a time.  Thread (ty, tx) of
// 16 x 16 owns rows ty + 16 i (i < RI, as many sixteens as the block has rows), of the scores keys tx + 16 j, of the output columns
// 4 tx .. 4 tx + 3 of every 64.  Scores: rows and keys lie with the features innermost, so four features of a row are one 16-byte
// read and two of them one operand of the packed multiply-add (fma.rn.f32x2: two float multiply-adds; the even and the odd features
// are two chains whose sums are added; heads of up to AF_NARROW features are one chain, which takes no longer there: 2,048 rows of 8 heads of
// 32, 188 and 194 us).  A row's sixteen threads lie in one half of a warp: maximum and sum are shuffles, and the weights pass through
// shared memory behind a warp's barrier only.  The keys of the next tile come (cp.async) under the value product, the values under the scores.  112 KB of shared memory for heads of 128, so that two CTAs share an SM.  FMA pipe, shared
// memory and issue are each used by half, a tile's phases in turn: heads of 128, which the tensor cores have taken over since, took 307 us for
// 550 rows of 12 heads over 1,536 to 3,000 held positions, 2,200 with a key a lane and two reads of shared memory for every multiply-add.
//
// A row's arithmetic depends on nothing but its own keys: tiles and splits lie at absolute positions, every sum has one order, and a
// value whose weight is nought is left out, so that an infinite one at a position that a row does not see does not reach it.  A warp
// looks at the weights that it has made of a tile; only where one is nought (the diagonal, a window's edge, a weight that underflowed)
// does it ask weight by weight (512 rows of 8 heads of 64 behind nothing, the diagonal in every eighth tile: 63 -> 65 us).
#pragma once

#include "common.cuh"
#include "float_pairs.cuh"

namespace bg {

constexpr int AF_ROWS = 64, AF_KEYS = 64, AF_THREADS = 256;
constexpr int AF_NARROW = 32;              // features of a head up to which a score is one chain of sums

// reductions over a row's sixteen threads (half a warp)
__device__ __forceinline__ float af_max16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float af_sum16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct AfShared { float *q, *k, *v, *w; int *page; int qld, kld, vld; };
// floats between rows: queries as wide as they are; keys in 16-byte pieces that are swapped by the row's number inside groups of
// eight, so a row takes whole groups; values a multiple of 64 columns
__host__ __device__ __forceinline__ int af_kld(int hd) { return (hd + 31) / 32 * 32; }
__host__ __device__ __forceinline__ int af_vld(int vd) { return (vd + 63) / 64 * 64; }
__host__ __device__ __forceinline__ size_t af_smem(int qhd, int hd, int vd) {
    return ((size_t)AF_ROWS * qhd + (size_t)AF_KEYS * (af_kld(hd) + af_vld(vd)) + (size_t)AF_ROWS * AF_KEYS + AF_KEYS) * sizeof(float);
}

template <bool V> struct AfAsk { static constexpr bool value = V; };

template <typename P, int RI, int NC, bool NARROW>
__device__ __forceinline__ void af_walk(const P& p, const AfShared& s, int req, int row0, int kvh, int sp, int n_rows,
                                        int k_first, int k_end, int lo_first) {
    const int tid = threadIdx.x, lane = tid & 31, ty = (tid >> 5) * 2 + (lane >> 4), tx = lane & 15;
    const int hd = p.hd, vd = p.vd, group = p.group, qhd = hd / p.maps;
    const float* pool = (const float*)p.kv_pool;
    const size_t page_elems = (size_t)p.nkv * p.page_size * (hd + vd), v_off = (size_t)p.nkv * p.page_size * hd;

    int pos[RI], lo[RI], qc[RI];           // of the thread's rows: position, first key seen, first piece of the row's map in a key row
    float slope[RI];
    unsigned long long acc[RI][2 * NC];
    float m[RI], l[RI];
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int r = ty + 16 * i, rr = r < n_rows ? r : 0;
        pos[i] = r < n_rows ? p.positions[row0 + rr / group] : -1;       // (a row that is not there sees no key)
        lo[i] = first_visible(pos[i] < 0 ? 0 : pos[i], p.window);
        qc[i] = (rr % group) % p.maps * qhd / 4;
        slope[i] = p.slopes ? p.slopes[kvh * group + rr % group] : 0.0f;
        m[i] = -INFINITY; l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < 2 * NC; ++c) acc[i][c] = 0ull;
    }

    auto skipped = [&](int t0) { return t0 + AF_KEYS <= lo_first && t0 >= p.keep; };
    auto next_tile = [&](int t0) { do t0 += AF_KEYS; while (t0 < k_end && skipped(t0)); return t0; };
    // the pages of a tile's keys, -1 for a key that no row of the block may see; the barrier behind it is the caller's
    auto look_up = [&](int t0) {
        if (tid < AF_KEYS) {
            const int key = t0 + tid;
            int page = -1;
            if (key < k_end && key_seen(key, lo_first, p.keep)) {
                page = p.block_table[(size_t)req * p.max_pages + key / p.page_size];
                if (page < 0 || page >= p.num_pages) {
                    if (p.status) atomicOr(p.status, BG_STATUS_BAD_PAGE);
                    page = -1;
                }
            }
            s.page[tid] = page;
        }
    };
    auto fetch_keys = [&](int t0) {
        const int n4 = hd >> 2;
        for (int idx = tid; idx < AF_KEYS * n4; idx += AF_THREADS) {
            const int j = idx / n4, c = idx - j * n4, page = s.page[j];
            const float* src = pool + (page >= 0 ? (size_t)page * page_elems + ((size_t)kvh * p.page_size + (t0 + j) % p.page_size) * hd + c * 4 : 0);
            async_copy<16>(s.k + j * s.kld + ((c & ~7) | ((c ^ j) & 7)) * 4, src, page >= 0);
        }
        async_commit();
    };
    auto fetch_values = [&](int t0) {
        const int n4 = vd >> 2;
        for (int idx = tid; idx < AF_KEYS * n4; idx += AF_THREADS) {
            const int j = idx / n4, c = idx - j * n4, page = s.page[j];
            const float* src = pool + (page >= 0 ? (size_t)page * page_elems + v_off + ((size_t)kvh * p.page_size + (t0 + j) % p.page_size) * vd + c * 4 : 0);
            async_copy<16>(s.v + j * s.vld + c * 4, src, page >= 0);
        }
        async_commit();
    };

    int t0 = k_first;
    if (skipped(t0)) t0 = next_tile(t0);
    if (t0 < k_end) {
        look_up(t0);
        __syncthreads();
        fetch_keys(t0);
    }
    while (t0 < k_end) {
        fetch_values(t0);
        async_wait<1>();                      // the keys are there
        __syncthreads();
        // ---- scores of the thread's rows against keys t0 + tx + 16 j
        unsigned long long sc[RI][4];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) sc[i][j] = 0ull;
        const float* qr = s.q + ty * s.qld;
        const float* kr = s.k + tx * s.kld;
        const int sw = tx & 7;             // (rows tx + 16 j have the same low bits)
        if constexpr (NARROW) {
            for (int c = 0; c < (qhd >> 2); ++c) {
                float4 a[RI], b[4];
#pragma unroll
                for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(qr + i * 16 * s.qld + c * 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(kr + j * 16 * s.kld + ((c & ~7) | ((c ^ sw) & 7)) * 4);
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j)            // (in the low half; the high one stays nought)
                        sc[i][j] = __float_as_uint(fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, __uint_as_float((unsigned)sc[i][j]))))));
            }
        } else if (p.maps == 1) {
#pragma unroll 4
            for (int c = 0; c < (qhd >> 2); ++c) {
                ulonglong2 a[RI], b[4];
#pragma unroll
                for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(qr + i * 16 * s.qld + c * 4);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(kr + j * 16 * s.kld + ((c & ~7) | ((c ^ sw) & 7)) * 4);
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int u = 0; u < RI; ++u) { const int i = j & 1 ? RI - 1 - u : u; sc[i][j] = fma2(a[i].x, b[j].x, sc[i][j]); }
#pragma unroll
                for (int j = 3; j >= 0; --j)
#pragma unroll
                    for (int u = 0; u < RI; ++u) { const int i = j & 1 ? u : RI - 1 - u; sc[i][j] = fma2(a[i].y, b[j].y, sc[i][j]); }
            }
        } else {                           // rows of different maps meet different columns of a key row: one row's keys at a time
            for (int c = 0; c < (qhd >> 2); ++c) {
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(qr + i * 16 * s.qld + c * 4);
                    const int kc = qc[i] + c;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(kr + j * 16 * s.kld + ((kc & ~7) | ((kc ^ sw) & 7)) * 4);
                        sc[i][j] = fma2(a.y, b.y, fma2(a.x, b.x, sc[i][j]));
                    }
                }
            }
        }
        // ---- weights
        bool nought = false;
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            float w[4], tmax = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = t0 + tx + 16 * j;
                w[j] = -INFINITY;
                if (key <= pos[i] && key < k_end && key_seen(key, lo[i], p.keep) && s.page[tx + 16 * j] >= 0) {
                    w[j] = sum2(sc[i][j]) * p.scale;
                    if (p.softcap > 0.0f) w[j] = p.softcap * tanhf(w[j] / p.softcap);
                    if (p.slopes) w[j] = fmaf(-slope[i], (float)(pos[i] - key), w[j]);
                }
                tmax = fmaxf(tmax, w[j]);
            }
            const float m_new = fmaxf(m[i], af_max16(tmax));
            const float corr = m[i] == -INFINITY ? 0.0f : expf(m[i] - m_new);
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                w[j] = w[j] == -INFINITY || m_new == -INFINITY ? 0.0f : expf(w[j] - m_new);
                nought |= w[j] == 0.0f && pos[i] >= 0;             // (rows that are not there are stored nowhere)
                sum += w[j];
                s.w[(ty + 16 * i) * AF_KEYS + tx + 16 * j] = w[j];
            }
            sum = af_sum16(sum);
            if (m_new != -INFINITY) {      // (else no key of this tile or of one before is seen: everything is still nought)
                m[i] = m_new;
                l[i] = fmaf(l[i], corr, sum);
                const unsigned long long cc = pair2(corr, corr);
#pragma unroll
                for (int c = 0; c < 2 * NC; ++c) acc[i][c] = fma2(acc[i][c], cc, 0ull);
            }
        }
        async_wait<0>();                      // the values are there; every warp is done with the keys and their pages
        __syncthreads();
        const int t1 = next_tile(t0);
        if (t1 < k_end) look_up(t1);
        // ---- the weights' sums of values (a row's weights were written by the same half of a warp)
        const float* wr = s.w + ty * AF_KEYS;
        const float* vr = s.v + tx * 4;
        const bool all_seen = !__any_sync(0xffffffffu, nought);            // (of the rows of both halves of the warp)
        auto values = [&](int j, auto ask) {
            float4 a[RI];
#pragma unroll
            for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const float4*>(wr + i * 16 * AF_KEYS + j);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ulonglong2 b[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) b[c] = *reinterpret_cast<const ulonglong2*>(vr + (j + e) * s.vld + c * 64);
#pragma unroll
                for (int u = 0; u < RI; ++u) {
                    const int i = e & 1 ? RI - 1 - u : u;
                    const float f = e == 0 ? a[i].x : e == 1 ? a[i].y : e == 2 ? a[i].z : a[i].w;
                    if (decltype(ask)::value && f == 0.0f) continue;
                    const unsigned long long ff = pair2(f, f);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        acc[i][2 * c] = fma2(ff, b[c].x, acc[i][2 * c]);
                        acc[i][2 * c + 1] = fma2(ff, b[c].y, acc[i][2 * c + 1]);
                    }
                }
            }
        };
        auto values_of = [&](int from, int to) {
            if (all_seen) {
#pragma unroll 1
                for (int j = from; j < to; j += 4) values(j, AfAsk<false>());
            } else {
#pragma unroll 1
                for (int j = from; j < to; j += 4) values(j, AfAsk<true>());
            }
        };
        if (t1 < k_end) {
            // the first sixteen keys, then the pages are known to all and the next keys set out under the rest
            values_of(0, 16);
            __syncthreads();
            fetch_keys(t1);
            values_of(16, AF_KEYS);
            __syncthreads();               // the values have been read
        } else {
            values_of(0, AF_KEYS);
        }
        t0 = t1;
    }
    // ---- partial results of the rows that see at least one key of this split
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int r = ty + 16 * i;
        if (r >= n_rows || pos[i] < sp * p.split || (lo[i] >= (sp + 1) * p.split && sp * p.split >= p.keep)) continue;
        const size_t prow = ((size_t)(row0 + r / group) * p.nh + (size_t)kvh * group + r % group) * p.max_splits + sp;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            const int d = tx * 4 + c * 64;
            if (d < vd) *reinterpret_cast<ulonglong2*>(p.part_o + prow * vd + d) = make_ulonglong2(acc[i][2 * c], acc[i][2 * c + 1]);
        }
        if (tx == 0) { p.part_ml[prow * 2 + 0] = m[i]; p.part_ml[prow * 2 + 1] = l[i]; }
    }
}

// (NARROW: one map of heads of up to AF_NARROW features)
template <typename P, int NC, bool NARROW>
__global__ void __launch_bounds__(AF_THREADS, NC <= 2 ? 2 : 1) attention_f32_kernel(P p) {
    extern __shared__ __align__(16) float af_s[];
    pdl_launch();
    pdl_wait();
    const int qb = blockIdx.x, kvh = blockIdx.y, sp = blockIdx.z;
    const int req = p.qblk[qb * 3 + 0], row0 = p.qblk[qb * 3 + 1], nq = p.qblk[qb * 3 + 2];
    if (nq <= 0) return;
    const int lo_first = first_visible(p.positions[row0], p.window);
    const int k_first = sp * p.split, k_end = min((sp + 1) * p.split, p.positions[row0 + nq - 1] + 1);       // exclusive
    if (k_first >= k_end || (lo_first >= k_end && k_first >= p.keep)) return;      // no key of the split is seen
    const int qhd = p.hd / p.maps, n_rows = nq * p.group;
    AfShared s;
    s.qld = qhd; s.kld = af_kld(p.hd); s.vld = af_vld(p.vd);
    s.q = af_s; s.k = s.q + AF_ROWS * s.qld; s.v = s.k + AF_KEYS * s.kld; s.w = s.v + AF_KEYS * s.vld;
    s.page = (int*)(s.w + AF_ROWS * AF_KEYS);
    // the queries, rows up to the next sixteen (zeros behind the last); columns of the values' tile that no value fills
    const int n4 = qhd >> 2, rows16 = (n_rows + 15) / 16 * 16;
    for (int idx = threadIdx.x; idx < rows16 * n4; idx += AF_THREADS) {
        const int r = idx / n4, c = idx - r * n4, qi = r / p.group, g = r - qi * p.group;
        const bool in = r < n_rows;
        const float* src = (const float*)p.q + (in ? (size_t)(row0 + qi) * p.q_stride + (size_t)(kvh * p.group + g) * qhd + c * 4 : 0);
        async_copy<16>(s.q + r * s.qld + c * 4, src, in);
    }
    async_commit();                           // (complete when the first keys are)
    if (s.vld > p.vd)
        for (int idx = threadIdx.x; idx < AF_KEYS * (s.vld - p.vd); idx += AF_THREADS)
            s.v[idx / (s.vld - p.vd) * s.vld + p.vd + idx % (s.vld - p.vd)] = 0.0f;
    if (n_rows <= 16) af_walk<P, 1, NC, NARROW>(p, s, req, row0, kvh, sp, n_rows, k_first, k_end, lo_first);
    else if (n_rows <= 32) af_walk<P, 2, NC, NARROW>(p, s, req, row0, kvh, sp, n_rows, k_first, k_end, lo_first);
    else af_walk<P, 4, NC, NARROW>(p, s, req, row0, kvh, sp, n_rows, k_first, k_end, lo_first);
}

}  // namespace bg
