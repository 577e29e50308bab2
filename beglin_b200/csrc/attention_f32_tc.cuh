// The partial results of float queries over a float cache on the tensor cores: heads of 48 to 128 features, a multiple of 16
// (attention_f32.cuh runs the other sizes, attention_partial_kernel in attention.cu the other types).
//
// Queries, keys, values and weights are cut into three bfloat16 numbers each, and of the nine products of the parts of two floats the six are
// made that are not below 2^-24 of theirs, the small ones added up before the large ones; gemm_f32_tc.cu says what that leaves out, and how far the sums
// are off (a row that sees few keys is a sum of few terms).
// A CTA takes up to 128 rows (queries x query heads of a kv head), a lane of tensor memory each, and one split of keys, 64 at a time:
// eight warps cut the keys and values of a tile into swizzled shared memory, one issues the MMAs, and eight warps, two threads a row with
// 32 keys each, make the weights and keep the row's sums of values in registers (a tile's sums leave tensor memory and are added in float).
// Queries and weights are left operands in tensor memory.  The scores of a tile are multiplied while the weights of the one before are made,
// its values while those of the one behind are.
// 550 rows of 12 heads of 128 (2 kv heads) behind 1,500 positions: 79 us, 87 with one tile of keys and of values in shared memory, 120 with
// all options in one unrolled loop and results stored a row a thread; the mixer of 550 rows over 1,536 to 3,000 held positions takes 179 us
// with its products, 399 with the float units' attention and the same products.  What bounds it: a tile's some 8,000 cycles are a chain of
// hand-overs and of instructions that are fetched once a tile (its MMAs take 3,072), on one CTA an SM.
//
// A row's arithmetic depends on nothing but its own keys: tiles and splits lie at absolute positions, and an MMA's rows do not meet.  Scores that
// are not finite (an operand that is infinite or not a number, a query above 2^90) are summed by floats instead.  Values of 2^72 and more go into
// the tile as nought and are added by floats to the rows whose weight for them is not nought, so that an infinite one at a position that a row
// does not see does not reach it.  Small operands take the usual way (see AX_Q_UP): 550 rows with a key, a query or a value of 1e-36 in every eighth
// row or less, 79 us; noticed where they are cut and summed by floats they took 940 to 980.  With NaN in every eighth key 330 us (16 bytes a load; a value
// a load 940), in one query 845, in every eighth value 183 (the float units' kernel: 293 to 308).
#pragma once

#include "float_parts.cuh"

namespace bg {

constexpr int AX_ROWS = 128, AX_KEYS = 64;
constexpr int AX_NONE = -2147483647 - 1;               // no key here (not an entry of a block table)
constexpr int AX_THREADS = 640;                        // two warpgroups of rows, two that cut, one with the warp that issues
constexpr unsigned AX_BLOCK = AX_KEYS * 128, AX_PART = 2 * AX_BLOCK, AX_TILE = 3 * AX_PART;       // 64 keys x 64 features; x 128; three parts
constexpr unsigned AX_Q = 0, AX_S = 192, AX_P = 256, AX_O = 352;                      // columns of tensor memory
constexpr int AX_REGS = 96, AX_REGS_ROW = 144, AX_REGS_CUT = 72, AX_REGS_OTHER = 48;
static_assert(2 * AX_REGS_ROW + 2 * AX_REGS_CUT + AX_REGS_OTHER <= 5 * AX_REGS);

__host__ __device__ __forceinline__ bool ax_takes(int rows, int hd, int vd, int maps) {
    return maps == 1 && rows <= AX_ROWS && hd >= 48 && hd <= 128 && hd % 16 == 0 && vd >= 16 && vd <= 128 && vd % 16 == 0;
}
// Powers of two that queries, weights and values are cut with.  Every weight and value has exact parts then (the smallest bit of a float times
// 2^24 is 2^-125), and so has every query below 2^90; larger ones have parts that are not numbers, which the scores show.  Keys are cut as they
// are: what is lost of the smallest, below 2^-133, moves a score of smaller queries by less than 2^-36.
constexpr float AX_Q_UP = 274877906944.0f, AX_PV_UP = 16777216.0f;     // 2^38, 2^24
// Values that are added by floats: 64 of the others times their weights stay finite.
__device__ __forceinline__ bool ax_large(float x) { return !(fabsf(x) < 4.722366e21f); }       // 2^72
// all 256 threads of the rows meet
__device__ __forceinline__ void ax_rows_meet() { asm volatile("barrier.cta.sync 1, 256;\n" ::: "memory"); }

// OD: output features of a thread where they are a constant (half a value's: 64 or 32), or 0.
template <typename P, int OD>
__global__ void __launch_bounds__(AX_THREADS, 1) attention_f32_tc_kernel(P p) {
    extern __shared__ unsigned char ax_raw[];
    unsigned char* kt = (unsigned char*)(((uintptr_t)ax_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* vt = kt + 2 * AX_TILE;              // two tiles of keys, two of values
    __shared__ __align__(8) unsigned long long q_full, k_full[2], k_empty[2], v_full[2], v_empty[2], s_full, s_empty, p_full, o_full, o_empty;
    __shared__ unsigned tmem_sh;
    __shared__ int failed;
    // of the last tiles, as many as cutting can be ahead of reading: pages of the keys, -1: none (asked for again when a tile's values have been summed), ..
    __shared__ int page_s[8][AX_KEYS];
    __shared__ unsigned char value_large[4][AX_KEYS];
    __shared__ float row_max[2][AX_ROWS];
    __shared__ int row_at[AX_ROWS];                    // a row's place among the partial results, -1: none

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int qb = blockIdx.x, kvh = blockIdx.y, sp = blockIdx.z;
    if (tid == 0) {
        mbar_init(&q_full, 8);
        for (int b = 0; b < 2; ++b) { mbar_init(&k_full[b], 8); mbar_init(&k_empty[b], 1); mbar_init(&v_full[b], 8); mbar_init(&v_empty[b], 1); }
        mbar_init(&s_full, 1); mbar_init(&s_empty, 8); mbar_init(&p_full, 8); mbar_init(&o_full, 1); mbar_init(&o_empty, 8);
        failed = 0;
        mbar_init_fence();
    }
    if (warp == 16) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();                                      // (the columns are held)
    const unsigned tmem = tmem_sh;
    pdl_wait();
    const int req = p.qblk[qb * 3 + 0], row0 = p.qblk[qb * 3 + 1], nq = p.qblk[qb * 3 + 2];
    const int lo_first = nq > 0 ? first_visible(p.positions[row0], p.window) : 0;
    const int k_first = sp * p.split, k_end = nq > 0 ? min((sp + 1) * p.split, p.positions[row0 + nq - 1] + 1) : 0;       // exclusive
    const bool seen = nq > 0 && k_first < k_end && !(lo_first >= k_end && k_first >= p.keep);       // (else no key of the split is seen)
    const int hd = p.hd, vd = p.vd, group = p.group, n_rows = nq * group;
    const float* pool = (const float*)p.kv_pool;
    const size_t page_elems = (size_t)p.nkv * p.page_size * (hd + vd), v_off = (size_t)p.nkv * p.page_size * hd;
    auto skipped = [&](int t0) { return t0 + AX_KEYS <= lo_first && t0 >= p.keep; };
    auto next_tile = [&](int t0) { do t0 += AX_KEYS; while (t0 < k_end && skipped(t0)); return t0; };
    const int t_first = skipped(k_first) ? next_tile(k_first) : k_first;

    if (warp >= 16) gt_regs<AX_REGS, AX_REGS_OTHER>();
    if (warp == 16) {
        // ---------------- the MMAs: a tile's scores before the values of the tile in front of it
        if (seen && t_first < k_end) {
            const unsigned s_desc = instr_desc_bf16(AX_ROWS, AX_KEYS), o_desc = instr_desc_bf16(AX_ROWS, vd, 1);
            const unsigned k0 = smem_u32(kt), v0 = smem_u32(vt);
            bool ok = mbar_wait(&q_full, 0, &failed);
            int i = 0;
            auto scores = [&](int tile) {
                ok = ok && mbar_wait(&k_full[tile & 1], (tile >> 1) & 1, &failed) && (tile == 0 || mbar_wait(&s_empty, (tile - 1) & 1, &failed));
                if (!ok) return;
                tc_fence_after();
                const unsigned ka = k0 + (tile & 1) * AX_TILE;
                if (elect_one()) {
#pragma unroll
                    for (int e = 0; e < 6; ++e) {
                        constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (j < hd / 16) tc_mma_ts(tmem + AX_S, tmem + AX_Q + PA[e] * 64 + j * 8, smem_desc_sw128(ka + PB[e] * AX_PART + (j >> 2) * AX_BLOCK + (j & 3) * 32), s_desc, e || j ? 1u : 0u);
                    }
                    tc_commit(&s_full);
                    tc_commit(&k_empty[tile & 1]);
                }
                __syncwarp();
            };
            scores(0);
            for (int t0 = t_first; t0 < k_end && ok; ++i) {
                const int t1 = next_tile(t0);
                if (t1 < k_end) scores(i + 1);
                ok = ok && mbar_wait(&v_full[i & 1], (i >> 1) & 1, &failed) && mbar_wait(&p_full, i & 1, &failed) && (i == 0 || mbar_wait(&o_empty, (i - 1) & 1, &failed));
                if (!ok) break;
                tc_fence_after();
                const unsigned va = v0 + (i & 1) * AX_TILE;
                if (elect_one()) {
#pragma unroll
                    for (int e = 0; e < 6; ++e) {
                        constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
                        for (int j = 0; j < AX_KEYS / 16; ++j)
                            tc_mma_ts(tmem + AX_O, tmem + AX_P + PA[e] * 32 + j * 8, smem_desc_sw128_nmajor(va + PB[e] * AX_PART + j * 2048, AX_BLOCK, 1024), o_desc, e || j ? 1u : 0u);
                    }
                    tc_commit(&o_full);
                    tc_commit(&v_empty[i & 1]);
                }
                __syncwarp();
                t0 = t1;
            }
        }
    } else if (warp >= 8 && warp < 16) {
        // ---------------- keys and values into parts: four threads a key, pieces of eight features
        gt_regs<AX_REGS, AX_REGS_CUT>();
        const int c0 = tid & 3, key = (tid - 256) >> 2;
        if (seen) {
            int i = 0;
            auto page_of = [&](int t0) {
                const int at = t0 + key;
                return at < k_end && key_seen(at, lo_first, p.keep) ? p.block_table[(size_t)req * p.max_pages + at / p.page_size] : AX_NONE;
            };
            int page_next = page_of(t_first);          // (asked for a tile ahead)
            for (int t0 = t_first; t0 < k_end; ++i) {
                const int at = t0 + key;
                int page = page_next;
                if (page != AX_NONE && (page < 0 || page >= p.num_pages)) {
                    if (p.status && c0 == 0) atomicOr(p.status, BG_STATUS_BAD_PAGE);
                    page = -1;
                }
                if (page < 0) page = -1;
                unsigned char *kb = kt + (i & 1) * AX_TILE, *vb = vt + (i & 1) * AX_TILE;
                const size_t slot = (size_t)kvh * p.page_size + at % p.page_size;
                const float* ks = pool + (page >= 0 ? (size_t)page * page_elems + slot * hd : 0);
                const float* vs = pool + (page >= 0 ? (size_t)page * page_elems + v_off + slot * vd : 0);
                auto fetch = [&](const float* src, int width, float4 (&v)[8]) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c = c0 + 4 * j;
                        v[2 * j] = v[2 * j + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (page >= 0 && c * 8 < width) {
                            v[2 * j] = *reinterpret_cast<const float4*>(src + c * 8);
                            v[2 * j + 1] = *reinterpret_cast<const float4*>(src + c * 8 + 4);
                        }
                    }
                };
                auto store = [&](unsigned char* tile, int c, const uint4& h, const uint4& m, const uint4& l) {
                    unsigned char* d = tile + (c >> 3) * AX_BLOCK + key * 128 + (((c ^ key) & 7) << 4);
                    *reinterpret_cast<uint4*>(d) = h;
                    *reinterpret_cast<uint4*>(d + AX_PART) = m;
                    *reinterpret_cast<uint4*>(d + 2 * AX_PART) = l;
                };
                auto split8 = [&](const float4& a, const float4& b, uint4& h, uint4& m, uint4& l, float up) {
                    gt_split(gt_up(pair2(a.x, a.y), up), h.x, m.x, l.x);
                    gt_split(gt_up(pair2(a.z, a.w), up), h.y, m.y, l.y);
                    gt_split(gt_up(pair2(b.x, b.y), up), h.z, m.z, l.z);
                    gt_split(gt_up(pair2(b.z, b.w), up), h.w, m.w, l.w);
                };
                float4 v[8];
                fetch(ks, hd, v);
                const int t1 = next_tile(t0);
                page_next = t1 < k_end ? page_of(t1) : AX_NONE;
                if (i > 1) mbar_wait(&k_empty[i & 1], ((i >> 1) - 1) & 1, &failed);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint4 h, m, l;
                    split8(v[2 * j], v[2 * j + 1], h, m, l, 1.0f);
                    if ((c0 + 4 * j) * 8 < hd) store(kb, c0 + 4 * j, h, m, l);
                }
                if (c0 == 0) page_s[i & 7][key] = page;
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&k_full[i & 1]);
                fetch(vs, vd, v);
                if (i > 1) mbar_wait(&v_empty[i & 1], ((i >> 1) - 1) & 1, &failed);
                unsigned long long squares = 0ull;     // not finite with a value of 2^64 and more
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const unsigned long long a = pair2(v[j].x, v[j].y), b = pair2(v[j].z, v[j].w);
                    squares = fma2(b, b, fma2(a, a, squares));
                }
                auto values = [&]() {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint4 h, m, l;
                        split8(v[2 * j], v[2 * j + 1], h, m, l, AX_PV_UP);
                        if ((c0 + 4 * j) * 8 < vd) store(vb, c0 + 4 * j, h, m, l);
                    }
                };
                values();
                unsigned large = !(sum2(squares) <= 3.402823466e38f);
                large |= __shfl_xor_sync(0xffffffffu, large, 1);
                large |= __shfl_xor_sync(0xffffffffu, large, 2);
                if (large) {                           // large values are nought here
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (ax_large(v[j].x)) v[j].x = 0.0f;
                        if (ax_large(v[j].y)) v[j].y = 0.0f;
                        if (ax_large(v[j].z)) v[j].z = 0.0f;
                        if (ax_large(v[j].w)) v[j].w = 0.0f;
                    }
                    values();
                }
                if (c0 == 0) value_large[i & 3][key] = large != 0;
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_full[i & 1]);
                t0 = t1;
            }
        }
    } else if (warp < 8) {
        // ---------------- the rows: lane and quarter are the row, the half says which keys and which output features
        gt_regs<AX_REGS, AX_REGS_ROW>();
        const int quarter = warp & 3, half = warp >> 2, row = quarter * 32 + lane;
        const unsigned lanes = tmem + ((unsigned)(quarter * 32) << 16);
        const bool in = row < n_rows;
        const int qi = in ? row / group : 0, head = kvh * group + (in ? row - qi * group : 0);
        const int pos = in ? p.positions[row0 + qi] : -1, lo = first_visible(pos < 0 ? 0 : pos, p.window);
        const float* q = (const float*)p.q + (size_t)(row0 + qi) * p.q_stride + (size_t)head * hd;
        const float slope = p.slopes && in ? p.slopes[head] : 0.0f, scale_down = p.scale / AX_Q_UP;
        const int od = OD ? OD : vd / 2;               // output features of a thread, a multiple of 8
        constexpr int MOST = OD ? OD : 64;
        float out[MOST];
        float m = -INFINITY, sum = 0.0f;
#pragma unroll
        for (int d = 0; d < MOST; ++d) out[d] = 0.0f;
        if (seen && t_first < k_end) {
            // the row's queries, half of their features a thread
            float4 x[16];                              // (all on their way together)
#pragma unroll
            for (int c = 0; c < 16; ++c) x[c] = in && c * 4 < hd / 2 ? *reinterpret_cast<const float4*>(q + half * (hd / 2) + c * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                if (c * 8 >= hd / 2) break;
                unsigned h[4], mm[4], l[4];
                gt_split(gt_up(pair2(x[2 * c].x, x[2 * c].y), AX_Q_UP), h[0], mm[0], l[0]);
                gt_split(gt_up(pair2(x[2 * c].z, x[2 * c].w), AX_Q_UP), h[1], mm[1], l[1]);
                gt_split(gt_up(pair2(x[2 * c + 1].x, x[2 * c + 1].y), AX_Q_UP), h[2], mm[2], l[2]);
                gt_split(gt_up(pair2(x[2 * c + 1].z, x[2 * c + 1].w), AX_Q_UP), h[3], mm[3], l[3]);
                const unsigned a = lanes + AX_Q + half * (hd / 4) + c * 4;
                gt_st4(a, h); gt_st4(a + 64, mm); gt_st4(a + 128, l);
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_full);
            float corr_before = 0.0f;                  // of the tile whose values are still being summed
            // adds the tile's sums of values to the row's
            auto add_values = [&](int i, int t0, float corr) {
                mbar_wait(&o_full, i & 1, &failed);
                __syncwarp();
                tc_fence_after();
                const unsigned long long cc = pair2(corr, corr), down = pair2(1.0f / AX_PV_UP / AX_PV_UP, 1.0f / AX_PV_UP / AX_PV_UP);
#pragma unroll
                for (int c = 0; c < MOST; c += 16) {
                    if (!OD && c >= od) break;
                    unsigned r[16];
                    if (OD || c + 16 <= od) gt_ld16(lanes + AX_O + half * od + c, r);
                    else gt_ld8(lanes + AX_O + half * od + c, r);
                    tc_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; e += 2)
                        if (OD || c + e < od) {
                            const unsigned long long y = fma2(pair2(out[c + e], out[c + e + 1]), cc, fma2((unsigned long long)r[e] | ((unsigned long long)r[e + 1] << 32), down, 0ull));
                            out[c + e] = low2(y); out[c + e + 1] = high2(y);
                        }
                }
                bool large = false;
#pragma unroll
                for (int j = 0; j < 2; ++j) large |= value_large[i & 3][j * 32 + lane] != 0;
                if (__any_sync(0xffffffffu, large)) {  // the weights come back from their parts
                    for (int j = 0; j < AX_KEYS; ++j) {
                        if (!value_large[i & 3][j]) continue;
                        __syncwarp();                  // (lanes come from the sums of the key before)
                        unsigned w[3];
#pragma unroll
                        for (int e = 0; e < 3; ++e)
                            asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(w[e]) : "r"(lanes + AX_P + e * 32 + (j >> 1)));
                        tc_wait_ld();
                        float f = 0.0f;
#pragma unroll
                        for (int e = 2; e >= 0; --e) f += __uint_as_float(j & 1 ? w[e] & 0xffff0000u : w[e] << 16);
                        f *= 1.0f / AX_PV_UP;
                        const int page = page_s[i & 7][j];
                        if (f != 0.0f && page >= 0) {
                            const float* src = pool + (size_t)page * page_elems + v_off + ((size_t)kvh * p.page_size + (t0 + j) % p.page_size) * vd + half * od;
#pragma unroll
                            for (int d = 0; d < MOST; ++d)
                                if (d < od && ax_large(src[d])) out[d] = fmaf(f, src[d], out[d]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&o_empty);
            };
            int i = 0, t_before = 0;
            for (int t0 = t_first; t0 < k_end; ++i) {
                mbar_wait(&s_full, i & 1, &failed);
                __syncwarp();
                tc_fence_after();
                float w[32];
                {
                    unsigned r[32];
                    tc_ld32_nowait(lanes + AX_S + half * 32, r);
                    tc_wait_ld();
#pragma unroll
                    for (int j = 0; j < 32; ++j) w[j] = __uint_as_float(r[j]);
                }
                // the keys that the row sees, a bit each, and the scores that the parts cannot make
                const int base = t0 + half * 32, last = min(pos, k_end - 1) - base;
                auto below = [](int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1; };       // bits 0 .. n - 1
                unsigned visible = __ballot_sync(0xffffffffu, page_s[i & 7][half * 32 + lane] >= 0) & below(last + 1) & (~below(lo - base) | below(p.keep - base));
                unsigned bad = 0;
                float nought = 0.0f;
#pragma unroll
                for (int j = 0; j < 32; ++j) nought = fmaf(w[j], 0.0f, nought);
                if (!(nought == 0.0f)) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (!(fabsf(w[j]) <= 3.402823466e38f)) bad |= 1u << j;
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) w[j] *= scale_down;
                bad &= visible;
                while (bad) {
                    const int jb = __ffs(bad) - 1, at = t0 + half * 32 + jb, page = page_s[i & 7][half * 32 + jb];
                    bad &= bad - 1;
                    const float* src = pool + (size_t)page * page_elems + ((size_t)kvh * p.page_size + at % p.page_size) * hd;
                    float even = 0.0f, odd = 0.0f;
#pragma unroll 2
                    for (int d = 0; d < hd; d += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(q + d), y = *reinterpret_cast<const float4*>(src + d);
                        even = fmaf(x.z, y.z, fmaf(x.x, y.x, even));
                        odd = fmaf(x.w, y.w, fmaf(x.y, y.y, odd));
                    }
                    even = (even + odd) * p.scale;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (j == jb) w[j] = even;
                }
                __syncwarp();
                // (the way that most tiles go is short: a warp's instructions are fetched once a tile, and with every option in one unrolled
                // loop the fetches were most of a tile's 12,500 cycles)
                float most = -INFINITY;
                if (p.softcap > 0.0f || p.slopes) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (p.softcap > 0.0f) w[j] = p.softcap * tanhf(w[j] / p.softcap);
                        if (p.slopes) w[j] = fmaf(-slope, (float)(pos - (base + j)), w[j]);
                    }
                }
                if (!__all_sync(0xffffffffu, visible == 0xffffffffu)) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (!(visible >> j & 1)) w[j] = -INFINITY;
                }
#pragma unroll
                for (int j = 0; j < 32; ++j) most = fmaxf(most, w[j]);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_empty);  // (the scores and the tile's pages have been read)
                row_max[half][row] = most;
                ax_rows_meet();
                const float m_new = fmaxf(m, fmaxf(row_max[0][row], row_max[1][row]));
                const float corr = m == -INFINITY ? 0.0f : expf(m - m_new);
                const float from = m_new == -INFINITY ? 0.0f : m_new;          // (no key seen so far: every weight is nought)
                float s = 0.0f;
#pragma unroll
                for (int j = 0; j < 32; ++j) { w[j] = expf(w[j] - from); s += w[j]; }
                sum = fmaf(sum, corr, s);
                m = m_new;
                if (i > 0) add_values(i - 1, t_before, corr_before);
                // row_max is free again; and neither of a row's two threads puts weights where the other may still read those of the tile before
                // (add_values, values without three parts)
                ax_rows_meet();
                tc_fence_after();
                corr_before = corr;
                // the weights' parts, where the values' products before have read theirs
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    unsigned h[4], mm[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) gt_split(gt_up(pair2(w[8 * c + 2 * e], w[8 * c + 2 * e + 1]), AX_PV_UP), h[e], mm[e], l[e]);
                    const unsigned a = lanes + AX_P + half * 16 + 4 * c;
                    gt_st4(a, h); gt_st4(a + 32, mm); gt_st4(a + 64, l);
                }
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full);
                t_before = t0;
                t0 = next_tile(t0);
            }
            add_values(i - 1, t_before, corr_before);
            // partial results of the rows that see at least one key of this split, through the tiles' room (their products are complete)
            row_max[half][row] = sum;
            if (half == 0) row_at[row] = in && !(pos < sp * p.split || (lo >= (sp + 1) * p.split && sp * p.split >= p.keep)) ? (row0 + qi) * p.nh + head : -1;
            float* stage = (float*)kt;
            const int ld = vd + 4;
#pragma unroll
            for (int d = 0; d < MOST; d += 4)
                if (OD || d < od) *reinterpret_cast<float4*>(stage + row * ld + half * od + d) = make_float4(out[d], out[d + 1], out[d + 2], out[d + 3]);
            ax_rows_meet();
            const bool lost = *(volatile int*)&failed != 0;                    // (a wait ran out)
            if (half == 0 && row_at[row] >= 0) {
                float* ml = p.part_ml + ((size_t)row_at[row] * p.max_splits + sp) * 2;
                ml[0] = m; ml[1] = lost ? NAN : row_max[0][row] + row_max[1][row];
            }
            for (int r = warp; r < n_rows; r += 8) {
                const int place = row_at[r];
                if (place >= 0 && lane * 4 < vd)
                    *reinterpret_cast<float4*>(p.part_o + ((size_t)place * p.max_splits + sp) * vd + lane * 4) = *reinterpret_cast<const float4*>(stage + r * ld + lane * 4);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
    if (tid == 0 && failed && p.status) atomicOr(p.status, BG_STATUS_TIMEOUT);
}

}  // namespace bg
