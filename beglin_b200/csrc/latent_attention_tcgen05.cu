// Attention through a latent on tcgen05, for single tokens of each request (decoding) in bfloat16: the arguments of
// latent_attention_mma.cu, ranges of keys that follow each request's own length, partial results for latent_attention_merge.
//
// A CTA takes one row (a request's token), up to NH = 16 or 32 of its heads and one range of its keys, 128 keys at a time.  What has
// to move is the cached rows, once: they come by TMA (boxes of 64 features x 64 positions of a page, 128-byte swizzle) into a ring,
// and both products read them there as they lie.  Keys and features are the M side, heads the N side, so that 16 or 32 heads leave
// no part of a 128-row MMA unused:
//     S^T [128 keys, NH]         = K [128, width] Q^T            (K: a box as it is, features innermost)
//     O^T [128 features, NH]     = V^T [128 features, 128 keys] P^T, of one tile, for every 128 features of the latent
// V is the first `rank` features of the same rows, read with the features as M (an M-major left operand).  Scores and a tile's results
// live in tensor memory, two of each.  Warps: 0 asks for the rows, 1 issues the score products, 2 the value products, 4 to 7 are the
// softmax, a thread per key: the maximum over the keys of a head is one redux over the warp and one exchange of the four warps through
// shared memory; P goes to shared memory as bfloat16, relative to the largest weight of its OWN tile, which is then one and not rounded;
// the sums of weights are of the rounded ones.  (A maximum kept over tiles left the weights that matter most between powers of two:
// scores with a deviation of six, 0.00081 of the result, 0.00013 so.)  A tile's results are added up by the softmax's threads, a thread
// per feature with all its heads in registers, when the next tile's weights are on their way.
//
// The ring is cut finer than a tile: slots of 128 features x 128 keys, given back one by one as the value products have read them, and
// one slot for the rotated part, given back by the score products.  A tile of 576 features is 147 KB, so that two of them do not fit
// an SM; with the finer slots the next tile sets out while the last one is used.  One CTA an SM; bound by the bytes of the cache.
// Measured (kernel and merge, 512 + 64 features, 32 heads): 64 requests of 4,000 keys 257.9 us with latent_attention_mma.cu -> 96.3 us
// (3.1 TB/s of cache; 91.7 with a maximum kept over tiles and sums in tensor memory, 10 us more with MMAs issued under a test of the lane's
// number), 8 requests 48.9 -> 35.4, 32 requests of 300 keys 38.7 -> 24.4; 12 heads of 384 + 64, 64 requests of 4,096 keys 127.7 -> 61.8,
// one request 30.6 -> 23.9.  What is left beside the bytes is a range's start and end (queries, the first rows, the results: 5 us of the
// whole when they left as 128 stores of 4 bytes a thread, whose instructions every CTA fetched for one use) and the chain of a tile, whose rows
// are held until its last value product while only a part of the next tile's fit.  Tiles of 64 keys, of which 2.5 fit, took 100 us against
// 92.6 then: half of every score product's rows are then not keys, and the chain is walked twice as often.
// Keys behind the range's last lie in pages that this request may never have written: their rows are zeroed in shared memory before
// the value products read them (0 x NaN would reach every head).
#include "tc_common.cuh"
#include "latent_range.cuh"

namespace bg {

constexpr int LT_THREADS = 256;
constexpr int LT_KEYS = LATENT_RANGE_STEP;               // keys of a tile
constexpr unsigned LT_BLOCK = LT_KEYS * 128;             // 64 features x 128 keys, bytes
constexpr unsigned LT_SLOT = 2 * LT_BLOCK;               // 128 features
constexpr int LT_MAX_SLOTS = 8;
constexpr float LT_LOG2E = 1.4426950408889634f, LT_LN2 = 0.6931471805599453f;
constexpr float LT_FALL = 60.0f;                         // how far (in powers of two) a tile's reference may lie under the largest score

struct LtParams {
    const float* q_lat; long long ql_head; int ql_row;
    const __nv_bfloat16* q_raw; int qr_row, qr_head, qr_off;
    const float* cos_sin;
    const int* block_table; int max_pages, num_pages, page_size;
    const int* positions; const int* qblk;
    float* part_o; float* part_ml; int max_splits;
    int H, rank, rot, rot_dims, window, slots;
    int ctas, sms;          // rows times chunks of heads, SMs: what the number of a row's ranges goes by (latent_range.cuh)
    float scale_log2;
    unsigned* status;
};

__device__ __forceinline__ float lt_warp_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;\n" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float lt_exp2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void lt_bar(int id, int threads) { asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory"); }
// Whether `ok` holds in all 128 threads of the softmax warps (which meet here)
__device__ __forceinline__ bool lt_all(bool ok) {
    unsigned r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n bar.red.and.pred q, 3, 128, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r) : "r"((unsigned)ok) : "memory");
    return r != 0;
}
template <int NH>
__device__ __forceinline__ void lt_load(unsigned taddr, float (&v)[NH]) {
    if constexpr (NH == 32) tc_ld32(taddr, v);
    else {
        unsigned r[16];
        tc_ld16(taddr, r);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
    }
}
template <int NH>
__global__ void __launch_bounds__(LT_THREADS, 1) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map, LtParams p) {
    extern __shared__ unsigned char lt_raw[];
    __shared__ __align__(8) unsigned long long slot_full[LT_MAX_SLOTS], slot_empty[LT_MAX_SLOTS], rot_full, rot_empty, s_full[2], s_empty[2],
        p_full, p_empty;
    __shared__ __align__(16) float wmax[2][4][32], mrow[4][32], frow[2][4][32], lsum[4][32];      // (mrow, frow: a warp's own copies)
    __shared__ unsigned tmem_sh;
    __shared__ int failed;
    constexpr unsigned TMEM_COLS = NH == 32 ? 512 : 256, O_COL = 2 * NH, O_COLS = 4 * NH;      // (a tile's results: up to four pairs)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // (the list and the positions are read in front of the wait, here as in the decoding attention: no kernel between a step's upload, or the
    // sampling kernel that ends a replay, and its last layer writes them)
    const int qb = blockIdx.x, h0 = blockIdx.y * NH, nh = min(NH, p.H - h0), sp = blockIdx.z;
    const int req = p.qblk[qb * 3 + 0], t = p.qblk[qb * 3 + 1];
    const int pos = p.positions[t], lo = first_visible(pos, p.window);
    const LatentRange range = latent_range(pos, lo, p.max_splits, p.ctas, p.sms);
    if (p.qblk[qb * 3 + 2] <= 0 || sp >= range.count) return;              // (the whole CTA)
    const int k_begin = range.begin + sp * range.per, k_end = min(k_begin + range.per, pos + 1);
    const int n_tiles = (k_end - k_begin + LT_KEYS - 1) / LT_KEYS;
    const int blocks = p.rank / 64, pairs = (blocks + 1) / 2, q_blocks = blocks + (p.rot > 0 ? 1 : 0);

    unsigned char* ring = (unsigned char*)(((uintptr_t)lt_raw + 1023) & ~(uintptr_t)1023);       // [slots][2][128 keys][64 features]
    unsigned char* rot_s = ring + (size_t)p.slots * LT_SLOT;                                       // [128 keys][64 features]
    unsigned char* q_s = rot_s + LT_BLOCK;                                                         // [q_blocks][NH][64 features]
    unsigned char* p_s = q_s + (size_t)q_blocks * NH * 128;                                        // [2][NH][64 keys]

    if (tid == 0) {
        for (int i = 0; i < p.slots; ++i) { mbar_init(&slot_full[i], 1); mbar_init(&slot_empty[i], 1); }
        mbar_init(&rot_full, 1); mbar_init(&rot_empty, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 128); }
        mbar_init(&p_full, 128); mbar_init(&p_empty, 1);
        failed = 0;
        mbar_init_fence();
        tma_prefetch_map(&map);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_sh;
    pdl_launch();
    pdl_wait();
    bool ok = true;

    if (warp == 0) {
        // ------------------------------------------------------------------ the cached rows: the warp walks, lane 0 asks
        const int rows_total = p.num_pages * p.page_size;
        int mine = 0;                                    // lane l: the pool row of the (l % 2)-th half of the (l / 2)-th of sixteen tiles
        int it = 0;
        for (int ti = 0; ti < n_tiles && ok; ++ti) {
            if ((ti & 15) == 0) {
                const int key = k_begin + (ti * 2 + lane) * 64;
                mine = rows_total;                       // out of bounds: zeros
                if (key < k_end && key + 63 >= lo) {
                    const int page = p.block_table[(size_t)req * p.max_pages + key / p.page_size];
                    if (page >= 0 && page < p.num_pages) mine = page * p.page_size + key % p.page_size;
                    else if (p.status) atomicOr(p.status, BG_STATUS_BAD_PAGE);
                }
            }
            const int row_a = __shfl_sync(0xffffffffu, mine, (ti & 15) * 2), row_b = __shfl_sync(0xffffffffu, mine, (ti & 15) * 2 + 1);
            for (int i = 0; i < pairs && ok; ++i, ++it) {
                const int slot = it % p.slots;
                if (it >= p.slots) ok = __all_sync(0xffffffffu, mbar_wait(&slot_empty[slot], ((it / p.slots) - 1) & 1, &failed)) != 0;
                if (!ok) break;
                if (lane == 0) {
                    unsigned char* dst = ring + (size_t)slot * LT_SLOT;
                    const bool two = 2 * i + 1 < blocks;
                    mbar_expect_tx(&slot_full[slot], two ? LT_SLOT : LT_BLOCK);
                    tma_load_2d(dst, &map, i * 128, row_a, &slot_full[slot]);
                    tma_load_2d(dst + LT_BLOCK / 2, &map, i * 128, row_b, &slot_full[slot]);
                    if (two) {
                        tma_load_2d(dst + LT_BLOCK, &map, i * 128 + 64, row_a, &slot_full[slot]);
                        tma_load_2d(dst + LT_BLOCK + LT_BLOCK / 2, &map, i * 128 + 64, row_b, &slot_full[slot]);
                    }
                }
                __syncwarp();
            }
            if (ok && p.rot > 0) {
                if (ti > 0) ok = __all_sync(0xffffffffu, mbar_wait(&rot_empty, (ti - 1) & 1, &failed)) != 0;
                if (ok && lane == 0) {
                    mbar_expect_tx(&rot_full, LT_BLOCK);
                    tma_load_2d(rot_s, &map, p.rank, row_a, &rot_full);
                    tma_load_2d(rot_s + LT_BLOCK / 2, &map, p.rank, row_b, &rot_full);
                }
                __syncwarp();
            }
        }
    } else {
        // the row's queries as bfloat16, heads that are not there as zeros
        const int half = p.rot_dims / 2, pieces = q_blocks * 8;
        for (int idx = tid - 32; idx < NH * pieces; idx += LT_THREADS - 32) {
            const int r = idx / pieces, c = idx - r * pieces, f = c * 8;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.0f;
            if (r < nh) {
                const int h = h0 + r;
                if (f < p.rank) {
                    load8(p.q_lat + (size_t)h * p.ql_head + (size_t)t * p.ql_row + f, v);
                } else {
                    const __nv_bfloat16* src = p.q_raw + (size_t)t * p.qr_row + (size_t)h * p.qr_head + p.qr_off;
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        const int d = f - p.rank + e;
                        if (d >= p.rot) continue;
                        const float u = __bfloat162float(src[d]), w = __bfloat162float(src[d + 1]);       // (rot is a multiple of 8)
                        if (d < p.rot_dims) {
                            const float2 cs = *reinterpret_cast<const float2*>(p.cos_sin + ((size_t)t * half + d / 2) * 2);
                            v[e] = u * cs.x - w * cs.y; v[e + 1] = w * cs.x + u * cs.y;
                        } else { v[e] = u; v[e + 1] = w; }
                    }
                }
            }
            store8(reinterpret_cast<__nv_bfloat16*>(q_s + (size_t)(c >> 3) * NH * 128 + r * 128 + (((c ^ r) & 7) << 4)), v);
        }
        fence_proxy_async();
        lt_bar(1, LT_THREADS - 32);
    }

    if (warp == 1 || warp == 2) {
        constexpr unsigned idesc_s = instr_desc_bf16(128, NH), idesc_o = instr_desc_bf16(128, NH) | (1u << 15);      // (A M-major)
        auto wait_all = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, &failed)) != 0; };
        const unsigned ring_a = smem_u32(ring), q_a = smem_u32(q_s), p_a = smem_u32(p_s), rot_a = smem_u32(rot_s);
        int it = 0;
        if (warp == 1) {
            // -------------------------------------------------------------- scores, block by block as the rows land
            for (int ti = 0; ti < n_tiles && ok; ++ti) {
                const int b = ti & 1;
                if (ti >= 2) ok = wait_all(&s_empty[b], ((ti >> 1) - 1) & 1);
                for (int i = 0; i < pairs && ok; ++i, ++it) {
                    const int slot = it % p.slots;
                    ok = wait_all(&slot_full[slot], (it / p.slots) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const unsigned k_a = ring_a + (unsigned)slot * LT_SLOT, q_i = q_a + (unsigned)(2 * i) * (NH * 128), d = tmem + (unsigned)b * NH;
#pragma unroll
                        for (int ks = 0; ks < 4; ++ks)
                            tc_mma(d, smem_desc_sw128(k_a + ks * 32), smem_desc_sw128(q_i + ks * 32), idesc_s, (i > 0 || ks > 0) ? 1u : 0u);
                        if (2 * i + 1 < blocks) {
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                tc_mma(d, smem_desc_sw128(k_a + LT_BLOCK + ks * 32), smem_desc_sw128(q_i + NH * 128 + ks * 32), idesc_s, 1u);
                        }
                        if (i == pairs - 1 && p.rot == 0) tc_commit(&s_full[b]);
                    }
                    __syncwarp();
                }
                if (ok && p.rot > 0) {
                    ok = wait_all(&rot_full, ti & 1);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
                        for (int ks = 0; ks * 16 < p.rot; ++ks)
                            tc_mma(tmem + (unsigned)b * NH, smem_desc_sw128(rot_a + ks * 32), smem_desc_sw128(q_a + (unsigned)blocks * (NH * 128) + ks * 32),
                                   idesc_s, 1u);
                        tc_commit(&s_full[b]);
                        tc_commit(&rot_empty);
                    }
                    __syncwarp();
                }
            }
        } else {
            // -------------------------------------------------------------- values
            for (int ti = 0; ti < n_tiles && ok; ++ti) {
                ok = wait_all(&p_full, ti & 1);
                if (!ok) break;
                tc_fence_after();
                for (int i = 0; i < pairs; ++i, ++it) {
                    if (elect_one()) {
                        const int slot = it % p.slots;
                        const unsigned v_a = ring_a + (unsigned)slot * LT_SLOT;
#pragma unroll
                        for (int ks = 0; ks < LT_KEYS / 16; ++ks)
                            tc_mma(tmem + O_COL + (unsigned)(ti & 1) * O_COLS + (unsigned)i * NH, smem_desc_sw128_nmajor(v_a + ks * 2048, LT_BLOCK, 1024),
                                   smem_desc_sw128(p_a + (ks >> 2) * (NH * 128) + (ks & 3) * 32), idesc_o, ks > 0 ? 1u : 0u);
                        tc_commit(&slot_empty[slot]);
                        if (i == pairs - 1) tc_commit(&p_empty);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------------ softmax: a thread per key of the tile
        const int quarter = warp & 3, kk = quarter * 32 + lane;
        const unsigned lane_addr = (unsigned)(quarter * 32) << 16;
        float m = -INFINITY, ref = -INFINITY;            // of head `lane`, alike in the four warps: the largest score, what l and acc are relative to
        float l[NH], acc[4][NH];                         // of this thread's keys, of this thread's features
#pragma unroll
        for (int h = 0; h < NH; ++h) l[h] = acc[0][h] = acc[1][h] = acc[2][h] = acc[3][h] = 0.0f;
#pragma unroll 1
        for (int ti = 0; ti <= n_tiles; ++ti) {          // (the last time round: the last tile's results)
            const int b = ti & 1, key = k_begin + ti * LT_KEYS + kk;
            const bool tile = ti < n_tiles;
            __nv_bfloat162 w2[NH / 2];                   // the key's weights
            if (tile) {
                float s[NH];
                ok = mbar_wait(&s_full[b], (ti >> 1) & 1, &failed);
                if (!lt_all(ok)) { ok = false; break; }
                tc_fence_after();
                lt_load<NH>(tmem + lane_addr + (unsigned)b * NH, s);
                tc_fence_before();
                mbar_arrive(&s_empty[b]);
                const bool seen = key >= lo && key < k_end;
                float top = -INFINITY;
#pragma unroll
                for (int h = 0; h < NH; ++h) {
                    s[h] = seen ? s[h] * p.scale_log2 : -INFINITY;
                    const float w = lt_warp_max(s[h]);
                    if (lane == h) top = w;
                }
                wmax[b][quarter][lane] = top;
                lt_bar(2, 128);
                top = fmaxf(fmaxf(wmax[b][0][lane], wmax[b][1][lane]), fmaxf(wmax[b][2][lane], wmax[b][3][lane]));
                // the tile's own maximum; far below the largest so far its weights count for nothing, and the sums before must not overflow
                m = fmaxf(m, top);
                const float now = fmaxf(top, m - LT_FALL);
                mrow[quarter][lane] = now;
                frow[b][quarter][lane] = ref == -INFINITY ? 0.0f : lt_exp2(ref - now);
                ref = now;
                __syncwarp();
#pragma unroll
                for (int h = 0; h < NH; h += 4) {
                    const float4 r = *reinterpret_cast<const float4*>(&mrow[quarter][h]), f = *reinterpret_cast<const float4*>(&frow[b][quarter][h]);
                    w2[h / 2] = __floats2bfloat162_rn(lt_exp2(s[h] - r.x), lt_exp2(s[h + 1] - r.y));
                    w2[h / 2 + 1] = __floats2bfloat162_rn(lt_exp2(s[h + 2] - r.z), lt_exp2(s[h + 3] - r.w));
                    const float2 u = __bfloat1622float2(w2[h / 2]), v = __bfloat1622float2(w2[h / 2 + 1]);
                    l[h] = fmaf(l[h], f.x, u.x); l[h + 1] = fmaf(l[h + 1], f.y, u.y);
                    l[h + 2] = fmaf(l[h + 2], f.z, v.x); l[h + 3] = fmaf(l[h + 3], f.w, v.y);
                }
                if (ti == n_tiles - 1) {                 // rows that this request has not written (the scores have read them), side by side
                    const unsigned from = (unsigned)(k_end - k_begin - ti * LT_KEYS) * 128;
                    for (int i = 0; i < pairs; ++i) {
                        unsigned char* slot = ring + (size_t)((ti * pairs + i) % p.slots) * LT_SLOT;
                        for (unsigned o = from + kk * 16; o < LT_BLOCK; o += 128 * 16) {
                            *reinterpret_cast<uint4*>(slot + o) = make_uint4(0u, 0u, 0u, 0u);
                            *reinterpret_cast<uint4*>(slot + LT_BLOCK + o) = make_uint4(0u, 0u, 0u, 0u);
                        }
                    }
                }
            }
            if (ti > 0) {                                // the value products of the last tile are done: P and their results are this group's
                ok = mbar_wait(&p_empty, (ti - 1) & 1, &failed);
                if (!lt_all(ok)) { ok = false; break; }
                tc_fence_after();
            }
            if (tile) {
                unsigned char* pk = p_s + (kk >> 6) * (NH * 128) + (kk & 7) * 2;
#pragma unroll
                for (int h = 0; h < NH; ++h)
                    *reinterpret_cast<__nv_bfloat16*>(pk + h * 128 + (((((kk & 63) >> 3) ^ h) & 7) << 4)) = h & 1 ? w2[h / 2].y : w2[h / 2].x;
                fence_proxy_async();
                tc_fence_before();
                mbar_arrive(&p_full);                    // (this tile's results go where those of the last but one were, which were added
            }                                            // up before the last tile's weights were handed over)
            if (ti > 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i >= pairs) break;
                    float o[NH];
                    lt_load<NH>(tmem + lane_addr + O_COL + (unsigned)(b ^ 1) * O_COLS + (unsigned)i * NH, o);
#pragma unroll
                    for (int h = 0; h < NH; h += 4) {
                        const float4 f = *reinterpret_cast<const float4*>(&frow[b ^ 1][quarter][h]);
                        acc[i][h] = fmaf(acc[i][h], f.x, o[h]); acc[i][h + 1] = fmaf(acc[i][h + 1], f.y, o[h + 1]);
                        acc[i][h + 2] = fmaf(acc[i][h + 2], f.z, o[h + 2]); acc[i][h + 3] = fmaf(acc[i][h + 3], f.w, o[h + 3]);
                    }
                }
            }
            __syncwarp();                                // (mrow, and the factors of the last tile, have been read)
        }
        if (ok) {
            // l[h] over the warp: every step halves the heads that a lane still holds
#pragma unroll
            for (int w = NH / 2, o = 16; o > 0; o >>= 1, w >>= 1) {
                if (w > 0) {
#pragma unroll
                    for (int h = 0; h < w; ++h) {
                        const float mine = lane & o ? l[h + w] : l[h], other = lane & o ? l[h] : l[h + w];
                        l[h] = mine + __shfl_xor_sync(0xffffffffu, other, o);
                    }
                } else l[0] += __shfl_xor_sync(0xffffffffu, l[0], o);
            }
            if (NH == 32 || (lane & 1) == 0) lsum[quarter][NH == 32 ? lane : lane >> 1] = l[0];
            // the results through the ring, which is free: rows of a head, 16 bytes a store (and few instructions: each is fetched once a CTA)
            float* o_s = reinterpret_cast<float*>(ring);             // [NH][512]
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int h = 0; h < NH; ++h) o_s[h * 512 + i * 128 + kk] = acc[i][h];
            lt_bar(2, 128);
            if (quarter == 0 && lane < nh) {
                const size_t prow = ((size_t)t * p.H + h0 + lane) * p.max_splits + sp;
                p.part_ml[prow * 2 + 0] = ref * LT_LN2;
                p.part_ml[prow * 2 + 1] = (lsum[0][lane] + lsum[1][lane]) + (lsum[2][lane] + lsum[3][lane]);
            }
            if (kk * 4 < p.rank) {
                float* to = p.part_o + (((size_t)t * p.H + h0) * p.max_splits + sp) * p.rank + kk * 4;
#pragma unroll 4
                for (int h = 0; h < nh; ++h)
                    *reinterpret_cast<float4*>(to + (size_t)h * p.max_splits * p.rank) = *reinterpret_cast<const float4*>(o_s + h * 512 + kk * 4);
            }
            tc_fence_before();
        }
    }
    if (!ok && lane == 0) atomicExch(&failed, 1);
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    if (tid == 0 && failed && p.status) atomicOr(p.status, BG_STATUS_TIMEOUT);
}

static size_t lt_fixed_smem(int nh, int rank, int rot) {
    return 1024 + LT_BLOCK + (size_t)(rank / 64 + (rot > 0 ? 1 : 0)) * nh * 128 + (size_t)2 * nh * 128;
}
static int lt_slots(int nh, int rank, int rot) {
    const size_t limit = 227 * 1024 - 4096;              // (4 KB: barriers and the exchanges between warps)
    const size_t fixed = lt_fixed_smem(nh, rank, rot);
    if (fixed >= limit) return 0;
    const int n = (int)((limit - fixed) / LT_SLOT);
    return n < LT_MAX_SLOTS ? n : LT_MAX_SLOTS;
}

}  // namespace bg

using namespace bg;

// Whether the tcgen05 kernel takes these sizes: whole boxes of 64 features and 64 positions of a page, room for a tile and a slot more.
extern "C" int bg_latent_attention_tc_plan(int H, int rank, int rot, int page_size) {
    if (H <= 0 || rank <= 0 || rank % 64 || rank > 512 || rot < 0 || rot > 64 || rot % 8 || page_size <= 0 || page_size % 64) return BG_ERR_UNSUPPORTED;
    const int nh = H <= 16 ? 16 : 32;
    return lt_slots(nh, rank, rot) > (rank / 64 + 1) / 2 ? BG_OK : BG_ERR_UNSUPPORTED;
}

// How many ranges the row that is cut into the most of them makes, of up to `keys` keys, with `ctas` rows (times chunks of heads) on `sms` SMs:
// what a grid and partial results are sized for.
extern "C" int bg_latent_attention_tc_ranges(int ctas, int keys, int sms) {
    const int tiles = (keys + LATENT_RANGE_STEP - 1) / LATENT_RANGE_STEP;
    int most = 1;
    for (int t = 2; t <= tiles; ++t) {
        const int n = latent_ranges(t, LATENT_MAX_RANGES, ctas, sms);
        if (n > most) most = n;
    }
    return most;
}

// The arguments of bg_latent_attention_mma_partial; query blocks of one row each; a request's keys are spread over `max_splits` ranges
// as latent_range.cuh says, at most LATENT_MAX_RANGES.
extern "C" int bg_latent_attention_tc_partial(const float* q_lat, long long ql_head, int ql_row, const void* q_raw, int qr_row, int qr_head,
                                              int qr_off, const float* cos_sin, const void* pool, int num_pages, int page_size,
                                              const int* block_table, int max_pages, const int* positions, const int* qblk, int n_qblk,
                                              float* part_o, float* part_ml, int max_splits, int H, int rank, int rot, int rot_dims,
                                              int window, float scale, unsigned* status, cudaStream_t stream) {
    if (n_qblk <= 0 || max_splits <= 0) return BG_OK;
    const int rc = bg_latent_attention_tc_plan(H, rank, rot, page_size);
    if (rc != BG_OK) return rc;
    if (rot_dims > rot || (rot_dims & 1) || max_splits > LATENT_MAX_RANGES || (long long)n_qblk * ((H + 31) / 32) > (1 << 25)) return BG_ERR_SHAPE;
    if ((uintptr_t)pool % 16 || (uintptr_t)q_lat % 16 || ql_head % 4 || ql_row % 4 || (uintptr_t)cos_sin % 8) return BG_ERR_ALIGN;
    if ((long long)num_pages * page_size > 0x7fffffffLL) return BG_ERR_SHAPE;
    CUtensorMap map;
    const int mrc = make_map(&map, pool, (long long)num_pages * page_size, rank + rot, rank + rot, 64);
    if (mrc != BG_OK) return mrc;
    LtParams p;
    p.q_lat = q_lat; p.ql_head = ql_head; p.ql_row = ql_row; p.q_raw = (const __nv_bfloat16*)q_raw; p.qr_row = qr_row; p.qr_head = qr_head;
    p.qr_off = qr_off; p.cos_sin = cos_sin; p.block_table = block_table; p.max_pages = max_pages; p.num_pages = num_pages;
    p.page_size = page_size; p.positions = positions; p.qblk = qblk; p.part_o = part_o; p.part_ml = part_ml; p.max_splits = max_splits;
    p.H = H; p.rank = rank; p.rot = rot; p.rot_dims = rot_dims; p.window = window; p.scale_log2 = scale * LT_LOG2E; p.status = status;
    const int nh = H <= 16 ? 16 : 32;
    p.slots = lt_slots(nh, rank, rot);
    p.ctas = n_qblk * ((H + nh - 1) / nh); p.sms = sm_count();
    const size_t smem = lt_fixed_smem(nh, rank, rot) + (size_t)p.slots * LT_SLOT;
    const dim3 grid(n_qblk, (H + nh - 1) / nh, max_splits);
#define BG_LT_LAUNCH(NH)                                                                                                   \
    do {                                                                                                                   \
        cudaError_t e = cudaFuncSetAttribute(latent_attention_tc_kernel<NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        if (e != cudaSuccess) return (int)e;                                                                               \
        launch(latent_attention_tc_kernel<NH>, grid, dim3(LT_THREADS), smem, stream, map, p);                              \
    } while (0)
    if (nh == 16) BG_LT_LAUNCH(16);
    else BG_LT_LAUNCH(32);
#undef BG_LT_LAUNCH
    BG_LAUNCH_CHECK();
    return BG_OK;
}
