// The float product C[M, N] (+)= A[M, K] W[N, K]^T (+ bias) on the tensor cores, for inner sizes above those of gemm_f32.cu's own kernel.
//
// Every operand is cut into three bfloat16 numbers, x = h + m + l exactly, and of the nine products of the parts of two floats the six are made
// that are not below 2^-24 of theirs (m l, l m and l l are left out; one with a single bit set times any float is exact).  64 of k are one
// stage: its five kinds of small products go into an accumulator in tensor memory first, so that their sums are not cut off at the size of
// the large ones, then h h; the stage's sum leaves tensor memory and is added to the range's in float, rounded to nearest.  (An
// accumulator cuts off instead of rounding, always towards nought: four MMAs on a large sum are four such cuts.)  Ranges of k lie at places that
// follow from N and K alone (gt_range); their sums are added in order, then the bias.  None of this depends on the number of rows, on
// tiles or on who adds the ranges, so a row's result does not depend on how many other rows the call has: all forms here give the
// same bits.
//
// Error against 64 bits (2-norm, normal operands), two chains of float multiply-adds over 1,024 of k in brackets: K of 192 0.85e-7 (1.8e-7),
// 1,536 1.0e-7 (3.7e-7), 9,000 1.3e-7 (4.1e-7).  It is smaller for dense rows and larger for those of few terms, whose chains have few
// roundings: one term in a row 4.5e-8 (2.5e-8), four 5.6e-8 (4.2e-8), sixteen 6.3e-8 (6.1e-8), 64 7.0e-8 (1.07e-7).  And sums of one sign lean
// towards nought, by 0.6 (one term) to 1.4 (dense) x 2^-24 of themselves, where the chains' do not lean.
//
// Operands are cut times 2^24 (GT_UP) and sums are scaled back, so that small ones keep their parts.  A range's sum that is not finite (an operand
// that is infinite, not a number or above some 2^103, or a sum above some 2^80) is made by floats instead, in two chains (even and odd k), which makes of
// it what floats make.  That, too, depends on the output's own row and column only.  550 x 1,536 with k of 8,960: 103 us, with an infinity in one
// row 180, with NaN in every row 2,510.  (Small operands noticed where they are cut and summed by floats: 1,900 us with one weight of 1e-36, 510 with one
// in a row of tokens, 30,000 with one in every row.)
//
// The weights' rows are the M side (128 a CTA), so a lane of tensor memory is an output feature and results leave in rows of 128 bytes;
// the tokens are the N side (NT = 16 to 160).  Weights come as floats (TMA, two boxes of 128 rows x 32 of k a stage); a warpgroup or
// several read them, a row a lane, cut them and put the parts into tensor memory (`tcgen05.st`) as left operands: they never return to
// shared memory, whose bandwidth the right operands need.  The tokens' parts are made once by gf_parts_kernel and come by bulk copies
// (the weights' tiles would each make them again).  Other warpgroups add up the stages' sums.
//
// What bounds it: with 144 and 160 tokens the tensor cores (a stage of 160 tokens takes 1,980 cycles, its MMAs 1,920; with 32 of k a stage, one
// warp that issued and one set of warps that cut and added it was 5,000), with fewer the instructions of the cut (some 12 a value:
// weights at 4.6 TB/s for 8 rows).  In us, the float units' kernels in brackets: 550 x 17,920 with k of 1,536 142 (930),
// 550 x 1,536 with 8,960 103 (498), 64 x 17,920 with 1,536 34 (116), 8 x 17,920 24 to 26 (31), 1 x 2,048 with 768 8.0 (13.2).
#include "gemm_f32.cuh"
#include "float_parts.cuh"

namespace bg {

constexpr int GT_BM = 128, GT_BK = 64;     // output features of a CTA; k of a stage
constexpr unsigned GT_W_BYTES = GT_BM * GT_BK * 4;
// Tokens and weights are cut times 2^24: no float is so small then that its parts are not exact (the smallest bit of any is 2^-125); what is
// infinite, not a number or above some 2^103 has parts that are not numbers, which every sum that they enter shows.
constexpr float GT_UP = 16777216.0f;
constexpr long long GT_SCRATCH = 32 << 20; // floats that a call's scratch may take
// Warpgroups: those that cut the weights, those that add the stages' sums, one for copies, MMAs and tokens.
constexpr int gt_threads(int gc, int gd) { return (gc + gd + 1) * 128; }

struct GtParams {
    const float* A; const float* W; const float* bias; float* C;
    float* part;                           // [ranges][batch][M][N]: a CTA has one range and leaves its sums here; or null: it walks them all
    float* run;                            // where a walk keeps the ranges' sum so far, [batch][M] rows of ldr
    const unsigned char* images;           // the tokens' parts (gf_parts_kernel)
    long long batch_a, batch_w, batch_c, batch_r;
    int lda, ldw, ldc, ldr, M, N, K, accumulate, range_len, ranges, r0, r1, batch, tok_tiles, feat_tiles, units, map_batch;      // (ranges: of all k; r0 to r1: of this launch)
    unsigned* status;
};

// The tokens' parts as the images of the stages' right operands, [batch][tile of nt tokens][stage][part][token][64 of k] with the swizzle of
// shared memory, noughts behind the last token and behind K.  One part of a stage is then one copy of contiguous bytes: boxes of a tensor map, 64 bytes a row, took the copy engine 2.4 cycles a row, 1,750 for 32 of k of 192 tokens.
// A CTA (or gridDim.y of them) per row, a warp per 512 of k, 16 values a lane.
template <bool VEC>
__global__ void __launch_bounds__(256) gf_parts_kernel(GtParams p, unsigned char* images, int nt) {
    pdl_launch();
    const int padded = p.tok_tiles * nt, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int k_first = p.r0 * p.range_len, k_all = min(p.K, p.r1 * p.range_len) - k_first, stages = (k_all + GT_BK - 1) / GT_BK;
    const int b = blockIdx.x / padded, m = blockIdx.x - b * padded, in = m % nt, most = m < p.M ? k_all : 0;
    const float* src = p.A + (size_t)b * p.batch_a + (size_t)m * p.lda + k_first;
    unsigned char* tile = images + ((size_t)b * p.tok_tiles + m / nt) * stages * 3 * nt * 128 + in * 128 + (((lane >> 1 & 7) ^ (in & 7)) << 4) + (lane & 1) * 8;
    pdl_wait();
    for (int k0 = ((int)blockIdx.y * (blockDim.x / 32) + warp) * 512; k0 < stages * GT_BK; k0 += gridDim.y * (blockDim.x / 32) * 512) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + i * 128 + lane * 4;
            if constexpr (VEC) v[i] = k < most ? *reinterpret_cast<const float4*>(src + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            else v[i] = make_float4(k < most ? src[k] : 0.0f, k + 1 < most ? src[k + 1] : 0.0f, k + 2 < most ? src[k + 2] : 0.0f, k + 3 < most ? src[k + 3] : 0.0f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int stage = (k0 + i * 128) / GT_BK + (lane >> 4);
            uint2 h, q, l;
            gt_split(gt_up(pair2(v[i].x, v[i].y), GT_UP), h.x, q.x, l.x);
            gt_split(gt_up(pair2(v[i].z, v[i].w), GT_UP), h.y, q.y, l.y);
            if (stage < stages) {
                unsigned char* d = tile + (size_t)stage * 3 * nt * 128;
                *reinterpret_cast<uint2*>(d) = h;
                *reinterpret_cast<uint2*>(d + (size_t)nt * 128) = q;
                *reinterpret_cast<uint2*>(d + (size_t)nt * 256) = l;
            }
        }
    }
}

// `bytes` contiguous ones (a multiple of 16, both sides on 16 bytes)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
// Two chains of multiply-adds over n of k (the even and the odd ones), and their sum.
__device__ __forceinline__ float gt_chain(const float* a, const float* w, int n) {
    unsigned long long sum = 0ull;
    int k = 0;
    if ((((uintptr_t)a | (uintptr_t)w) & 15) == 0) {
#pragma unroll 8
        for (; k + 3 < n; k += 4) {
            const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(a + k), y = *reinterpret_cast<const ulonglong2*>(w + k);
            sum = fma2(x.y, y.y, fma2(x.x, y.x, sum));
        }
    }
#pragma unroll 8
    for (; k + 1 < n; k += 2) sum = fma2(pair2(a[k], a[k + 1]), pair2(w[k], w[k + 1]), sum);
    if (k < n) sum = fma2(pair2(a[k], 0.0f), pair2(w[k], 0.0f), sum);
    return sum2(sum);
}

// What a form of the kernel takes: tokens NT; warpgroups that cut (GC: 64 / GC of a stage's k each) and that add (GD: NT / GD columns each);
// stages whose parts (DA) and sums (DS) tensor memory holds, of weights (WS) and tokens (BS) in shared memory; registers of a thread
// at launch, of one that cuts, that adds, and of the others: their sum over the warpgroups is not above the launch's.
template <int NT_, int GC_, int GD_, int DA_, int DS_, int WS_, int BS_, int REGS_, int RC_, int RD_, int RO_>
struct GtForm {
    static constexpr int NT = NT_, GC = GC_, GD = GD_, DA = DA_, DS = DS_, WS = WS_, BS = BS_, REGS = REGS_, RC = RC_, RD = RD_, RO = RO_;
    static_assert(GC * RC + GD * RD + RO <= (GC + GD + 1) * REGS);
};

template <typename F, bool DIRECT>
__global__ void __launch_bounds__(gt_threads(F::GC, F::GD), 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, GtParams p) {
    constexpr int NT = F::NT, GC = F::GC, GD = F::GD, DA = F::DA, DS = F::DS, WS = F::WS, BS = F::BS;
    constexpr int CG = NT / GD, KG = GT_BK / GC, ADDERS = 128 * GD;
    constexpr unsigned PLANE = NT * 128, B_BYTES = 3 * PLANE;
    constexpr unsigned PARTS0 = DS * NT, WANT = PARTS0 + DA * 96, COLS = 512;
    static_assert(WANT <= 512 && CG % 8 == 0 && KG % 8 == 0);
    extern __shared__ unsigned char gt_raw[];
    unsigned char* wt = (unsigned char*)(((uintptr_t)gt_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* bt = wt + WS * GT_W_BYTES;
    __shared__ __align__(8) unsigned long long w_full[WS], w_empty[WS], b_full[BS * 3], b_empty[BS * 3], a_full[DA], a_empty[DA], done[DS], sum_empty[DS];
    __shared__ unsigned tmem_sh;
    __shared__ int failed;

    constexpr int W_WARP = 4 * (GC + GD), MMA_WARP = W_WARP + 1, TOKEN_WARP = W_WARP + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, STAGES = p.range_len / GT_BK;
    // The CTA's units, blockIdx.x + i gridDim.x: a tile of tokens (they vary fastest: the weights' tile is in the second-level cache) and of
    // features over one range of k, or all of them.  Every role walks them with a count of stages of its own, so copies, cuts and MMAs of a
    // unit go on while the one before is added and stored.
    struct Unit { int t0, n0, b, range, k_begin, k_end, n, tok; };
    auto unit_of = [&](int u) {
        Unit x;
        x.tok = u % p.tok_tiles; u /= p.tok_tiles;
        const int cuts = p.part ? p.r1 - p.r0 : 1, cut = u % cuts; u /= cuts;
        x.n0 = u % p.feat_tiles * GT_BM;
        x.b = u / p.feat_tiles;
        x.t0 = x.tok * NT;
        x.range = p.r0 + cut;
        x.k_begin = x.range * p.range_len;
        x.k_end = min(p.K, (p.part ? x.range + 1 : p.r1) * p.range_len);
        x.n = (x.k_end - x.k_begin + GT_BK - 1) / GT_BK;
        return x;
    };

    if (threadIdx.x == 0) {
        for (int i = 0; i < WS; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 4 * GC); }
        for (int i = 0; i < BS * 3; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < DA; ++i) { mbar_init(&a_full[i], 4 * GC); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < DS; ++i) { mbar_init(&done[i], 1); mbar_init(&sum_empty[i], 4 * GD); }
        failed = 0;
        mbar_init_fence();
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_sh)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_launch();                                              // (the columns are held)
    const unsigned tmem = tmem_sh;

    if (warp >= W_WARP) gt_regs<F::REGS, F::RO>();
    if (warp == W_WARP) {
        // ---------------- the weights' copies
        if (lane == 0 && !DIRECT) {
            // (for few rows the weights depend on no kernel of the step, as in the other products of few rows)
            if (NT > 16) pdl_wait();
            bool ok = true;
            for (int u = blockIdx.x, g = 0; u < p.units && ok; u += gridDim.x) {
                const Unit x = unit_of(u);
                for (int s = 0; s < x.n; ++s, ++g) {
                    if (g >= WS && !(ok = mbar_wait(&w_empty[g % WS], (g / WS - 1) & 1, &failed))) break;
                    mbar_expect_tx(&w_full[g % WS], GT_W_BYTES);
#pragma unroll
                    for (int q = 0; q < 2; ++q)        // (boxes of 32 columns; one that begins behind K brings noughts)
                        tma_load_3d(wt + (g % WS) * GT_W_BYTES + q * (GT_W_BYTES / 2), &map_w, x.k_begin + s * GT_BK + q * 32, x.n0, p.map_batch ? x.b : 0, &w_full[g % WS]);
                }
            }
        }
    } else if (warp == MMA_WARP || warp == MMA_WARP + 2) {
        // ---------------- the MMAs: two warps in turns, so that one's waits (some 130 cycles each, ready or not) lie under the other's MMAs.
        // The tokens' third parts are needed for the first sixth of a stage only, the second ones up to its half, the first ones from there
        // on: each is copied by itself, under the stage's other products.
        constexpr unsigned idesc = instr_desc_bf16(GT_BM, NT);
        bool ok = true;
        for (int u = blockIdx.x, g = 0; u < p.units && ok; u += gridDim.x) {
            const int to = g + unit_of(u).n;
            for (; g < to && ok; ++g) {
                if ((g & 1) != (warp == MMA_WARP ? 0 : 1)) continue;
                const int d = g % DS, o = g % DA, i = g % BS;
                ok = g < DS || mbar_wait(&sum_empty[d], (g / DS - 1) & 1, &failed);
                ok = ok && mbar_wait(&a_full[o], (g / DA) & 1, &failed);
                const unsigned acc = tmem + d * NT, a = tmem + PARTS0 + o * 96, bb = smem_u32(bt + i * B_BYTES);
#pragma unroll
                for (int q = 2; q >= 0; --q) {
                    ok = ok && mbar_wait(&b_full[i * 3 + q], (g / BS) & 1, &failed);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {
#pragma unroll
                        for (int e = 2 - q; e >= 0; --e)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                tc_mma_ts(acc, a + e * 32 + j * 8, smem_desc_sw128(bb + q * PLANE + j * 32), idesc, q < 2 || j ? 1u : 0u);
                        tc_commit(&b_empty[i * 3 + q]);
                        if (q == 0) {
                            tc_commit(&done[d]);
                            tc_commit(&a_empty[o]);
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp == TOKEN_WARP) {
        // ---------------- the copies of the tokens' parts
        if (lane == 0) {
            const int stages = (min(p.K, p.r1 * p.range_len) - p.r0 * p.range_len + GT_BK - 1) / GT_BK;
            pdl_wait();
            bool ok = true;
            for (int u = blockIdx.x, g = 0; u < p.units && ok; u += gridDim.x) {
                const Unit x = unit_of(u);
                const unsigned char* src = p.images + (((size_t)x.b * p.tok_tiles + x.tok) * stages + (x.k_begin - p.r0 * p.range_len) / GT_BK) * B_BYTES;
                for (int s = 0; s < x.n && ok; ++s, ++g)
#pragma unroll
                    for (int q = 2; q >= 0; --q) {
                        const int i = g % BS * 3 + q;
                        if (g >= BS && !(ok = mbar_wait(&b_empty[i], (g / BS - 1) & 1, &failed))) break;
                        mbar_expect_tx(&b_full[i], PLANE);
                        bulk_load(bt + g % BS * B_BYTES + q * PLANE, src + (size_t)s * B_BYTES + q * PLANE, PLANE, &b_full[i]);
                    }
            }
        }
    } else if (warp < 4 * GC) {
        // ---------------- weights into parts, a row a lane
        gt_regs<F::REGS, F::RC>();
        const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane;
        const unsigned parts = tmem + ((unsigned)(quarter * 32) << 16) + PARTS0 + group * (KG / 2);
        unsigned long long v[KG / 2];
        auto fetch = [&](int g) {
            mbar_wait(&w_full[g % WS], (g / WS) & 1, &failed);
            const unsigned char* src = wt + (g % WS) * GT_W_BYTES + group * KG / 32 * (GT_W_BYTES / 2) + row * 128;
#pragma unroll
            for (int i = 0; i < KG / 4; ++i) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(src + (((group * (KG / 4) % 8 + i) ^ (row & 7)) << 4));
                v[2 * i] = x.x; v[2 * i + 1] = x.y;
            }
        };
        if (DIRECT) pdl_wait();
        if (!DIRECT && (int)blockIdx.x < p.units) fetch(0);
        for (int u = blockIdx.x, g = 0; u < p.units; u += gridDim.x) {
            const Unit x = unit_of(u);
#pragma unroll 1
            for (int s = 0; s < x.n; ++s, ++g) {
                if constexpr (DIRECT) {
                    const int k = x.k_begin + s * GT_BK + group * KG;
                    const bool in = x.n0 + row < p.N;
                    const float* w_row = p.W + (size_t)x.b * p.batch_w + (size_t)(in ? x.n0 + row : 0) * p.ldw;
#pragma unroll
                    for (int i = 0; i < KG / 2; ++i)
                        v[i] = pair2(in && k + 2 * i < x.k_end ? w_row[k + 2 * i] : 0.0f, in && k + 2 * i + 1 < x.k_end ? w_row[k + 2 * i + 1] : 0.0f);
                }
                // (what the registers hold is cut before the wait for room)
                constexpr int AHEAD = 2;
                unsigned h[AHEAD][4], m[AHEAD][4], l[AHEAD][4];
                // (packed or one by one: 550 x 17,920 with k of 1,536 143.4 and 145.2 us; sixteen products of 8 x 512 with 256 8.0 and 7.3)
                auto cut = [&](int c, int to) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const unsigned long long x = v[4 * c + i];
                        gt_split(GC == 2 ? fma2(x, pair2(GT_UP, GT_UP), 0ull) : gt_up(x, GT_UP), h[to][i], m[to][i], l[to][i]);
                    }
                };
                const unsigned a = parts + g % DA * 96;
                auto put = [&](int c, int from) { gt_st4(a + 4 * c, h[from]); gt_st4(a + 32 + 4 * c, m[from]); gt_st4(a + 64 + 4 * c, l[from]); };
#pragma unroll
                for (int c = 0; c < AHEAD; ++c) cut(c, c);
                if (g >= DA) {                                 // (the products of stage g - DA have read its parts)
                    mbar_wait(&a_empty[g % DA], (g / DA - 1) & 1, &failed);
                    __syncwarp();
                    tc_fence_after();
                }
#pragma unroll
                for (int c = 0; c < AHEAD; ++c) put(c, c);
#pragma unroll
                for (int c = AHEAD; c < KG / 8; ++c) { cut(c, c % AHEAD); put(c, c % AHEAD); }
                __syncwarp();
                if (lane == 0 && !DIRECT) mbar_arrive(&w_empty[g % WS]);
                const bool more = s + 1 < x.n;
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[g % DA]);
                if (!DIRECT && (more || u + (int)gridDim.x < p.units)) fetch(g + 1);
            }
        }
    } else if (warp < W_WARP) {
        // ---------------- the stages' sums
        gt_regs<F::REGS, F::RD>();
        const int quarter = warp & 3, group = (warp >> 2) - GC, row = quarter * 32 + lane;
        const unsigned sums = tmem + ((unsigned)(quarter * 32) << 16) + group * CG;
        unsigned long long total[CG / 2];
        pdl_wait();
        for (int u = blockIdx.x, g = 0; u < p.units; u += gridDim.x) {
          const Unit x = unit_of(u);
          const int t0 = x.t0, b = x.b, n = x.n, feature = x.n0 + row;
#pragma unroll 1
          for (int e = 0; e < n; ++e, ++g) {
            const bool first = e % STAGES == 0, last = (e + 1) % STAGES == 0 || e + 1 == n;
            const unsigned acc = sums + g % DS * NT;
            mbar_wait(&done[g % DS], (g / DS) & 1, &failed);
            __syncwarp();                                      // (the loads of tensor memory want the whole warp: not all lanes store a range's sums)
            tc_fence_after();
            auto add = [&](int c, const unsigned* r, int count) {
#pragma unroll
                for (int j = 0; j < count / 2; ++j) {
                    const unsigned long long one = (unsigned long long)r[2 * j] | ((unsigned long long)r[2 * j + 1] << 32);
                    total[c / 2 + j] = first ? one : gt_add2(total[c / 2 + j], one);
                }
            };
            constexpr int STEP = CG >= 64 && GC == 4 ? 16 : 32, WHOLE = CG / STEP * STEP;
#pragma unroll
            for (int c = 0; c < WHOLE; c += STEP) {
                unsigned r[STEP];
                if constexpr (STEP == 32) tc_ld32_nowait(acc + c, r);
                else gt_ld16(acc + c, r);
                tc_wait_ld();
                add(c, r, STEP);
            }
            if constexpr (CG - WHOLE >= 16) { unsigned r[16]; gt_ld16(acc + WHOLE, r); tc_wait_ld(); add(WHOLE, r, 16); }
            if constexpr (CG % 16 == 8) { unsigned r[8]; gt_ld8(acc + CG - 8, r); tc_wait_ld(); add(CG - 8, r, 8); }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[g % DS]);
            if (!last) continue;
            // ---- the sums of a range
            const int range = x.range + e / STAGES;
            unsigned long long nought = 0ull;                  // not nought if a sum is not finite
#pragma unroll
            for (int j = 0; j < CG / 2; ++j) {
                nought = fma2(total[j], 0ull, nought);
                total[j] = gt_up(total[j], 1.0f / GT_UP / GT_UP);
            }
            const bool lost = *(volatile int*)&failed != 0;    // (a wait ran out)
            if (!(sum2(nought) == 0.0f) || lost) {
                const int kr = range * p.range_len, nr = min(p.K - kr, p.range_len);
                const float* w_row = p.W + (size_t)b * p.batch_w + (size_t)(feature < p.N ? feature : 0) * p.ldw;
#pragma unroll 1
                for (int c = 0; c < CG; ++c) {
                    const int t = t0 + group * CG + c;
                    if (t >= p.M) break;
                    float y = 0.0f;
#pragma unroll
                    for (int j = 0; j < CG; ++j) y = j == c ? (j & 1 ? high2(total[j / 2]) : low2(total[j / 2])) : y;
                    if (feature < p.N && !(fabsf(y) <= 3.402823466e38f)) y = gt_chain(p.A + (size_t)b * p.batch_a + (size_t)t * p.lda + kr, w_row + kr, nr);
                    if (lost) y = __uint_as_float(0x7fffffffu);
#pragma unroll
                    for (int j = 0; j < CG; ++j)
                        if (j == c) total[j / 2] = j & 1 ? pair2(low2(total[j / 2]), y) : pair2(y, high2(total[j / 2]));
                }
            }
            if (feature < p.N) {
                const int rows = min(CG, p.M - t0 - group * CG);
                const bool end = !p.part && range + 1 == p.ranges, sums_before = !p.part && range > 0, add_old = end && p.accumulate;
                const size_t at = (size_t)(t0 + group * CG);
                float* run = p.run + (size_t)b * p.batch_r + at * p.ldr + feature;
                float* out = p.part ? p.part + (((size_t)range * p.batch + b) * p.M + at) * p.N + feature : end ? p.C + (size_t)b * p.batch_c + at * p.ldc + feature : run;
                size_t step = p.part ? p.N : end ? p.ldc : p.ldr, step_r = p.ldr;
                const float bias = end && p.bias ? p.bias[feature] : 0.0f;
#pragma unroll
                for (int j0 = 0; j0 < CG; j0 += 8) {           // (eight loads on their way at a time)
                    asm volatile("" : "+l"(run), "+l"(out), "+l"(step), "+l"(step_r));         // (no address is made ahead and kept)
                    float y[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) y[j] = j & 1 ? high2(total[(j0 + j) / 2]) : low2(total[(j0 + j) / 2]);
                    if (sums_before) {
                        float old[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) old[j] = j0 + j < rows ? run[j * step_r] : 0.0f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) y[j] = old[j] + y[j];
                    }
                    if (end && p.bias) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) y[j] += bias;
                    }
                    if (add_old) {
                        float old[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) old[j] = j0 + j < rows ? out[j * step] : 0.0f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) y[j] = old[j] + y[j];
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (j0 + j < rows) out[j * step] = y[j];
                    run += 8 * step_r;
                    out += 8 * step;
                }
            }
            __syncwarp();
          }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(COLS) : "memory");
    }
    if (threadIdx.x == 0 && failed && p.status) atomicOr(p.status, BG_STATUS_TIMEOUT);
}

// C = (old C +) ((part 0 + part 1) + ...) (+ bias), a thread per output or, where rows are whole 16-byte pieces (V = 4), per four neighbours: the
// parts' bytes at 16 a load, a thread's place by a 32-bit division (a piece's scratch is at most 128 MB).
// With one output a thread and a 64-bit division: 550 x 1,536 over three ranges 11.0 us, now 5.2; over twelve 14.9, now 8.4; eight rows 3.4 (level).
constexpr int GR_THREADS = 64;             // (few rows: as many SMs as there are blocks)
template <int V>
__global__ void __launch_bounds__(GR_THREADS) gemm_f32_ranges_kernel(GtParams p) {
    using Piece = typename std::conditional<V == 4, float4, float>::type;
    pdl_launch();
    const size_t total = (size_t)p.M * p.N, step = total * p.batch / V;
    const unsigned e = blockIdx.x * GR_THREADS + threadIdx.x, wide = (unsigned)(p.N / V);
    const unsigned m = e / wide, n = (e - m * wide) * V;
    pdl_wait();
    if (e >= (unsigned)(total / V)) return;
    const Piece* s = reinterpret_cast<const Piece*>(p.part + (size_t)blockIdx.y * total) + e;
    auto add = [](float* v, const Piece& x) {
        if constexpr (V == 4) { v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w; } else v[0] += x;
    };
    float v[V];
    {
        const Piece x = s[0];
        if constexpr (V == 4) { v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; } else v[0] = x;
    }
    for (int r0 = 1; r0 < p.ranges; r0 += 8) {             // eight loads on their way at a time
        Piece a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (r0 + u < p.ranges) a[u] = s[(size_t)(r0 + u) * step];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (r0 + u < p.ranges) add(v, a[u]);
    }
#pragma unroll
    for (int i = 0; i < V; ++i)
        if (p.bias) v[i] += p.bias[n + i];
    Piece* c = reinterpret_cast<Piece*>(p.C + (size_t)blockIdx.y * p.batch_c + (size_t)m * p.ldc + n);
    if constexpr (V == 4) {
        const float4 o = p.accumulate ? *c : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        *c = p.accumulate ? make_float4(o.x + v[0], o.y + v[1], o.z + v[2], o.w + v[3]) : make_float4(v[0], v[1], v[2], v[3]);
    } else {
        *c = p.accumulate ? *c + v[0] : v[0];
    }
}

// ------------------------------------------------------------------------------------------------ host
// How a call is cut: tiles of nt tokens; pieces of `rows` rows of `batches` products (and, for very long k, of `at_once` ranges) whose scratch
// fits; the ranges to units of their own or not.
struct GtPlan { int nt, rows, batches, range_len, ranges, at_once; bool cut; };

// The length of a range.  It depends on the product's own sizes only: as many ranges as give few rows a unit for each of the device's 148
// SMs, of 512 of k at the least (256 up to 1,024 of k; 8,192 at the most); a product whose features alone do that is summed in one.
static int gt_range(int N, int K) {
    const int tiles = (N + GT_BM - 1) / GT_BM;
    int ranges = (148 + tiles / 2) / tiles;
    const int least = K > 1024 ? 512 : 256;
    if (ranges > (K + least - 1) / least) ranges = (K + least - 1) / least;
    if (ranges < (K + 8191) / 8192) ranges = (K + 8191) / 8192;
    return ((K + ranges - 1) / ranges + GT_BK - 1) / GT_BK * GT_BK;
}

// Cycles of a call, roughly, from those that a stage of each form was seen to take with most SMs at it: up to 96 tokens a stage waits for its bytes
// (weights as floats and the tokens' parts, some 23 a cycle and SM), above for the tensor cores at the clock that their power leaves.  The sums of
// ranges pass through memory.  In us, planned by 1,000 cycles a stage or the tensor cores' if that is more, and by these: 550 x 1,536 with k of
// 1,536 33.4 and 29.3, 550 x 1,536 with 8,960 111 and 102, 424 x 3,136 with 3,072 77.7 and 71.6, 200 x 8,192 with 2,048 56.5 and 52.4,
// 128 x 4,096 with 4,096 51.2 and 48.0.
static double gt_stage(int nt) { return nt <= 16 ? 1430.0 : nt <= 32 ? 1900.0 : nt <= 64 ? 2250.0 : nt <= 96 ? 2650.0 : nt <= 128 ? 3000.0 : nt <= 144 ? 2750.0 : 2950.0; }
static double gt_cost(int M, int N, int K, int batch, int range_len, int ranges, int nt, bool cut) {
    const long long slots = sm_count(), units = (long long)((M + nt - 1) / nt) * ((N + GT_BM - 1) / GT_BM) * batch * (cut ? ranges : 1);
    const double stages = (double)((cut ? range_len : K) + GT_BK - 1) / GT_BK;
    const double rounds = (double)((units + slots - 1) / slots);
    return 2000.0 + rounds * (stages * gt_stage(nt) + 600.0 + (cut ? 0 : 20.0 * nt * (ranges - 1))) + (cut ? 5000.0 + 8.0 * M * N * ranges * batch / 2500.0 : 0.0);
}

static GtPlan gt_plan(int M, int N, int K, int batch) {
    GtPlan g;
    g.range_len = gt_range(N, K);
    g.ranges = g.at_once = (K + g.range_len - 1) / g.range_len;
    double best = 0.0;
    g.nt = 0;
    for (int nt : {16, 32, 64, 96, 128, 144, 160}) {
        if (nt == 16 && M > 16) continue;
        for (int cut = 0; cut < (g.ranges > 1 ? 2 : 1); ++cut) {
            const double c = gt_cost(M, N, K, batch, g.range_len, g.ranges, nt, cut);
            if (g.nt == 0 || c < best) { best = c; g.nt = nt; g.cut = cut; }
        }
    }
    const long long part = (long long)g.ranges * N, all = (M + g.nt - 1) / g.nt * (long long)g.nt, token = (long long)g.range_len * 3 / 2;
    if (g.cut && all * token * g.ranges + M * part > GT_SCRATCH) g.cut = false;
    const long long each = all * token * g.ranges + (g.cut ? M * part : 0), tile = g.nt * token * g.ranges;
    g.rows = M;
    g.batches = batch;
    if (each > GT_SCRATCH) {                               // (never a cut one: the tokens' parts)
        g.batches = 1;
        g.rows = (int)(GT_SCRATCH / tile * g.nt);
        if (g.rows == 0) {
            g.rows = g.nt;
            g.at_once = (int)(GT_SCRATCH / (g.nt * token));
            if (g.at_once < 1) g.at_once = 1;
        }
    } else if (GT_SCRATCH / each < batch) g.batches = (int)(GT_SCRATCH / each);
    return g;
}
static long long gt_token_floats(const GtPlan& g, long long padded, int ranges) { return padded * ranges * (g.range_len * 3 / 2); }
long long gt_scratch(int M, int N, int K, int batch) {
    const GtPlan g = gt_plan(M, N, K, batch);
    const long long padded = (long long)(g.rows + g.nt - 1) / g.nt * g.nt * g.batches;
    return gt_token_floats(g, padded, g.at_once) + (g.cut ? (long long)g.rows * g.batches * g.ranges * N : 0);
}

// A batch of float matrices, boxes of 32 columns x 128 rows.
static int gt_weight_map(CUtensorMap* map, const GfParams& p, int batch) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return BG_ERR_UNSUPPORTED;
    const long long apart = batch > 1 ? p.batch_w : (long long)p.N * p.ldw;
    cuuint64_t dims[3] = {(cuuint64_t)p.K, (cuuint64_t)p.N, (cuuint64_t)batch};
    cuuint64_t strides[2] = {(cuuint64_t)p.ldw * 4, (cuuint64_t)apart * 4};
    cuuint32_t box[3] = {32u, (cuuint32_t)GT_BM, 1u}, elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p.W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? BG_OK : BG_ERR_SHAPE;
}
template <typename F>
static cudaError_t gt_launch(const CUtensorMap& mw, const GtParams& p, bool direct, cudaStream_t stream) {
    constexpr size_t smem = (size_t)F::WS * GT_W_BYTES + (size_t)F::BS * 3 * F::NT * 128 + 1024;
    static_assert(smem + 5 * 1024 <= 227 * 1024);
    auto kern = direct ? gemm_f32_tc_kernel<F, true> : gemm_f32_tc_kernel<F, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    static const bool fits = F::RC == F::REGS && F::RD == F::REGS && F::RO == F::REGS ? true : [] {      // (the split of the registers counts on as many at launch)
        cudaFuncAttributes a, b;
        return cudaFuncGetAttributes(&a, gemm_f32_tc_kernel<F, true>) == cudaSuccess && cudaFuncGetAttributes(&b, gemm_f32_tc_kernel<F, false>) == cudaSuccess &&
               a.numRegs >= F::REGS && b.numRegs >= F::REGS;
    }();
    if (!fits) return cudaErrorInvalidConfiguration;
    const int slots = sm_count();
    const dim3 grid(p.units < slots ? p.units : slots);
    return launch(kern, grid, dim3(gt_threads(F::GC, F::GD)), smem, stream, mw, p);
}

static int gt_piece(const GfParams& f, const GtPlan& g, int r0, int r1, cudaStream_t stream) {
    GtParams p = {};
    p.A = f.A; p.W = f.W; p.bias = f.bias; p.C = f.C; p.batch_a = f.batch_a; p.batch_w = f.batch_w; p.batch_c = f.batch_c;
    p.lda = f.lda; p.ldw = f.ldw; p.ldc = f.ldc; p.M = f.M; p.N = f.N; p.K = f.K; p.accumulate = f.accumulate; p.batch = f.batch;
    p.range_len = g.range_len; p.ranges = g.ranges; p.r0 = r0; p.r1 = r1; p.status = f.status;
    p.tok_tiles = (f.M + g.nt - 1) / g.nt;
    // (Weights off 16 bytes are read value by value, a row a lane.  In us, by 4-byte asynchronous copies on the float units in brackets:
    // 1 x 768 with k of 201 11.6 (16.1), 8 x 2,048 with 513 11.8 (38.4), 8 x 8,192 with 1,537 36.6 (76), 64 x 2,048 36.3 (78), 550 x 4,096 104 (281).)
    const bool direct = !(f.ldw % 4 == 0 && f.batch_w % 4 == 0 && (uintptr_t)f.W % 16 == 0);
    p.map_batch = f.batch > 1 && f.batch_w != 0;
    CUtensorMap mw = {};
    if (!direct) {
        const int rc = gt_weight_map(&mw, f, p.map_batch ? f.batch : 1);
        if (rc != BG_OK) return rc;
    }
    const long long padded = (long long)p.tok_tiles * g.nt * f.batch;
    unsigned char* images = (unsigned char*)f.scratch;
    float* behind = f.scratch + gt_token_floats(g, padded, g.at_once);         // (the running sums stay in one place from launch to launch)
    p.images = images;
    p.feat_tiles = (f.N + GT_BM - 1) / GT_BM;
    const long long units = (long long)p.tok_tiles * p.feat_tiles * f.batch * (g.cut ? r1 - r0 : 1);
    if (units > 0x3fffffff) return BG_ERR_SHAPE;
    p.units = (int)units;
    const bool vec = f.K % 4 == 0 && f.lda % 4 == 0 && f.batch_a % 4 == 0 && (uintptr_t)f.A % 16 == 0 && p.r0 * (long long)g.range_len % 4 == 0;
    // (a row's pieces of 512 go to more CTAs where the rows leave SMs idle)
    const int pieces = ((r1 - r0) * g.range_len + 511) / 512, threads = 32 * (pieces < 8 ? pieces : 8), slices = padded <= 64 ? (pieces + 7) / 8 : 1;
    cudaError_t e = vec ? launch(gf_parts_kernel<true>, dim3((unsigned)padded, slices), dim3(threads), 0, stream, p, images, g.nt)
                        : launch(gf_parts_kernel<false>, dim3((unsigned)padded, slices), dim3(threads), 0, stream, p, images, g.nt);
    if (e != cudaSuccess) return (int)e;
    if (g.cut) p.part = behind;
    else if (f.accumulate && g.ranges > 1) { p.run = behind; p.ldr = f.N; p.batch_r = (long long)f.M * f.N; }
    else { p.run = f.C; p.ldr = f.ldc; p.batch_r = f.batch_c; }
    switch (g.nt) {
        //                               NT GC GD DA DS WS BS regs cut add others
        case 16: e = gt_launch<GtForm<16, 4, 1, 4, 4, 5, 4, 80, 72, 64, 72>>(mw, p, direct, stream); break;
        case 32: e = gt_launch<GtForm<32, 4, 1, 4, 3, 5, 3, 80, 72, 88, 72>>(mw, p, direct, stream); break;
        case 64: e = gt_launch<GtForm<64, 4, 2, 3, 3, 3, 4, 72, 64, 88, 56>>(mw, p, direct, stream); break;
        case 96: e = gt_launch<GtForm<96, 4, 2, 3, 2, 3, 3, 72, 64, 96, 56>>(mw, p, direct, stream); break;
        case 128: e = gt_launch<GtForm<128, 4, 2, 2, 2, 3, 2, 72, 64, 104, 40>>(mw, p, direct, stream); break;
        case 144: e = gt_launch<GtForm<144, 2, 2, 2, 2, 3, 2, 96, 80, 128, 64>>(mw, p, direct, stream); break;
        default: e = gt_launch<GtForm<160, 2, 2, 2, 2, 3, 2, 96, 80, 128, 64>>(mw, p, direct, stream); break;
    }
    if (e == cudaSuccess && g.cut) {
        const bool pieces = f.N % 4 == 0 && p.ldc % 4 == 0 && p.batch_c % 4 == 0 && (uintptr_t)p.C % 16 == 0 && (uintptr_t)p.part % 16 == 0;
        const size_t outputs = (size_t)f.M * f.N / (pieces ? 4 : 1);
        const dim3 grid((unsigned)((outputs + GR_THREADS - 1) / GR_THREADS), f.batch);
        e = pieces ? launch(gemm_f32_ranges_kernel<4>, grid, dim3(GR_THREADS), 0, stream, p) : launch(gemm_f32_ranges_kernel<1>, grid, dim3(GR_THREADS), 0, stream, p);
    }
    return e == cudaSuccess ? BG_OK : (int)e;
}

int gt_run(const GfParams& f, cudaStream_t stream) {
    const GtPlan g = gt_plan(f.M, f.N, f.K, f.batch);
    for (int b0 = 0; b0 < f.batch; b0 += g.batches)
        for (int m0 = 0; m0 < f.M; m0 += g.rows) {
            GfParams p = f;
            p.A += b0 * f.batch_a + (long long)m0 * f.lda;
            p.W += b0 * f.batch_w;
            p.C += b0 * f.batch_c + (long long)m0 * f.ldc;
            p.M = f.M - m0 < g.rows ? f.M - m0 : g.rows;
            p.batch = f.batch - b0 < g.batches ? f.batch - b0 : g.batches;
            for (int r0 = 0; r0 < g.ranges; r0 += g.at_once) {
                const int rc = gt_piece(p, g, r0, r0 + g.at_once < g.ranges ? r0 + g.at_once : g.ranges, stream);
                if (rc != BG_OK) return rc;
            }
        }
    return BG_OK;
}

}  // namespace bg
