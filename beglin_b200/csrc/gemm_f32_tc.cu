// The float product C[M, N] (+)= A[M, K] W[N, K]^T (+ bias) on the tensor cores, for inner sizes above those of gemm_f32.cu's own kernel.
//
// No precision is given up for it: every operand is cut into three bfloat16 numbers, x = h + m + l exactly, and a product of two floats is
// the six products of parts that are not below 2^-24 of it (one with a single bit set times any float is exact).  32 of k are one
// stage: its five kinds of small products go into an accumulator in tensor memory first, so that their sums are not cut off at the size of
// the large ones, then h h; the stage's sum leaves tensor memory and is added to the range's in float, rounded to nearest.  (An
// accumulator cuts off instead of rounding, always towards nought: two MMAs on a large sum are two such cuts.)  Ranges of GF_RANGE of k lie
// at fixed places; their sums are added in order, then the bias.  None of this depends on the number of rows, on tiles or on who
// adds the ranges, so a row's result does not depend on how many other rows the call has: all forms here give the same bits.
//
// An operand that has no three parts (infinite, not a number, next to the largest float, or below some 2^-110) is noticed where it is cut;
// the outputs of its row and range, and those whose sum is not finite, are summed by floats in two chains (even and odd k) instead, which
// makes of them what floats make.  That, too, depends on the output's own row and column only.
//
// The weights' rows are the M side (128 a CTA), so a lane of tensor memory is an output feature and results leave in rows of 128 bytes;
// the tokens are the N side (NT = 16 to 192).  Weights come as floats (TMA, 128 rows x 32 of k a stage); a warpgroup or two read them, a row a
// lane, cut them and put the parts into tensor memory (`tcgen05.st`) as left operands: they never return to shared memory, whose
// bandwidth the right operands need.  The tokens' parts are made once by gf_parts_kernel and come by bulk copies (the weights' tiles would each
// make them again); up to 16 tokens a warp of the CTA's own makes them.  Other warpgroups add up the stages' sums.
#include "gemm_f32.cuh"
#include "float_pairs.cuh"
#include "ptx.cuh"

namespace bg {

constexpr int GT_BM = 128, GT_BK = 32;     // output features of a CTA; k of a stage
constexpr unsigned GT_W_BYTES = GT_BM * GT_BK * 4;
constexpr int GT_RING = 4;                 // entries of the operands' marks, by range
constexpr long long GT_SCRATCH = 32 << 20; // floats that a call's scratch may take
// Warpgroups: those that cut the weights, those that add the stages' sums, one for copies, MMAs and tokens.
constexpr int gt_threads(int gc, int gd) { return (gc + gd + 1) * 128; }

struct GtParams {
    const float* A; const float* W; const float* bias; float* C;
    float* part;                           // [ranges][batch][M][N]: a CTA has one range and leaves its sums here; or null: it walks them all
    float* run;                            // where a walk keeps the ranges' sum so far, [batch][M] rows of ldr
    const unsigned char* images;           // the tokens' parts (gf_parts_kernel)
    const unsigned char* odd;              // [batch][tokens of all tiles][r1 - r0]: rows with an operand that has no three parts
    long long batch_a, batch_w, batch_c, batch_r;
    int lda, ldw, ldc, ldr, M, N, K, accumulate, ranges, r0, r1, batch, tok_tiles, map_batch;      // (ranges: of all k; r0 to r1: of this launch)
    unsigned* status;
};

// Two floats into their three parts, two bfloat16 a word (the first one low).  `odd` collects what is left over in the low halves:
// nought there if the third part is exact.  (An infinity leaves a NaN, whose low half is not nought.)
__device__ __forceinline__ unsigned gt_pack(unsigned long long v) {
    unsigned r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(high2(v)), "f"(low2(v)));
    return r;
}
__device__ __forceinline__ unsigned long long gt_unpack(unsigned p) {
    return (unsigned long long)(p << 16) | ((unsigned long long)(p & 0xffff0000u) << 32);
}
__device__ __forceinline__ void gt_split(unsigned long long v, unsigned& h, unsigned& m, unsigned& l, unsigned& odd) {
    const unsigned long long minus = pair2(-1.0f, -1.0f);
    h = gt_pack(v);
    const unsigned long long r = fma2(gt_unpack(h), minus, v);
    m = gt_pack(r);
    const unsigned long long q = fma2(gt_unpack(m), minus, r);
    l = __byte_perm((unsigned)q, (unsigned)(q >> 32), 0x7632);
    odd |= (unsigned)q | (unsigned)(q >> 32);
}
__device__ __forceinline__ unsigned long long gt_add2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The tokens' parts as the images of the stages' right operands, [batch][tile of nt tokens][stage][part][token][32 of k] with the swizzle of
// shared memory, noughts behind the last token and behind K; and the rows' marks.  One stage is then one copy of contiguous bytes:
// boxes of a tensor map, 64 bytes a row, took the copy engine 2.4 cycles a row, 1,750 a stage of 192 tokens.  A warp per row and range.
template <bool VEC>
__global__ void __launch_bounds__(256) gf_parts_kernel(GtParams p, unsigned char* images, unsigned char* odd, int nt) {
    pdl_launch();
    const int padded = p.tok_tiles * nt, lane = threadIdx.x & 31, ranges = p.r1 - p.r0, k_all = min(p.K, p.r1 * GF_RANGE) - p.r0 * GF_RANGE, stages = (k_all + GT_BK - 1) / GT_BK;
    const long long job = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (job >= (long long)p.batch * padded * ranges) return;
    const long long row = job / ranges;
    const int range = (int)(job - row * ranges), b = (int)(row / padded), m = (int)(row - (long long)b * padded), in = m % nt;
    const float* src = p.A + (size_t)b * p.batch_a + (size_t)m * p.lda + p.r0 * GF_RANGE;
    pdl_wait();
    float4 v[GF_RANGE / 128];
#pragma unroll
    for (int i = 0; i < GF_RANGE / 128; ++i) {
        const int k = range * GF_RANGE + i * 128 + lane * 4, most = m < p.M ? k_all : 0;
        if constexpr (VEC) v[i] = k < most ? *reinterpret_cast<const float4*>(src + k) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        else v[i] = make_float4(k < most ? src[k] : 0.0f, k + 1 < most ? src[k + 1] : 0.0f, k + 2 < most ? src[k + 2] : 0.0f, k + 3 < most ? src[k + 3] : 0.0f);
    }
    unsigned left = 0;
#pragma unroll
    for (int i = 0; i < GF_RANGE / 128; ++i) {
        const int stage = (range * GF_RANGE + i * 128) / GT_BK + (lane >> 3);
        uint2 h, q, l;
        gt_split(pair2(v[i].x, v[i].y), h.x, q.x, l.x, left);
        gt_split(pair2(v[i].z, v[i].w), h.y, q.y, l.y, left);
        if (stage < stages) {
            unsigned char* d = images + (((size_t)b * p.tok_tiles + m / nt) * stages + stage) * 3 * nt * 64 + in * 64 + (((lane >> 1 & 3) ^ (in >> 1 & 3)) << 4) + (lane & 1) * 8;
            *reinterpret_cast<uint2*>(d) = h;
            *reinterpret_cast<uint2*>(d + (size_t)nt * 64) = q;
            *reinterpret_cast<uint2*>(d + (size_t)nt * 128) = l;
        }
    }
    const unsigned any = __ballot_sync(0xffffffffu, (left & 0xffffu) != 0);
    if (lane == 0) odd[job] = any != 0;
}

// Loads and stores of tensor memory; the caller waits.
__device__ __forceinline__ void gt_ld8(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void gt_ld16(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}
__device__ __forceinline__ void gt_st4(unsigned taddr, const unsigned (&v)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
}
// The descriptor of a K-major right operand in rows of 64 bytes (32 of k), 64-byte swizzle: groups of 8 rows 512 bytes apart.
__device__ __forceinline__ unsigned long long smem_desc_sw64(unsigned smem_addr) {
    return (unsigned long long)((smem_addr & 0x3FFFFu) >> 4) | (unsigned long long)(512u >> 4) << 32 | 1ull << 46 | 4ull << 61;
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
template <int HAS, int WANTS>
__device__ __forceinline__ void gt_regs() {
    if constexpr (WANTS > HAS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(WANTS));
    if constexpr (WANTS < HAS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(WANTS));
}

// Whether any of the THREADS that add says so; they all meet.
template <int THREADS>
__device__ __forceinline__ bool gt_any(bool mine) {
    unsigned r;
    asm volatile("{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.cta.red.or.pred q, 1, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(r) : "r"(mine ? 1u : 0u), "n"(THREADS) : "memory");
    return r != 0;
}

// Two chains of multiply-adds over n of k, and their sum.
__device__ __forceinline__ float gt_chain(const float* a, const float* w, int n) {
    float even = 0.0f, odd = 0.0f;
    int k = 0;
    for (; k + 1 < n; k += 2) { even = fmaf(a[k], w[k], even); odd = fmaf(a[k + 1], w[k + 1], odd); }
    if (k < n) even = fmaf(a[k], w[k], even);
    return even + odd;
}

// What a form of the kernel takes: tokens NT; warpgroups that cut (GC: 32 / GC of a stage's k each) and that add (GD: NT / GD columns each);
// stages whose parts (DA) and sums (DS) tensor memory holds, of weights (WS) and tokens (BS) in shared memory; CTAs an SM; registers of a thread
// at launch, of one that cuts, that adds, and of the others: their sum over the warpgroups is not above the launch's.
template <int NT_, int GC_, int GD_, int DA_, int DS_, int WS_, int BS_, int PER_SM_, int REGS_, int RC_, int RD_, int RO_>
struct GtForm {
    static constexpr int NT = NT_, GC = GC_, GD = GD_, DA = DA_, DS = DS_, WS = WS_, BS = BS_, PER_SM = PER_SM_, REGS = REGS_, RC = RC_, RD = RD_, RO = RO_;
    static constexpr bool OWN = NT == 16;              // the tokens are cut by a warp of the CTA
    static_assert(GC * RC + GD * RD + RO <= (GC + GD + 1) * REGS);
};

template <typename F, bool DIRECT>
__global__ void __launch_bounds__(gt_threads(F::GC, F::GD), F::PER_SM)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, GtParams p) {
    constexpr int NT = F::NT, GC = F::GC, GD = F::GD, DA = F::DA, DS = F::DS, WS = F::WS, BS = F::BS;
    constexpr bool OWN = F::OWN;
    constexpr int CG = NT / GD, KG = GT_BK / GC, ADDERS = 128 * GD, STAGES = GF_RANGE / GT_BK;
    constexpr unsigned PLANE = NT * 64, B_BYTES = 3 * PLANE;
    constexpr unsigned PARTS0 = DS * NT, WANT = PARTS0 + DA * 48, COLS = WANT > 256 ? 512 : WANT > 128 ? 256 : 128;
    static_assert(WANT <= 512 && COLS * F::PER_SM <= 512 && CG % 8 == 0 && KG % 8 == 0);
    extern __shared__ unsigned char gt_raw[];
    unsigned char* wt = (unsigned char*)(((uintptr_t)gt_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* bt = wt + WS * GT_W_BYTES;
    __shared__ __align__(8) unsigned long long w_full[WS], w_empty[WS], b_full[BS], b_empty[BS], a_full[DA], a_empty[DA], done[DS], sum_empty[DS];
    __shared__ unsigned tmem_sh;
    __shared__ int failed;
    __shared__ unsigned char row_odd[GT_RING][GC][GT_BM], tok_odd[GT_RING][NT], tok_now[NT];

    constexpr int W_WARP = 4 * (GC + GD), MMA_WARP = W_WARP + 1, TOKEN_WARP = W_WARP + 2;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tok = blockIdx.x % p.tok_tiles, feat = blockIdx.x / p.tok_tiles, b = blockIdx.y;
    const int t0 = tok * NT, n0 = feat * GT_BM;
    const int r_begin = p.part ? blockIdx.z : p.r0, r_end = p.part ? r_begin + 1 : p.r1;
    const int k_begin = r_begin * GF_RANGE, k_end = min(p.K, r_end * GF_RANGE), n = (k_end - k_begin + GT_BK - 1) / GT_BK;

    if (threadIdx.x == 0) {
        for (int i = 0; i < WS; ++i) { mbar_init(&w_full[i], 1); mbar_init(&w_empty[i], 4 * GC); }
        for (int i = 0; i < BS; ++i) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
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
            if (!OWN) pdl_wait();
            for (int s = 0; s < n; ++s) {
                if (s >= WS && !mbar_wait(&w_empty[s % WS], (s / WS - 1) & 1, &failed)) break;
                mbar_expect_tx(&w_full[s % WS], GT_W_BYTES);
                tma_load_3d(wt + (s % WS) * GT_W_BYTES, &map_w, k_begin + s * GT_BK, n0, p.map_batch ? b : 0, &w_full[s % WS]);
            }
        }
    } else if (warp == MMA_WARP || warp == MMA_WARP + 2) {
        // ---------------- the MMAs: two warps in turns, so that one's three waits (some 130 cycles each, ready or not) lie under the other's MMAs
        constexpr unsigned idesc = instr_desc_bf16(GT_BM, NT);
        for (int s = warp == MMA_WARP ? 0 : 1; s < n; s += 2) {
            const int d = s % DS, o = s % DA, i = s % BS;
            bool ok = mbar_wait(&b_full[i], (s / BS) & 1, &failed);
            ok = ok && (s < DS || mbar_wait(&sum_empty[d], (s / DS - 1) & 1, &failed));
            ok = ok && mbar_wait(&a_full[o], (s / DA) & 1, &failed);
            if (!ok) break;
            tc_fence_after();
            if (elect_one()) {
                const unsigned acc = tmem + d * NT, a = tmem + PARTS0 + o * 48, bb = smem_u32(bt + i * B_BYTES);
#pragma unroll
                for (int e = 0; e < 6; ++e) {
                    constexpr int PA[6] = {2, 1, 0, 1, 0, 0}, PB[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        tc_mma_ts(acc, a + PA[e] * 16 + j * 8, smem_desc_sw64(bb + PB[e] * PLANE + j * 32), idesc, e || j ? 1u : 0u);
                }
                tc_commit(&done[d]);
                tc_commit(&a_empty[o]);
                tc_commit(&b_empty[i]);
            }
            __syncwarp();
        }
    } else if (warp == TOKEN_WARP) {
        if constexpr (!OWN) {
            // ---------------- the copies of the tokens' parts
            if (lane == 0) {
                const unsigned char* src = p.images + (((size_t)b * p.tok_tiles + tok) * ((min(p.K, p.r1 * GF_RANGE) - p.r0 * GF_RANGE + GT_BK - 1) / GT_BK) + (k_begin - p.r0 * GF_RANGE) / GT_BK) * B_BYTES;
                pdl_wait();
                for (int s = 0; s < n; ++s) {
                    const int i = s % BS;
                    if (s >= BS && !mbar_wait(&b_empty[i], (s / BS - 1) & 1, &failed)) break;
                    mbar_expect_tx(&b_full[i], B_BYTES);
                    bulk_load(bt + i * B_BYTES, src + (size_t)s * B_BYTES, B_BYTES, &b_full[i]);
                }
            }
        } else {
            // ---------------- up to 16 tokens: two lanes a row, 16 of k each, asked for two stages ahead
            const int row = lane >> 1, m = t0 + row;
            const float* src = p.A + (size_t)b * p.batch_a + (size_t)(m < p.M ? m : 0) * p.lda;
            const bool vec = p.lda % 4 == 0 && p.batch_a % 4 == 0 && (uintptr_t)p.A % 16 == 0;
            unsigned left = 0;
            auto fetch = [&](int s, float4 (&v)[4]) {
                const int k0 = k_begin + s * GT_BK + (lane & 1) * 16;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int k = k0 + u * 4;
                    v[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (m >= p.M) continue;
                    if (vec && k + 3 < k_end) v[u] = *reinterpret_cast<const float4*>(src + k);
                    else {
                        if (k < k_end) v[u].x = src[k];
                        if (k + 1 < k_end) v[u].y = src[k + 1];
                        if (k + 2 < k_end) v[u].z = src[k + 2];
                        if (k + 3 < k_end) v[u].w = src[k + 3];
                    }
                }
            };
            auto put = [&](int s, const float4 (&v)[4]) {
                const int i = s % BS;
                if (s >= BS && !mbar_wait(&b_empty[i], (s / BS - 1) & 1, &failed)) return false;
                unsigned char* d = bt + i * B_BYTES + row * 64;
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    uint4 h, q, l;
                    gt_split(pair2(v[2 * u].x, v[2 * u].y), h.x, q.x, l.x, left);
                    gt_split(pair2(v[2 * u].z, v[2 * u].w), h.y, q.y, l.y, left);
                    gt_split(pair2(v[2 * u + 1].x, v[2 * u + 1].y), h.z, q.z, l.z, left);
                    gt_split(pair2(v[2 * u + 1].z, v[2 * u + 1].w), h.w, q.w, l.w, left);
                    unsigned char* at = d + ((((lane & 1) * 2 + u) ^ (row >> 1 & 3)) << 4);
                    *reinterpret_cast<uint4*>(at) = h;
                    *reinterpret_cast<uint4*>(at + PLANE) = q;
                    *reinterpret_cast<uint4*>(at + 2 * PLANE) = l;
                }
                if ((s + 1) % STAGES == 0 || s + 1 == n) {
                    const unsigned mine = (left & 0xffffu) != 0, other = __shfl_xor_sync(0xffffffffu, mine, 1);
                    if (!(lane & 1)) tok_odd[(s / STAGES) % GT_RING][row] = (unsigned char)(mine | other);
                    left = 0;
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&b_full[i]);
                return true;
            };
            float4 v0[4], v1[4];
            pdl_wait();
            fetch(0, v0);
            fetch(1, v1);
#pragma unroll 1
            for (int s = 0; s < n; s += 2) {
                if (!put(s, v0)) break;
                fetch(s + 2, v0);
                if (s + 1 < n && !put(s + 1, v1)) break;
                fetch(s + 3, v1);
            }
        }
    } else if (warp < 4 * GC) {
        // ---------------- weights into parts, a row a lane
        gt_regs<F::REGS, F::RC>();
        const int quarter = warp & 3, group = warp >> 2, row = quarter * 32 + lane;
        const unsigned parts = tmem + ((unsigned)(quarter * 32) << 16) + PARTS0 + group * (KG / 2);
        const float* w_row = p.W + (size_t)b * p.batch_w + (size_t)(n0 + row < p.N ? n0 + row : 0) * p.ldw;
        unsigned long long v[KG / 2];
        unsigned left = 0;
        auto fetch = [&](int s) {
            if constexpr (DIRECT) {
                const int k = k_begin + s * GT_BK + group * KG;
                const bool in = n0 + row < p.N;
#pragma unroll
                for (int u = 0; u < KG / 2; ++u) v[u] = pair2(in && k + 2 * u < k_end ? w_row[k + 2 * u] : 0.0f, in && k + 2 * u + 1 < k_end ? w_row[k + 2 * u + 1] : 0.0f);
            } else {
                mbar_wait(&w_full[s % WS], (s / WS) & 1, &failed);
                const unsigned char* src = wt + (s % WS) * GT_W_BYTES + row * 128;
#pragma unroll
                for (int u = 0; u < KG / 4; ++u) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(src + (((group * (KG / 4) + u) ^ (row & 7)) << 4));
                    v[2 * u] = x.x; v[2 * u + 1] = x.y;
                }
            }
        };
        if (DIRECT && !OWN) pdl_wait();
        fetch(0);
#pragma unroll 1
        for (int s = 0; s < n; ++s) {
            if (s >= DA) {                                     // (the products of stage s - DA have read its parts)
                mbar_wait(&a_empty[s % DA], (s / DA - 1) & 1, &failed);
                tc_fence_after();
            }
            const unsigned a = parts + s % DA * 48;
#pragma unroll
            for (int u = 0; u < KG / 8; ++u) {
                unsigned h[4], m[4], l[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) gt_split(v[4 * u + i], h[i], m[i], l[i], left);
                gt_st4(a + 4 * u, h); gt_st4(a + 16 + 4 * u, m); gt_st4(a + 32 + 4 * u, l);
            }
            __syncwarp();
            if (lane == 0 && !DIRECT) mbar_arrive(&w_empty[s % WS]);
            if ((s + 1) % STAGES == 0 || s + 1 == n) {
                row_odd[(s / STAGES) % GT_RING][group][row] = (left & 0xffffu) != 0;
                left = 0;
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[s % DA]);
            if (s + 1 < n) fetch(s + 1);
        }
    } else if (warp < W_WARP) {
        // ---------------- the stages' sums
        gt_regs<F::REGS, F::RD>();
        const int quarter = warp & 3, group = (warp >> 2) - GC, row = quarter * 32 + lane, feature = n0 + row, adder = threadIdx.x - 128 * GC;
        const unsigned sums = tmem + ((unsigned)(quarter * 32) << 16) + group * CG;
        const float* w_row = p.W + (size_t)b * p.batch_w + (size_t)(feature < p.N ? feature : 0) * p.ldw;
        unsigned long long total[CG / 2];
        bool waited = false;
#pragma unroll 1
        for (int e = 0; e < n; ++e) {
            const bool first = e % STAGES == 0, last = (e + 1) % STAGES == 0 || e + 1 == n;
            const unsigned acc = sums + e % DS * NT;
            mbar_wait(&done[e % DS], (e / DS) & 1, &failed);
            tc_fence_after();
            constexpr int STEP = CG % 32 == 0 ? 32 : CG % 16 == 0 ? 16 : 8;
#pragma unroll
            for (int c = 0; c < CG; c += STEP) {
                unsigned r[STEP];
                if constexpr (STEP == 32) tc_ld32_nowait(acc + c, r);
                else if constexpr (STEP == 16) gt_ld16(acc + c, r);
                else gt_ld8(acc + c, r);
                tc_wait_ld();
#pragma unroll
                for (int j = 0; j < STEP / 2; ++j) {
                    const unsigned long long x = (unsigned long long)r[2 * j] | ((unsigned long long)r[2 * j + 1] << 32);
                    total[c / 2 + j] = first ? x : gt_add2(total[c / 2 + j], x);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sum_empty[e % DS]);
            if (!last) continue;
            // ---- the sums of a range
            const int ring = e / STAGES, range = r_begin + ring;
            if (!waited) { pdl_wait(); waited = true; }
            bool w_odd = false, t_odd = false;
#pragma unroll
            for (int g = 0; g < GC; ++g) w_odd |= row_odd[ring % GT_RING][g][row] != 0;
            if (adder < NT) {
                if constexpr (OWN) t_odd = tok_odd[ring % GT_RING][adder];
                else t_odd = p.odd[((size_t)b * p.tok_tiles * NT + t0 + adder) * (p.r1 - p.r0) + range - p.r0];
            }
            unsigned long long nought = 0ull;                  // not nought if a sum is not finite
#pragma unroll
            for (int j = 0; j < CG / 2; ++j) nought = fma2(total[j], 0ull, nought);
            if (gt_any<ADDERS>(w_odd || t_odd || !(sum2(nought) == 0.0f) || *(volatile int*)&failed)) {
                if (adder < NT) tok_now[adder] = t_odd;
                gt_any<ADDERS>(false);
                const int kr = range * GF_RANGE, nr = min(p.K - kr, GF_RANGE);
#pragma unroll 1
                for (int c = 0; c < CG; ++c) {
                    const int t = t0 + group * CG + c;
                    if (t >= p.M) break;
                    float x = 0.0f;
#pragma unroll
                    for (int j = 0; j < CG; ++j) x = j == c ? (j & 1 ? high2(total[j / 2]) : low2(total[j / 2])) : x;
                    if (feature < p.N && (w_odd || tok_now[group * CG + c] || !(fabsf(x) <= 3.402823466e38f)))
                        x = gt_chain(p.A + (size_t)b * p.batch_a + (size_t)t * p.lda + kr, w_row + kr, nr);
                    if (*(volatile int*)&failed) x = __uint_as_float(0x7fffffffu);         // (a wait ran out)
#pragma unroll
                    for (int j = 0; j < CG; ++j)
                        if (j == c) total[j / 2] = j & 1 ? pair2(low2(total[j / 2]), x) : pair2(x, high2(total[j / 2]));
                }
                gt_any<ADDERS>(false);
            }
            if (feature >= p.N) continue;
            const int rows = min(CG, p.M - t0 - group * CG);
            const bool end = !p.part && range + 1 == p.ranges, sums_before = !p.part && range > 0, add_old = end && p.accumulate;
            const size_t at = (size_t)(t0 + group * CG);
            float* run = p.run + (size_t)b * p.batch_r + at * p.ldr + feature;
            float* out = p.part ? p.part + (((size_t)range * p.batch + b) * p.M + at) * p.N + feature : end ? p.C + (size_t)b * p.batch_c + at * p.ldc + feature : run;
            size_t step = p.part ? p.N : end ? p.ldc : p.ldr, step_r = p.ldr;
            const float bias = end && p.bias ? p.bias[feature] : 0.0f;
#pragma unroll
            for (int j0 = 0; j0 < CG; j0 += 8) {               // (eight loads on their way at a time)
                asm volatile("" : "+l"(run), "+l"(out), "+l"(step), "+l"(step_r));         // (no address is made ahead and kept)
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = j & 1 ? high2(total[(j0 + j) / 2]) : low2(total[(j0 + j) / 2]);
                if (sums_before) {
                    float old[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) old[j] = j0 + j < rows ? run[j * step_r] : 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = old[j] + x[j];
                }
                if (end && p.bias) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] += bias;
                }
                if (add_old) {
                    float old[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) old[j] = j0 + j < rows ? out[j * step] : 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) x[j] = old[j] + x[j];
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (j0 + j < rows) out[j * step] = x[j];
                run += 8 * step_r;
                out += 8 * step;
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

// C = (old C +) ((part 0 + part 1) + ...) (+ bias), a thread per output.
__global__ void __launch_bounds__(256) gemm_f32_ranges_kernel(GtParams p) {
    pdl_launch();
    pdl_wait();
    const size_t total = (size_t)p.M * p.N, step = total * p.batch;
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const int m = (int)(e / p.N), n = (int)(e - (size_t)m * p.N);
    const float* s = p.part + (size_t)blockIdx.y * total + e;
    float v = s[0];
    for (int r0 = 1; r0 < p.ranges; r0 += 8) {             // eight loads on their way at a time
        float a[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = r0 + u < p.ranges ? s[(size_t)(r0 + u) * step] : 0.0f;
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (r0 + u < p.ranges) v += a[u];
    }
    if (p.bias) v += p.bias[n];
    float* c = p.C + (size_t)blockIdx.y * p.batch_c + (size_t)m * p.ldc + n;
    *c = p.accumulate ? *c + v : v;
}

// ------------------------------------------------------------------------------------------------ host
// How a call is cut: tiles of nt tokens; pieces of `rows` rows of `batches` products whose scratch fits; the ranges to CTAs of their own or not.
struct GtPlan { int nt, rows, batches, ranges, at_once; bool own, cut; };
constexpr long long GT_TOKEN = GF_RANGE / GT_BK * 48 + 1;        // floats of a token's parts and mark of a range

static long long gt_tiles(int M, int N, int batch, int nt) { return (long long)((M + nt - 1) / nt) * ((N + GT_BM - 1) / GT_BM) * batch; }

static double gt_cost(int M, int N, int batch, int ranges, int nt, bool cut) {
    const long long sms = sm_count(), units = gt_tiles(M, N, batch, nt) * (cut ? ranges : 1);
    const int per_sm = nt <= 32 ? 2 : 1;
    const double stage = 770.0 + 8.5 * nt, rounds = (double)((units + sms * per_sm - 1) / (sms * per_sm));
    const double work = rounds * stage * (per_sm == 2 && units > sms ? 1.4 : 1.0) * 16.0 * (cut ? 1 : ranges) + 3000.0 * rounds;
    return work + (cut ? 4000.0 + 8.0 * M * N * ranges * batch / 2000.0 : 0.0);
}

static GtPlan gt_plan(int M, int N, int K, int batch) {
    GtPlan g;
    g.ranges = (K + GF_RANGE - 1) / GF_RANGE;
    g.own = M <= 16;                                       // (the tokens are cut in the kernel)
    g.at_once = g.ranges;
    double best = 0.0;
    g.nt = 0;
    for (int nt : {16, 32, 64, 96, 128, 160, 192}) {
        if ((nt == 16) != (M <= 16)) continue;
        for (int cut = 0; cut < (g.ranges > 1 ? 2 : 1); ++cut) {
            const double c = gt_cost(M, N, batch, g.ranges, nt, cut);
            if (g.nt == 0 || c < best) { best = c; g.nt = nt; g.cut = cut; }
        }
    }
    const long long part = (long long)g.ranges * N, all = (M + g.nt - 1) / g.nt * (long long)g.nt, token = g.own ? 0 : GT_TOKEN;
    if (g.cut && all * token * g.ranges + M * part > GT_SCRATCH) g.cut = false;
    const long long each = all * token * g.ranges + (g.cut ? M * part : 0), tile = g.nt * token;
    g.rows = M;
    g.batches = batch;
    if (each > GT_SCRATCH) {                               // (never a cut one: the tokens' parts)
        g.batches = 1;
        g.rows = (int)(GT_SCRATCH / (tile * g.ranges) * g.nt);
        if (g.rows == 0) { g.rows = g.nt; g.at_once = (int)(GT_SCRATCH / tile); }
    } else if (each > 0 && GT_SCRATCH / each < batch) g.batches = (int)(GT_SCRATCH / each);
    return g;
}
static long long gt_floats(const GtPlan& g, int N) {
    const long long padded = (long long)(g.rows + g.nt - 1) / g.nt * g.nt * g.batches;
    return (g.own ? 0 : padded * GT_TOKEN * g.at_once) + (g.cut ? (long long)g.rows * g.batches * g.ranges * N : 0);
}
long long gt_scratch(int M, int N, int K, int batch) {
    const GtPlan g = gt_plan(M, N, K, batch);
    return gt_floats(g, N);
}

// A batch of float matrices, boxes of 32 columns x 128 rows.
static int gt_weight_map(CUtensorMap* map, const GfParams& p, int batch) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return BG_ERR_UNSUPPORTED;
    const long long apart = batch > 1 ? p.batch_w : (long long)p.N * p.ldw;
    cuuint64_t dims[3] = {(cuuint64_t)p.K, (cuuint64_t)p.N, (cuuint64_t)batch};
    cuuint64_t strides[2] = {(cuuint64_t)p.ldw * 4, (cuuint64_t)apart * 4};
    cuuint32_t box[3] = {(cuuint32_t)GT_BK, (cuuint32_t)GT_BM, 1u}, elem[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p.W), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? BG_OK : BG_ERR_SHAPE;
}
template <typename F>
static cudaError_t gt_launch(const CUtensorMap& mw, const GtParams& p, bool direct, cudaStream_t stream) {
    constexpr size_t smem = (size_t)F::WS * GT_W_BYTES + (size_t)F::BS * 3 * F::NT * 64 + 1024;
    static_assert((smem + 3072) * F::PER_SM <= 227 * 1024);
    auto kern = direct ? gemm_f32_tc_kernel<F, true> : gemm_f32_tc_kernel<F, false>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    static const bool fits = F::RC == F::REGS && F::RD == F::REGS && F::RO == F::REGS ? true : [] {      // (the split of the registers counts on as many at launch)
        cudaFuncAttributes a, b;
        return cudaFuncGetAttributes(&a, gemm_f32_tc_kernel<F, true>) == cudaSuccess && cudaFuncGetAttributes(&b, gemm_f32_tc_kernel<F, false>) == cudaSuccess &&
               a.numRegs >= F::REGS && b.numRegs >= F::REGS;
    }();
    if (!fits) return cudaErrorInvalidConfiguration;
    const dim3 grid((unsigned)((p.N + GT_BM - 1) / GT_BM * p.tok_tiles), p.batch, p.part ? p.ranges : 1);
    return launch(kern, grid, dim3(gt_threads(F::GC, F::GD)), smem, stream, mw, p);
}

static int gt_piece(const GfParams& f, const GtPlan& g, int r0, int r1, cudaStream_t stream) {
    GtParams p = {};
    p.A = f.A; p.W = f.W; p.bias = f.bias; p.C = f.C; p.batch_a = f.batch_a; p.batch_w = f.batch_w; p.batch_c = f.batch_c;
    p.lda = f.lda; p.ldw = f.ldw; p.ldc = f.ldc; p.M = f.M; p.N = f.N; p.K = f.K; p.accumulate = f.accumulate; p.batch = f.batch;
    p.ranges = g.ranges; p.r0 = r0; p.r1 = r1; p.status = f.status;
    p.tok_tiles = (f.M + g.nt - 1) / g.nt;
    const bool direct = !(f.ldw % 4 == 0 && f.batch_w % 4 == 0 && (uintptr_t)f.W % 16 == 0);
    p.map_batch = f.batch > 1 && f.batch_w != 0;
    float* behind = f.scratch;
    CUtensorMap mw = {};
    if (!direct) {
        const int rc = gt_weight_map(&mw, f, p.map_batch ? f.batch : 1);
        if (rc != BG_OK) return rc;
    }
    cudaError_t e = cudaSuccess;
    if (!g.own) {
        const long long padded = (long long)p.tok_tiles * g.nt * f.batch, here = r1 - r0;
        unsigned char *images = (unsigned char*)behind, *odd = (unsigned char*)(behind + padded * (GT_TOKEN - 1) * here);
        behind += padded * GT_TOKEN * here;
        p.images = images;
        p.odd = odd;
        const bool vec = f.K % 4 == 0 && f.lda % 4 == 0 && f.batch_a % 4 == 0 && (uintptr_t)f.A % 16 == 0;
        const dim3 grid((unsigned)((padded * here + 7) / 8));
        e = vec ? launch(gf_parts_kernel<true>, grid, dim3(256), 0, stream, p, images, odd, g.nt)
                : launch(gf_parts_kernel<false>, grid, dim3(256), 0, stream, p, images, odd, g.nt);
        if (e != cudaSuccess) return (int)e;
    }
    if (g.cut) p.part = behind;
    else if (f.accumulate && g.ranges > 1) { p.run = behind; p.ldr = f.N; p.batch_r = (long long)f.M * f.N; }
    else { p.run = f.C; p.ldr = f.ldc; p.batch_r = f.batch_c; }
    switch (g.nt) {
        //                               NT GC GD DA DS WS BS SM regs cut add others
        case 16: {
            // three CTAs an SM where there are so many
            const long long units = gt_tiles(f.M, f.N, f.batch, 16) * (g.cut ? g.ranges : 1);
            e = units > 2LL * sm_count() ? gt_launch<GtForm<16, 1, 1, 2, 2, 3, 4, 3, 56, 64, 48, 56>>(mw, p, direct, stream)
                                         : gt_launch<GtForm<16, 1, 1, 4, 4, 4, 4, 2, 80, 80, 80, 80>>(mw, p, direct, stream);
            break;
        }
        case 32: e = gt_launch<GtForm<32, 2, 1, 4, 2, 4, 4, 2, 64, 64, 72, 56>>(mw, p, direct, stream); break;
        case 64: e = gt_launch<GtForm<64, 4, 2, 4, 4, 4, 8, 1, 72, 56, 88, 56>>(mw, p, direct, stream); break;
        case 96: e = gt_launch<GtForm<96, 4, 2, 4, 3, 4, 6, 1, 72, 56, 104, 56>>(mw, p, direct, stream); break;
        case 128: e = gt_launch<GtForm<128, 2, 4, 5, 2, 4, 6, 1, 72, 64, 80, 56>>(mw, p, direct, stream); break;
        case 160: e = gt_launch<GtForm<160, 2, 4, 4, 2, 4, 4, 1, 72, 56, 88, 40>>(mw, p, direct, stream); break;
        default: e = gt_launch<GtForm<192, 2, 4, 2, 2, 4, 4, 1, 72, 56, 88, 40>>(mw, p, direct, stream); break;
    }
    if (e == cudaSuccess && g.cut)
        e = launch(gemm_f32_ranges_kernel, dim3((unsigned)(((size_t)f.M * f.N + 255) / 256), f.batch), dim3(256), 0, stream, p);
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
