// C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]) in true float: CUDA-core FFMA, no tensor cores and no
// reduced-precision mode (the tensor cores have no float x float kind; their tf32 kind drops
// mantissa bits).  This is the reference's linear, y[o] = bias[o] + sum_i W[o,i] x[i] with W
// row-major [out, in] (qwen_infer.c:688-691), for a batch of rows.
//
// K is cut into ranges of GF_RANGE, at the same places whatever the call.  Every output is, per range, TWO chains of fused
// multiply-adds, over the even and over the odd k in order, each starting from nought, and their sum; the ranges' sums are added in
// order, then the bias.  Which kernel runs, how its tiles lie and whether the ranges go to CTAs of their own changes none of that, so
// a row's result does not depend on how many other rows the call has or where the row stands among them: all the kernels here give
// the same bits.  Two chains because an even k and the odd one behind it lie side by side in both operands, which is what the packed
// multiply-add takes (fma.rn.f32x2: two independent float multiply-adds).  In a product's inner loop the register file, not the
// float units, is what an 8 x 8 block of single multiply-adds waits for: 51 TFLOP/s on 148 SMs from registers alone, 68 with packed
// ones whose rows are walked to and fro, so that each shares an operand with the one before.
//
// Inner sizes of up to GF_SHORT are summed in one chain, k = 0 .. K-1 in order, whatever the rows: two chains and a pipeline over k gain
// nothing there.
//
//   gemm_f32_short_kernel  inner sizes of up to 64, and of up to 128 with more than 16 rows
//   gemm_f32_tile_kernel   tiles of 128 (or 64) rows x 128 columns, for more than 16 rows
//   gemm_f32_few_kernel    up to 16 rows: the product is a stream of weights
//   gemm_f32_ranges_kernel adds the sums of ranges that went to CTAs of their own
#include "common.cuh"
#include "float_pairs.cuh"

namespace bg {

constexpr int GF_RANGE = 1024;             // a multiple of every step of k below
constexpr int GF_BN = 128, GF_BK = 16, GF_LD = GF_BK + 4, GF_STAGES = 4, GF_THREADS = 256;
constexpr int GF_FEW = 16;                 // rows up to which the product is treated as a stream of weights
constexpr int GF_SHORT = 64;               // inner sizes up to which a product is one chain of sums
constexpr long long GF_SCRATCH = 32 << 20; // floats that the sums of ranges may take

struct GfParams {
    const float* A; const float* W; const float* bias; float* C;
    float* part;                           // [ranges][batch][M][N] sums of the ranges, or null: a CTA walks them all
    long long batch_a, batch_w, batch_c;   // a batch of independent products
    int lda, ldw, ldc, M, N, K, accumulate, ranges, batch;
};

// ROWS rows of GF_BK values from column k on into a tile of row stride GF_LD (`src`: the tile's first row, of which `rows` exist);
// what lies behind `rows` or K becomes zeros.
template <int ROWS, bool VEC>
__device__ __forceinline__ void gf_fetch(float* dst, const float* src, int ld, int rows, int k, int K) {
    constexpr int W = VEC ? 4 : 1, PER_ROW = GF_BK / W;                  // values of a copy, copies of a row
#pragma unroll
    for (int i = 0; i < ROWS * PER_ROW / GF_THREADS; ++i) {
        const int r = threadIdx.x / PER_ROW + i * (GF_THREADS / PER_ROW), c = threadIdx.x % PER_ROW * W;
        const bool in = r < rows && k + c < K;
        async_copy<W * 4>(dst + r * GF_LD + c, src + (in ? (size_t)((unsigned)r * (unsigned)ld + (unsigned)(k + c)) : 0), in);
    }
}

// Short inner sizes (narrow models, small heads): both operands come whole, BM rows and 64 columns, and a thread sums rows ty + 16 i
// and columns tx + 16 j, four k of a row at a read (rows 68 or 132 floats apart: eight neighbouring ones in different banks).  Above GF_SHORT
// in two chains, as the kernels of larger inner sizes, whose bits these are.
// Bound by its reads of shared memory and by the results it writes.  2,048 x 4,096 with k of 64: 36 us, 51 in two chains by the pipelined
// tiles; sixteen products of 2,048 x 512: 71 and 89, with k of 32 43 and 63; 64 x 640 with k of 72 5.4 and 8.8 (7.5 in tiles of 64 x 64 without
// a pipeline), 2,048 x 640 10.4 and 16.8, 8,192 x 2,048 with k of 128 121 and 141, 300 x 2,048 14.0 and 12.0.
constexpr int GS_BN = 64;
template <int BM, bool TWO>
__global__ void __launch_bounds__(GF_THREADS) gemm_f32_short_kernel(GfParams p) {
    constexpr int RI = BM / 16, CJ = GS_BN / 16, EACH = GF_THREADS / 32;          // EACH: rows that the threads bring at a time
    constexpr int MOST = TWO ? 2 * GF_SHORT : GF_SHORT, LD = MOST + 4;
    extern __shared__ __align__(16) float gf_s[];
    float *As = gf_s, *Ws = gf_s + BM * LD;
    pdl_launch();
    pdl_wait();
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * GS_BN, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const float* A = p.A + (size_t)blockIdx.z * p.batch_a;
    const float* W = p.W + (size_t)blockIdx.z * p.batch_w;
#pragma unroll
    for (int h = 0; h < MOST; h += 32) {                 // (zeros behind K, the rows and the columns)
        const int k = h + lane;
        if (h >= p.K) break;
#pragma unroll
        for (int r = warp; r < BM; r += EACH) As[r * LD + k] = k < p.K && m0 + r < p.M ? A[(size_t)(m0 + r) * p.lda + k] : 0.0f;
#pragma unroll
        for (int r = warp; r < GS_BN; r += EACH) Ws[r * LD + k] = k < p.K && n0 + r < p.N ? W[(size_t)(n0 + r) * p.ldw + k] : 0.0f;
    }
    __syncthreads();
    unsigned long long acc[RI][CJ];                      // (one chain: in the low half, the high one stays nought)
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < CJ; ++j) acc[i][j] = 0ull;
#pragma unroll 4
    for (int k = 0; k < p.K; k += 4) {
        ulonglong2 a[RI], w[CJ];
#pragma unroll
        for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(As + (ty + 16 * i) * LD + k);
#pragma unroll
        for (int j = 0; j < CJ; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(Ws + (tx + 16 * j) * LD + k);
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < CJ; ++j) {
                if constexpr (TWO) acc[i][j] = fma2(a[i].y, w[j].y, fma2(a[i].x, w[j].x, acc[i][j]));
                else acc[i][j] = __float_as_uint(fmaf(high2(a[i].y), high2(w[j].y), fmaf(low2(a[i].y), low2(w[j].y),
                                                 fmaf(high2(a[i].x), high2(w[j].x), fmaf(low2(a[i].x), low2(w[j].x), low2(acc[i][j]))))));
            }
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
        const int m = m0 + ty + 16 * i;
        if (m >= p.M) continue;
#pragma unroll
        for (int j = 0; j < CJ; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n >= p.N) continue;
            float v = TWO ? sum2(acc[i][j]) : low2(acc[i][j]);
            if (p.bias) v += p.bias[n];
            float* c = p.C + (size_t)blockIdx.z * p.batch_c + (size_t)m * p.ldc + n;
            *c = p.accumulate ? *c + v : v;
        }
    }
}

// A thread owns rows ty + 16 i and columns tx + 16 j, 8 x 8 outputs (4 x 8 with BM = 64), an even and an odd sum each.  Both operands
// lie in shared memory as they do in memory, k innermost, so they come by 16-byte asynchronous copies and a thread reads four k of a
// row at a time: 16 reads of 16 bytes for 128 packed multiply-adds.  A warp covers 4 x 8 (ty, tx); rows 20 floats apart put eight
// neighbouring rows into different banks.  One CTA an SM (the sums take 128 registers).  550 rows of 1,536 x 17,920: 930 us, 32.5
// TFLOP/s, where tiles of 64 x 64 with 4-byte loads and no pipeline took 1,720 us; its two warps a scheduler wait for the FMA pipe's
// queue and for fixed latencies as long as they issue (FMA pipe 54 %, reads of shared memory 40 % of their rates).
template <int BM, int BN, bool VEC>
__global__ void __launch_bounds__(GF_THREADS, 1) gemm_f32_tile_kernel(GfParams p) {
    extern __shared__ __align__(16) float gf_s[];
    constexpr int RI = BM / 16, CJ = BN / 16, STAGE = (BM + BN) * GF_LD;
    float* total = gf_s + GF_STAGES * STAGE + threadIdx.x;       // [RI * CJ][GF_THREADS]: the ranges' sums so far, a thread's own
    pdl_launch();
    pdl_wait();
    const int b = blockIdx.z % p.batch, own = blockIdx.z / p.batch;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const float* A = p.A + (size_t)b * p.batch_a + (size_t)m0 * p.lda;
    const float* W = p.W + (size_t)b * p.batch_w + (size_t)n0 * p.ldw;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
    const int r_begin = p.part ? own : 0, r_end = p.part ? own + 1 : p.ranges;
    for (int range = r_begin; range < r_end; ++range) {
        const int k_begin = range * GF_RANGE, k_end = min(p.K, k_begin + GF_RANGE);
        const int steps = (k_end - k_begin + GF_BK - 1) / GF_BK;
        auto fetch = [&](int s) {
            if (s < steps) {
                float* st = gf_s + (s % GF_STAGES) * STAGE;
                gf_fetch<BM, VEC>(st, A, p.lda, p.M - m0, k_begin + s * GF_BK, k_end);
                gf_fetch<BN, VEC>(st + BM * GF_LD, W, p.ldw, p.N - n0, k_begin + s * GF_BK, k_end);
            }
            async_commit();
        };
        unsigned long long acc[RI][CJ];
#pragma unroll
        for (int i = 0; i < RI; ++i)
#pragma unroll
            for (int j = 0; j < CJ; ++j) acc[i][j] = 0ull;
        __syncthreads();                   // (the last range's tiles have been read)
#pragma unroll
        for (int s = 0; s < GF_STAGES - 1; ++s) fetch(s);
        for (int s = 0; s < steps; ++s) {
            async_wait<GF_STAGES - 2>();
            __syncthreads();
            fetch(s + GF_STAGES - 1);      // into the stage that was read in the step before
            const float* As = gf_s + (s % GF_STAGES) * STAGE + ty * GF_LD;
            const float* Ws = gf_s + (s % GF_STAGES) * STAGE + (BM + tx) * GF_LD;
#pragma unroll
            for (int k = 0; k < GF_BK; k += 4) {
                ulonglong2 a[RI], w[CJ];
#pragma unroll
                for (int i = 0; i < RI; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(As + i * 16 * GF_LD + k);
#pragma unroll
                for (int j = 0; j < CJ; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(Ws + j * 16 * GF_LD + k);
                // rows to and fro under the columns
#pragma unroll
                for (int j = 0; j < CJ; ++j)
#pragma unroll
                    for (int u = 0; u < RI; ++u) { const int i = j & 1 ? RI - 1 - u : u; acc[i][j] = fma2(a[i].x, w[j].x, acc[i][j]); }
#pragma unroll
                for (int j = CJ - 1; j >= 0; --j)
#pragma unroll
                    for (int u = 0; u < RI; ++u) { const int i = j & 1 ? u : RI - 1 - u; acc[i][j] = fma2(a[i].y, w[j].y, acc[i][j]); }
            }
        }
        async_wait<0>();
        if (range + 1 < r_end) {           // more ranges follow in this CTA
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < CJ; ++j) {
                    float* t = total + (i * CJ + j) * GF_THREADS;
                    *t = range == r_begin ? sum2(acc[i][j]) : *t + sum2(acc[i][j]);
                }
            continue;
        }
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int m = m0 + ty + 16 * i;
            if (m >= p.M) continue;
#pragma unroll
            for (int j = 0; j < CJ; ++j) {
                const int n = n0 + tx + 16 * j;
                if (n >= p.N) continue;
                float v = sum2(acc[i][j]);
                if (p.part) {
                    p.part[(((size_t)range * p.batch + b) * p.M + m) * p.N + n] = v;
                    continue;
                }
                if (range > r_begin) v = total[(i * CJ + j) * GF_THREADS] + v;
                if (p.bias) v += p.bias[n];
                float* c = p.C + (size_t)b * p.batch_c + (size_t)m * p.ldc + n;
                *c = p.accumulate ? *c + v : v;
            }
        }
    }
}

// C = (old C +) ((part 0 + part 1) + ...) (+ bias), a thread per output.
__global__ void __launch_bounds__(256) gemm_f32_ranges_kernel(GfParams p) {
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

// Up to 2 RPL rows.  A warp takes 32 columns over one range of k: lane (g, c) owns columns c and c + 16 of rows g RPL .. g RPL + RPL - 1.
// The weights' rows and those of A come through a ring of the warp's own (GW_STAGES steps of 32 k, 16-byte asynchronous copies of
// 128 contiguous bytes a row), so no warp waits for another, and nine warps' rings fit an SM.  (A read through the first-level cache
// instead, beside rings that leave it no room, made every read a trip to L2; 16 columns a warp made five reads of shared memory
// for every eight packed multiply-adds, and those reads the bound: 71 us for 8 rows of 1,536 x 17,920, 33.5 us now, 355 before.)  The
// warps of a CTA take the ranges of the same columns and the sums meet in shared memory; where the columns leave SMs idle the ranges
// are spread over up to gridDim.z CTAs, which leave their sums in `part`.  Bound by the stream of weights.
constexpr int GW_BK = 32, GW_LD = GW_BK + 4, GW_STAGES = 4, GW_COLS = 32, GW_WARPS = 8;

template <int RPL>
__global__ void __launch_bounds__(GW_WARPS * 32) gemm_f32_few_kernel(GfParams p, int groups) {
    extern __shared__ __align__(16) float gf_s[];
    constexpr int ROWS = GW_COLS + 2 * RPL, STAGE = ROWS * GW_LD;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    float* ring = gf_s + warp * (GW_STAGES * STAGE);
    float* sums = gf_s + warps * (GW_STAGES * STAGE);                      // [groups][ranges][2 RPL][GW_COLS]
    const int c = lane & 15, g = lane >> 4, b = blockIdx.y;
    const int fr = lane >> 3, fk = (lane & 7) * 4;                         // the row of four, and its four k, that the lane copies
    const float* A = p.A + (size_t)b * p.batch_a;
    const float* W = p.W + (size_t)b * p.batch_w;
    const int each = (p.ranges + gridDim.z - 1) / gridDim.z, r0 = blockIdx.z * each, n_ranges = min(each, p.ranges - r0);
    const int jobs = groups * n_ranges, first = blockIdx.x * groups * GW_COLS;
    pdl_launch();
    bool waited = false;
    for (int job = warp; job < jobs; job += warps) {
        const int group = job / n_ranges, range = job - group * n_ranges;
        const int n0 = first + group * GW_COLS;
        if (n0 >= p.N) continue;
        const int k_begin = (r0 + range) * GF_RANGE, k_end = min(p.K, k_begin + GF_RANGE);
        const int steps = (k_end - k_begin + GW_BK - 1) / GW_BK;
        auto fetch_w = [&](int s) {
            float* st = ring + (s % GW_STAGES) * STAGE + fr * GW_LD + fk;
            const int k = k_begin + s * GW_BK + fk;
#pragma unroll
            for (int r = 0; r < GW_COLS; r += 4) {
                const bool in = n0 + r + fr < p.N && k < k_end;
                async_copy<16>(st + r * GW_LD, in ? W + (size_t)(n0 + r + fr) * p.ldw + k : W, in);
            }
        };
        auto fetch_a = [&](int s) {
            float* st = ring + (s % GW_STAGES) * STAGE + (GW_COLS + fr) * GW_LD + fk;
            const int k = k_begin + s * GW_BK + fk;
#pragma unroll
            for (int r = 0; r < 2 * RPL; r += 4) {
                if (r + fr >= 2 * RPL) continue;
                const bool in = r + fr < p.M && k < k_end;
                async_copy<16>(st + r * GW_LD, in ? A + (size_t)(r + fr) * p.lda + k : A, in);
            }
        };
        __syncwarp();                      // (the last job's ring has been read)
#pragma unroll
        for (int s = 0; s < GW_STAGES - 1; ++s)
            if (s < steps) fetch_w(s);
        if (!waited) { pdl_wait(); waited = true; }                        // the weights depend on no kernel of the step
#pragma unroll
        for (int s = 0; s < GW_STAGES - 1; ++s) {                          // (the first group holds all the weights asked for above)
            if (s < steps) fetch_a(s);
            async_commit();
        }
        unsigned long long acc[2][RPL];
#pragma unroll
        for (int r = 0; r < RPL; ++r) acc[0][r] = acc[1][r] = 0ull;
        for (int s = 0; s < steps; ++s) {
            async_wait<GW_STAGES - 2>();
            __syncwarp();
            if (s + GW_STAGES - 1 < steps) { fetch_w(s + GW_STAGES - 1); fetch_a(s + GW_STAGES - 1); }
            async_commit();
            const float* ws = ring + (s % GW_STAGES) * STAGE + c * GW_LD;
            const float* as = ring + (s % GW_STAGES) * STAGE + (GW_COLS + g * RPL) * GW_LD;
            // (k behind the range's end: zeros on both sides)
#pragma unroll 4
            for (int k = 0; k < GW_BK; k += 4) {
                const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + k), w1 = *reinterpret_cast<const ulonglong2*>(ws + 16 * GW_LD + k);
                ulonglong2 a[RPL];
#pragma unroll
                for (int r = 0; r < RPL; ++r) a[r] = *reinterpret_cast<const ulonglong2*>(as + r * GW_LD + k);
#pragma unroll
                for (int r = 0; r < RPL; ++r) { acc[0][r] = fma2(a[r].x, w0.x, acc[0][r]); acc[1][r] = fma2(a[r].x, w1.x, acc[1][r]); }
#pragma unroll
                for (int r = 0; r < RPL; ++r) { acc[0][r] = fma2(a[r].y, w0.y, acc[0][r]); acc[1][r] = fma2(a[r].y, w1.y, acc[1][r]); }
            }
        }
        async_wait<0>();
        float* out = sums + (size_t)((group * n_ranges + range) * 2 * RPL + g * RPL) * GW_COLS + c;
#pragma unroll
        for (int r = 0; r < RPL; ++r) { out[r * GW_COLS] = sum2(acc[0][r]); out[r * GW_COLS + 16] = sum2(acc[1][r]); }
    }
    if (!waited) pdl_wait();               // (no warp goes on to the sums before it)
    __syncthreads();
    for (int idx = threadIdx.x; idx < groups * 2 * RPL * GW_COLS; idx += blockDim.x) {
        const int group = idx / (2 * RPL * GW_COLS), e = idx - group * 2 * RPL * GW_COLS;
        const int m = e / GW_COLS, n = first + group * GW_COLS + e % GW_COLS;
        if (m >= p.M || n >= p.N) continue;
        const float* s = sums + (size_t)group * n_ranges * 2 * RPL * GW_COLS + e;
        if (p.part) {
            for (int r = 0; r < n_ranges; ++r) p.part[(((size_t)(r0 + r) * p.batch + b) * p.M + m) * p.N + n] = s[(size_t)r * 2 * RPL * GW_COLS];
            continue;
        }
        float v = s[0];
        for (int r = 1; r < n_ranges; ++r) v += s[(size_t)r * 2 * RPL * GW_COLS];
        if (p.bias) v += p.bias[n];
        float* cc = p.C + (size_t)b * p.batch_c + (size_t)m * p.ldc + n;
        *cc = p.accumulate ? *cc + v : v;
    }
}

// Columns (in groups of GW_COLS) of a CTA of the kernel of few rows: with several ranges its warps take those of one group, with one
// range a group each as far as every SM keeps two CTAs.
static int gf_few_groups(int N, int ranges, int batch) {
    const int all = (N + GW_COLS - 1) / GW_COLS;
    int groups = ranges >= GW_WARPS ? 1 : GW_WARPS / ranges;
    while (groups > 1 && (long long)((all + groups - 1) / groups) * batch < 2LL * sm_count()) --groups;
    return groups;
}

// How many CTAs share the ranges of a group of columns: one, unless the groups alone leave SMs idle.
static int gf_few_shares(int N, int ranges, int batch) {
    const long long ctas = (long long)((N + GW_COLS - 1) / GW_COLS) * batch;
    int shares = 1;
    while (shares < ranges && ctas * (shares + 1) <= sm_count()) ++shares;
    const int each = (ranges + shares - 1) / shares;
    return (ranges + each - 1) / each;                   // no CTA without a range
}

// Rows at a time whose ranges of K go to CTAs of their own (and through `part`), 0: none, a CTA walks all its ranges.  They do where the
// tiles alone make fewer than two rounds of the SMs, the last of them partly empty (550 x 1,536 with k of 8,960: 60 tiles, 540 with their
// ranges), in pieces of rows whose sums fit GF_SCRATCH.  Where they go changes no bit.
static int gf_cuts(int M, int N, int ranges, int batch, int bm) {
    if (ranges < 2) return 0;
    const long long tiles = (long long)((M + bm - 1) / bm) * ((N + GF_BN - 1) / GF_BN) * batch;
    if (tiles >= 2LL * sm_count()) return 0;
    const long long rows = GF_SCRATCH / ((long long)ranges * batch * N);
    return rows >= M ? M : (int)(rows / bm * bm);
}

// Inner sizes that go to the short kernel; from 16 rows down, longer than GF_SHORT, the product is a stream of weights as others.
static bool gf_short(int M, int K) { return K <= GF_SHORT || (K <= 2 * GF_SHORT && M > GF_FEW); }
static bool gf_few(int M, int ranges, bool vec) { return vec && M <= GF_FEW && ranges <= 64; }
// Tiles of 64 rows where 128 would be half empty, or leave SMs without a tile.
static int gf_bm(int M, int N, int ranges, int batch) {
    const long long tiles = (long long)((M + 127) / 128) * ((N + GF_BN - 1) / GF_BN) * batch * ranges;
    return M <= 64 || ((M - 1) % 128 < 64 && M < 512) || tiles < sm_count() ? 64 : 128;
}

template <int RPL>
static cudaError_t gf_launch_few(const GfParams& p, cudaStream_t stream) {
    constexpr size_t ring = (size_t)GW_STAGES * (GW_COLS + 2 * RPL) * GW_LD * sizeof(float), most = 220 * 1024;
    const int shares = p.part ? gf_few_shares(p.N, p.ranges, p.batch) : 1, each = (p.ranges + shares - 1) / shares;
    const int groups = gf_few_groups(p.N, each, p.batch * shares);
    const size_t sums = (size_t)groups * each * 2 * RPL * GW_COLS * sizeof(float);
    int warps = groups * each < GW_WARPS ? groups * each : GW_WARPS;
    while (warps > 1 && warps * ring + sums > most) --warps;
    const size_t smem = warps * ring + sums;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<RPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const unsigned x = (unsigned)((p.N + groups * GW_COLS - 1) / (groups * GW_COLS));
    return launch(gemm_f32_few_kernel<RPL>, dim3(x, p.batch, shares), dim3(warps * 32), smem, stream, p, groups);
}
template <int BM, int BN, bool VEC>
static cudaError_t gf_launch_tile(const GfParams& p, cudaStream_t stream) {
    constexpr size_t tiles = (size_t)GF_STAGES * (BM + BN) * GF_LD * sizeof(float), totals = (size_t)BM * BN * sizeof(float);
    const size_t smem = p.part || p.ranges == 1 ? tiles : tiles + totals;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<BM, BN, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(tiles + totals));
    if (e != cudaSuccess) return e;
    const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, p.batch * (p.part ? p.ranges : 1));
    return launch(gemm_f32_tile_kernel<BM, BN, VEC>, grid, dim3(GF_THREADS), smem, stream, p);
}

template <int BM, bool TWO>
static cudaError_t gf_launch_short(const GfParams& p, cudaStream_t stream) {
    constexpr size_t smem = (size_t)(BM + GS_BN) * ((TWO ? 2 * GF_SHORT : GF_SHORT) + 4) * sizeof(float);
    const dim3 grid((p.N + GS_BN - 1) / GS_BN, (p.M + BM - 1) / BM, p.batch);
    if (grid.y > 65535) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_short_kernel<BM, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch(gemm_f32_short_kernel<BM, TWO>, grid, dim3(GF_THREADS), smem, stream, p);
}

static cudaError_t gf_add_ranges(const GfParams& p, cudaStream_t stream) {
    const size_t total = (size_t)p.M * p.N;
    return launch(gemm_f32_ranges_kernel, dim3((unsigned)((total + 255) / 256), p.batch), dim3(256), 0, stream, p);
}

static int gf_run(GfParams p, cudaStream_t stream) {
    const bool vec = p.K % 4 == 0 && p.lda % 4 == 0 && p.ldw % 4 == 0 && p.batch_a % 4 == 0 && p.batch_w % 4 == 0 &&
                     (uintptr_t)p.A % 16 == 0 && (uintptr_t)p.W % 16 == 0;
    p.ranges = (p.K + GF_RANGE - 1) / GF_RANGE;
    if (gf_short(p.M, p.K)) {
        const cudaError_t e = p.K > GF_SHORT ? gf_launch_short<64, true>(p, stream)
                            : p.M <= 16 ? gf_launch_short<16, false>(p, stream) : gf_launch_short<64, false>(p, stream);
        return e == cudaSuccess ? BG_OK : (int)e;
    }
    if (gf_few(p.M, p.ranges, vec)) {
        if (gf_few_shares(p.N, p.ranges, p.batch) == 1) p.part = nullptr;
        cudaError_t e = p.M <= 2 ? gf_launch_few<1>(p, stream) : p.M <= 4 ? gf_launch_few<2>(p, stream)
                      : p.M <= 8 ? gf_launch_few<4>(p, stream) : gf_launch_few<8>(p, stream);
        if (e == cudaSuccess && p.part) e = gf_add_ranges(p, stream);
        return e == cudaSuccess ? BG_OK : (int)e;
    }
    const int bm = gf_bm(p.M, p.N, p.ranges, p.batch);
    const int cut = gf_cuts(p.M, p.N, p.ranges, p.batch, bm), rows = cut > 0 ? cut : p.M, M = p.M;
    if (cut > 0 && !p.part) return BG_ERR_SHAPE;
    if (cut == 0) p.part = nullptr;
    if ((rows + bm - 1) / bm > 65535 || (long long)p.batch * (cut > 0 ? p.ranges : 1) > 65535) return BG_ERR_SHAPE;
    for (int m0 = 0; m0 < M; m0 += rows) {
        p.M = M - m0 < rows ? M - m0 : rows;
        cudaError_t e;
        // (as many columns as there are: 32 products of 2,048 x 64, k of 192, 61 us, half empty 105; 300 x 64, k of 4,096, 39 and 67)
        if (p.N <= 64)
            e = bm == 64 ? (vec ? gf_launch_tile<64, 64, true>(p, stream) : gf_launch_tile<64, 64, false>(p, stream))
                         : (vec ? gf_launch_tile<128, 64, true>(p, stream) : gf_launch_tile<128, 64, false>(p, stream));
        else
            e = bm == 64 ? (vec ? gf_launch_tile<64, GF_BN, true>(p, stream) : gf_launch_tile<64, GF_BN, false>(p, stream))
                         : (vec ? gf_launch_tile<128, GF_BN, true>(p, stream) : gf_launch_tile<128, GF_BN, false>(p, stream));
        if (e == cudaSuccess && cut > 0) e = gf_add_ranges(p, stream);
        if (e != cudaSuccess) return (int)e;
        p.A += (size_t)rows * p.lda;
        p.C += (size_t)rows * p.ldc;
    }
    return BG_OK;
}

}  // namespace bg

// Floats of scratch that a product of these sizes wants (0: none): the ranges' sums, where they go to CTAs of their own.
extern "C" long long bg_gemm_f32_scratch(int M, int N, int K, int batch) {
    if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return 0;
    const int ranges = (K + bg::GF_RANGE - 1) / bg::GF_RANGE;
    // (asked without the operands' alignment: both kernels' wants count)
    const bool few = bg::gf_few(M, ranges, true) && bg::gf_few_shares(N, ranges, batch) > 1;
    const int cut = bg::gf_cuts(M, N, ranges, batch, bg::gf_bm(M, N, ranges, batch)), rows = few ? M : cut;
    return (long long)ranges * batch * rows * N;
}

extern "C" int bg_gemm_f32_nt(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc,
                              int M, int N, int K, int accumulate, float* scratch, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return BG_OK;
    if (K <= 0) return BG_ERR_SHAPE;
    bg::GfParams p = {};
    p.A = A; p.W = W; p.bias = bias; p.C = C; p.part = scratch; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.accumulate = accumulate; p.batch = 1;
    return bg::gf_run(p, stream);
}

// `batch` products of the same shape: product b reads A + b * batch_a and W + b * batch_w and writes C + b * batch_c
// (element counts).  No bias.  The per-head products of an attention that works in a latent space are of this kind.
extern "C" int bg_gemm_f32_nt_batched(const float* A, int lda, long long batch_a, const float* W, int ldw, long long batch_w,
                                      float* C, int ldc, long long batch_c, int batch, int M, int N, int K, float* scratch,
                                      cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return BG_OK;
    if (K <= 0 || batch > 65535) return BG_ERR_SHAPE;
    bg::GfParams p = {};
    p.A = A; p.W = W; p.C = C; p.part = scratch; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.batch_a = batch_a; p.batch_w = batch_w; p.batch_c = batch_c; p.batch = batch;
    return bg::gf_run(p, stream);
}
