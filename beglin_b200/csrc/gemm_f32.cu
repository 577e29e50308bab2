// C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]) of floats, no operand in fewer bits.  This is the
// reference's linear, y[o] = bias[o] + sum_i W[o,i] x[i] with W row-major [out, in] (qwen_infer.c:688-691), for a batch of rows.
//
// Inner sizes above 2 GF_SHORT run on the tensor cores, every operand in three bfloat16 parts (gemm_f32_tc.cu).  Shorter ones come whole and
// are summed on the float units here: up to GF_SHORT in one chain of fused multiply-adds, k = 0 .. K-1 in order, above it in two, over
// the even and over the odd k, each starting from nought, and their sum (an even k and the odd one behind it lie side by side in both
// operands, which is what the packed multiply-add takes: fma.rn.f32x2, two independent float multiply-adds).  Which way a product goes is
// its K's alone, so a row's result does not depend on how many other rows the call has or where the row stands among them.
// (The line lies at 128: with 136 of k 300 x 128 takes 7.9 us on the tensor cores and 12.8 on the float units, 2,048 x 256 10.1 and 12.9, but
// 16 x 1,536 6.0 and 5.4, and 2,048 x 64 with 192 of k 10.1 and 9.1.)
#include "gemm_f32.cuh"
#include "float_pairs.cuh"

namespace bg {

constexpr int GF_THREADS = 256;
constexpr int GF_SHORT = 64;               // inner sizes up to which a product is one chain of sums; twice that come whole

// Short inner sizes (narrow models, small heads): both operands come whole, BM rows and 64 columns, and a thread sums rows ty + 16 i
// and columns tx + 16 j, four k of a row at a read (rows 68 or 132 floats apart: eight neighbouring ones in different banks).  Above GF_SHORT
// in two chains.  Tiles of 16 rows for up to as many, of 64 else.
// Bound by its reads of shared memory and by the results it writes.  2,048 x 4,096 with k of 64: 36 us, 51 in two chains by pipelined
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

template <int BM, bool TWO>
static cudaError_t gf_launch_short(const GfParams& p, cudaStream_t stream) {
    constexpr size_t smem = (size_t)(BM + GS_BN) * ((TWO ? 2 * GF_SHORT : GF_SHORT) + 4) * sizeof(float);
    const dim3 grid((p.N + GS_BN - 1) / GS_BN, (p.M + BM - 1) / BM, p.batch);
    if (grid.y > 65535) return cudaErrorInvalidConfiguration;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_short_kernel<BM, TWO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch(gemm_f32_short_kernel<BM, TWO>, grid, dim3(GF_THREADS), smem, stream, p);
}

static int gf_run(const GfParams& p, cudaStream_t stream) {
    if (p.K > 2 * GF_SHORT) return gt_run(p, stream);
    const cudaError_t e = p.K > GF_SHORT ? (p.M <= 16 ? gf_launch_short<16, true>(p, stream) : gf_launch_short<64, true>(p, stream))
                                         : (p.M <= 16 ? gf_launch_short<16, false>(p, stream) : gf_launch_short<64, false>(p, stream));
    return e == cudaSuccess ? BG_OK : (int)e;
}

}  // namespace bg

// Floats of scratch that a product of these sizes wants (0: none); one that accumulates wants M N more.
extern "C" long long bg_gemm_f32_scratch(int M, int N, int K, int batch) {
    if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return 0;
    return K > 2 * bg::GF_SHORT ? bg::gt_scratch(M, N, K, batch) : 0;
}

extern "C" int bg_gemm_f32_nt(const float* A, int lda, const float* W, int ldw, const float* bias, float* C, int ldc,
                              int M, int N, int K, int accumulate, float* scratch, unsigned* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return BG_OK;
    if (K <= 0) return BG_ERR_SHAPE;
    bg::GfParams p = {};
    p.A = A; p.W = W; p.bias = bias; p.C = C; p.scratch = scratch; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.accumulate = accumulate; p.batch = 1; p.status = status;
    return bg::gf_run(p, stream);
}

// `batch` products of the same shape: product b reads A + b * batch_a and W + b * batch_w and writes C + b * batch_c
// (element counts).  No bias.  The per-head products of an attention that works in a latent space are of this kind.
extern "C" int bg_gemm_f32_nt_batched(const float* A, int lda, long long batch_a, const float* W, int ldw, long long batch_w,
                                      float* C, int ldc, long long batch_c, int batch, int M, int N, int K, float* scratch,
                                      unsigned* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return BG_OK;
    if (K <= 0 || batch > 65535) return BG_ERR_SHAPE;
    bg::GfParams p = {};
    p.A = A; p.W = W; p.C = C; p.scratch = scratch; p.lda = lda; p.ldw = ldw; p.ldc = ldc; p.M = M; p.N = N; p.K = K;
    p.batch_a = batch_a; p.batch_w = batch_w; p.batch_c = batch_c; p.batch = batch; p.status = status;
    return bg::gf_run(p, stream);
}

// The float feed-forward out[T, hidden] = (act(gate) * up) down^T as one call: gate/up product, activation, down product.  up [2 ff, hidden] (gate and up
// rows in turns of `block`, or halves), down [hidden, ff], both one row behind the other; act and limit as bg_swiglu's.  (silu made where the down
// product cuts its tokens, a kernel less, was no gain: 550 x 1,536 by 8,960 246.6 us and 248, 8 rows 60.5 and 53, whose down product has less time
// to fetch its weights ahead.)
extern "C" long long bg_mlp_f32_scratch(int T, int hidden, int ff) {
    const long long a = bg_gemm_f32_scratch(T, 2 * ff, hidden, 1), b = bg_gemm_f32_scratch(T, hidden, ff, 1);
    return 3LL * T * ff + (a > b ? a : b);
}
extern "C" int bg_mlp_f32(const float* h, int ldh, int T, int hidden, int ff, const float* up, int block, const float* down, int act, float limit, float* scratch,
                          long long scratch_floats, float* out, unsigned* status, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (hidden <= 0 || ff <= 0 || ff % 4) return BG_ERR_SHAPE;
    if (scratch_floats < bg_mlp_f32_scratch(T, hidden, ff)) return BG_ERR_SHAPE;
    float* gu = scratch;
    float* rows = gu + 2LL * T * ff;
    float* rest = rows + (long long)T * ff;
    int rc = bg_gemm_f32_nt(h, ldh, up, hidden, nullptr, gu, 2 * ff, T, 2 * ff, hidden, 0, rest, status, stream);
    if (rc == BG_OK) rc = bg_swiglu(gu, BG_DTYPE_F32, 1, 0, rows, BG_DTYPE_F32, T, ff, block, act, limit, stream);
    if (rc == BG_OK) rc = bg_gemm_f32_nt(rows, ff, down, ff, nullptr, out, hidden, T, hidden, ff, 0, rest, status, stream);
    return rc;
}
