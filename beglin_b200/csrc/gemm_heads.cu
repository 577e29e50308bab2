// The products of attention through a latent that every head has of its own, for steps of few rows:
//   out[h][t][n] = sum_k X[h][t][k] W[h][n][k]  (* sigmoid(gate[t][h]), or of the feature's own gate)
// bfloat16 operands, float accumulation, on tcgen05 as gemm_tcgen05.cu: a CTA takes 128 of a head's output features (the M side) and up to 64
// rows (the N side).  A head's rows of X begin at column h x_col and row h x_row of one matrix, so a product's rows and the attention's
// results by head are both read where they lie; boxes that run past a head's rows or features read a neighbour's, whose results are not stored.
// The whole inner size (a multiple of 64) is on its way at once, the weights while the kernel ahead still runs: what bounds these products is their
// start and the way from L2, not the tensor cores.  With the gates and the row-by-row order in the epilogue the step saves a kernel.
// Two products and the gates, us, the library's kernels and the gates' first: 64 rows of 32 heads, 64 -> 512 features and back to 128: 3.0 and 2.8, 4.8 and
// 5.3; 41 rows of 20 heads, 448 and 64: 2.9 and 2.5, 5.1 and 4.4; 14 rows of 32 heads, 320 and 64: 2.6 and 2.0, 4.9 and 3.7.
// Every wait is bounded and records BG_STATUS_TIMEOUT.
#include "tc_common.cuh"

namespace bg {

constexpr int GH_STAGES = 8;

struct HeadsParams {
    void* out; long long out_head; int out_row;
    const void* gate; int gate_float, gate_stride, gate_col, per_feature;
    int n_out, T, H, n_kb, stages;
    int x_col, x_row;
    unsigned* status;
};

template <int BN, typename TO>
__global__ void __launch_bounds__(TC_THREADS)
gemm_heads_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, HeadsParams p) {
    constexpr unsigned A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr unsigned TMEM_COLS = BN < 32 ? 32 : BN;
    extern __shared__ unsigned char gh_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)gh_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[GH_STAGES], empty_bar[GH_STAGES], acc_bar;
    __shared__ unsigned tmem_base_sh;
    __shared__ int failed;
    __shared__ float gate_s[BN < 16 ? 16 : BN];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * TC_BM, h = blockIdx.y, t0 = blockIdx.z * BN;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(&acc_bar, 1);
        failed = 0;
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_sh)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem_base = tmem_base_sh;
    pdl_launch();

    if (warp == 0) {
        if (lane == 0) {
            const int w_row = h * p.n_out + m0, x = h * p.x_col, y = h * p.x_row + t0;
            for (int i = 0; i < p.stages; ++i) {
                mbar_expect_tx(&full_bar[i], STAGE_BYTES);
                tma_load_2d(tiles + (size_t)i * STAGE_BYTES, &map_w, i * TC_BK, w_row, &full_bar[i]);
            }
            pdl_wait();
            for (int i = 0; i < p.stages; ++i) tma_load_2d(tiles + (size_t)i * STAGE_BYTES + A_BYTES, &map_x, x + i * TC_BK, y, &full_bar[i]);
            for (int i = p.stages; i < p.n_kb; ++i) {
                const int s = i % p.stages;
                if (!mbar_wait(&empty_bar[s], ((i / p.stages) - 1) & 1)) { atomicExch(&failed, 1); break; }
                unsigned char* a = tiles + (size_t)s * STAGE_BYTES;
                mbar_expect_tx(&full_bar[s], STAGE_BYTES);
                tma_load_2d(a, &map_w, i * TC_BK, w_row, &full_bar[s]);
                tma_load_2d(a + A_BYTES, &map_x, x + i * TC_BK, y, &full_bar[s]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr unsigned idesc = instr_desc_bf16(TC_BM, BN);
            for (int i = 0; i < p.n_kb; ++i) {
                const int s = i % p.stages;
                if (!mbar_wait(&full_bar[s], (i / p.stages) & 1)) { atomicExch(&failed, 1); break; }
                tc_fence_after();
                const unsigned a_addr = smem_u32(tiles + (size_t)s * STAGE_BYTES), b_addr = a_addr + A_BYTES;
#pragma unroll
                for (int k = 0; k < TC_BK / 16; ++k)
                    tc_mma(tmem_base, smem_desc_sw128(a_addr + k * 32), smem_desc_sw128(b_addr + k * 32), idesc, (i > 0 || k > 0) ? 1u : 0u);
                tc_commit(&empty_bar[s]);
            }
            tc_commit(&acc_bar);
        }
    } else {
        // warps 2..5 own tensor-memory lanes 32 (warp % 4) .. + 31: a lane is an output feature, a column a row of the step
        const int quarter = warp & 3, n = m0 + quarter * 32 + lane;
        pdl_wait();
        auto sigmoid = [&](size_t at) {
            const float g = p.gate_float ? ((const float*)p.gate)[at] : __bfloat162float(((const __nv_bfloat16*)p.gate)[at]);
            return 1.0f / (1.0f + expf(-g));
        };
        const int rows = min(BN, p.T - t0);
        if (p.gate && !p.per_feature) {
            const int i = threadIdx.x - 64;
            if (i < BN) gate_s[i] = i >= rows ? 1.0f : sigmoid((size_t)(t0 + i) * p.gate_stride + p.gate_col + h);
            asm volatile("bar.sync 1, 128;\n" ::: "memory");
        }
        const bool ok = mbar_wait(&acc_bar, 0);
        if (!ok) atomicExch(&failed, 1);
        tc_fence_after();
        if (__all_sync(0xffffffffu, ok)) {
            TO* to = (TO*)p.out + (size_t)h * p.out_head + (size_t)t0 * p.out_row + n;
            const unsigned t_addr = tmem_base + ((unsigned)(quarter * 32) << 16);
            // a load of tensor memory is the whole warp's: where features end inside a warp, lanes without one wait for the others
            const bool ragged = p.n_out % 32 != 0 && m0 + TC_BM > p.n_out;
#pragma unroll 1
            for (int c = 0; c < rows; c += 16, to += (size_t)16 * p.out_row) {
                unsigned r[16];
                tc_ld16(t_addr + (unsigned)c, r);
                if (p.gate) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float g = 1.0f;
                        if (!p.per_feature) g = gate_s[c + j];
                        else if (c + j < rows && n < p.n_out) g = sigmoid((size_t)(t0 + c + j) * p.gate_stride + p.gate_col + (size_t)h * p.n_out + n);
                        r[j] = __float_as_uint(__uint_as_float(r[j]) * g);
                    }
                }
                if (n < p.n_out) {
                    if (c + 16 <= rows) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) to[(size_t)j * p.out_row] = from_float<TO>(__uint_as_float(r[j]));
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (c + j < rows) to[(size_t)j * p.out_row] = from_float<TO>(__uint_as_float(r[j]));
                    }
                }
                if (ragged) __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
    if (threadIdx.x == 0 && failed && p.status) atomicOr(p.status, BG_STATUS_TIMEOUT);
}

template <int BN, typename TO>
static int gh_launch(const CUtensorMap& mw, const CUtensorMap& mx, const HeadsParams& p, cudaStream_t stream) {
    auto kern = gemm_heads_kernel<BN, TO>;
    constexpr size_t STAGE = (size_t)(TC_BM + BN) * TC_BK * 2;
    static std::once_flag once;
    static cudaError_t set = cudaSuccess;
    std::call_once(once, [&] { set = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(GH_STAGES * STAGE + 1024)); });
    if (set != cudaSuccess) return (int)set;
    const dim3 grid((p.n_out + TC_BM - 1) / TC_BM, p.H, (p.T + BN - 1) / BN);
    const cudaError_t e = launch(kern, grid, dim3(TC_THREADS), p.stages * STAGE + 1024, stream, mw, mx, p);
    return e == cudaSuccess ? BG_OK : (int)e;
}

}  // namespace bg

using namespace bg;

// W [H * n_out, K] bfloat16, rows one behind the other; X a bfloat16 matrix of x_rows x x_cols with row stride ldx, in which head h's T rows of K begin at
// row h x_row and column h x_col; out: element (h, t, n) at h out_head + t out_row + n, float or bfloat16; gate (either type) or null: its rows hold a
// number per head from gate_col on, or, per_feature, H n_out of them.
extern "C" int bg_gemm_heads(const void* W, int H, int n_out, int K, const void* X, long long x_rows, int x_cols, int ldx, int x_row, int x_col, int T, void* out,
                             int out_dtype, long long out_head, int out_row, const void* gate, int gate_dtype, int gate_stride, int gate_col, int per_feature,
                             unsigned* status, cudaStream_t stream) {
    if (T <= 0 || n_out <= 0 || H <= 0) return BG_OK;
    if (K <= 0 || x_row < 0 || x_col < 0) return BG_ERR_SHAPE;
    if (K % TC_BK || H > 65535 || (long long)H * n_out > 0x7fffffffLL || x_rows > 0x7fffffffLL) return BG_ERR_UNSUPPORTED;
    if ((long long)(H - 1) * x_row + T > x_rows || (long long)(H - 1) * x_col + K > x_cols) return BG_ERR_SHAPE;
    if (ldx % 8 || x_col % 8 || (uintptr_t)W % 16 || (uintptr_t)X % 16) return BG_ERR_ALIGN;
    if ((out_dtype != BG_DTYPE_F32 && out_dtype != BG_DTYPE_BF16) || (gate && gate_dtype != BG_DTYPE_F32 && gate_dtype != BG_DTYPE_BF16)) return BG_ERR_DTYPE;
    // rows a CTA: as few as leave every CTA an SM of its own (64 rows of 32 heads, 512 -> 128 features: 5.4 us on 32 CTAs of 64 rows)
    const long long tiles = (long long)((n_out + TC_BM - 1) / TC_BM) * H;
    int bn = 16;
    while (bn < 64 && bn < T && tiles * ((T + bn - 1) / bn) > sm_count()) bn *= 2;
    HeadsParams p;
    p.out = out; p.out_head = out_head; p.out_row = out_row;
    p.gate = gate; p.gate_float = gate_dtype == BG_DTYPE_F32; p.gate_stride = gate_stride; p.gate_col = gate_col; p.per_feature = per_feature;
    p.n_out = n_out; p.T = T; p.H = H; p.n_kb = K / TC_BK; p.stages = p.n_kb < GH_STAGES ? p.n_kb : GH_STAGES; p.x_col = x_col; p.x_row = x_row;
    p.status = status;
    CUtensorMap mw, mx;
    int rc = weight_map(&mw, W, H * n_out, K, K);
    if (rc == BG_OK) rc = make_map(&mx, X, x_rows, x_cols, ldx, bn);
    if (rc != BG_OK) return rc;
    BG_DISPATCH_DTYPE(out_dtype, TO, {
        if (bn == 16) return gh_launch<16, TO>(mw, mx, p, stream);
        if (bn == 32) return gh_launch<32, TO>(mw, mx, p, stream);
        return gh_launch<64, TO>(mw, mx, p, stream);
    });
    return BG_OK;
}
