// The experts' products of a routed feed-forward for many rows an expert, on PAIRS of CTAs:
//   out[row, n] = act(sum_k X[row, k] * W[e][n, k])     for the rows offsets[e] .. offsets[e + 1] of expert e,
// the arguments and results of gemm_grouped_tc.cu, whose kernel takes the steps with fewer rows.  Bound by the tensor cores.
//
// A persistent kernel, one pair (a cluster of two CTAs) per tile of 256 output features of one expert x up to 256 of its rows.
// The features are the M side (128 for each CTA), the rows the N side, so that a tile is only as wide as the expert has rows for:
// one thread of the first CTA issues tcgen05.mma.cta_group::2 of M = 256 and N = 64 .. 256, each CTA brings its own features and HALF
// of the rows (32 KB a stage at most, six stages), and the accumulator, the CTA's own 128 features x N rows, is double-buffered in
// tensor memory, so that the epilogue of a tile runs under the MMAs of the next.
//
// Which rows an expert has is known on the device only.  Every CTA lays the tiles out for itself, alike: an expert's rows are cut
// evenly into the least number of tiles of at most `width` rows, and `width` is that one of 256, 192 and 128 whose rounds of tiles
// over the pairs cost least (a k-block's operands reach an SM at 64 bytes a cycle: 512, 448 and 384 cycles).  A box that runs past
// its expert's rows or features reads the neighbour's, whose columns or lanes are not stored.
//
// 4,096 rows of 8 experts: 1,536 -> 3,072 features 57.4 us on single CTAs -> 42.1 (0.92 PFLOP/s), 3,072 -> 1,536 53.1 -> 36.7; 1,200
// rows of 4 experts, 1,536 -> 2,048 and back: 18.0 -> 16.1 and 20.1 -> 14.1.  What is left: the last round of tiles (240 of them on 74
// pairs) and tiles narrower than 256.
//
// Barriers as in gemm_pair.cu; every wait is bounded and records BG_STATUS_TIMEOUT.
#include "tc_pair.cuh"

namespace bg {

constexpr int GGP_THREADS = 192;           // warp 0: TMA, warp 1: MMA + tensor memory, warps 2-5: epilogue
constexpr int GGP_STAGES = 6, GGP_ROWS = 256, GGP_BOX = 32, GGP_MAX_EXPERTS = 512;
constexpr unsigned GGP_A_BYTES = TC_BM * TC_BK * 2;
constexpr unsigned GGP_STAGE = GGP_A_BYTES + GGP_ROWS / 2 * TC_BK * 2;
constexpr size_t GGP_SMEM = 1024 + (size_t)GGP_STAGES * GGP_STAGE;

struct GroupedPairParams {
    void* out;              // [rows][ldo] float or bfloat16
    int ldo, out_dtype;
    int n_out, K, E;
    int act;                // 0: none; 1: the square of relu
    const int* offsets;     // [E + 1]
    unsigned* status;
};

// The rows under boxes of 32, 64, 96 and 128 rows: whatever a tile's width, a CTA's half of it is one copy (a copy costs the thread
// that asks for it a good part of what the MMAs of a k-block take: 45.0 us with one box, 47.0 with four of 32 rows, in the example below)
struct GroupedPairMaps { CUtensorMap box[4]; };

__global__ void __launch_bounds__(GGP_THREADS, 1)
gemm_grouped_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ GroupedPairMaps map_x, GroupedPairParams p) {
    extern __shared__ unsigned char ggp_raw[];
    unsigned char* tiles = (unsigned char*)(((uintptr_t)ggp_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) unsigned long long full_bar[GGP_STAGES], empty_bar[GGP_STAGES], acc_full[2], acc_empty[2];
    __shared__ int row_s[GGP_MAX_EXPERTS + 1];       // the experts' first rows
    __shared__ int tile_s[GGP_MAX_EXPERTS + 1];      // row tiles of the experts before
    __shared__ int total_s[3];
    __shared__ unsigned tmem_base_sh;
    __shared__ int failed;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const int n_pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
    const int n_kb = (p.K + TC_BK - 1) / TC_BK, tiles_m = (p.n_out + 2 * TC_BM - 1) / (2 * TC_BM);

    if (threadIdx.x == 0) {
        for (int s = 0; s < GGP_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 8); }
        total_s[0] = total_s[1] = total_s[2] = 0;
        failed = 0;
        mbar_init_fence();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_sh)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                     // the peer's barriers are initialised before anything is signalled there
    tc_fence_after();
    const unsigned tmem_base = tmem_base_sh;
    pdl_launch();
    pdl_wait();                             // the offsets are this step's

    // ---------------- the tiles of this distribution of the rows
    for (int e = threadIdx.x; e <= p.E; e += GGP_THREADS) {
        row_s[e] = p.offsets[e];
        if (e == p.E) continue;
        const int cnt = p.offsets[e + 1] - p.offsets[e];
        if (cnt <= 0) continue;
        atomicAdd(&total_s[0], (cnt + 255) / 256);
        atomicAdd(&total_s[1], (cnt + 191) / 192);
        atomicAdd(&total_s[2], (cnt + 127) / 128);
    }
    __syncthreads();
    int width = 256;
    {
        const int r0 = (total_s[0] * tiles_m + n_pairs - 1) / n_pairs * 512, r1 = (total_s[1] * tiles_m + n_pairs - 1) / n_pairs * 448,
                  r2 = (total_s[2] * tiles_m + n_pairs - 1) / n_pairs * 384;
        if (r1 < r0) width = 192;
        if (r2 < min(r0, r1)) width = 128;
    }
    if (warp == 0) {
        int run = 0;
        for (int e0 = 0; e0 < p.E; e0 += 32) {
            const int e = e0 + lane;
            const int n = e < p.E ? (max(row_s[e + 1] - row_s[e], 0) + width - 1) / width : 0;
            int upto = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (e < p.E) tile_s[e] = run + upto - n;
            run += __shfl_sync(0xffffffffu, upto, 31);
        }
        if (lane == 0) tile_s[p.E] = run;
    }
    __syncthreads();
    const int n_tiles = tile_s[p.E] * tiles_m;
    struct Tile { int m0, w_row, row0, rows, n; };      // features from m0, weight row, first row, its rows, N of the MMA
    auto tile_of = [&](int i) {
        const int j = i / tiles_m;                       // row tile: the last expert whose first tile is not behind it
        int lo = 0, hi = p.E - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (tile_s[mid] <= j) lo = mid; else hi = mid - 1;
        }
        const int cnt = row_s[lo + 1] - row_s[lo], parts = tile_s[lo + 1] - tile_s[lo];
        const int each = ((cnt + parts - 1) / parts + 63) & ~63, at = (j - tile_s[lo]) * each;
        Tile t;
        t.m0 = (i - j * tiles_m) * 2 * TC_BM;
        t.w_row = lo * p.n_out + t.m0;
        t.row0 = row_s[lo] + at;
        t.rows = max(min(each, cnt - at), 0);
        t.n = max((t.rows + 63) & ~63, 64);
        return t;
    };

    bool ok = true;
    if (warp == 0) {
        // ---------------- TMA producer (in both CTAs: own features, own half of the rows)
        if (lane == 0) {
            int it = 0;
            for (int i = pair; i < n_tiles && ok; i += n_pairs) {
                const Tile t = tile_of(i);
                const int half = t.n / 2;
                const CUtensorMap* rows_map = &map_x.box[half / GGP_BOX - 1];
                const int w_row = t.w_row + (int)rank * TC_BM, x_row = t.row0 + (int)rank * half;
                const unsigned bytes = 2 * (GGP_A_BYTES + (unsigned)half * TC_BK * 2);
                for (int kb = 0; kb < n_kb; ++kb, ++it) {
                    const int s = it % GGP_STAGES;
                    if (it >= GGP_STAGES && !mbar_wait(&empty_bar[s], ((it / GGP_STAGES) - 1) & 1, &failed)) { ok = false; break; }
                    unsigned char* a = tiles + (size_t)s * GGP_STAGE;
                    if (rank == 0) mbar_expect_tx(&full_bar[s], bytes);
                    const unsigned bar = peer_addr(smem_u32(&full_bar[s]), 0);
                    tma_load_2d_pair(a, &map_w, kb * TC_BK, w_row, bar);
                    tma_load_2d_pair(a + GGP_A_BYTES, rows_map, kb * TC_BK, x_row, bar);
                }
            }
            if (!ok) atomicExch(&failed, 1);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: one thread of the pair's first CTA
        if (rank == 0) {
            int it = 0, t_idx = 0;
            auto wait_all = [&](unsigned long long* bar, unsigned parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, &failed)) != 0; };
            for (int i = pair; i < n_tiles && ok; i += n_pairs, ++t_idx) {
                const int b = t_idx & 1;
                const unsigned idesc = instr_desc_bf16(2 * TC_BM, tile_of(i).n);
                if (t_idx >= 2) ok = wait_all(&acc_empty[b], ((t_idx >> 1) - 1) & 1);
                if (!ok) break;
                tc_fence_after();
                const unsigned d = tmem_base + (unsigned)(b * GGP_ROWS);
                for (int kb = 0; kb < n_kb; ++kb, ++it) {
                    const int s = it % GGP_STAGES;
                    ok = wait_all(&full_bar[s], (it / GGP_STAGES) & 1);
                    if (!ok) break;
                    tc_fence_after();
                    const unsigned a_addr = smem_u32(tiles + (size_t)s * GGP_STAGE), b_addr = a_addr + GGP_A_BYTES;
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k)
                            tc_mma_pair(d, smem_desc_sw128(a_addr + k * 32), smem_desc_sw128(b_addr + k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        tc_commit_pair(&empty_bar[s]);  // the stage is free in both CTAs once these MMAs have read it
                        if (kb == n_kb - 1) tc_commit_pair(&acc_full[b]);
                    }
                    __syncwarp();
                }
            }
            if (!ok && lane == 0) atomicExch(&failed, 1);
        }
    } else {
        // ---------------- epilogue: warps 2..5 own tensor-memory lanes 32 * (warp % 4) .. + 31: a lane is a feature, a column a row
        const int quarter = warp & 3;
        const unsigned acc_empty_first = peer_addr(smem_u32(&acc_empty[0]), 0);
        int t_idx = 0;
        for (int i = pair; i < n_tiles && ok; i += n_pairs, ++t_idx) {
            const Tile t = tile_of(i);
            const int b = t_idx & 1, m = t.m0 + (int)rank * TC_BM + quarter * 32 + lane;
            ok = mbar_wait(&acc_full[b], (t_idx >> 1) & 1, &failed);
            ok = __all_sync(0xffffffffu, ok) != 0;
            if (!ok) break;
            tc_fence_after();
            const unsigned t_addr = tmem_base + ((unsigned)(quarter * 32) << 16) + (unsigned)(b * GGP_ROWS);
            // where features end inside a warp, lanes without one wait for the others, since a load of tensor memory is the whole warp's (a loop of its own:
            // with a condition in it the other one lost 1 to 3 %)
            auto drain = [&](auto wait) {
                for (int c = 0; c < t.rows; c += 32) {
                    float v[32];
                    tc_ld32(t_addr + (unsigned)c, v);
                    if (p.act == 1) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) { v[j] = fmaxf(v[j], 0.0f); v[j] *= v[j]; }
                    }
                    if (m < p.n_out) {
                        const int left = t.rows - c;
                        const size_t o = (size_t)(t.row0 + c) * p.ldo + m;
                        if (p.out_dtype == BG_DTYPE_F32) {
                            float* to = (float*)p.out + o;
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (j < left) to[(size_t)j * p.ldo] = v[j];
                        } else {
                            __nv_bfloat16* to = (__nv_bfloat16*)p.out + o;
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (j < left) to[(size_t)j * p.ldo] = __float2bfloat16_rn(v[j]);
                        }
                    }
                    if constexpr (decltype(wait)::value) __syncwarp();
                }
            };
            if (p.n_out % 32 != 0 && t.m0 + (int)rank * TC_BM + TC_BM > p.n_out) drain(std::true_type{});
            else drain(std::false_type{});
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_empty_first + (unsigned)(b * sizeof(unsigned long long)));
        }
        if (!ok) atomicExch(&failed, 1);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                     // neither CTA frees tensor memory or leaves while its peer may still signal it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base), "r"(512u) : "memory");
    }
    if (threadIdx.x == 0 && failed && p.status) atomicOr(p.status, BG_STATUS_TIMEOUT);
}

}  // namespace bg

using namespace bg;

// The arguments of bg_gemm_grouped_tc; BG_ERR_UNSUPPORTED (before anything is launched) for more than 512 experts.
extern "C" int bg_gemm_grouped_pair(const void* W, int E, int n_out, int K, int ldw, const void* X, int rows, int ldx, void* out,
                                    int out_dtype, int ldo, const int* offsets, int act, unsigned* status, cudaStream_t stream) {
    if (rows <= 0 || n_out <= 0) return BG_OK;
    if (K <= 0 || E <= 0) return BG_ERR_SHAPE;
    if (E > GGP_MAX_EXPERTS) return BG_ERR_UNSUPPORTED;
    if ((ldw % 8) || (ldx % 8) || ((uintptr_t)W % 16) || ((uintptr_t)X % 16)) return BG_ERR_ALIGN;
    if (out_dtype != BG_DTYPE_F32 && out_dtype != BG_DTYPE_BF16) return BG_ERR_DTYPE;
    CUtensorMap mw;
    GroupedPairMaps mx;
    int rc = weight_map(&mw, W, E * n_out, K, ldw);
    for (int i = 0; i < 4 && rc == BG_OK; ++i) rc = make_map(&mx.box[i], X, rows, K, ldx, (i + 1) * GGP_BOX);
    if (rc != BG_OK) return rc;
    GroupedPairParams p;
    p.out = out; p.ldo = ldo; p.out_dtype = out_dtype; p.n_out = n_out; p.K = K; p.E = E; p.act = act; p.offsets = offsets; p.status = status;
    const long long most = (long long)((n_out + 2 * TC_BM - 1) / (2 * TC_BM)) * (rows / 128 + E);
    int pairs = sm_count() / 2;
    if (pairs > most) pairs = (int)most;
    if (pairs < 1) return BG_ERR_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(gemm_grouped_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GGP_SMEM);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs); cfg.blockDim = dim3(GGP_THREADS); cfg.dynamicSmemBytes = GGP_SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 2; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
    ++n;
    cfg.attrs = attr; cfg.numAttrs = n;
    e = cudaLaunchKernelEx(&cfg, gemm_grouped_pair_kernel, mw, mx, p);
    if (e != cudaSuccess) return (int)e;
    BG_LAUNCH_CHECK();
    return BG_OK;
}
