// Routed experts: what stands around the experts' products.
//
//   route_topk     per token, the `top` experts of largest score (score = sigmoid of the router's float logit, or the
//                  logit itself), ties to the lower index; the logits are what is compared, since sigmoid keeps their
//                  order but rounds large ones to equal scores.  The weight of a choice is its score, divided by the
//                  sum of the chosen scores when `renorm`.
//   route_sort     the step's assignments (token t, rank j) -> a = t * top + j are laid out expert by expert:
//                  offsets[e] .. offsets[e + 1] are expert e's rows; row_of[a] is where assignment a went and
//                  src_of[row] the assignment that row holds.  ONE CTA; the order inside an expert is whatever the
//                  atomics give, which no result depends on (a row's product is a function of that row alone).
//   route_rows     the three above and below for a step of few tokens in one kernel, a cluster of CTAs.
//   route_place    route_sort and route_gather in one kernel, from counts that the router's kernel leaves: for many outputs.
//   route_gather   xp[row] = (weight * x[token]) rounded to the compute type (or x[token] as it is).
//   gemm_grouped   yp[row] = act(xp[row] W[e]^T) on CUDA cores, float accumulation, every output summed over k in index
//                  order by one thread: the float32 path, and the sizes the tensor-core product does not take.
//   route_combine  out[t] = sum_j (weight *) yp[row_of[t * top + j]], ranks added in index order, float.
//
// Nothing here is read back to the host: the grids depend on the step's shapes alone (the grouped products are launched
// with as many row tiles as any distribution of the tokens could need, and a CTA without rows returns), so a step with
// routed experts can be captured in a graph.
#include "common.cuh"

namespace bg {

// How the router's logits become scores (`mode`): 0 the logit itself, 1 its sigmoid, 2 the softmax over all E logits, 3 the
// softmax over the chosen logits only (the choice is made on the logits themselves).
struct RouteRule {
    int mode;
    int renorm;             // the chosen scores are divided by their sum
    const float* bias;      // [E] or null: added to the scores for the CHOICE only; the weights are the scores without it
    float scale;            // multiplies the weights
    const float* logit_bias;    // [E] or null: part of the logits
};

// One warp chooses for one token: `sc` holds the token's E logits in shared memory and is used up.  Without a bias and
// without the softmax the choice is made on the logits: sigmoid keeps their order, but rounds large ones to the same
// score.  Otherwise it is made on score + bias, the scores formed anew from the logits each time; a logit of -inf marks
// an expert that is taken.  Ties go to the lower index.
__device__ __forceinline__ void choose_experts(float* sc, int E, int top, RouteRule rule, int* __restrict__ ids,
                                               float* __restrict__ weights, size_t t, int lane) {
    float total = 0.0f;
    float zmax = 0.0f, inv = 1.0f;
    if (rule.logit_bias) {
        for (int e = lane; e < E; e += 32) sc[e] += rule.logit_bias[e];
        __syncwarp();
    }
    if (rule.mode == 2) {                                  // softmax over all experts, float
        float m = -INFINITY;
        for (int e = lane; e < E; e += 32) m = fmaxf(m, sc[e]);
        zmax = warp_max(m);
        float s = 0.0f;
        for (int e = lane; e < E; e += 32) s += expf(sc[e] - zmax);
        inv = 1.0f / warp_sum(s);
    }
    const bool on_scores = rule.mode == 2 || rule.bias != nullptr;
    auto score_of = [&](float z) {
        return rule.mode >= 2 ? expf(z - zmax) * inv : (rule.mode == 1 ? 1.0f / (1.0f + expf(-z)) : z);
    };
    for (int j = 0; j < top; ++j) {
        float best = -INFINITY;
        int arg = 0x7fffffff;
        for (int e = lane; e < E; e += 32) {
            float v = sc[e];
            if (on_scores && v != -INFINITY) v = score_of(v) + (rule.bias ? rule.bias[e] : 0.0f);
            if (v > best) { best = v; arg = e; }            // ascending e: the first of equal scores stays
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
        }
        if (arg == 0x7fffffff) arg = 0;                     // (every score NaN or -inf: a defined choice)
        if (rule.mode == 3 && j == 0) zmax = sc[arg];           // (without a choice bias the first choice is the largest)
        const float score = score_of(on_scores ? sc[arg] : best);
        __syncwarp();
        if (lane == 0) {
            ids[(size_t)t * top + j] = arg;
            weights[(size_t)t * top + j] = score * rule.scale;
            sc[arg] = -INFINITY;
        }
        total += score;
        __syncwarp();
    }
    if ((rule.renorm || rule.mode == 3) && lane < top) weights[(size_t)t * top + lane] /= total;
}

__global__ void route_topk_kernel(const float* __restrict__ logits, int T, int E, int top, RouteRule rule,
                                  int* __restrict__ ids, float* __restrict__ weights) {
    extern __shared__ float score_s[];                     // [warps][E]
    pdl_launch();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= T) return;
    float* sc = score_s + (size_t)warp * E;
    for (int e = lane; e < E; e += 32) sc[e] = logits[(size_t)t * E + e];
    __syncwarp();
    choose_experts(sc, E, top, rule, ids, weights, (size_t)t, lane);
}

// The router of a step in one kernel: a block takes ROUTE_TOKENS tokens; each of its warps takes experts in turn and
// forms the float logits of all the block's tokens against that expert's row (the row is read once per block; a lane
// walks the features 32 apart and the warp adds up, so a logit's order of summation depends on nothing but the width);
// then warp w chooses for token w.  `logits_out`, when given, also receives the logits.
constexpr int ROUTE_LOG = 3, ROUTE_TOKENS = 1 << ROUTE_LOG, ROUTE_UNROLL = 8;
template <typename TI>
__global__ void __launch_bounds__(32 * ROUTE_TOKENS)
route_kernel(const TI* __restrict__ h, int ldh, const float* __restrict__ W, int T, int d, int E, int top, RouteRule rule,
             int* __restrict__ ids, float* __restrict__ weights, float* __restrict__ logits_out) {
    extern __shared__ float logit_s[];                     // [ROUTE_TOKENS][E]
    pdl_launch();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t0 = blockIdx.x * ROUTE_TOKENS;
    const int n = min(ROUTE_TOKENS, T - t0);
    for (int e = warp; e < E; e += ROUTE_TOKENS) {
        float acc[ROUTE_TOKENS];
#pragma unroll
        for (int j = 0; j < ROUTE_TOKENS; ++j) acc[j] = 0.0f;
        const float* w = W + (size_t)e * d;
        // ROUTE_UNROLL features a lane at a time: all their loads go out before the first product (one feature at a time
        // cost a trip to memory per feature: 58 us for 1,536 features, whatever the number of tokens)
        for (int k0 = lane; k0 < d; k0 += 32 * ROUTE_UNROLL) {
            float wk[ROUTE_UNROLL], hv[ROUTE_UNROLL][ROUTE_TOKENS];
#pragma unroll
            for (int u = 0; u < ROUTE_UNROLL; ++u) {
                const int k = k0 + 32 * u;
                wk[u] = k < d ? w[k] : 0.0f;
#pragma unroll
                for (int j = 0; j < ROUTE_TOKENS; ++j)
                    hv[u][j] = (k < d && j < n) ? to_float(h[(size_t)(t0 + j) * ldh + k]) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < ROUTE_UNROLL; ++u)
#pragma unroll
                for (int j = 0; j < ROUTE_TOKENS; ++j) acc[j] = fmaf(hv[u][j], wk[u], acc[j]);
        }
#pragma unroll
        for (int j = 0; j < ROUTE_TOKENS; ++j) {
            const float v = warp_sum(acc[j]);
            if (lane == 0 && j < n) {
                logit_s[j * E + e] = v;
                if (logits_out) logits_out[(size_t)(t0 + j) * E + e] = v;
            }
        }
    }
    __syncthreads();
    if (warp < n) choose_experts(logit_s + warp * E, E, top, rule, ids, weights, (size_t)(t0 + warp), lane);
}

// The logits of TPW tokens' rows (row, row + ldh, ..; those from `live` on are the first one's again and not stored) by `warps` warps of a block
// (this is the `warp`-th), each a group of G experts at a time: a lane walks the features in chunks of eight, 32 chunks apart (16-byte
// loads), and the warp adds up.  An expert's row is fetched once for all the tokens; a logit's sum does not depend on TPW, G or `warps`.
// Several tokens: experts from E on are the last one again and not stored, since a condition on the loads keeps them from being on their way
// together.  One token: loads under conditions, which fetch nothing twice (18 outputs of 4,096 features 9.8 us, without conditions 10.4).
template <typename TI, int TPW, int G>
__device__ __forceinline__ void route_logits_of(const TI* row, int ldh, int live, const float* __restrict__ W, int d8, int d, int E, float* sc,
                                                float* logits_out, int warp, int warps, int lane) {
    for (int e0 = warp * G; e0 < E; e0 += warps * G) {
        float acc[TPW][G];
#pragma unroll
        for (int q = 0; q < TPW; ++q)
#pragma unroll
            for (int u = 0; u < G; ++u) acc[q][u] = 0.0f;
#pragma unroll 2
        for (int c = lane; c < d8; c += 32) {
            float hv[TPW][8], wv[G][8];
#pragma unroll
            for (int q = 0; q < TPW; ++q) load8(row + (size_t)(q < live ? q : 0) * ldh + 8 * c, hv[q]);
            if constexpr (TPW == 1) {
#pragma unroll
                for (int u = 0; u < G; ++u)
                    if (e0 + u < E) {
                        load8(W + (size_t)(e0 + u) * d + 8 * c, wv[u]);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[0][u] = fmaf(hv[0][i], wv[u][i], acc[0][u]);
                    }
            } else {
#pragma unroll
            for (int u = 0; u < G; ++u) load8(W + (size_t)min(e0 + u, E - 1) * d + 8 * c, wv[u]);
#pragma unroll
            for (int u = 0; u < G; ++u)
#pragma unroll
                for (int q = 0; q < TPW; ++q)
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[q][u] = fmaf(hv[q][i], wv[u][i], acc[q][u]);
            }
        }
#pragma unroll
        for (int q = 0; q < TPW; ++q)
#pragma unroll
            for (int u = 0; u < G; ++u) {
                const float v = warp_sum(acc[q][u]);
                if (lane == 0 && e0 + u < E && q < live) {
                    sc[q * E + e0 + u] = v;
                    if (logits_out) logits_out[(size_t)q * E + e0 + u] = v;
                }
            }
    }
}

// The same for a width that is a multiple of 8 and 16-byte aligned rows.  A block of eight warps takes TPW x 8 / wpt tokens: `wpt` warps share
// TPW tokens' experts in groups of G, and every warp then chooses for some of the block's tokens.  Steps of few tokens: a block per token and
// an expert per warp at a time, so that a decoding step spreads over as many SMs as it has tokens and a warp's chain of loads is one
// expert long.  Steps of many: four tokens a warp, four experts at a time.  What bounds it is the router's float rows, which every token needs
// whole: with a warp to one token they came through the first-level cache once a token (2,048 tokens, 8 experts, 1,536 features: 17.0 -> 8.9 us).
// `hist`, when given, receives how many of the block's assignments each expert has, [blocks][E].
template <typename TI, int TPW, int G>
__global__ void __launch_bounds__(32 * ROUTE_TOKENS)
route_vec8_kernel(const TI* __restrict__ h, int ldh, const float* __restrict__ W, int T, int d, int E, int top, RouteRule rule, int wpt_log,
                  int* __restrict__ ids, float* __restrict__ weights, float* __restrict__ logits_out, int* __restrict__ hist) {
    extern __shared__ float logit_s[];                     // [tokens][E], then the experts' counts
    pdl_launch();
    const int wpt = 1 << wpt_log;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tokens = TPW << (ROUTE_LOG - wpt_log), t0 = blockIdx.x * tokens, n = min(tokens, T - t0);
    const int first = (warp >> wpt_log) * TPW;                // of this warp's tokens, in the block
    const int live = min(TPW, n - first);
    int* count_s = (int*)(logit_s + tokens * E);
    if (hist) for (int e = threadIdx.x; e < E; e += blockDim.x) count_s[e] = 0;
    pdl_wait();
    if (live > 0)
        route_logits_of<TI, TPW, G>(h + (size_t)(t0 + first) * ldh, ldh, live, W, d >> 3, d, E, logit_s + first * E,
                                    logits_out ? logits_out + (size_t)(t0 + first) * E : nullptr, warp & (wpt - 1), wpt, lane);
    __syncthreads();                                       // every warp comes here, with or without a token
    for (int tl = warp; tl < n; tl += ROUTE_TOKENS) {
        choose_experts(logit_s + tl * E, E, top, rule, ids, weights, (size_t)(t0 + tl), lane);
        if (hist) {
            __syncwarp();
            if (lane < top) atomicAdd(&count_s[ids[(size_t)(t0 + tl) * top + lane]], 1);
        }
    }
    if (!hist) return;
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += blockDim.x) hist[(size_t)blockIdx.x * E + e] = count_s[e];
}

// What route_sort and route_gather do, for the same blocks of `tokens` tokens as the router's kernel ahead, from its counts: every block adds up the
// counts (RL_MAX of them at most) for itself, so an expert's rows begin behind those of smaller experts, a block's behind those of the
// blocks before it, and inside a block they stand in the order of the assignments.  No atomics: the order is the same every time.
// gridDim.y blocks share the columns of a block's rows.  Bound by bytes and by the chain of counts, prefix and rows in front of them
// (bg_route_layout_wins says where that chain is worth the sort that it saves).
constexpr int RL_MAX = 8192, RL_MAX_E = 256, RL_MAX_A = 512;
template <typename TI>
__global__ void __launch_bounds__(256)
route_place_kernel(const TI* __restrict__ h, int ldh, const float* __restrict__ weights, const int* __restrict__ ids, const int* __restrict__ hist,
                   int T, int d, int E, int top, int tokens, int* __restrict__ offsets, int* __restrict__ row_of, int* __restrict__ src_of,
                   TI* __restrict__ xp, int scale) {
    __shared__ int before_s[RL_MAX_E], total_s[RL_MAX_E], expert_s[RL_MAX_A], row_s[RL_MAX_A];
    __shared__ float weight_s[RL_MAX_A];
    pdl_launch();
    const int tid = threadIdx.x, t0 = blockIdx.x * tokens, n = min(tokens, T - t0), A = n * top, a0 = t0 * top;
    for (int e = tid; e < E; e += blockDim.x) { before_s[e] = 0; total_s[e] = 0; }
    pdl_wait();
    for (int a = tid; a < A; a += blockDim.x) { expert_s[a] = ids[a0 + a]; weight_s[a] = scale ? weights[a0 + a] : 1.0f; }
    __syncthreads();
    {
        int ep = 1;                                        // threads of the same expert: ep apart
        while (ep < E) ep *= 2;
        const int e = tid & (ep - 1), step = 256 / ep;
        int total = 0, before = 0;
        if (e < E) {
#pragma unroll 8
            for (int b = tid / ep; b < (int)gridDim.x; b += step) {
                const int c = hist[b * E + e];
                total += c;
                before += b < (int)blockIdx.x ? c : 0;
            }
        }
        for (int o = ep; o < 32; o *= 2) { total += __shfl_xor_sync(0xffffffffu, total, o); before += __shfl_xor_sync(0xffffffffu, before, o); }
        if (e < E && (tid & 31) < ep) { atomicAdd(&total_s[e], total); atomicAdd(&before_s[e], before); }
    }
    __syncthreads();
    if (tid < 32) {                                        // totals become the experts' first rows
        int run = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int c = e0 + tid < E ? total_s[e0 + tid] : 0;
            int up = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, up, o);
                if (tid >= o) up += u;
            }
            if (e0 + tid < E) {
                total_s[e0 + tid] = run + up - c;
                if (blockIdx.x == 0 && blockIdx.y == 0) offsets[e0 + tid] = run + up - c;
            }
            run += __shfl_sync(0xffffffffu, up, 31);
        }
        if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) offsets[E] = run;
    }
    __syncthreads();
    for (int a = tid; a < A; a += blockDim.x) {
        const int e = expert_s[a];
        int row = total_s[e] + before_s[e];
#pragma unroll 8
        for (int b = 0; b < a; ++b) row += expert_s[b] == e ? 1 : 0;
        row_s[a] = row;
        if (blockIdx.y == 0) { row_of[a0 + a] = row; src_of[row] = a0 + a; }
    }
    __syncthreads();
    // a warp to a token at a time, its share of the columns four pieces a lane on their way together
    const int d8 = d >> 3, c0 = (int)((long long)d8 * blockIdx.y / gridDim.y), c1 = (int)((long long)d8 * (blockIdx.y + 1) / gridDim.y);
    for (int tl = tid >> 5; tl < n; tl += 8) {
        const TI* from = h + (size_t)(t0 + tl) * ldh;
        for (int c = c0 + (tid & 31); c < c1; c += 128) {
            float x[4][8];
#pragma unroll
            for (int u = 0; u < 4; ++u) load8(from + 8 * min(c + 32 * u, c1 - 1), x[u]);
            for (int j = 0; j < top; ++j) {
                const float wt = weight_s[tl * top + j];
                TI* to = xp + (size_t)row_s[tl * top + j] * d;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float v[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) v[q] = wt * x[u][q];
                    if (c + 32 * u < c1) store8(to + 8 * (c + 32 * u), v);
                }
            }
        }
    }
}

// Routing, layout and gather of a step of few tokens as ONE kernel: three dependent launches cost more than their work, on
// the device (eight tokens, ten router outputs: 8.0 us as three kernels, 6.4 as one) and most of all, outside a graph, on the host (a
// gated layer with identity and shared experts: 138 -> 125 us).  A cluster of eight CTAs, a token each, routed as in the kernel above
// (the same sums, so the same choice); with two tokens a CTA, one after the other, it lost (10.7 against 8.1 us).  The CTAs read each other's choices through the cluster, each lays out all
// assignments for itself (an assignment's row: those of smaller experts and the earlier ones of its own, counted) and gathers its own
// tokens' rows.  Inside an expert the rows stand in the order of the assignments.
constexpr int RR_CTAS = 8, RR_TOKENS = 8, RR_MAX_A = 256;
template <typename TI, int G>
__global__ void __launch_bounds__(32 * ROUTE_TOKENS)
route_rows_kernel(const TI* __restrict__ h, int ldh, const float* __restrict__ W, int T, int d, int E, int top, RouteRule rule,
                  int* __restrict__ ids, float* __restrict__ weights, int* __restrict__ offsets, int* __restrict__ row_of,
                  int* __restrict__ src_of, TI* __restrict__ xp, int scale) {
    extern __shared__ float logit_s[];                     // [E]
    __shared__ int all_s[RR_MAX_A], row_s[RR_MAX_A];       // every assignment's expert (own tokens' first), its row
    pdl_launch();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    const int rank = blockIdx.z, A = T * top, d8 = d >> 3;
    const int t = rank;                                    // this CTA's token
    if (t < T) {
        route_logits_of<TI, 1, G>(h + (size_t)t * ldh, ldh, 1, W, d8, d, E, logit_s, nullptr, warp, ROUTE_TOKENS, lane);
        __syncthreads();
        if (warp == 0) {
            choose_experts(logit_s, E, top, rule, ids, weights, (size_t)t, lane);
            if (lane < top) all_s[t * top + lane] = ids[(size_t)t * top + lane];
        }
    }
    cluster_sync_all();
    for (int a = tid; a < A; a += blockDim.x) {            // the other CTAs' tokens, from where they were routed
        const int owner = a / top;
        if (owner == rank) continue;
        int v;
        asm volatile("ld.shared::cluster.s32 %0, [%1];\n" : "=r"(v) : "r"(peer_addr((unsigned)__cvta_generic_to_shared(&all_s[a]), (unsigned)owner)) : "memory");
        all_s[a] = v;
    }
    cluster_sync_all();                                    // (nobody leaves, or is read, before all have read)
    for (int a = tid; a < A; a += blockDim.x) {
        const int e = all_s[a];
        int row = 0;
        for (int b = 0; b < A; ++b) row += all_s[b] < e || (all_s[b] == e && b < a) ? 1 : 0;
        row_s[a] = row;
        if (rank == 0) { row_of[a] = row; src_of[row] = a; }
    }
    if (rank == 0) {
        for (int e = tid; e <= E; e += blockDim.x) {
            int n = 0;
            for (int b = 0; b < A; ++b) n += all_s[b] < e ? 1 : 0;
            offsets[e] = n;
        }
    }
    __syncthreads();
    for (int c = tid; t < T && c < d8; c += blockDim.x) {
        float x[8];
        load8(h + (size_t)t * ldh + 8 * c, x);
        for (int j = 0; j < top; ++j) {
            const int a = t * top + j;
            const float w = scale ? weights[a] : 1.0f;
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = w * x[i];
            store8(xp + (size_t)row_s[a] * d + 8 * c, v);
        }
    }
}

__global__ void __launch_bounds__(1024)
route_sort_kernel(const int* __restrict__ ids, int A, int E, int* __restrict__ offsets, int* __restrict__ row_of,
                  int* __restrict__ src_of) {
    extern __shared__ int count_s[];                       // [E] counts, then [E] cursors
    int* cursor_s = count_s + E;
    pdl_launch();
    for (int e = threadIdx.x; e < E; e += blockDim.x) count_s[e] = 0;
    pdl_wait();
    __syncthreads();
    for (int a = threadIdx.x; a < A; a += blockDim.x) {
        const int e = ids[a];
        if (e >= 0 && e < E) atomicAdd(&count_s[e], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < E; ++e) { offsets[e] = run; cursor_s[e] = run; run += count_s[e]; }
        offsets[E] = run;
    }
    __syncthreads();
    for (int a = threadIdx.x; a < A; a += blockDim.x) {
        const int e = ids[a];
        if (e < 0 || e >= E) continue;
        const int row = atomicAdd(&cursor_s[e], 1);
        row_of[a] = row;
        src_of[row] = a;
    }
}

template <typename TI, typename TO>
__global__ void route_gather_kernel(const TI* __restrict__ x, const float* __restrict__ weights, const int* __restrict__ src_of,
                                    TO* __restrict__ xp, int A, int d, int top, int scale) {
    pdl_launch();
    pdl_wait();
    const int row = blockIdx.x;
    const int a = src_of[row];
    const float w = scale ? weights[a] : 1.0f;
    const TI* src = x + (size_t)(a / top) * d;
    TO* dst = xp + (size_t)row * d;
    for (int i = threadIdx.x; i < d; i += blockDim.x) dst[i] = from_float<TO>(w * to_float(src[i]));
}

// The same with 16-byte accesses (d a multiple of 8, rows on 16-byte boundaries), a warp to a row, four of a lane's loads on their way
// together.  Bound by bytes (4,096 rows of 1,536: 8.5 -> 4.2 us).
template <typename TI, typename TO>
__global__ void __launch_bounds__(256)
route_gather_vec8_kernel(const TI* __restrict__ x, const float* __restrict__ weights, const int* __restrict__ src_of, TO* __restrict__ xp,
                         int A, int d, int top, int scale) {
    pdl_launch();
    pdl_wait();
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), d8 = d >> 3;
    if (row >= A) return;
    const int a = src_of[row];
    const float w = scale ? weights[a] : 1.0f;
    const TI* src = x + (size_t)(a / top) * d;
    TO* dst = xp + (size_t)row * d;
    for (int c0 = threadIdx.x & 31; c0 < d8; c0 += 128) {
        float v[4][8];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + 32 * u < d8) load8(src + (size_t)(c0 + 32 * u) * 8, v[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (c0 + 32 * u < d8) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[u][i] = w * v[u][i];
                store8(dst + (size_t)(c0 + 32 * u) * 8, v[u]);
            }
    }
}

template <typename TY>
__global__ void route_combine_kernel(const TY* __restrict__ yp, const float* __restrict__ weights, const int* __restrict__ row_of,
                                     float* __restrict__ out, int T, int d, int top, int scale) {
    pdl_launch();
    pdl_wait();
    const int t = blockIdx.x;
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float acc = 0.0f;
        for (int j = 0; j < top; ++j) {
            const int a = t * top + j;
            const float v = to_float(yp[(size_t)row_of[a] * d + i]);
            acc += scale ? weights[a] * v : v;
        }
        out[(size_t)t * d + i] = acc;
    }
}

// The same for float results, four columns a thread (d a multiple of 4, rows on 16-byte boundaries); the columns of all tokens in one
// row of threads.  Bound by bytes (2,048 tokens, two rows of 1,536 each: 9.7 -> 5.1 us).
__global__ void __launch_bounds__(256)
route_combine_vec4_kernel(const float* __restrict__ yp, const float* __restrict__ weights, const int* __restrict__ row_of,
                          float* __restrict__ out, int T, int d, int top, int scale) {
    pdl_launch();
    pdl_wait();
    const int d4 = d >> 2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int t = (int)(idx / d4), i = (int)(idx - (long long)t * d4) * 4;
    if (t >= T) return;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int j = 0; j < top; ++j) {
        const int a = t * top + j;
        const float w = scale ? weights[a] : 1.0f;
        const float4 v = *reinterpret_cast<const float4*>(yp + (size_t)row_of[a] * d + i);
        acc.x += w * v.x; acc.y += w * v.y; acc.z += w * v.z; acc.w += w * v.w;
    }
    *reinterpret_cast<float4*>(out + (size_t)t * d + i) = acc;
}

// The same sum for a layer that also has experts without weights and a shared expert:
//   out[t] = sum_j w_j (id_j < n_real ? yp[row_of[t top + j]] : h[t])  +  sigmoid(sg[t]) shared[t].
// An expert whose index is n_real or more returns its input (the step's rows h in the compute type).  `shared` [T][d]
// float is the result of an expert that every token passes, `sg` one number per token (element t at sg[t * sg_stride], float
// or bfloat16), whose sigmoid multiplies it; without `sg` the shared result is added as it is.  Ranks in index order, float.
template <typename TY, typename TH>
__global__ void route_combine_ext_kernel(const TY* __restrict__ yp, const float* __restrict__ weights, const int* __restrict__ row_of,
                                         const int* __restrict__ ids, int n_real, const TH* __restrict__ h, int ldh,
                                         const float* __restrict__ shared, const void* __restrict__ sg, int sg_float, int sg_stride,
                                         float* __restrict__ out, int T, int d, int top) {
    pdl_launch();
    pdl_wait();
    const int t = blockIdx.x;
    float sgate = shared ? 1.0f : 0.0f;
    if (shared && sg) {
        const float z = sg_float ? ((const float*)sg)[(size_t)t * sg_stride] : __bfloat162float(((const __nv_bfloat16*)sg)[(size_t)t * sg_stride]);
        sgate = 1.0f / (1.0f + expf(-z));
    }
    for (int i = threadIdx.x; i < d; i += blockDim.x) {
        float acc = 0.0f;
        for (int j = 0; j < top; ++j) {
            const int a = t * top + j;
            const float v = ids[a] < n_real ? to_float(yp[(size_t)row_of[a] * d + i]) : to_float(h[(size_t)t * ldh + i]);
            acc = fmaf(weights[a], v, acc);
        }
        if (shared) acc = fmaf(sgate, shared[(size_t)t * d + i], acc);
        out[(size_t)t * d + i] = acc;
    }
}

// The same, four columns a thread (d a multiple of 4, float results of the experts, 16-byte aligned rows).
template <typename TH>
__global__ void route_combine_ext_vec4_kernel(const float* __restrict__ yp, const float* __restrict__ weights,
                                              const int* __restrict__ row_of, const int* __restrict__ ids, int n_real,
                                              const TH* __restrict__ h, int ldh, const float* __restrict__ shared,
                                              const void* __restrict__ sg, int sg_float, int sg_stride, float* __restrict__ out, int T,
                                              int d, int top) {
    pdl_launch();
    pdl_wait();
    const int t = blockIdx.x;
    float sgate = shared ? 1.0f : 0.0f;
    if (shared && sg) {
        const float z = sg_float ? ((const float*)sg)[(size_t)t * sg_stride] : __bfloat162float(((const __nv_bfloat16*)sg)[(size_t)t * sg_stride]);
        sgate = 1.0f / (1.0f + expf(-z));
    }
    for (int i = threadIdx.x * 4; i < d; i += blockDim.x * 4) {
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float4 hv;
        {
            const TH* hp = h + (size_t)t * ldh + i;
            hv = make_float4(to_float(hp[0]), to_float(hp[1]), to_float(hp[2]), to_float(hp[3]));
        }
        for (int j = 0; j < top; ++j) {
            const int a = t * top + j;
            const float w = weights[a];
            const float4 v = ids[a] < n_real ? *reinterpret_cast<const float4*>(yp + (size_t)row_of[a] * d + i) : hv;
            acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y); acc.z = fmaf(w, v.z, acc.z); acc.w = fmaf(w, v.w, acc.w);
        }
        if (shared) {
            const float4 s = *reinterpret_cast<const float4*>(shared + (size_t)t * d + i);
            acc.x = fmaf(sgate, s.x, acc.x); acc.y = fmaf(sgate, s.y, acc.y); acc.z = fmaf(sgate, s.z, acc.z); acc.w = fmaf(sgate, s.w, acc.w);
        }
        *reinterpret_cast<float4*>(out + (size_t)t * d + i) = acc;
    }
}

// A gated expert's activation with clamps: from a row [gate (n) | up (n)] of the product,
//   g = min(gate, limit), u = clamp(up, -limit, limit), out = g sigmoid(alpha g) (u + 1).
// Float arithmetic; the input in either type with `ld` elements between rows, the output contiguous.
template <typename TI, typename TO>
__global__ void glu_clamped_kernel(const TI* __restrict__ gu, int ld, TO* __restrict__ out, size_t total, int n, float limit,
                                   float alpha) {
    pdl_launch();
    pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const size_t r = idx / n;
    const int i = (int)(idx - r * n);
    const float g = fminf(to_float(gu[r * ld + i]), limit);
    const float u = fminf(fmaxf(to_float(gu[r * ld + n + i]), -limit), limit);
    out[idx] = from_float<TO>(g / (1.0f + expf(-alpha * g)) * (u + 1.0f));
}

// The same, eight columns a thread (n and ld multiples of 8, 16-byte aligned rows).
template <typename TI, typename TO>
__global__ void glu_clamped_vec8_kernel(const TI* __restrict__ gu, int ld, TO* __restrict__ out, size_t total8, int n, float limit,
                                        float alpha) {
    pdl_launch();
    pdl_wait();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total8) return;
    const int n8 = n >> 3;
    const size_t r = idx / n8;
    const int i = (int)(idx - r * n8) * 8;
    float g[8], u[8];
    load8(gu + r * ld + i, g);
    load8(gu + r * ld + n + i, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float gg = fminf(g[e], limit);
        const float uu = fminf(fmaxf(u[e], -limit), limit);
        g[e] = gg / (1.0f + expf(-alpha * gg)) * (uu + 1.0f);
    }
    store8(out + r * n + i, g);
}

// ------------------------------------------------------------------------------------------------ grouped product
// The expert and the rows of row tile `tile` (tiles of `bm` rows, expert after expert); false when there is none.
__device__ __forceinline__ bool group_tile(const int* offsets, int E, int bm, int tile, int* e_out, int* row0, int* n_rows) {
    int before = 0;
    for (int e = 0; e < E; ++e) {
        const int lo = offsets[e], n = offsets[e + 1] - lo;
        const int tiles = (n + bm - 1) / bm;
        if (tile < before + tiles) {
            const int r = (tile - before) * bm;
            *e_out = e; *row0 = lo + r; *n_rows = min(bm, n - r);
            return true;
        }
        before += tiles;
    }
    return false;
}

constexpr int GG_BM = 32, GG_BN = 64, GG_BK = 16, GG_THREADS = 256;

// C[row, n] = act(sum_k A[row, k] W[e][n, k]); ACT 1: the square of relu.
template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(GG_THREADS)
gemm_grouped_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W, int ldw, long long w_expert, TC* __restrict__ C,
                    int ldc, const int* __restrict__ offsets, int E, int N, int K, int act) {
    __shared__ float As[GG_BK][GG_BM + 4];
    __shared__ float Ws[GG_BK][GG_BN + 4];
    __shared__ int where[3];
    pdl_launch();
    pdl_wait();
    if (threadIdx.x == 0) {
        int e = -1, r0 = 0, n = 0;
        if (!group_tile(offsets, E, GG_BM, blockIdx.y, &e, &r0, &n)) e = -1;
        where[0] = e; where[1] = r0; where[2] = n;
    }
    __syncthreads();
    const int e = where[0], row0 = where[1], n_rows = where[2];
    if (e < 0) return;
    W += (size_t)e * w_expert;
    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * GG_BN;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, each 2 rows x 4 columns of C
    float acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += GG_BK) {
        // A tile: 32 rows x 16 k = 512 values, two a thread; W tile: 64 rows x 16 k = 1024 values, four a thread
        for (int idx = tid; idx < GG_BM * GG_BK; idx += GG_THREADS) {
            const int r = idx / GG_BK, k = idx - r * GG_BK;
            As[k][r] = (r < n_rows && k0 + k < K) ? to_float(A[(size_t)(row0 + r) * lda + k0 + k]) : 0.0f;
        }
        for (int idx = tid; idx < GG_BN * GG_BK; idx += GG_THREADS) {
            const int r = idx / GG_BK, k = idx - r * GG_BK;
            Ws[k][r] = (n0 + r < N && k0 + k < K) ? to_float(W[(size_t)(n0 + r) * ldw + k0 + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GG_BK; ++kk) {
            float a[2], w[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = As[kk][ty * 2 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = ty * 2 + i;
        if (r >= n_rows) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (act == 1) { v = fmaxf(v, 0.0f); v *= v; }
            C[(size_t)(row0 + r) * ldc + n] = from_float<TC>(v);
        }
    }
}

// C[M, N] = A[M, K] W[N, K]^T with A of either type and float W and C: the router's logits, float from a step's rows
// in the compute type.  Every output is summed over k in index order by one thread.
template <typename TA>
__global__ void __launch_bounds__(256)
gemm_rows_f32w_kernel(const TA* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C, int ldc,
                      int M, int N, int K) {
    __shared__ float As[16][64 + 4];
    __shared__ float Ws[16][64 + 4];
    pdl_launch();
    pdl_wait();
    const int tid = threadIdx.x, m0 = blockIdx.y * 64, n0 = blockIdx.x * 64;
    const int tx = tid & 15, ty = tid >> 4;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += 16) {
        for (int idx = tid; idx < 64 * 16; idx += 256) {
            const int r = idx >> 4, k = idx & 15;
            As[k][r] = (m0 + r < M && k0 + k < K) ? to_float(A[(size_t)(m0 + r) * lda + k0 + k]) : 0.0f;
            Ws[k][r] = (n0 + r < N && k0 + k < K) ? W[(size_t)(n0 + r) * ldw + k0 + k] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[i] = As[kk][ty * 4 + i]; w[i] = Ws[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m < M && n < N) C[(size_t)m * ldc + n] = acc[i][j];
        }
}

}  // namespace bg

using namespace bg;

extern "C" int bg_route_logits(const void* A, int a_dtype, int lda, const float* W, int ldw, float* C, int ldc, int M, int N,
                               int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return BG_OK;
    if (K <= 0) return BG_ERR_SHAPE;
    dim3 grid((N + 63) / 64, (M + 63) / 64);
    if (grid.y > 65535) return BG_ERR_SHAPE;
    BG_DISPATCH_DTYPE(a_dtype, TA, launch(gemm_rows_f32w_kernel<TA>, grid, dim3(256), 0, stream, (const TA*)A, lda, W, ldw, C, ldc,
                                          M, N, K));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_route_topk(const float* logits, int T, int E, int top, int mode, int renorm, const float* bias, float scale,
                             const float* logit_bias, int* ids, float* weights, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (E <= 0 || top <= 0 || top > E || top > 32 || mode < 0 || mode > 3 || (mode == 3 && bias)) return BG_ERR_SHAPE;
    const RouteRule rule = {mode, renorm, bias, scale, logit_bias};
    const int warps = 4;
    const size_t smem = (size_t)warps * E * sizeof(float);
    if (smem > 40 * 1024) return BG_ERR_UNSUPPORTED;
    launch(route_topk_kernel, dim3((T + warps - 1) / warps), dim3(32 * warps), smem, stream, logits, T, E, top, rule, ids,
           weights);
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// How the router's kernel of 16-byte loads cuts a step: `tpw` tokens and `g` experts a warp at a time, 2^`wpt_log` warps to the same tokens, `tokens` a
// block.  Few tokens: a block each, and as many experts a warp as let them go through in one pass (the loads of a pass are all on their way
// together; ten router outputs: 9.3 -> 7.8 us).  More than 256: four tokens a warp, where there are more than four experts: for four a block of eight
// warps would be 32 tokens (300 to 2,048 tokens of four outputs: 1,536 features 5.7 to 10.6 us with a token a warp, 11.6 to 12.4 with four).
struct RouteCut { int tpw, g, wpt_log, tokens; };
static RouteCut route_cut(int T, int E) {
    if (T <= 256) return {1, E <= ROUTE_TOKENS ? 1 : E <= 2 * ROUTE_TOKENS ? 2 : 4, ROUTE_LOG, 1};
    if (E <= 4) return {1, 4, 0, ROUTE_TOKENS};
    int log = 0;
    while (log < ROUTE_LOG && (4 << log) < E) ++log;
    return {4, 4, log, 4 << (ROUTE_LOG - log)};
}
static bool route_vec(const void* h, int ldh, const float* W, int d) {
    return d % 8 == 0 && ldh % 8 == 0 && (uintptr_t)h % 16 == 0 && (uintptr_t)W % 16 == 0;
}
static int route_launch(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, RouteRule rule, int* ids,
                        float* weights, float* logits_out, int* hist, cudaStream_t stream) {
    const RouteCut c = route_cut(T, E);
    const size_t smem = (size_t)(c.tokens + (hist ? 1 : 0)) * E * sizeof(float);
    if (smem > 40 * 1024) return BG_ERR_UNSUPPORTED;
#define BG_ROUTE_VEC(TPW, G)                                                                                                     \
    BG_DISPATCH_DTYPE(h_dtype, TI, launch(route_vec8_kernel<TI, TPW, G>, dim3((T + c.tokens - 1) / c.tokens), dim3(32 * ROUTE_TOKENS), smem, \
                                          stream, (const TI*)h, ldh, W, T, d, E, top, rule, c.wpt_log, ids, weights, logits_out, hist))
    if (c.tpw == 4) BG_ROUTE_VEC(4, 4);
    else if (c.g == 1) BG_ROUTE_VEC(1, 1);
    else if (c.g == 2) BG_ROUTE_VEC(1, 2);
    else BG_ROUTE_VEC(1, 4);
#undef BG_ROUTE_VEC
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// The router in one kernel: float logits of h [T, d] (either type, row stride ldh) against W [E, d] float, and the choice.
extern "C" int bg_route(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, int mode, int renorm,
                        const float* bias, float scale, const float* logit_bias, int* ids, float* weights, float* logits_out,
                        cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (E <= 0 || top <= 0 || top > E || top > 32 || d <= 0 || mode < 0 || mode > 3 || (mode == 3 && bias)) return BG_ERR_SHAPE;
    const RouteRule rule = {mode, renorm, bias, scale, logit_bias};
    const size_t smem = (size_t)ROUTE_TOKENS * E * sizeof(float);
    if (smem > 40 * 1024) return BG_ERR_UNSUPPORTED;
    if (route_vec(h, ldh, W, d)) return route_launch(h, h_dtype, ldh, W, T, d, E, top, rule, ids, weights, logits_out, nullptr, stream);
    BG_DISPATCH_DTYPE(h_dtype, TI, launch(route_kernel<TI>, dim3((T + ROUTE_TOKENS - 1) / ROUTE_TOKENS), dim3(32 * ROUTE_TOKENS), smem, stream,
                                          (const TI*)h, ldh, W, T, d, E, top, rule, ids, weights, logits_out));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// The integers of scratch that bg_route_layout wants for a step of T tokens; nought where it does not take the sizes: rows that are not whole 16-byte
// pieces, more than RL_MAX counts (every block of the second kernel adds them all up: 2,048 tokens of 8 experts are 1,024), more assignments to a
// block than fit.  (Besides sizes it wants its rows on 16 bytes.)
extern "C" int bg_route_layout_counts(int T, int d, int E, int top) {
    if (T <= 0 || E <= 0 || E > RL_MAX_E || top <= 0 || top > E || top > 32 || d <= 0 || d % 8) return 0;
    const RouteCut c = route_cut(T, E);
    const long long counts = (long long)((T + c.tokens - 1) / c.tokens) * E;
    return c.tokens * top > RL_MAX_A || counts > RL_MAX ? 0 : (int)counts;
}
// The same where the two kernels are no slower than three.  Every block of the second one adds up the counts and lays out its own rows, which takes
// longer than one block's sort and a gather as long as the sort has few experts or the blocks are many
// (us for three and two kernels: 10 outputs, 768 features, 64 tokens 6.8 and 8.1, 1,536 features, 512 tokens 12.1 and 13.1; 32 outputs, 1,536 features, 64
// tokens 11.2 and 11.0, 256 15.3 and 16.2, 1,024 17.9 and 16.6; 64 outputs, 4,096 features, 300 tokens 35.9 and 30.7).
extern "C" int bg_route_layout_wins(int T, int d, int E, int top) {
    return E >= 32 && d >= 1024 && (T <= 128 || T > 256) ? bg_route_layout_counts(T, d, E, top) : 0;
}
// Whether bg_route_rows takes the sizes (it wants its rows on 16 bytes, too).
extern "C" int bg_route_rows_takes(int T, int d, int E, int top) { return T > 0 && T <= RR_TOKENS && T * top <= RR_MAX_A && E <= 1024 && d % 8 == 0; }

// bg_route, bg_route_sort and bg_route_gather (xp in h's type) of a step of any number of tokens as two kernels; hist: `n_hist` integers of
// scratch, bg_route_layout_counts of them at least.  BG_ERR_UNSUPPORTED, with nothing launched, where they do not take the sizes.
extern "C" int bg_route_layout(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, int mode, int renorm,
                               const float* bias, float scale, const float* logit_bias, int* ids, float* weights, int* offsets, int* row_of,
                               int* src_of, void* xp, int scale_input, int* hist, int n_hist, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (E <= 0 || top <= 0 || top > E || top > 32 || d <= 0 || mode < 0 || mode > 3 || (mode == 3 && bias)) return BG_ERR_SHAPE;
    const RouteCut c = route_cut(T, E);
    const int blocks = (T + c.tokens - 1) / c.tokens, counts = bg_route_layout_counts(T, d, E, top);
    if (!counts || counts > n_hist || !route_vec(h, ldh, W, d) || (uintptr_t)xp % 16) return BG_ERR_UNSUPPORTED;
    const RouteRule rule = {mode, renorm, bias, scale, logit_bias};
    const int rc = route_launch(h, h_dtype, ldh, W, T, d, E, top, rule, ids, weights, nullptr, hist, stream);
    if (rc != BG_OK) return rc;
    const int cols = blocks >= 296 || d < 1024 ? 1 : 2;
    BG_DISPATCH_DTYPE(h_dtype, TI, launch(route_place_kernel<TI>, dim3(blocks, cols), dim3(256), 0, stream, (const TI*)h, ldh, weights, ids, hist, T, d,
                                          E, top, c.tokens, offsets, row_of, src_of, (TI*)xp, scale_input));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// bg_route, bg_route_sort and bg_route_gather (xp in h's type) in one kernel, for up to 8 tokens whose width is a multiple of 8 on 16-byte
// rows; BG_ERR_UNSUPPORTED, with nothing launched, where it does not take the sizes.
extern "C" int bg_route_rows(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, int mode, int renorm,
                             const float* bias, float scale, const float* logit_bias, int* ids, float* weights, int* offsets, int* row_of,
                             int* src_of, void* xp, int scale_input, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    if (E <= 0 || top <= 0 || top > E || top > 32 || d <= 0 || mode < 0 || mode > 3 || (mode == 3 && bias)) return BG_ERR_SHAPE;
    if (!bg_route_rows_takes(T, d, E, top) || ldh % 8 || (uintptr_t)h % 16 || (uintptr_t)W % 16 || (uintptr_t)xp % 16) return BG_ERR_UNSUPPORTED;
    const RouteRule rule = {mode, renorm, bias, scale, logit_bias};
    const size_t smem = (size_t)E * sizeof(float);
#define BG_ROUTE_ROWS(G)                                                                                                    \
    BG_DISPATCH_DTYPE(h_dtype, TI, launch_cluster(route_rows_kernel<TI, G>, dim3(1, 1, RR_CTAS), dim3(32 * ROUTE_TOKENS), smem, stream, RR_CTAS, (const TI*)h, \
                                                  ldh, W, T, d, E, top, rule, ids, weights, offsets, row_of, src_of, (TI*)xp, scale_input))
    if (E <= ROUTE_TOKENS) BG_ROUTE_ROWS(1);
    else if (E <= 2 * ROUTE_TOKENS) BG_ROUTE_ROWS(2);
    else BG_ROUTE_ROWS(4);
#undef BG_ROUTE_ROWS
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_route_sort(const int* ids, int A, int E, int* offsets, int* row_of, int* src_of, cudaStream_t stream) {
    if (E <= 0 || A < 0) return BG_ERR_SHAPE;
    const size_t smem = (size_t)2 * E * sizeof(int);
    if (smem > 40 * 1024) return BG_ERR_UNSUPPORTED;
    launch(route_sort_kernel, dim3(1), dim3(1024), smem, stream, ids, A, E, offsets, row_of, src_of);
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_route_gather(const void* x, int x_dtype, const float* weights, const int* src_of, void* xp, int xp_dtype, int A,
                               int d, int top, int scale, cudaStream_t stream) {
    if (A <= 0) return BG_OK;
    const int threads = d >= 256 ? 256 : ((d + 31) / 32) * 32;
    if (d % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)xp % 16 == 0)
        BG_DISPATCH_DTYPE(x_dtype, TI, BG_DISPATCH_DTYPE(xp_dtype, TO,
            launch(route_gather_vec8_kernel<TI, TO>, dim3((A + 7) / 8), dim3(256), 0, stream, (const TI*)x, weights, src_of, (TO*)xp, A, d, top,
                   scale)));
    else
    BG_DISPATCH_DTYPE(x_dtype, TI, BG_DISPATCH_DTYPE(xp_dtype, TO,
        launch(route_gather_kernel<TI, TO>, dim3(A), dim3(threads), 0, stream, (const TI*)x, weights, src_of, (TO*)xp, A, d, top, scale)));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// Routing, layout and gather of a step from one call: as one kernel (bg_route_rows), as two (bg_route_layout, with `n_hist` integers of scratch that are
// bg_route_layout_wins of the sizes or more) or as three, whichever takes the step and is no slower.  `launched` counts the kernels.
extern "C" int bg_route_place(const void* h, int h_dtype, int ldh, const float* W, int T, int d, int E, int top, int mode, int renorm,
                              const float* bias, float scale, const float* logit_bias, int* ids, float* weights, int* offsets, int* row_of,
                              int* src_of, void* xp, int scale_input, int* hist, int n_hist, int* launched, cudaStream_t stream) {
    int n = 0, rc = BG_ERR_UNSUPPORTED;
    if (launched) *launched = 0;
    if (T <= 0) return BG_OK;
    if (bg_route_rows_takes(T, d, E, top)) {
        rc = bg_route_rows(h, h_dtype, ldh, W, T, d, E, top, mode, renorm, bias, scale, logit_bias, ids, weights, offsets, row_of, src_of, xp, scale_input, stream);
        n = 1;
    }
    if (rc == BG_ERR_UNSUPPORTED && bg_route_layout_wins(T, d, E, top)) {
        rc = bg_route_layout(h, h_dtype, ldh, W, T, d, E, top, mode, renorm, bias, scale, logit_bias, ids, weights, offsets, row_of, src_of, xp, scale_input, hist, n_hist, stream);
        n = 2;
    }
    if (rc == BG_ERR_UNSUPPORTED) {
        rc = bg_route(h, h_dtype, ldh, W, T, d, E, top, mode, renorm, bias, scale, logit_bias, ids, weights, nullptr, stream);
        if (rc == BG_OK) rc = bg_route_sort(ids, T * top, E, offsets, row_of, src_of, stream);
        if (rc == BG_OK) rc = bg_route_gather(h, h_dtype, weights, src_of, xp, h_dtype, T * top, d, top, scale_input, stream);
        n = 3;
    }
    if (launched) *launched = rc == BG_OK ? n : 0;
    return rc;
}

extern "C" int bg_route_combine(const void* yp, int y_dtype, const float* weights, const int* row_of, float* out, int T, int d,
                                int top, int scale, cudaStream_t stream) {
    if (T <= 0) return BG_OK;
    const int threads = d >= 256 ? 256 : ((d + 31) / 32) * 32;
    if (y_dtype == BG_DTYPE_F32 && d % 4 == 0 && (uintptr_t)yp % 16 == 0 && (uintptr_t)out % 16 == 0)
        launch(route_combine_vec4_kernel, dim3((unsigned)(((long long)T * (d / 4) + 255) / 256)), dim3(256), 0, stream, (const float*)yp, weights,
               row_of, out, T, d, top, scale);
    else
    BG_DISPATCH_DTYPE(y_dtype, TY, launch(route_combine_kernel<TY>, dim3(T), dim3(threads), 0, stream, (const TY*)yp, weights, row_of,
                                          out, T, d, top, scale));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_route_combine_ext(const void* yp, int y_dtype, const float* weights, const int* row_of, const int* ids, int n_real,
                                    const void* h, int h_dtype, int ldh, const float* shared, const void* sg, int sg_dtype,
                                    int sg_stride, float* out, int T, int d, int top, cudaStream_t stream) {
    const int sg_float = sg_dtype == BG_DTYPE_F32 ? 1 : 0;
    if (T <= 0) return BG_OK;
    if (!ids || !h || top <= 0) return BG_ERR_SHAPE;
    const int threads = d >= 256 ? 256 : ((d + 31) / 32) * 32;
    if (y_dtype == BG_DTYPE_F32 && d % 4 == 0 && ldh % 4 == 0 && (uintptr_t)yp % 16 == 0 && (uintptr_t)out % 16 == 0 &&
        (!shared || (uintptr_t)shared % 16 == 0)) {
        const int tv = d / 4 >= 384 ? 384 : ((d / 4 + 31) / 32) * 32;
        BG_DISPATCH_DTYPE(h_dtype, TH, launch(route_combine_ext_vec4_kernel<TH>, dim3(T), dim3(tv), 0, stream, (const float*)yp, weights,
                                              row_of, ids, n_real, (const TH*)h, ldh, shared, sg, sg_float, sg_stride, out, T, d, top));
        BG_LAUNCH_CHECK();
        return BG_OK;
    }
    BG_DISPATCH_DTYPE(y_dtype, TY, BG_DISPATCH_DTYPE(h_dtype, TH,
        launch(route_combine_ext_kernel<TY, TH>, dim3(T), dim3(threads), 0, stream, (const TY*)yp, weights, row_of, ids, n_real,
               (const TH*)h, ldh, shared, sg, sg_float, sg_stride, out, T, d, top)));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

extern "C" int bg_glu_clamped(const void* gu, int gu_dtype, int ld, void* out, int out_dtype, int rows, int n, float limit,
                              float alpha, cudaStream_t stream) {
    if (rows <= 0 || n <= 0) return BG_OK;
    if (ld < 2 * n) return BG_ERR_SHAPE;
    const size_t total = (size_t)rows * n;
    if ((total + 255) / 256 > 0x7fffffffULL) return BG_ERR_SHAPE;
    if (n % 8 == 0 && ld % 8 == 0 && (uintptr_t)gu % 16 == 0 && (uintptr_t)out % 16 == 0) {
        const size_t total8 = total / 8;
        BG_DISPATCH_DTYPE(gu_dtype, TI, BG_DISPATCH_DTYPE(out_dtype, TO,
            launch(glu_clamped_vec8_kernel<TI, TO>, dim3((unsigned)((total8 + 255) / 256)), dim3(256), 0, stream, (const TI*)gu, ld,
                   (TO*)out, total8, n, limit, alpha)));
        BG_LAUNCH_CHECK();
        return BG_OK;
    }
    BG_DISPATCH_DTYPE(gu_dtype, TI, BG_DISPATCH_DTYPE(out_dtype, TO,
        launch(glu_clamped_kernel<TI, TO>, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, (const TI*)gu, ld, (TO*)out,
               total, n, limit, alpha)));
    BG_LAUNCH_CHECK();
    return BG_OK;
}

// A [rows, K] (float or bfloat16), W [E][N, K] of the same type with w_expert elements between experts, C [rows, N] float or of
// A's type.  `rows` is the number of assignments: the grid has a row tile for every tile any distribution could need.
extern "C" int bg_gemm_grouped(const void* A, int a_dtype, int lda, const void* W, int ldw, long long w_expert, void* C, int c_dtype,
                               int ldc, const int* offsets, int E, int rows, int N, int K, int act, cudaStream_t stream) {
    if (rows <= 0 || N <= 0) return BG_OK;
    if (K <= 0 || E <= 0) return BG_ERR_SHAPE;
    const int row_tiles = rows / GG_BM + E;
    if (row_tiles > 65535) return BG_ERR_SHAPE;
    dim3 grid((N + GG_BN - 1) / GG_BN, row_tiles);
    if (a_dtype == BG_DTYPE_F32 && c_dtype == BG_DTYPE_F32)
        launch(gemm_grouped_kernel<float, float, float>, grid, dim3(GG_THREADS), 0, stream, (const float*)A, lda, (const float*)W, ldw,
               w_expert, (float*)C, ldc, offsets, E, N, K, act);
    else if (a_dtype == BG_DTYPE_BF16 && c_dtype == BG_DTYPE_BF16)
        launch(gemm_grouped_kernel<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>, grid, dim3(GG_THREADS), 0, stream,
               (const __nv_bfloat16*)A, lda, (const __nv_bfloat16*)W, ldw, w_expert, (__nv_bfloat16*)C, ldc, offsets, E, N, K, act);
    else if (a_dtype == BG_DTYPE_BF16 && c_dtype == BG_DTYPE_F32)
        launch(gemm_grouped_kernel<__nv_bfloat16, __nv_bfloat16, float>, grid, dim3(GG_THREADS), 0, stream,
               (const __nv_bfloat16*)A, lda, (const __nv_bfloat16*)W, ldw, w_expert, (float*)C, ldc, offsets, E, N, K, act);
    else return BG_ERR_DTYPE;
    BG_LAUNCH_CHECK();
    return BG_OK;
}
