// The pass over a request's chunks that turns their sums into the states at the chunks' starts, four neighbouring values a thread: what the recurrences
// that run in chunks share.  Bound by bytes (every sum is read, every state written, mostly in the second-level cache), so two batches of four
// chunks are on their way at a time: one value a thread and one batch of eight left the memory idle while a batch was walked.
// 2,048 tokens in chunks of 64: 32 heads of 128 x 128 with a decay per channel 52 us -> 19, 24 heads of Mamba-2 24 -> 13, 12 of a constant decay
// 16.5 -> 9.7.
#pragma once

#include "common.cuh"

namespace bg {

constexpr int CS_THREADS = 256, CS_BATCH = 4;

// a0: four values of the first chunk's sum, `step` floats from chunk to chunk, n chunks; decay(c): what the state is multiplied with over chunk c.
// Returns the state behind the last.
template <typename D>
__device__ __forceinline__ float4 chunk_walk4(float* a0, size_t step, int n, D decay, float4 S) {
    float4 A[2][CS_BATCH];
    float d[2][CS_BATCH];
    // (chunks behind the last are the last once more: a condition would keep the loads from leaving together)
    auto load = [&](int b, int c) {
#pragma unroll
        for (int u = 0; u < CS_BATCH; ++u) {
            const int at = min(c + u, n - 1);
            A[b][u] = *reinterpret_cast<const float4*>(a0 + (size_t)at * step);
            d[b][u] = decay(at);
        }
    };
    auto walk = [&](int b, int c) {
#pragma unroll
        for (int u = 0; u < CS_BATCH; ++u)
            if (c + u < n) {
                *reinterpret_cast<float4*>(a0 + (size_t)(c + u) * step) = S;
                const float4 a = A[b][u];
                const float f = d[b][u];
                S = make_float4(fmaf(f, S.x, a.x), fmaf(f, S.y, a.y), fmaf(f, S.z, a.z), fmaf(f, S.w, a.w));
            }
    };
    load(0, 0);
    if (n > CS_BATCH) load(1, CS_BATCH);
#pragma unroll 1
    for (int c = 0; c < n; c += 2 * CS_BATCH) {
        walk(0, c);
        if (c + 2 * CS_BATCH < n) load(0, c + 2 * CS_BATCH);
        walk(1, c + CS_BATCH);
        if (c + 3 * CS_BATCH < n) load(1, c + 3 * CS_BATCH);
    }
    return S;
}

}  // namespace bg
