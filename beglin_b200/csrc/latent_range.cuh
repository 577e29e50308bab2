// How a request's keys are spread over CTAs in decoding through a latent: evenly, in whole tiles of LATENT_RANGE_STEP keys, from the tile
// in which the row's window begins, in as many ranges as suit the row's OWN number of tiles (a grid is sized for the longest row that
// may come, in a captured step for the longest context).  The attention kernel and the merge behind it work it out alike.
#pragma once

namespace bg {

constexpr int LATENT_RANGE_STEP = 128, LATENT_MAX_RANGES = 64;

struct LatentRange { int begin, per, count; };      // the first range's first key, keys of a range, ranges that hold keys

// What `s` ranges of a row of `tiles` tiles cost: the waves of one CTA an SM that `ctas` such rows make, times a range's tiles and three more
// for a CTA's start, queries and results.  (64 rows of 4,000 keys in 1, 2, 3, 4, 6 and 9 ranges: 169, 103, 140, 120, 141, 157 us)
__host__ __device__ __forceinline__ long long latent_range_cost(int tiles, int s, int ctas, int sms) {
    const unsigned per = (unsigned)(tiles + s - 1) / (unsigned)s, n = ((unsigned)tiles + per - 1) / per;
    return (long long)(((unsigned)ctas * n + (unsigned)sms - 1) / (unsigned)sms) * (per + 3);
}
// The least number of ranges of the least cost, of at most `most` (1 .. LATENT_MAX_RANGES)
__host__ inline int latent_ranges(int tiles, int most, int ctas, int sms) {
    int best = 1;
    for (int s = 2; s <= most && s <= tiles; ++s)
        if (latent_range_cost(tiles, s, ctas, sms) < latent_range_cost(tiles, best, ctas, sms)) best = s;
    return best;
}

#ifdef __CUDACC__
// The same and the ranges themselves, by a whole warp: every lane tries two numbers.
__device__ __forceinline__ LatentRange latent_range(int pos, int lo, int most, int ctas, int sms) {
    LatentRange r;
    r.begin = lo / LATENT_RANGE_STEP * LATENT_RANGE_STEP;
    const int tiles = (pos + 1 - r.begin + LATENT_RANGE_STEP - 1) / LATENT_RANGE_STEP, top = min(min(most, tiles), LATENT_MAX_RANGES);
    int best = 1;
    if (top > 1) {
        const int lane = threadIdx.x & 31;
        best = min(lane + 1, top);
        long long cost = latent_range_cost(tiles, best, ctas, sms);
        if (lane + 33 <= top) {
            const long long c = latent_range_cost(tiles, lane + 33, ctas, sms);
            if (c < cost) { cost = c; best = lane + 33; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const long long c = __shfl_xor_sync(0xffffffffu, cost, o);
            const int b = __shfl_xor_sync(0xffffffffu, best, o);
            if (c < cost || (c == cost && b < best)) { cost = c; best = b; }
        }
    }
    const int each = (tiles + best - 1) / best;
    r.per = each * LATENT_RANGE_STEP;
    r.count = (tiles + each - 1) / each;
    return r;
}
#endif

}  // namespace bg
