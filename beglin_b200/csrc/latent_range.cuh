// How a request's keys are spread over `max_splits` CTAs in decoding through a latent: evenly, in whole tiles of LATENT_RANGE_STEP keys,
// from the tile in which the row's window begins.  The attention kernel and the merge behind it work it out from the row's position.
#pragma once

namespace bg {

constexpr int LATENT_RANGE_STEP = 128;

struct LatentRange { int begin, per, count; };      // the first range's first key, keys of a range, ranges that hold keys

__host__ __device__ __forceinline__ LatentRange latent_range(int pos, int lo, int max_splits) {
    LatentRange r;
    r.begin = lo / LATENT_RANGE_STEP * LATENT_RANGE_STEP;
    const int tiles = (pos + 1 - r.begin + LATENT_RANGE_STEP - 1) / LATENT_RANGE_STEP;
    const int each = (tiles + max_splits - 1) / max_splits;
    r.per = each * LATENT_RANGE_STEP;
    r.count = (tiles + each - 1) / each;
    return r;
}

}  // namespace bg
