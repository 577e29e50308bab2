// What the two files of the float product share: its parameters, the length of a range of k, and the tensor-core part's host interface.
#pragma once

#include "common.cuh"

namespace bg {

struct GfParams {
    const float* A; const float* W; const float* bias; float* C;
    float* scratch;                        // as many floats as gt_scratch asks for (with `accumulate` M N more)
    long long batch_a, batch_w, batch_c;   // a batch of independent products
    int lda, ldw, ldc, M, N, K, accumulate, batch;
    unsigned* status;
};

long long gt_scratch(int M, int N, int K, int batch);
int gt_run(const GfParams& p, cudaStream_t stream);

}  // namespace bg
