// Launch interface of the per-query radix selection (radix_select.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ivf.cuh"

namespace annb {

struct RadixSelectArgs {
    const float* keys;      // query q's stream: keys[offs[q] + p] (or keys[q * ld + p]), p < len
    int64_t ld;             // row stride when offs is null; also the upper bound of len
    const int64_t* offs;    // optional
    const int64_t* lens;    // optional int64 lengths
    const int* lens32;      // optional int32 lengths (clamped to ld)
    const int* ids;         // optional explicit ids (ids[offs[q] + p]); else plan rows; else p
    IvfPlan plan;           // ids from the candidate-stream plan when use_plan is set
    int use_plan;
    int R;
    float* out_key;         // [nq, R] the set (unsorted), padded with +inf / kNoId
    int* out_id;            // [nq, R]
    const int* out_rows = nullptr;  // optional: query q writes output row out_rows[q]
};

int launch_radix_select(const RadixSelectArgs& a, int nq, cudaStream_t st);

}  // namespace annb
