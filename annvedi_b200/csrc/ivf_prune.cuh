// Launch interfaces of the pruned exact SQ8 selection (ivf_prune.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "flat_prune.cuh"
#include "ivf.cuh"

namespace annb {

// *max2: the bit pattern of the largest |y|^2, y = scale (code - 127.5), over the rows (a NaN leaves a NaN pattern).
int launch_sq8_max_norm(const IvfView& ix, unsigned* max2, cudaStream_t st);
// FP16 operand rows of the codes, [n, kpad]: (code - 127.5) / 128 (exact), then 1024 |g y|^2 in three pieces; g is the
// power of two that brings the largest |y| into [1, 2).
int launch_sq8_operand(const IvfView& ix, float g, __half* out, int kpad, cudaStream_t st);

struct IvfPruneArgs {
    IvfView ix;
    IvfPlan plan;
    const float* q;      // [nq, ldq]
    int64_t ldq;
    int R;
    float cmax, g;       // upper bound of |y| over the rows, and the operands' scale
    __half* qop;         // [nq, kpad] the queries' operand rows
    int kpad;
    float2* win;         // [nq] twice the keys' error bound (NaN: the query is not covered by it) and |u|^2, as scaled
    const float* tauF;   // [nq] sampled bars
    float* tauX;         // [nq] filter bars: tauF and its window
    int cap;             // survivors kept per query
    const float* fkey;   // [nq, cap] survivors: key, list-order row
    const int* frow;
    int* rcount;         // [nq] survivors met
    int* fails;          // [1] queries that the pruned pass leaves
    const int* err;      // [1] set where a wait of the key passes gave up: every query is left
    float* keyR;         // [nq, R] the best R (SQ8 distance, row), in no order, padded with (+inf, kNoId)
    int* idR;
};
// Survivors kept per query, and whether a batch's sizes fit.
constexpr int kIvfPruneMaxLists = 32;
inline int ivf_prune_cap(int R) { return 16 * R; }
bool ivf_prune_fits(int R, int npc, int dpad8);
int launch_ivf_prune_queries(const IvfPruneArgs& a, cudaStream_t st);  // qop and win
int launch_ivf_prune_bars(const IvfPruneArgs& a, cudaStream_t st);     // tauX; rcount and fails zeroed
int launch_ivf_prune_finish(const IvfPruneArgs& a, cudaStream_t st);   // keyR, idR and fails

}  // namespace annb
