// Launch interfaces of the pruned exact scan (flat_prune.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace annb {

// Bounds of the BF16 keys' error over a base (launch_base_norms): the largest row norm and the largest norm of a
// row's BF16 rounding residual x - bf16(x).
struct PruneBounds {
    float cmax = 0.f;
    float rmax = 0.f;
};
// Norms outside this range leave the error bound's assumptions (no overflow, nothing lost to underflow).
constexpr float kPruneNormMin = 1e-12f, kPruneNormMax = 1e15f;

// Smaller bases are scanned: from here on every batch measured faster pruned (32768 x 64, one query: 67 us against
// 105 us), and the sample (an eighth of a small base) still holds enough rows for the bar.
constexpr int64_t kPruneMinRows = 32768;

// out2 = bit patterns (uint32) of {largest squared norm, largest squared residual norm} over rows [n, dim] of
// stride ld; a NaN anywhere leaves a NaN pattern. rows (optional): each row's norm and residual norm.
int launch_base_norms(const float* x, int64_t n, int dim, int64_t ld, unsigned* out2, cudaStream_t st,
                      float2* rows = nullptr);

struct PruneArgs {
    const float* base;  // [n, dpad]
    int64_t n;
    int dim, dpad;
    int64_t mult;       // position p of the BF16 copy holds row (p * mult) mod n
    const float* q;     // [nq, dpad]
    int nq, k, metric;
    int stream_form;    // 1: the sums of the streaming scan, 0: of the staged scan
    PruneBounds b;
    float* win;         // [nq] window: 2 eps + delta (NaN: the query is not covered by the bound)
    const float* tauF;  // [nq] sampled bar
    float* tauX;        // [nq] filter bar tauF + win
    int cap;            // survivors kept per query
    float* fkey;        // [nq, cap] survivors: key, position
    int* fcol;
    int* rcount;        // [nq] survivors met
    int* list;          // [nq] queries left to the scan
    int* count;         // [1]
    int64_t* out_ids;   // [nq, k]
    float* out_dists;   // [nq, k] or null
};
// Survivors kept per query, and whether their kernel's shared memory fits.
int prune_cap(int k);
bool prune_fits(int k, int dpad);
// Rank of the sampled bar: with S of n keys sampled, the smallest rank r for which the k smallest keys lie at or
// below the r-th smallest sampled key with probability of about 1 - 1e-7.
int prune_bar_rank(int k, int64_t S, int64_t n);
int launch_prune_windows(const PruneArgs& a, cudaStream_t st);  // win
int launch_prune_bars(const PruneArgs& a, cudaStream_t st);     // tauX; rcount and count zeroed
int launch_prune_finish(const PruneArgs& a, cudaStream_t st);   // results, list and count
// qg[j] = q[list[j]] for j < *count.
int launch_prune_gather(const float* q, int dpad, const int* list, const int* count, int nq, float* qg, cudaStream_t st);

}  // namespace annb
