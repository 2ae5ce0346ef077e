// Launch interfaces of the pruned exact scan (flat_prune.cu).
#pragma once
#include <cuda_bf16.h>
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

// Bases that are scanned. Measured over dims 64 to 4,096, k = 10 and 100, scanned / pruned, us a call:
// one query at k = 100 8,192 rows 1.6 to 1.9 times faster pruned; at k = 10 even up to 200,000 rows (50,000 x 768 93 / 105,
// 100,000 x 384 80 / 78, 100,000 x 1,536 149 / 156, clustered data up to 25% slower), but for some 20,000, whose pass is one
// tile an SM (70 / 70 at dim 384, 90 / 82 at 768, 152 / 118 at 2,048); 300,000 x 384 125 / 117, x 768 189 / 161;
// 3 queries 3,000 rows 89 / 66, 8,192 rows 1.3 to 3.1 times; 8 and more 3,000 rows 1.04 to 3.1 times, 24,000 rows 1.2 to
// 21 times. The sample (an eighth of a small base) still holds enough rows for the bar.
inline bool prune_rows(int64_t n, int nq, int k) {
    if (nq == 1 && k < 64) return n >= 200000 || (n >= 16384 && n < 32768);
    return n >= (nq <= 4 ? 8192 : 4096);
}

// The window of the BF16 keys (tc_gemm.cuh) of vector q against rows x: 2 eps + delta. With x^, q^ the BF16 operands,
//   |x.q - x^.q^| <= |x - x^| |q| + |x^| |q - q^| <= rmax |q| + (cmax + rmax) |q - q^|,
// (residual norms taken, not bounded by 2^-9: about 0.4 of that), and the FP32 accumulation of the dim + 3 products
// (truncating adds allowed for: 2^-21 each, of the terms' absolute sum) adds acc * sum. delta bounds the rounding
// of two FP32 distances summed over dim terms. The norms passed in are FP32 sums too: the factor 1.002 covers them.
// qn, rq: |q| and |q - q^|; cm, rm: upper bounds of |x| and |x - x^|.
__host__ __device__ __forceinline__ float key_window_l2(float qn, float rq, float cm, float rm, int dim) {
    const float acc = (float)(dim + 19) * 4.76837158e-7f;  // (dim + 19) 2^-21
    const float cross = rm * qn + (cm + rm) * rq;
    return 1.002f * (2.f * (2.f * cross + acc * (2.f * (cm + rm) * (qn + rq) + cm * cm)) + acc * (qn + cm) * (qn + cm));
}
__host__ __device__ __forceinline__ float key_window_ip(float qn, float rq, float cm, float rm, int dim) {
    const float acc = (float)(dim + 19) * 4.76837158e-7f;
    const float cross = rm * qn + (cm + rm) * rq;
    return 1.002f * (2.f * (cross + acc * (cm + rm) * (qn + rq)) + 2.f * acc * qn * cm);
}

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
    int cap;            // survivors kept per query
    float* fkey;        // [nq, cap] survivors: key, position
    int* fcol;
    int* rcount;        // [nq] survivors met
    int* list;          // [nq] queries left to the scan
    int* count;         // [1]
    int* err;           // [1] set where a wait of the sample or filter pass gave up: every query is left to the scan
    int64_t* out_ids;   // [nq, k]
    float* out_dists;   // [nq, k] or null
    // few queries (prune_split(nq)): a query's rows shared by several blocks (null: by one)
    unsigned long long* words;  // [nq, cap] the formed (distance, row)
    int2* joined;               // [nq] words written, blocks done
    unsigned long long* wide;   // optional, page-locked: set to 1 by a query that has rows for several blocks, where one forms them
};
// Whether a pass of nq queries may use words and joined (its blocks would leave most of the chip idle).
bool prune_split(int nq);
// Survivors kept per query, and whether their kernel's shared memory fits.
int prune_cap(int k);
bool prune_fits(int k, int dpad);
// Rank of the sampled bar: with S of n keys sampled, the smallest rank r for which the k smallest keys lie at or
// below the r-th smallest sampled key with probability of about 1 - 1e-7.
int prune_bar_rank(int k, int64_t S, int64_t n);
// win and the queries' operand rows qb [nq, kpad] (launch_tc_operand's); rcount, count and err zeroed.
int launch_prune_queries(const PruneArgs& a, __nv_bfloat16* qb, int kpad, cudaStream_t st);
int launch_prune_finish(const PruneArgs& a, cudaStream_t st);  // results, list and count
// qg[j] = q[list[j]] for j < *count; where *count > 0 or report, *word (page-locked host memory, optional) =
// pass << 32 | nq << 16 | *count (nq <= 65,535).
int launch_prune_gather(const float* q, int dpad, const int* list, const int* count, int nq, float* qg,
                        unsigned long long* word, uint32_t pass, int report, cudaStream_t st);

}  // namespace annb
