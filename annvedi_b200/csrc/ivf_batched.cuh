// Launch interface of the batched, list-major SQ8 pass (ivf_batched.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "ivf.cuh"

namespace annb {

constexpr int64_t kItemRows = 2048;  // list rows per work item

struct IvfBatchArgs {
    IvfView ix;
    IvfPlan plan;
    const int32_t* pair_vals;   // (q * npc + j) of each probe, grouped by list
    const int32_t* pair_lists;  // the list of each pair
    const int64_t* lq_off;      // [C + 1] first pair of each list
    const int64_t* item_off;    // [C + 1] first work item of each list
    const int64_t* total_items; // device scalar (item_off[C])
    const int64_t* cand_off;    // [nq + 1] first candidate-stream slot of each query in D
    unsigned* counter;          // work-item counter (zeroed by batched_prepare)
    const float* qs;            // [nq, dpad] q - offset
    float* D;                   // [sum of n_cands] SQ8 distances in stream order
};

// What the tensor-core forms want of the set-up beside IvfBatchArgs (null arrays are left out).
struct IvfBatchTiles {
    int64_t* titem = nullptr;  // [C + 1] first 128 x 256 tile of each list (pairs x rows)
    // the sampled form: with div > 0 the first ceil(size / div) rows of each list are its sampled head
    int div = 0;
    int64_t* lcap = nullptr;   // [C] rows of the heads
    int64_t* sitem = nullptr;  // [C + 1] first tile of each head
    int64_t* sseg = nullptr;   // [nq, npc] each query's sample stream: where its lists' heads start, its length and
    int64_t* slen = nullptr;   // [nq]      its first slot
    int64_t* soff = nullptr;   // [nq + 1]
    // the pairs' operand rows: A[i] = the row (row_bytes) of pair i's query in qrows, row_query[i] = the query, sdbase[i] =
    // the sample-stream slot of its list's row 0, pfac[i] = qfac[query]
    const void* qrows = nullptr;
    int row_bytes = 0;
    void* A = nullptr;
    int32_t* row_query = nullptr;
    int64_t* sdbase = nullptr;
    const float* qfac = nullptr;
    float* pfac = nullptr;
};

// Scratch of batched_prepare for nq queries x npc probes over C lists.
size_t batched_scratch_bytes(int nq, int npc, int C);
// Groups the plan's probes by list (in no order within one), counts work items and candidate offsets; host_totals[0..4] =
// {work items, total candidates, whether a query's stream is every row, queries set apart, *a.key_err}. Synchronises the stream.
// With sync = false the totals are copied to host_totals (which must then be page-locked) without waiting: they
// are valid after the caller's next synchronisation of st.
int batched_prepare(const IvfQueryArgs& a, void* scratch, IvfBatchArgs* out, int64_t* host_totals, cudaStream_t st,
                    bool sync = true, const IvfBatchTiles& tiles = IvfBatchTiles{});
int launch_batched(const IvfBatchArgs& b, const float* qdev, float* qs, float* D, cudaStream_t st);

}  // namespace annb
