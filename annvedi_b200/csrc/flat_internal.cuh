// The flat index handle, shared by the C ABI translation units.
#pragma once
#include <atomic>

#include <cuda_bf16.h>

#include "common.cuh"
#include "flat_prune.cuh"
#include "runtime.cuh"

struct ann_flat {
    int device = 0;
    int64_t n = 0;
    int dim = 0;
    int dpad = 0;
    int metric = ANN_METRIC_L2;
    float* base = nullptr;  // [n, dpad]
    std::atomic<int64_t> ndist{0};
    ann_workspace ws;       // default workspace
    annb::StageProfiler prof;     // stage 0: scan kernel(s); stage 1: merge / selection
    __nv_bfloat16* base_bf16 = nullptr;  // [n, kpad] BF16 operand form for the tensor-core scan (built on first use)
    int64_t row_mult = 1;                // position p of base_bf16 holds row (p * row_mult) mod n
    int kpad = 0;                        // operand columns: dim plus the key columns, rounded up to 64
    int query_tile = 0;                  // the exact scan's queries per CTA (0: chosen by the batch size)
    int* d_err = nullptr;                // device flag of bounded waits
    int tc_kind = 0;                     // element kind of the tensor-core search (0 BF16, 1 E4M3)
    uint8_t* base_e4m3 = nullptr;        // [n, kpad8] E4M3 operand form, Weyl order, built on first use
    float2* fac_e4m3 = nullptr;          // [n] its per-row key factors
    int kpad8 = 0;                       // dim rounded up to 32
    bool prune = true;                   // the exact search may prune by tensor-core keys
    uint64_t wait_ns = 0;                // > 0: the self-test of the bounded waits, with this limit
    std::mutex tc_mu;                    // serialises the first use of the operand forms above
    annb::PruneBounds bounds;            // of the BF16 copy's keys (cmax 0: the rows are not covered)
    bool bounds_known = false;
    double prune_credit_us = 0.0;        // what pruning would have saved the exact searches so far (estimated)
    bool prune_refused = false;          // the BF16 copy for them did not fit beside what the card holds (until the next fit)
    size_t prune_ws_refused = SIZE_MAX;  // scratch of this size did not fit
    // how the latest pruned pass ended, written by the device into page-locked memory where it left queries or the host waits
    // for a better end (pass << 32 | queries << 16 | queries left to the scan), and the back-off that follows from it
    // (flat_prune_open)
    unsigned long long* prune_word = nullptr;  // two words: that, and whether a query had rows for several blocks (PruneArgs::wide)
    uint32_t prune_pass = 0;             // passes launched
    int prune_nq = 0;                    // queries of the latest
    uint32_t prune_seen = 0;             // the latest whose end has been read
    int prune_streak = 0;                // passes in a row that left too many queries
    int prune_skip = 0;                  // calls that the scan still answers
};

namespace annb {
// Number of row splits (and rows per split) for an exact scan of n rows by nq queries in tiles of bq.
// ctas_per_sm: resident CTAs per SM of the scan form used (one wave = kNumSMs * ctas_per_sm CTAs).
int flat_choose_nsplit(int64_t n, int nq, int bq, int64_t* rows_per_split, int ctas_per_sm = 1);
}  // namespace annb
