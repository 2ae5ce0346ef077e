// Launch interface of the dense tensor-core filter pass (tc_filter.cu).
#pragma once
#include "tc_gemm.cuh"

namespace annb {

struct TcFilterArgs {
    int M, N, K;           // A [M, K] queries, B [N, K] base rows in operand form (tc_gemm.cuh); K as launch_tc_gemm takes it
    int kind;              // kTcBF16 or kTcE4M3
    const float* tau;      // [M] bars: keys <= tau[m] are kept (NaN: none)
    float* fkey;           // [M, cap] kept keys of row m, in no particular order
    int* fcol;             // [M, cap] their columns
    int cap;
    int* rcount;           // [M] keys kept (zeroed by the caller); may exceed cap: nothing is written past it
    const float2* col_fac; // E4M3: per B row, per A row (TcGemmArgs)
    const float* row_fac;
    int* err;              // device flag set (to 2) if a bounded wait gives up
    uint64_t wait_ns = 0;  // limit of the waits (0: 2 s)
    int test_no_loads = 0; // self-test: the producers issue no copies, so that the waits run out with nothing in flight
    // Sample pass (launch_tc_sample): N sampled columns in whole tiles of 256, tile j holding B rows
    // j * 256 * b_tile_stride ..; out_min [M, N / 8] receives the smallest key of each 8 columns.
    float* out_min = nullptr;
    int b_tile_stride = 1;
    int64_t b_rows = 0;    // rows of B
};
int launch_tc_filter(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st);
// The r-th smallest of a row's minima is at or above the r-th smallest of its sampled keys, and close to it while r is
// a small share of N / 8: bars are taken from the minima, an eighth of the keys to write and read.
int launch_tc_sample(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st);

}  // namespace annb
