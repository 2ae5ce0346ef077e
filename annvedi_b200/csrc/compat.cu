// Reference-semantics linear scan: reproduces the ranking LinearIndex::query returns
// (competitors/linear/src/linear_index.cpp:27-60, 100-121), including its 64-entry early-abandon
// heap, bit for bit.
//
// The reference ranks point i by v_i, where T_i is the 64th-smallest exact distance among points
// 0..i-1 (FLT_MAX before 64 are seen): v_i = d_i when d_i < T_i, else the first checkpoint partial
// sum of compute_l2_distance (competitors/linear/src/simd.h:32-64) that reached T_i. It returns
// the k smallest (v_i, i) pairs.
//
// Pass 1 (compat_partials_kernel) is parallel: each group of 16 threads plays the 16 AVX-512
// lanes of one (query, row) pair -- lane j sums elements j, j+16, ... with an unfused multiply
// and add -- and folds the lanes in the compiled reference's order at every checkpoint (after
// 96, 192, ... elements and after the last full 16-chunk). The remainder (dim % 16) follows the
// compiled reference too: one fused 8-wide chunk folded the same way, then scalar fused steps.
// It writes the full distance D[q][i] and the checkpoint values P[q][c][i].
//
// Pass 2, the thresholds: T_i is a prefix order statistic, so the rows are cut into up to 128 segments. Each
// segment's `lim` smallest distances are found on their own (compat_segments_kernel), merged into the heap the
// reference holds at every segment's first row (compat_prefix_kernel), and one warp a segment walks its rows from
// there, replaying insertions (rows with D < T, rare once T settles) and recording each row's threshold
// (compat_threshold_kernel). As one walk of all rows by one warp this took 248 of a query's 436 us at 100k x 384. The
// walk inserts 64 ln(b / a) rows of [a, b) on random data, 290 clocks each, so the first segment's alone is most of it
// (240 insertions, 32 us of 163): it is cut again at 128, 256, 512 and 1024, five warps that make their own starting heap
// from the rows before (a few chunks of 64, sorted and merged): 44 insertions each, 15 us.
// Pass 3 (compat_values_kernel) picks v_i from D, P and T_i, and each segment's k best (v_i, i) by block; the k best of
// those, sorted, are the result (compat_final_kernel).
#include <cfloat>

#include "block_select.cuh"
#include "common.cuh"
#include "compat.cuh"
#include "refmath.cuh"

namespace annb {

// grid: (row blocks, query groups); block: 256 threads = 16 rows x 16 lanes. PIECES: the row's 16-chunks held in
// registers (dim <= 16 PIECES; 0: any dim), so that a row's loads are in flight together. As many as the dimension needs,
// to a few: with 32 at every dimension up to 512, 127 queries over 46,245 x 4 took 818 us here, 313 by the loop before it
// (a call: 971, 532; 473 now), and 500 over 100,000 x 100 8,335 us a call (7,290; 5,760 now).
template <int PIECES>
__global__ void __launch_bounds__(256) compat_partials_kernel(CompatArgs a, int q_begin) {
    extern __shared__ float sQ[];  // [QG][dim]
    const int grp = threadIdx.x >> 4;
    const int qg0 = q_begin + blockIdx.y * kCompatQG;
    const int nqg = min(kCompatQG, a.q_end - qg0);
    for (int e = threadIdx.x; e < nqg * a.dim; e += blockDim.x) sQ[e] = a.q[(int64_t)(qg0 + e / a.dim) * a.ldq + e % a.dim];
    __syncthreads();
    const int ncp = a.ncp;
    const bool leader = (threadIdx.x & 15) == 0;
    for (int64_t r0 = (int64_t)blockIdx.x * 16; r0 < a.n; r0 += (int64_t)gridDim.x * 16) {
        const int64_t row = r0 + grp;
        const bool valid = row < a.n;
        const float* x = a.base + (valid ? row : 0) * a.ldb;
        float xr[PIECES > 0 ? PIECES : 1];  // the row's full 16-chunks, loaded once for the queries
#pragma unroll
        for (int c = 0; c < PIECES; ++c) xr[c] = c < (a.dim >> 4) ? x[c * 16 + (threadIdx.x & 15)] : 0.f;
        for (int qq = 0; qq < nqg; ++qq) {
            const int64_t qi = qg0 + qq - q_begin;  // index within this chunk of queries
            float* P = a.P + (int64_t)qi * ncp * a.n + row;
            auto emit = [&](int c, float v) {
                if (leader && valid) P[(int64_t)c * a.n] = v;
            };
            const float* qv = sQ + qq * a.dim;
            float d;
            if constexpr (PIECES > 0)
                d = ref_l2_f32_pieces(xr, x, qv, a.dim, emit);
            else
                d = ref_l2_f32(x, qv, a.dim, emit);
            if (leader && valid) a.D[(int64_t)qi * a.n + row] = d;
        }
    }
}

constexpr int kCompatAhead = 8;  // 32-row steps of distances loaded ahead of the walk

constexpr int kCompatWarps = 4;

// Walks rows [begin, end) of D through the heap in row order; out(i, T_i, valid) per row.
template <class Out>
__device__ __forceinline__ void compat_walk(const float* __restrict__ D, int64_t begin, int64_t end, WarpHeap64& heap,
                                            Out&& out) {
    const int lane = threadIdx.x & 31;
    const float inf = __int_as_float(0x7f800000);
    float Tcur = heap.worst();
    float nxt[kCompatAhead];
#pragma unroll
    for (int j = 0; j < kCompatAhead; ++j) {
        const int64_t i = begin + (int64_t)j * 32 + lane;
        nxt[j] = i < end ? D[i] : inf;
    }
    for (int64_t base = begin; base < end; base += 32 * kCompatAhead) {
        float cur[kCompatAhead];
#pragma unroll
        for (int j = 0; j < kCompatAhead; ++j) {
            cur[j] = nxt[j];
            const int64_t i = base + 32 * kCompatAhead + (int64_t)j * 32 + lane;
            nxt[j] = i < end ? D[i] : inf;
        }
#pragma unroll
        for (int j = 0; j < kCompatAhead; ++j) {
            const int64_t i = base + (int64_t)j * 32 + lane;
            const bool valid = i < end;
            const float d = cur[j];
            // rows enter the heap in row order; a row's threshold is the heap's before its own insertion
            float myT = Tcur;
            int last = -1;
            while (true) {
                const unsigned cand = __ballot_sync(0xffffffffu, valid && lane > last && d < myT);
                if (cand == 0) break;
                const int l0 = __ffs(cand) - 1;
                heap.insert(__shfl_sync(0xffffffffu, d, l0));
                Tcur = heap.worst();
                if (lane > l0) myT = Tcur;
                last = l0;
            }
            out(i, myT, valid);
        }
    }
}

// One block per (segment, query): the segment's `lim` smallest distances, ascending (FLT_MAX where fewer than lim are
// below it, as the heap's empty slots).
__global__ void __launch_bounds__(256) compat_segments_kernel(CompatArgs a) {
    __shared__ int sHist[256];
    __shared__ int sMisc[12];
    __shared__ int sN;
    __shared__ unsigned long long sR[64];
    const int s = blockIdx.x, qi = blockIdx.y;
    const float* D = a.D + (int64_t)qi * a.n + (int64_t)s * a.seg_rows;
    const int m = (int)a.seg_rows;  // the last, shorter segment's list serves no later one and is not made
    const int lim = a.k < 64 ? a.k : 64;
    if (threadIdx.x == 0) sN = 0;
    if (threadIdx.x < 64) sR[threadIdx.x] = ~0ull;
    __syncthreads();
    auto at = [&](int i) { return select_word(D[i], i); };
    const SelectBound b = block_select_bound(at, m, lim, sHist, sMisc);
    for (int i = threadIdx.x; i < m; i += 256) {
        const unsigned long long w = at(i);
        if (b.in(w)) sR[atomicAdd(&sN, 1)] = w;
    }
    block_sort_u64(sR, 64);
    if (threadIdx.x < 64) {
        const float v = threadIdx.x < lim ? f32_ord((uint32_t)(sR[threadIdx.x] >> 32)) : FLT_MAX;
        a.seg_heap[((int64_t)qi * a.nseg + s) * 64 + threadIdx.x] = v < FLT_MAX ? v : FLT_MAX;  // inf, NaN: never held
    }
}

// The `lim` smallest of two ascending lists of 64 values (FLT_MAX: none), (lo, hi) and (b0, b1): lane l holds values l and
// l + 32. min(a[i], b[63 - i]) are the 64 smallest, a bitonic sequence, which six exchange steps sort.
__device__ __forceinline__ void heap_merge(float& lo, float& hi, float b0, float b1, int lim) {
    const int lane = threadIdx.x & 31;
    // value i meets value 63 - i: lane l's lo meets lane 31 - l's hi, and its hi meets that lane's lo
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, b1, 31));
    hi = fminf(hi, __shfl_xor_sync(0xffffffffu, b0, 31));
    const float t = fminf(lo, hi);  // step 32
    hi = fmaxf(lo, hi);
    lo = t;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        const float ol = __shfl_xor_sync(0xffffffffu, lo, d), oh = __shfl_xor_sync(0xffffffffu, hi, d);
        const bool low = (lane & d) == 0;
        lo = low ? fminf(lo, ol) : fmaxf(lo, ol);
        hi = low ? fminf(hi, oh) : fmaxf(hi, oh);
    }
    if (lane >= lim) lo = FLT_MAX;
    if (lane + 32 >= lim) hi = FLT_MAX;
}

// Ascending order of a warp's 64 values, lane l holding values l and l + 32.
__device__ __forceinline__ void heap_sort(float& lo, float& hi) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int size = 2; size <= 64; size <<= 1) {
        if (size == 64) {  // step 32
            const float t = fminf(lo, hi);
            hi = fmaxf(lo, hi);
            lo = t;
        }
#pragma unroll
        for (int d = size == 64 ? 16 : size >> 1; d > 0; d >>= 1) {
            const float ol = __shfl_xor_sync(0xffffffffu, lo, d), oh = __shfl_xor_sync(0xffffffffu, hi, d);
            const bool low = (lane & d) == 0;
            const bool up_lo = (lane & size) == 0, up_hi = ((lane + 32) & size) == 0;  // ascending runs
            lo = low == up_lo ? fminf(lo, ol) : fmaxf(lo, ol);
            hi = low == up_hi ? fminf(hi, oh) : fmaxf(hi, oh);
        }
    }
}

// One block per query: seg_heap[s] := the heap the reference holds at segment s's first row, the `lim` smallest of the
// earlier segments' lists. Staged in shared memory: a list's load from L2 takes longer than its merge. Eight warps: each
// merges its run of lists, then the runs before it, then those into its own heaps: 13 + 7 + 13 merges in a chain
// instead of 97 (98 segments: 15.8 -> 7.8 us).
__global__ void __launch_bounds__(256) compat_prefix_kernel(CompatArgs a) {
    __shared__ float sL[kSelectSegs * 64];
    __shared__ float sRun[8 * 64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, qi = blockIdx.x;
    const int lim = a.k < 64 ? a.k : 64;
    float* L = a.seg_heap + (int64_t)qi * a.nseg * 64;
    for (int i = threadIdx.x; i < (a.nseg - 1) * 64; i += 256) sL[i] = L[i];  // the last segment has no list
    __syncthreads();
    const int per = (a.nseg + 7) / 8, s0 = min(a.nseg, warp * per), s1 = min(a.nseg, s0 + per);
    float lo = FLT_MAX, hi = FLT_MAX;
    for (int s = s0; s < s1; ++s) {  // the heap of the run's earlier lists, in place
        float* l = sL + s * 64;
        const bool has = s + 1 < a.nseg;
        const float b0 = has ? l[lane] : FLT_MAX, b1 = has ? l[lane + 32] : FLT_MAX;
        l[lane] = lo;
        l[lane + 32] = hi;
        heap_merge(lo, hi, b0, b1, lim);
    }
    sRun[warp * 64 + lane] = lo;
    sRun[warp * 64 + lane + 32] = hi;
    __syncthreads();
    lo = hi = FLT_MAX;
    for (int r = 0; r < warp; ++r) heap_merge(lo, hi, sRun[r * 64 + lane], sRun[r * 64 + lane + 32], lim);
#pragma unroll 2
    for (int s = s0; s < s1; ++s) {
        float h0 = sL[s * 64 + lane], h1 = sL[s * 64 + lane + 32];
        heap_merge(h0, h1, lo, hi, lim);
        L[s * 64 + lane] = h0;
        L[s * 64 + lane + 32] = h1;
    }
}

// One warp per (segment, query), several for the first segment: each row's threshold, from the starting heap.
constexpr int kFirstCuts = 5;  // the first segment's rows from 0, 128, 256, 512 and 1024
__global__ void __launch_bounds__(32 * kCompatWarps) compat_threshold_kernel(CompatArgs a) {
    const int w = blockIdx.x * kCompatWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31, qi = blockIdx.y;
    const int s = w < kFirstCuts ? 0 : w - (kFirstCuts - 1);
    if (s >= a.nseg) return;  // the whole warp
    const int lim = a.k < 64 ? a.k : 64;
    const float* D = a.D + (int64_t)qi * a.n;
    float* T = a.T + (int64_t)qi * a.n;
    int64_t begin = (int64_t)s * a.seg_rows, end = min(a.n, begin + a.seg_rows);
    WarpHeap64 heap;
    heap.init(lim);
    if (s > 0) {
        const float* L = a.seg_heap + ((int64_t)qi * a.nseg + s) * 64;
        heap.lo = L[lane];
        heap.hi = L[lane + 32];
    } else {
        if (w > 0) begin = (int64_t)64 << w;
        if (begin >= end) return;  // the whole warp
        if (w + 1 < kFirstCuts) end = min(end, (int64_t)128 << w);
        if (w == 0 && lim == 64) {  // no threshold before 64 rows are seen
            const int64_t m = min((int64_t)64, end);
            if (lane < m) T[lane] = FLT_MAX;
            if (lane + 32 < m) T[lane + 32] = FLT_MAX;
            begin = 64;
        }
        for (int64_t r = 0; r < begin; r += 64) {
            const float d0 = r + lane < end ? D[r + lane] : FLT_MAX, d1 = r + lane + 32 < end ? D[r + lane + 32] : FLT_MAX;
            float b0 = d0 < FLT_MAX ? d0 : FLT_MAX, b1 = d1 < FLT_MAX ? d1 : FLT_MAX;  // inf, NaN: never held
            heap_sort(b0, b1);
            heap_merge(heap.lo, heap.hi, b0, b1, lim);
        }
    }
    compat_walk(D, begin, end, heap, [&](int64_t i, float t, bool valid) {
        if (valid) T[i] = t;
    });
}

// v_i = d_i when d_i < T_i, else the first checkpoint value >= T_i (d_i if none), written over T_i; then the segment's
// best min(k, rows) (v_i, i), in no order. One block per (segment, query).
__global__ void __launch_bounds__(256) compat_values_kernel(CompatArgs a) {
    __shared__ int sHist[256];
    __shared__ int sMisc[12];
    __shared__ int sN;
    const int s = blockIdx.x, qi = blockIdx.y;
    const int64_t n = a.n, begin = (int64_t)s * a.seg_rows;
    const int m = (int)min(a.seg_rows, n - begin);
    const float* D = a.D + (int64_t)qi * n + begin;
    float* T = a.T + (int64_t)qi * n + begin;
    const float* P0 = a.P + (int64_t)qi * a.ncp * n + begin;
    for (int e = threadIdx.x; e < m; e += 256) {
        const float d = D[e];
        const float t = T[e];
        float v = d;
        if (!(d < t)) {
            for (int c = 0; c < a.ncp; ++c) {
                const float p = P0[(int64_t)c * n + e];
                if (p >= t) {
                    v = p;
                    break;
                }
            }
        }
        T[e] = v;
    }
    segment_select(T, begin, m, a.k, a.seg_best + ((int64_t)qi * a.nseg + s) * a.k, sHist, sMisc, &sN);
}

// The k best of the segments' best, in order. One block per query; the words are read once into shared memory where
// they fit (98 segments of 100: 20 -> 13 us), which six passes over them follow.
constexpr int kFinalThreads = 1024, kFinalStaged = 20480;
__global__ void __launch_bounds__(kFinalThreads) compat_final_kernel(CompatArgs a, int q_begin) {
    extern __shared__ __align__(16) unsigned long long sW[];
    __shared__ int sHist[256];
    __shared__ int sMisc[12];
    __shared__ int sN;
    __shared__ unsigned long long sR[512];
    const int qi = blockIdx.x;
    const unsigned long long* w = a.seg_best + (int64_t)qi * a.nseg * a.k;
    const int m = a.nseg * a.k;
    if (m <= kFinalStaged) {
        for (int i = threadIdx.x; i < m; i += blockDim.x) sW[i] = w[i];
        w = sW;
    }
    if (threadIdx.x == 0) sN = 0;
    __syncthreads();
    const SelectBound b = block_select_bound<true>([&](int i) { return w[i]; }, m, a.k, sHist, sMisc);
    const int p2 = pow2_ceil(a.k);
    for (int i = threadIdx.x; i < m; i += blockDim.x)
        if (b.in(w[i])) sR[atomicAdd(&sN, 1)] = w[i];
    for (int i = a.k + threadIdx.x; i < p2; i += blockDim.x) sR[i] = ~0ull;
    block_sort_u64(sR, p2);
    const int64_t o = (int64_t)(q_begin + qi) * a.k;
    for (int e = threadIdx.x; e < a.k; e += blockDim.x) {
        if (a.out_ids) a.out_ids[o + e] = (int64_t)(unsigned)sR[e];
        if (a.out_dists) a.out_dists[o + e] = f32_ord((uint32_t)(sR[e] >> 32));
    }
}

int compat_num_checkpoints(int dim) { return ref_num_checkpoints(dim); }

int launch_compat(CompatArgs a, int q_begin, int q_count, cudaStream_t st) {
    ANN_CHECK_ARG(a.k >= 1 && a.k <= 512, "reference mode: k=%d outside [1, 512]", a.k);
    ANN_CHECK_ARG(a.dim >= 1 && a.dim <= 4096, "reference mode: dim=%d outside [1, 4096]", a.dim);
    if (q_count <= 0 || a.n == 0) return ANN_OK;
    a.q_end = q_begin + q_count;
    const size_t smem = sizeof(float) * kCompatQG * a.dim;
    ANN_CHECK_ARG(a.k <= a.n, "reference mode: k=%d above n", a.k);
    // Many queries over few rows fill the chip by themselves, and a segment's lists only cost: one segment (1,000 queries over
    // 10,000 x 100, k = 10: 28 us of a call less; 346 over 15,323 would take 28 us more).
    a.seg_rows = select_seg_rows(a.n, q_count >= 256 && a.n <= 10240 ? 1 : kSelectSegs);
    a.nseg = (int)ceil_div(a.n, a.seg_rows);
    // the fewest registers that hold the row: the steps past its last piece are walked all the same
    const int full16 = a.dim / 16;
    auto partials = full16 <= 1    ? compat_partials_kernel<1>
                    : full16 <= 2  ? compat_partials_kernel<2>
                    : full16 <= 4  ? compat_partials_kernel<4>
                    : full16 <= 8  ? compat_partials_kernel<8>
                    : full16 <= 16 ? compat_partials_kernel<16>
                    : full16 <= 24 ? compat_partials_kernel<24>
                    : full16 <= 32 ? compat_partials_kernel<32>
                                   : compat_partials_kernel<0>;
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(partials)));
    const int64_t rblocks = std::min<int64_t>(ceil_div(a.n, 16), kNumSMs * 8);
    dim3 g1((unsigned)rblocks, (unsigned)ceil_div(q_count, kCompatQG));
    partials<<<g1, 256, smem, st>>>(a, q_begin);
    ANN_LAUNCH_CHECK();
    const dim3 gw((unsigned)ceil_div(a.nseg + kFirstCuts - 1, kCompatWarps), (unsigned)q_count);
    if (a.nseg > 1) {
        compat_segments_kernel<<<dim3(a.nseg - 1, (unsigned)q_count), 256, 0, st>>>(a);
        ANN_LAUNCH_CHECK();
        compat_prefix_kernel<<<(unsigned)q_count, 256, 0, st>>>(a);
        ANN_LAUNCH_CHECK();
    }
    compat_threshold_kernel<<<gw, 32 * kCompatWarps, 0, st>>>(a);
    ANN_LAUNCH_CHECK();
    compat_values_kernel<<<dim3(a.nseg, (unsigned)q_count), 256, 0, st>>>(a);
    ANN_LAUNCH_CHECK();
    const int64_t words = (int64_t)a.nseg * a.k;
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(compat_final_kernel)));
    // (a few words a query are as soon done by 256 threads, of which eight blocks fit an SM)
    compat_final_kernel<<<(unsigned)q_count, words <= 1024 ? 256 : kFinalThreads, words <= kFinalStaged ? words * 8 : 0, st>>>(a, q_begin);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace annb
