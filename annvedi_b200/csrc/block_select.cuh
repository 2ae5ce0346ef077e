// Block-wide selection of the k smallest (key, id) pairs, held as 64-bit words (ordered key bits, then id).
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace annb {

// The order-preserving integer image of a float (no NaN) and back.
__device__ __forceinline__ uint32_t ord_f32(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float f32_ord(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
// The digit (8 bits) of rank `rem` (1-based) of the block's 256-bin histogram: every thread gets the digit, the
// count below it and the digit's own count. One bin per thread of the first 256; sMisc: 12 ints.
__device__ __forceinline__ void block_pick(const int* hist, int rem, int* sMisc, int* digit, int* before, int* own) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = threadIdx.x < 256 ? hist[threadIdx.x] : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31 && warp < 8) sMisc[warp] = incl;
    __syncthreads();
    for (int w = 0; w < min(warp, 8); ++w) incl += sMisc[w];
    if (threadIdx.x < 256 && incl - c < rem && rem <= incl) {
        sMisc[8] = threadIdx.x;
        sMisc[9] = incl - c;
        sMisc[10] = c;
    }
    __syncthreads();
    *digit = sMisc[8];
    *before = sMisc[9];
    *own = sMisc[10];
}

// The k smallest of a set of distinct words are those with (word & mask) <= prefix.
struct SelectBound {
    unsigned long long prefix, mask;
    __device__ __forceinline__ bool in(unsigned long long w) const { return (w & mask) <= prefix; }
};

// The highest bit in which the words at(0..m) differ (0 where none does). Whole block; sOr: two ints. Distances and keys
// of a selection share their leading bits, whose digits would leave everything in one bin: a pass over the words in
// place of one to three passes, each with its histogram, prefix and three barriers. It pays where the words are in shared
// memory (flat_prune.cu's finish kernel, 1,000 queries over 1M x 384: 177 -> 163 us); a few read from L2 each time do
// not (compat_segments_kernel: 9.5 -> 10.3).
template <class At>
__device__ __forceinline__ int block_top_bit(At&& at, int m, unsigned* sOr) {
    if (threadIdx.x < 2) sOr[threadIdx.x] = 0u;
    const unsigned long long w0 = at(0);
    unsigned long long x = 0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) x |= at(i) ^ w0;
    const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)x), hi = __reduce_or_sync(0xffffffffu, (unsigned)(x >> 32));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        if (lo) atomicOr(&sOr[0], lo);
        if (hi) atomicOr(&sOr[1], hi);
    }
    __syncthreads();
    const unsigned long long all = ((unsigned long long)sOr[1] << 32) | sOr[0];
    return all ? 63 - __clzll((long long)all) : 0;
}

// The bound of the k smallest (1 <= k <= m) of the words at(0..m): 8-bit digits from the top (SKIP: the highest bit that
// differs) until one ends at the k-th exactly, or the last (words that may be equal: all of the k-th's value are in). Whole block of >= 256 threads; sHist:
// 256 ints, sMisc: 12 ints. Ends with a barrier passed.
template <bool SKIP = false, class At>
__device__ __forceinline__ SelectBound block_select_bound(At&& at, int m, int k, int* sHist, int* sMisc) {
    int shift = SKIP ? max(0, block_top_bit(at, m, reinterpret_cast<unsigned*>(sMisc)) - 7) : 56;
    SelectBound b{0, shift + 8 < 64 ? ~0ull << (shift + 8) : 0ull};
    if (SKIP) b.prefix = at(0) & b.mask;
    int rem = k;
    while (true) {
        if (threadIdx.x < 256) sHist[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const unsigned long long w = at(i);
            if ((w & b.mask) == b.prefix) atomicAdd(&sHist[(int)(w >> shift) & 255], 1);
        }
        __syncthreads();
        int d, before, own;
        block_pick(sHist, rem, sMisc, &d, &before, &own);
        rem -= before;
        b.prefix |= (unsigned long long)d << shift;
        b.mask |= 255ull << shift;
        if (rem == own || shift == 0) break;  // uniform
        shift = max(0, shift - 8);  // (a last digit repeats known bits, the same in every word left)
    }
    return b;
}

// The k-th smallest (1 <= k <= m) of the 32-bit values at(0..m), which may be equal; as block_select_bound<true>.
template <class At>
__device__ __forceinline__ uint32_t block_kth(At&& at, int m, int k, int* sHist, int* sMisc) {
    int shift = max(0, block_top_bit([&](int i) { return (unsigned long long)at(i); }, m, reinterpret_cast<unsigned*>(sMisc)) - 7);
    uint32_t mask = shift + 8 < 32 ? ~0u << (shift + 8) : 0u;
    uint32_t prefix = at(0) & mask;
    int rem = k;
    while (true) {
        if (threadIdx.x < 256) sHist[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
            const uint32_t o = at(i);
            if ((o & mask) == prefix) atomicAdd(&sHist[(o >> shift) & 255u], 1);
        }
        __syncthreads();
        int d, before, own;
        block_pick(sHist, rem, sMisc, &d, &before, &own);
        rem -= before;
        prefix |= (uint32_t)d << shift;
        mask |= 255u << shift;
        if (shift == 0) break;
        shift = max(0, shift - 8);
    }
    return prefix;
}

// Exclusive prefix of v over the block's 1,024 threads; *total = the sum. sWarp: 32 words.
__device__ __forceinline__ int64_t block_prefix(int64_t v, int64_t* sWarp, int64_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) sWarp[warp] = incl;
    __syncthreads();
    int64_t w = sWarp[lane];  // every warp sums the warps' totals
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
    }
    *total = __shfl_sync(0xffffffffu, w, 31);
    const int64_t before = __shfl_sync(0xffffffffu, w, warp > 0 ? warp - 1 : 0);
    __syncthreads();  // sWarp is free
    return (warp > 0 ? before : 0) + incl - v;
}

// Ascending bitonic sort of n words (a power of two) in shared memory by the block; starts and ends with a barrier.
__device__ __forceinline__ void block_sort_u64(unsigned long long* w, int n) {
    __syncthreads();
    for (int size = 2; size <= n; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int t = threadIdx.x; t < n / 2; t += blockDim.x) {
                const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
                const unsigned long long x = w[lo], y = w[hi];
                if ((x > y) == ((lo & size) == 0)) {
                    w[lo] = y;
                    w[hi] = x;
                }
            }
            __syncthreads();
        }
}

// The word of a distance and its row; NaN orders after +inf, -0 with +0. By the bits alone: with the NaN passed through
// an FP32 addition the compiled word came out below every distance's.
__device__ __forceinline__ unsigned long long select_word(float v, int64_t row) {
    uint32_t u = __float_as_uint(v);
    if ((u & 0x7fffffffu) > 0x7f800000u)
        u = 0x7fffffffu;
    else if (u == 0x80000000u)
        u = 0u;
    return ((unsigned long long)((u & 0x80000000u) ? ~u : (u | 0x80000000u)) << 32) | (unsigned)row;
}

// Rows of a segment when n rows are selected from in up to `segs` segments (a multiple of 1024).
constexpr int kSelectSegs = 128;
inline int64_t select_seg_rows(int64_t n, int segs = kSelectSegs) { return ceil_div(ceil_div(n, segs), 1024) * 1024; }

// The segment's best min(k, m) of the values T[0..m) of rows row0.., as words in no order into out[0..k), the rest
// filled with ~0. Whole block; sN: one int.
__device__ __forceinline__ void segment_select(const float* T, int64_t row0, int m, int k, unsigned long long* out,
                                               int* sHist, int* sMisc, int* sN) {
    if (threadIdx.x == 0) *sN = 0;
    __syncthreads();
    const int kk = min(k, m);
    auto at = [&](int i) { return select_word(T[i], row0 + i); };
    const SelectBound b = block_select_bound(at, m, kk, sHist, sMisc);
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const unsigned long long w = at(i);
        if (b.in(w)) out[atomicAdd(sN, 1)] = w;
    }
    for (int i = kk + threadIdx.x; i < k; i += blockDim.x) out[i] = ~0ull;
}

}  // namespace annb
