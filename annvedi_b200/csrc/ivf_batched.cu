// Batched, list-major SQ8 pass of the exact-mode IVF query: the batch's (query, probed list) pairs
// grouped by list, scored in one persistent launch.
//
// A query batch probes each list from many queries at once (queries are drawn in proportion to list
// size, so the big lists are shared by hundreds of queries). Scanning query by query decodes every
// code once per query; here a work item is (list, up to 32 of the queries probing it, a range of up to
// kItemRows of its rows): the rows stream through shared memory in tiles of 256 rows x 32 dimensions,
// are decoded once (the exact integer of each code, FP32) and scored against the item's queries with a
// register-tiled micro-kernel (8 queries x 4, 2 or 1 rows per thread by the item's queries, two fused
// multiply-adds per element pair). Each distance lands at its position in its query's candidate stream (the positions the plan
// assigns, lsh_index_optimized.cpp:372-405 order), so a per-query selection and the FP32 re-rank
// follow unchanged. Items are taken from a global counter by a persistent grid (uneven list lengths and
// query counts balance dynamically).
//
// The SQ8 distance is the per-query scan kernel's arithmetic (ivf.cu), so a query's keys do not depend
// on the batch it came in: diff_d = fma(code_d, scale_d, -(q_d - offset_d)), the squares summed by fused
// multiply-adds in dimension order separately over the two halves of the padded code row, then
// low + high. The FP32 re-rank that follows decides the final order.
#include "block_select.cuh"
#include "common.cuh"
#include "ivf.cuh"
#include "ivf_batched.cuh"
#include "runtime.cuh"

namespace annb {

namespace {

constexpr int kBQ = 32, kTQ = 8;
constexpr int kThreads = 256;
constexpr int kBR = 256;             // rows per tile
constexpr int kKC = 32;              // dimensions per step
constexpr int kPitch = kKC + 4;      // floats

__device__ __forceinline__ void cp16(void* smem, const void* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// The set-up of a batch: its pairs (query, probed list) grouped by list. Three launches -- each pair's rank among its
// list's, the offsets by a block per array, each pair (and its operand row) to its place -- in place of a radix sort of the pairs,
// three scans and the kernels between them: for 10,000 queries x 2 lists over 2,048 with the sampled form's arrays,
// 22 launches and copies and 115 us of the GPU's time before, 37 us now. The order of a list's pairs is that of the atomics
// and of no consequence: every pair's results go to its own query.
// One thread per pair; the pair of a query's first probe also lays out its sample stream.
__global__ void pair_rank_kernel(IvfPlan p, int* __restrict__ cnt, int32_t* __restrict__ rank, int* fallback,
                                 const int64_t* __restrict__ list_off, IvfBatchTiles t) {
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= (int64_t)p.nq * p.npc) return;
    const int q = (int)(e / p.npc), j = (int)(e % p.npc);
    const int ns = p.n_seg[q];
    if (ns < 0 && j == 0) atomicExch(fallback, 1);
    rank[e] = j < ns ? atomicAdd(&cnt[p.probes[e]], 1) : -1;
    if (t.div == 0 || j != 0) return;
    int64_t run = 0;
    for (int i = 0; i < p.npc; ++i) {
        t.sseg[e + i] = run;
        if (i >= ns) continue;
        const int l = p.probes[e + i];
        run += (list_off[l + 1] - list_off[l] + t.div - 1) / t.div;
    }
    t.slen[q] = run;
}

// out[0..n] = the exclusive sums of v(0..n) by one block, a run of them a thread.
template <class V>
__device__ __forceinline__ int64_t block_offsets(int n, int64_t* out, int64_t* sWarp, V&& v) {
    const int per = (n + 1023) / 1024, i0 = min(n, (int)threadIdx.x * per), i1 = min(n, i0 + per);
    int64_t sum = 0, total;
    for (int i = i0; i < i1; ++i) sum += v(i);
    int64_t run = block_prefix(sum, sWarp, &total);
    for (int i = i0; i < i1; ++i) {
        out[i] = run;
        run += v(i);
    }
    if (threadIdx.x == 0) out[n] = total;
    return total;
}

// One block per offset array. Latency-bound: a few loads a thread and one prefix (one block for all six: 28 us).
__global__ void __launch_bounds__(1024) batch_offsets_kernel(IvfPlan p, const int* __restrict__ cnt, int C,
                                                             const int64_t* __restrict__ list_off, int64_t* lq_off,
                                                             int64_t* item_off, int64_t* cand_off, const int* fallback,
                                                             const int* apart_count, const int* key_err, int64_t* totals,
                                                             IvfBatchTiles t) {
    __shared__ int64_t sWarp[32];
    auto rows = [&](int l) { return list_off[l + 1] - list_off[l]; };
    const bool first = threadIdx.x == 0;
    if (blockIdx.x == 0) {
        block_offsets(C, lq_off, sWarp, [&](int l) -> int64_t { return cnt[l]; });
        if (t.div > 0)
            for (int l = threadIdx.x; l < C; l += 1024) t.lcap[l] = ceil_div(rows(l), t.div);
    } else if (blockIdx.x == 1) {
        const int64_t items =
            block_offsets(C, item_off, sWarp, [&](int l) { return ceil_div(cnt[l], kBQ) * ceil_div(rows(l), kItemRows); });
        if (first) {
            totals[0] = items;
            totals[2] = *fallback;
            totals[4] = key_err ? *key_err : 0;
        }
    } else if (blockIdx.x == 2) {
        const int64_t cands = block_offsets(p.nq, cand_off, sWarp, [&](int q) { return p.n_cands[q]; });
        if (first) {
            totals[1] = cands;
            totals[3] = apart_count ? *apart_count : 0;
        }
    } else if (blockIdx.x == 3) {
        if (t.titem) block_offsets(C, t.titem, sWarp, [&](int l) { return ceil_div(cnt[l], 128) * ceil_div(rows(l), 256); });
    } else if (blockIdx.x == 4) {
        if (t.div > 0)
            block_offsets(C, t.sitem, sWarp,
                          [&](int l) { return ceil_div(cnt[l], 128) * ceil_div(ceil_div(rows(l), t.div), 256); });
    } else if (t.div > 0) {
        block_offsets(p.nq, t.soff, sWarp, [&](int q) { return t.slen[q]; });
    }
}

// One warp per pair.
__global__ void __launch_bounds__(256) pair_place_kernel(IvfPlan p, const int32_t* __restrict__ rank,
                                                         const int64_t* __restrict__ lq_off,
                                                         const int64_t* __restrict__ list_off,
                                                         int32_t* __restrict__ pair_vals, int32_t* __restrict__ pair_lists,
                                                         IvfBatchTiles t) {
    const int lane = threadIdx.x & 31;
    for (int64_t e = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; e < (int64_t)p.nq * p.npc;
         e += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int r = rank[e];
        if (r < 0) continue;
        const int q = (int)(e / p.npc), l = p.probes[e];
        const int64_t i = lq_off[l] + r;
        if (t.A) {
            const uint4* src = reinterpret_cast<const uint4*>(static_cast<const char*>(t.qrows) + (size_t)q * t.row_bytes);
            uint4* dst = reinterpret_cast<uint4*>(static_cast<char*>(t.A) + (size_t)i * t.row_bytes);
            for (int c = lane; c < t.row_bytes / 16; c += 32) dst[c] = src[c];
        }
        if (lane != 0) continue;
        pair_vals[i] = (int32_t)e;
        pair_lists[i] = l;
        if (t.row_query) t.row_query[i] = q;
        // (the grouped epilogue adds the tile's absolute list row)
        if (t.sdbase) t.sdbase[i] = t.soff[q] + t.sseg[e] - list_off[l];
        if (t.pfac) t.pfac[i] = t.qfac[q];
    }
}

// qs = q - offset (zero past dim), the shifted query the SQ8 distance compares against
__global__ void shift_queries_kernel(const float* q, int nq, int dpad, int dim, const float* offset, float* qs) {
    const int64_t total = (int64_t)nq * dpad;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        const int d = (int)(e % dpad);
        qs[e] = d < dim ? __fsub_rn(q[e], offset[d]) : 0.f;
    }
}

// The shared memory of a CTA.
struct ItemSmem {
    float* q;            // [kBQ][dpad] shifted queries
    float* x;            // [kBR][kPitch] decoded rows
    float* scale;        // [dpad]
    unsigned char* raw;  // [2][kBR][kKC] codes
    int64_t* base;       // [kBQ] D position of row 0
};

// One work item: rows [r_begin, r_end) against nqi <= 8 WQ queries. WQ query groups of 8 queries; a thread holds 8
// queries x TR = WQ rows, so that an item of few queries spreads its rows over all threads instead of multiplying
// padding: at 2,000 queries x 8 lists over 2,048 lists a list has about 7 queries beside its own cluster's, and 32-query
// tiles did 1.8 times the useful work. Warps whose rows or queries lie past the item's skip the sums.
template <int WQ>
__device__ __forceinline__ void score_item(const IvfBatchArgs& a, const ItemSmem& sm, int64_t r_begin, int64_t r_end,
                                           int nqi) {
    constexpr int TR = WQ, WR = kThreads / WQ;
    static_assert(WR * TR == kBR, "a tile's rows");
    const int dpad = a.ix.dpad, dpad8 = a.ix.dpad8;
    const int tid = threadIdx.x;
    const int tq = tid / WR, tr = tid % WR;
    const int nkc = dpad8 / kKC;  // code chunks (>= dpad / kKC; extra chunks hold zero codes and scale)
    const int half_kc = nkc / 2;  // first chunk of the high half of the padded code row (dpad8 / 2)
    const int64_t ntiles = ceil_div(r_end - r_begin, kBR);
    const int64_t nsteps = ntiles * nkc;
    auto issue = [&](int64_t step) {
        if (step < nsteps) {
            const int64_t t = step / nkc;
            const int kc = (int)(step % nkc);
            unsigned char* dst = sm.raw + (size_t)(step & 1) * kBR * kKC;
            for (int c = tid; c < kBR * 2; c += kThreads) {  // 256 rows x 2 pieces of 16 codes
                const int r = c >> 1, piece = c & 1;
                const int64_t row = r_begin + t * kBR + r;
                const bool ok = row < r_end;
                cp16(dst + r * kKC + piece * 16, a.ix.codes + (ok ? row : r_begin) * dpad8 + kc * kKC + piece * 16, ok);
            }
        }
        cp_commit();
    };
    issue(0);
    float acc[kTQ][TR], lowh[kTQ][TR];
#pragma unroll
    for (int j = 0; j < kTQ; ++j)
#pragma unroll
        for (int i = 0; i < TR; ++i) acc[j][i] = lowh[j][i] = 0.f;
    int kc = 0;
    int64_t t0 = r_begin;  // first row of the tile
    for (int64_t step = 0; step < nsteps; ++step) {
        cp_wait0();
        __syncthreads();  // raw codes of this step (and the queries) landed; last step's reads are done
        issue(step + 1);
        const int rows = (int)min((int64_t)kBR, r_end - t0);  // of this tile
        // decode the rows' 32 codes: the exact integer of each byte
        {
            const unsigned char* raw = sm.raw + (size_t)(step & 1) * kBR * kKC;
            for (int e = tid; e < rows * (kKC / 4); e += kThreads) {
                const int r = e / (kKC / 4), w4 = e % (kKC / 4);
                const uint32_t w = *reinterpret_cast<const uint32_t*>(raw + r * kKC + w4 * 4);
                float4 v;
                v.x = __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u)), 8388608.f);
                v.y = __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7541u)), 8388608.f);
                v.z = __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7542u)), 8388608.f);
                v.w = __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7543u)), 8388608.f);
                *reinterpret_cast<float4*>(sm.x + r * kPitch + w4 * 4) = v;
            }
        }
        __syncthreads();
        const bool busy = tq * kTQ < nqi && (tr & ~31) < rows;  // uniform across the warp (WR is a multiple of 32)
        if (kc == half_kc) {  // the high half starts: keep the low half's sums apart
#pragma unroll
            for (int j = 0; j < kTQ; ++j)
#pragma unroll
                for (int i = 0; i < TR; ++i) {
                    lowh[j][i] = acc[j][i];
                    acc[j][i] = 0.f;
                }
        }
        if (busy && kc * kKC < dpad) {
            const float* qbase = sm.q + kc * kKC;
#pragma unroll
            for (int kk = 0; kk < kKC; kk += 4) {
                float4 xv[TR], qv[kTQ];
                const float4 sc = *reinterpret_cast<const float4*>(sm.scale + kc * kKC + kk);
#pragma unroll
                for (int i = 0; i < TR; ++i) xv[i] = *reinterpret_cast<const float4*>(sm.x + (tr + i * WR) * kPitch + kk);
#pragma unroll
                for (int j = 0; j < kTQ; ++j)
                    qv[j] = *reinterpret_cast<const float4*>(qbase + (size_t)(tq * kTQ + j) * dpad + kk);
#pragma unroll
                for (int j = 0; j < kTQ; ++j)
#pragma unroll
                    for (int i = 0; i < TR; ++i) {
                        const float d0 = __fmaf_rn(xv[i].x, sc.x, -qv[j].x);
                        const float d1 = __fmaf_rn(xv[i].y, sc.y, -qv[j].y);
                        const float d2 = __fmaf_rn(xv[i].z, sc.z, -qv[j].z);
                        const float d3 = __fmaf_rn(xv[i].w, sc.w, -qv[j].w);
                        acc[j][i] = __fmaf_rn(d0, d0, acc[j][i]);
                        acc[j][i] = __fmaf_rn(d1, d1, acc[j][i]);
                        acc[j][i] = __fmaf_rn(d2, d2, acc[j][i]);
                        acc[j][i] = __fmaf_rn(d3, d3, acc[j][i]);
                    }
            }
        }
        if (++kc == nkc) {
            kc = 0;
#pragma unroll
            for (int j = 0; j < kTQ; ++j) {
                const int qq = tq * kTQ + j;
#pragma unroll
                for (int i = 0; i < TR; ++i) {
                    const int64_t row = t0 + tr + i * WR;
                    if (qq < nqi && row < r_end) a.D[sm.base[qq] + row] = __fadd_rn(lowh[j][i], acc[j][i]);
                    acc[j][i] = 0.f;
                    lowh[j][i] = 0.f;
                }
            }
            t0 += kBR;
        }
    }
    cp_wait0();
}

__global__ void __launch_bounds__(kThreads, 2) ivf_batched_kernel(IvfBatchArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int dpad = a.ix.dpad;
    ItemSmem sm;
    sm.q = reinterpret_cast<float*>(smem_raw);
    sm.x = sm.q + (size_t)kBQ * dpad;
    sm.scale = sm.x + (size_t)kBR * kPitch;
    sm.raw = reinterpret_cast<unsigned char*>(sm.scale + dpad);
    sm.base = reinterpret_cast<int64_t*>(sm.raw + 2 * kBR * kKC);
    int* sItem = reinterpret_cast<int*>(sm.base + kBQ);

    const int tid = threadIdx.x;
    for (int d = tid; d < dpad; d += kThreads) sm.scale[d] = a.ix.scale[d];
    while (true) {
        __syncthreads();
        if (tid == 0) sItem[0] = (int)atomicAdd(a.counter, 1u);
        __syncthreads();
        const int64_t item = sItem[0];
        if (item >= a.total_items[0]) break;
        // item -> (list, query tile, row range)
        int lo = 0, hi = a.ix.C - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.item_off[mid] <= item)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int l = lo;
        const int64_t local = item - a.item_off[l];
        const int64_t nrange = ceil_div(a.ix.list_off[l + 1] - a.ix.list_off[l], kItemRows);
        const int64_t qt = local / nrange, rr = local % nrange;
        const int64_t q0 = a.lq_off[l] + qt * kBQ;
        const int nqi = (int)min((int64_t)kBQ, a.lq_off[l + 1] - q0);
        const int64_t lstart = a.ix.list_off[l];
        const int64_t r_begin = lstart + rr * kItemRows;
        const int64_t r_end = min(a.ix.list_off[l + 1], r_begin + kItemRows);
        // the item's queries (zeros up to a multiple of 8): shifted query rows and the stream position of this list's row 0
        const int nq8 = (nqi + kTQ - 1) / kTQ * kTQ;
        for (int e = tid; e < nq8 * (dpad / 4); e += kThreads) {
            const int qq = e / (dpad / 4), piece = e % (dpad / 4);
            const bool ok = qq < nqi;
            const int32_t v = ok ? a.pair_vals[q0 + qq] : 0;
            const int qi = v / a.plan.npc;
            cp16(sm.q + (size_t)qq * dpad + piece * 4, a.qs + (int64_t)qi * dpad + piece * 4, ok);
        }
        cp_commit();
        if (tid < kBQ) {
            int64_t base = 0;
            if (tid < nqi) {
                const int32_t v = a.pair_vals[q0 + tid];
                const int qi = v / a.plan.npc, j = v % a.plan.npc;
                base = a.cand_off[qi] + a.plan.seg_pref[(int64_t)qi * (a.plan.npc + 1) + j] - lstart;
            }
            sm.base[tid] = base;
        }
        if (nqi <= kTQ)
            score_item<1>(a, sm, r_begin, r_end, nqi);
        else if (nqi <= 2 * kTQ)
            score_item<2>(a, sm, r_begin, r_end, nqi);
        else
            score_item<4>(a, sm, r_begin, r_end, nqi);
    }
}

}  // namespace

size_t batched_scratch_bytes(int nq, int npc, int C) {
    const size_t n = (size_t)nq * npc;
    Sizer sz;
    for (int i = 0; i < 3; ++i) sz.take<int32_t>(n);  // ranks, pair_vals, pair_lists
    sz.take<int>((size_t)C + 2);                      // pairs per list, fallback flag, item counter
    sz.take<int64_t>((size_t)C + 1);                  // lq_off
    sz.take<int64_t>((size_t)C + 1);                  // item_off
    sz.take<int64_t>((size_t)nq + 1);                 // cand_off
    sz.take<int64_t>(5);                              // totals
    return sz.bytes();
}

int batched_prepare(const IvfQueryArgs& a, void* scratch, IvfBatchArgs* out, int64_t* host_totals, cudaStream_t st,
                    bool sync, const IvfBatchTiles& tiles) {
    const int nq = a.plan.nq, npc = a.plan.npc, C = a.ix.C;
    const int64_t n = (int64_t)nq * npc;
    ANN_CHECK_ARG(tiles.A == nullptr || tiles.row_bytes % 16 == 0, "batch set-up: operand rows of %d bytes", tiles.row_bytes);
    ANN_CHECK_ARG((tiles.pfac == nullptr) == (tiles.qfac == nullptr), "batch set-up: pair factors need query factors");
    Carver cv(scratch);
    int32_t* rank = cv.take<int32_t>(n);
    int32_t* vals = cv.take<int32_t>(n);
    int32_t* lists = cv.take<int32_t>(n);
    int* cnt = cv.take<int>((size_t)C + 2);
    int64_t* lq_off = cv.take<int64_t>((size_t)C + 1);
    int64_t* item_off = cv.take<int64_t>((size_t)C + 1);
    int64_t* cand_off = cv.take<int64_t>((size_t)nq + 1);
    int64_t* totals = cv.take<int64_t>(5);
    ANN_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int) * ((size_t)C + 2), st));
    pair_rank_kernel<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(a.plan, cnt, rank, cnt + C, a.ix.list_off, tiles);
    ANN_LAUNCH_CHECK();
    batch_offsets_kernel<<<6, 1024, 0, st>>>(a.plan, cnt, C, a.ix.list_off, lq_off, item_off, cand_off, cnt + C,
                                             a.apart ? a.apart_count : nullptr, a.key_err, totals, tiles);
    ANN_LAUNCH_CHECK();
    pair_place_kernel<<<(unsigned)std::min<int64_t>(ceil_div(n, 8), 16 * kNumSMs), 256, 0, st>>>(
        a.plan, rank, lq_off, a.ix.list_off, vals, lists, tiles);
    ANN_LAUNCH_CHECK();
    ANN_CUDA_TRY(cudaMemcpyAsync(host_totals, totals, 5 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    if (sync) ANN_CUDA_TRY(cudaStreamSynchronize(st));
    IvfBatchArgs b{};
    b.ix = a.ix;
    b.plan = a.plan;
    b.pair_vals = vals;
    b.pair_lists = lists;
    b.lq_off = lq_off;
    b.item_off = item_off;
    b.total_items = item_off + C;
    b.cand_off = cand_off;
    b.counter = reinterpret_cast<unsigned*>(cnt + C + 1);
    *out = b;
    return ANN_OK;
}

int launch_batched(const IvfBatchArgs& b, const float* qdev, float* qs, float* D, cudaStream_t st) {
    IvfBatchArgs a = b;
    a.D = D;
    a.qs = qs;
    const int nq = a.plan.nq;
    shift_queries_kernel<<<(unsigned)std::min<int64_t>(ceil_div((int64_t)nq * a.ix.dpad, 256), kNumSMs * 16), 256, 0,
                           st>>>(qdev, nq, a.ix.dpad, a.ix.dim, a.ix.offset, qs);
    ANN_LAUNCH_CHECK();
    const size_t smem = sizeof(float) * ((size_t)kBQ * a.ix.dpad + (size_t)kBR * kPitch + a.ix.dpad) +
                        (size_t)2 * kBR * kKC + sizeof(int64_t) * kBQ + 16;
    ANN_CHECK_ARG(smem <= 227 * 1024, "batched SQ8 pass: dim %d needs %zu bytes of shared memory", a.ix.dim, smem);
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(ivf_batched_kernel)));
    int per_sm = 0;
    ANN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ivf_batched_kernel, kThreads, smem));
    const int grid = kNumSMs * std::max(1, per_sm);
    ivf_batched_kernel<<<grid, kThreads, smem, st>>>(a);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace annb
