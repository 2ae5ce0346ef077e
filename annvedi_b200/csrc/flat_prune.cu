// The exact scan of a query batch with its rows pruned by tensor-core keys.
//
// The exact scan (flat_scan.cu) forms every (query, row) distance on the FP32 units: 2 N dim instructions a query,
// 45.3 ms for 1,000 queries over 1M x 384 with the tensor cores idle (0.88 ms pruned); a single query reads 4 bytes
// an element (0.37 ms, 0.19 ms pruned). Only about k distances a query are kept. Here the BF16 tensor-core keys
// (tc_gemm.cuh) say which rows can be among them, and only those rows' FP32 distances are formed, with the scan's own
// sums, so that ids and distances are the scan's bit for bit:
//   1. a BF16 key differs from the real |x|^2 - 2 x.q (or -x.q) by at most eps (launch_prune_queries);
//   2. a sampled bar tauF that about a few k keys pass, and a filter pass that keeps every key <= tauF + w,
//      w = 2 eps + delta, delta covering the rounding of the FP32 distances themselves;
//   3. per query: T, the k-th smallest kept key, is the k-th smallest of all if T <= tauF. A row whose key exceeds
//      T + w is farther, in the scan's FP32 arithmetic as in real arithmetic, than the k rows of smallest key, so
//      the best k by (distance, id) are among the kept keys <= T + w; those rows' distances are formed and the
//      best k taken.
// A query that the bound does not cover (norms out of range, NaN), whose bar was too low, or with more survivors
// than fit goes to a list that the plain scan answers right after, its length read on the device: no step waits
// for the host. Every query does if a bounded wait of the passes gave up, since their keys may then be incomplete.
#include "block_select.cuh"
#include "common.cuh"
#include "flat_prune.cuh"

#include <cmath>

#include <cuda_bf16.h>

namespace annb {

namespace {

constexpr int kFinPitch = 36;  // floats per staged row of 32: 16-byte reads of 8 rows fall in different banks
constexpr int kFinStages = 2;

__device__ __forceinline__ int row_of_pos(int64_t p, int64_t n, int64_t mult) {
    return (int)(((unsigned __int128)p * (uint64_t)mult) % (uint64_t)n);
}
__device__ __forceinline__ void cp_async16_pr(float* smem, const float* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
                 : "memory");
}

// one warp per row, grid-stride
__global__ void __launch_bounds__(256) base_norms_kernel(const float* __restrict__ x, int64_t n, int dim, int64_t ld,
                                                         unsigned* out2, float2* __restrict__ rows) {
    const int lane = threadIdx.x & 31;
    unsigned ms = 0, mr = 0;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        float s = 0.f, e = 0.f;
        for (int d = lane; d < dim; d += 32) {
            const float v = x[r * ld + d];
            const float t = v - __bfloat162float(__float2bfloat16_rn(v));  // exact
            s = fmaf(v, v, s);
            e = fmaf(t, t, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, o);
            e += __shfl_xor_sync(0xffffffffu, e, o);
        }
        if (rows && lane == 0) rows[r] = make_float2(sqrtf(s), sqrtf(e));
        // non-negative floats order as their bit patterns, NaN above them all (its sign cleared)
        ms = max(ms, __float_as_uint(s) & 0x7fffffffu);
        mr = max(mr, __float_as_uint(e) & 0x7fffffffu);
    }
    if (lane == 0) {
        atomicMax(&out2[0], ms);
        atomicMax(&out2[1], mr);
    }
}

// One warp per query: its window w = 2 eps + delta (key_window_l2 / _ip), its operand row and its counter.
__global__ void __launch_bounds__(256) prune_queries_kernel(PruneArgs a, __nv_bfloat16* __restrict__ qb, int kpad) {
    const int q = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (q >= a.nq) return;
    const bool l2 = a.metric == ANN_METRIC_L2;
    float s = 0.f, e = 0.f;
    const float* __restrict__ x = a.q + (int64_t)q * a.dpad;
    for (int d = lane; d < kpad; d += 32) {
        const float v = d < a.dim ? x[d] : 0.f;
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        const float t = v - __bfloat162float(b);
        s = fmaf(v, v, s);
        e = fmaf(t, t, e);
        qb[(int64_t)q * kpad + d] = l2 && d >= a.dim && d < a.dim + 3 ? __float2bfloat16_rn(1.f)
                                                                      : __float2bfloat16_rn(l2 ? -2.f * v : -v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if (lane != 0) return;
    // Squares of components below 2^-74 are lost, so s = 0 does not say that the query is zero. Under L2 norms below
    // kPruneNormMin count as that, their share of the window nil beside the rows' own; under inner product every term
    // of the window is the query's, and such queries, zero among them (every key the same), are left to the scan.
    const float qn = fmaxf(sqrtf(s), kPruneNormMin), rq = fmaxf(sqrtf(e), kPruneNormMin);
    const float w = l2 ? key_window_l2(qn, rq, a.b.cmax, a.b.rmax, a.dim)
                       : key_window_ip(sqrtf(s), sqrtf(e), a.b.cmax, a.b.rmax, a.dim);
    const bool ok = s < kInf && qn <= kPruneNormMax && (l2 || sqrtf(s) >= kPruneNormMin);  // false for NaN
    a.win[q] = ok ? w : __int_as_float(0x7fffffff);
    a.rcount[q] = 0;
    if (a.joined) a.joined[q] = make_int2(0, 0);
    if (q == 0) *a.count = *a.err = 0;
}

// One block per query (file comment, step 3). Bound by the gather of the kept rows (about 500 rows of 1.5 KB a query
// at 1M x 384, k = 100): each warp takes 32 rows at a time, 128 bytes of each by coalesced asynchronous copies into
// its own stage, and each lane then sums its own row in the scan's order -- a row's terms are one serial chain, so
// 32 rows a warp, not 32 lanes a row, keep the FP32 pipe fed.
//   staged scan: one chain over d; streaming scan: 8 chains (floats 4o .. 4o + 3 of every 32), added pairwise.
// Warps: 8, two blocks per SM; 16 where a launch has no second block for an SM (launch_prune_finish): one query over
// 1M x 384, 33 -> 25 us.
// With gridDim.y > 1 (few queries) a query's rows beyond those of one round of the warps go to further blocks, each taking
// its run of the survivors; the block that ends last selects. A round is a chain of dim / 32 steps of about 1 us: clustered
// data of many dimensions, whose windows hold thousands of rows, took up to eight rounds in one block (one query over
// 20,000 x 2,048 normal / clustered: 118 / 152 us; 5 over 20,000 x 4,096: 216 / 880, scanned 438). The code and the blocks that
// mostly have nothing to do cost a single query 2 us (a kernel of one block fetches its instructions anew each call), so an
// index's passes have them (SPLIT) from the first query on that would use one.
template <bool STREAM, int METRIC, int kFinWarps, bool SPLIT>
__global__ void __launch_bounds__(kFinWarps * 32) prune_finish_kernel(PruneArgs a) {
    constexpr int kFinThreads = kFinWarps * 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int cap = a.cap, k = a.k, dpad = a.dpad;
    float* sX = reinterpret_cast<float*>(smem_raw);                                  // [warps][stages][32 pitch]
    float* sQ = sX + kFinWarps * kFinStages * 32 * kFinPitch;                        // [dpad]
    unsigned long long* sE = reinterpret_cast<unsigned long long*>(sQ + dpad);       // [cap] (distance, row)
    uint32_t* sO = reinterpret_cast<uint32_t*>(sE);                                  // [cap] keys, before sE is filled
    __shared__ int sHist[256];
    __shared__ int sMisc[12];
    __shared__ int sN;
    const int q = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cnt = a.rcount[q];
    const float w = a.win[q], tauF = a.tauF[q];
    const int gave_up = *a.err;  // (with the loads above, not a round trip of its own behind them)
    if (SPLIT && blockIdx.y > 0 && cnt <= (int)blockIdx.y * kFinThreads) return;  // no more than the blocks before take
    const float* fk = a.fkey + (int64_t)q * cap;
    const int* fc = a.fcol + (int64_t)q * cap;
    bool fail = cnt > cap || cnt < k || !(w < kInf) || gave_up != 0;
    float T = 0.f;
    if (!fail) {  // the k-th smallest kept key
        for (int i = tid; i < cnt; i += kFinThreads) sO[i] = ord_f32(fk[i]);
        __syncthreads();
        T = f32_ord(block_kth([&](int i) { return sO[i]; }, cnt, k, sHist, sMisc));
        fail = !(T <= tauF);
    }
    if (fail) {  // uniform
        if (tid == 0 && (!SPLIT || blockIdx.y == 0)) a.list[atomicAdd(a.count, 1)] = q;
        return;
    }
    const float lim = __fadd_ru(T, w);  // <= tauX: every key at or below it was kept
    auto collect = [&](int i0, int i1, bool first) {  // the rows of survivors [i0, i1) within the window; returns their number
        if (tid == 0) sN = 0;
        __syncthreads();
        if (first)  // (behind the barrier, beside the survivors' loads)
            for (int d = tid; d < dpad; d += kFinThreads) sQ[d] = a.q[(int64_t)q * dpad + d];
        for (int i = i0 + tid; i < i1; i += kFinThreads)
            if (fk[i] <= lim) sE[atomicAdd(&sN, 1)] = (unsigned)row_of_pos(fc[i], a.n, a.mult);
        __syncthreads();
        return sN;
    };
    const int total = collect(0, cnt, true);  // >= k, the same in every block of the query
    const int blocks = SPLIT ? min((int)gridDim.y, (total + kFinThreads - 1) / kFinThreads) : 1;
    if (SPLIT && (int)blockIdx.y >= blocks) return;
    if (!SPLIT && a.wide && total > kFinThreads && tid == 0) *static_cast<volatile unsigned long long*>(a.wide) = 1ull;
    int m = total;
    if (SPLIT && blocks > 1) {
        __syncthreads();
        m = collect((int)((int64_t)cnt * blockIdx.y / blocks), (int)((int64_t)cnt * (blockIdx.y + 1) / blocks), false);
    }
    float* myX = sX + warp * kFinStages * 32 * kFinPitch;
    const int nch = dpad / 32;
    for (int g = warp * 32; g < m; g += kFinWarps * 32) {
        const int row = (int)(unsigned)sE[min(g + lane, m - 1)];
        const int rows = min(32, m - g);
        auto issue = [&](int c) {
            if (c < nch) {
                float* dst = myX + (c % kFinStages) * 32 * kFinPitch;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = 4 * i + (lane >> 3);
                    const int rr = __shfl_sync(0xffffffffu, row, r);
                    if (r < rows)
                        cp_async16_pr(dst + r * kFinPitch + (lane & 7) * 4,
                                      a.base + (int64_t)rr * dpad + c * 32 + (lane & 7) * 4);
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        float acc[STREAM ? 8 : 1];
#pragma unroll
        for (int o = 0; o < (STREAM ? 8 : 1); ++o) acc[o] = 0.f;
        __syncwarp();  // every lane is done with the last group's stages
        issue(0);
        for (int c = 0; c < nch; ++c) {
            issue(c + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncwarp();
            const float* x = myX + (c % kFinStages) * 32 * kFinPitch + lane * kFinPitch;
            const float* qc = sQ + c * 32;
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                const float4 xv = *reinterpret_cast<const float4*>(x + 4 * o);
                const float4 qv = *reinterpret_cast<const float4*>(qc + 4 * o);
                float& s = acc[STREAM ? o : 0];
                if (METRIC == ANN_METRIC_L2) {
                    const float d0 = xv.x - qv.x, d1 = xv.y - qv.y, d2 = xv.z - qv.z, d3 = xv.w - qv.w;
                    s = fmaf(d0, d0, s);
                    s = fmaf(d1, d1, s);
                    s = fmaf(d2, d2, s);
                    s = fmaf(d3, d3, s);
                } else {
                    s = fmaf(xv.x, qv.x, s);
                    s = fmaf(xv.y, qv.y, s);
                    s = fmaf(xv.z, qv.z, s);
                    s = fmaf(xv.w, qv.w, s);
                }
            }
            __syncwarp();  // the stage is free for the copies issued next
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        float v = acc[0];
        if (STREAM)
            v = ((acc[0] + acc[1 % (STREAM ? 8 : 1)]) + (acc[2 % (STREAM ? 8 : 1)] + acc[3 % (STREAM ? 8 : 1)])) +
                ((acc[4 % (STREAM ? 8 : 1)] + acc[5 % (STREAM ? 8 : 1)]) +
                 (acc[6 % (STREAM ? 8 : 1)] + acc[7 % (STREAM ? 8 : 1)]));
        // + 0: a key of -0 orders with +0, by row
        if (lane < rows)
            sE[g + lane] = ((unsigned long long)ord_f32((METRIC == ANN_METRIC_L2 ? v : -v) + 0.f) << 32) | (unsigned)row;
    }
    __syncthreads();
    if (SPLIT && blocks > 1) {
        unsigned long long* gw = a.words + (int64_t)q * cap;
        __shared__ int sAt;
        if (tid == 0) sAt = atomicAdd(&a.joined[q].x, m);
        __syncthreads();
        for (int i = tid; i < m; i += kFinThreads) gw[sAt + i] = sE[i];
        __threadfence();
        __syncthreads();
        if (tid == 0) sAt = atomicAdd(&a.joined[q].y, 1);
        __syncthreads();
        if (sAt != blocks - 1) return;  // uniform: another block of the query is still to come
        __threadfence();
        m = total;
        for (int i = tid; i < m; i += kFinThreads) sE[i] = __ldcg(gw + i);
        __syncthreads();
    }
    const SelectBound bound = block_select_bound<true>([&](int i) { return sE[i]; }, m, k, sHist, sMisc);
    unsigned long long* sR = reinterpret_cast<unsigned long long*>(sX);  // the best k, then sorted
    const int p2 = pow2_ceil(k);
    if (tid == 0) sN = 0;
    __syncthreads();
    for (int i = tid; i < m; i += kFinThreads)
        if (bound.in(sE[i])) sR[atomicAdd(&sN, 1)] = sE[i];
    for (int i = k + tid; i < p2; i += kFinThreads) sR[i] = ~0ull;
    block_sort_u64(sR, p2);
    for (int e = tid; e < k; e += kFinThreads) {
        a.out_ids[(int64_t)q * k + e] = (int64_t)(unsigned)sR[e];
        if (a.out_dists) {
            const float key = f32_ord((uint32_t)(sR[e] >> 32));
            a.out_dists[(int64_t)q * k + e] = METRIC == ANN_METRIC_L2 ? key : 0.f - key;
        }
    }
}

__global__ void prune_gather_kernel(const float* __restrict__ q, int dpad, const int* __restrict__ list,
                                    const int* __restrict__ count, float* __restrict__ qg, int nq,
                                    volatile unsigned long long* word, uint32_t pass, int report) {
    const int n = *count;
    if (word && (n > 0 || report) && blockIdx.x == 0 && threadIdx.x == 0)  // over PCIe, and the kernels that follow wait for it
        *word = ((unsigned long long)pass << 32) | ((unsigned)nq << 16) | (unsigned)n;
    for (int j = blockIdx.x; j < n; j += gridDim.x)
        for (int d = threadIdx.x; d < dpad; d += blockDim.x) qg[(int64_t)j * dpad + d] = q[(int64_t)list[j] * dpad + d];
}

size_t finish_smem(int cap, int dpad, int warps) {
    return sizeof(float) * ((size_t)warps * kFinStages * 32 * kFinPitch + dpad) + sizeof(unsigned long long) * cap;
}
template <int W, bool SPLIT>
int run_finish(const PruneArgs& a, cudaStream_t st) {
    auto kern = a.metric == ANN_METRIC_L2
                    ? (a.stream_form ? prune_finish_kernel<true, ANN_METRIC_L2, W, SPLIT> : prune_finish_kernel<false, ANN_METRIC_L2, W, SPLIT>)
                    : (a.stream_form ? prune_finish_kernel<true, ANN_METRIC_IP, W, SPLIT> : prune_finish_kernel<false, ANN_METRIC_IP, W, SPLIT>);
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(kern)));
    const int blocks = SPLIT ? (int)std::min<int64_t>(ceil_div(a.cap, W * 32), std::max(1, kNumSMs / a.nq)) : 1;
    kern<<<dim3(a.nq, blocks), W * 32, finish_smem(a.cap, a.dpad, W), st>>>(a);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace

int prune_cap(int k) { return k <= 128 ? 4096 : 8192; }
bool prune_split(int nq) { return nq <= kNumSMs / 2; }
bool prune_fits(int k, int dpad) { return k <= 512 && finish_smem(prune_cap(k), dpad, 8) <= 200 * 1024; }

int prune_bar_rank(int k, int64_t S, int64_t n) {
    // keys of the k best met in the sample: about Poisson(k S / n); the rank past its 1 - 1e-7 quantile
    const double lam = (double)k * (double)S / (double)n;
    double term = std::exp(-lam), cdf = term;
    int r = 1;
    while (r < k && 1.0 - cdf > 1e-7) {
        term *= lam / r;
        cdf += term;
        ++r;
    }
    return r;
}

int launch_base_norms(const float* x, int64_t n, int dim, int64_t ld, unsigned* out2, cudaStream_t st, float2* rows) {
    ANN_CUDA_TRY(cudaMemsetAsync(out2, 0, 2 * sizeof(unsigned), st));
    if (n == 0) return ANN_OK;
    base_norms_kernel<<<(unsigned)std::min<int64_t>(ceil_div(n, 8), 16 * kNumSMs), 256, 0, st>>>(x, n, dim, ld, out2, rows);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_prune_queries(const PruneArgs& a, __nv_bfloat16* qb, int kpad, cudaStream_t st) {
    prune_queries_kernel<<<(unsigned)ceil_div(a.nq, 8), 256, 0, st>>>(a, qb, kpad);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_prune_finish(const PruneArgs& a, cudaStream_t st) {
    ANN_CHECK_ARG(a.k >= 1 && prune_fits(a.k, a.dpad) && a.dpad % 32 == 0 && a.cap == prune_cap(a.k),
                  "pruned scan: k=%d, padded dim %d", a.k, a.dpad);
    ANN_CHECK_ARG((a.words == nullptr) == (a.joined == nullptr), "pruned scan: shared rows need both arrays");
    const bool wide = a.nq <= kNumSMs && finish_smem(a.cap, a.dpad, 16) <= 220 * 1024;
    if (a.words) return wide ? run_finish<16, true>(a, st) : run_finish<8, true>(a, st);
    return wide ? run_finish<16, false>(a, st) : run_finish<8, false>(a, st);
}

int launch_prune_gather(const float* q, int dpad, const int* list, const int* count, int nq, float* qg,
                        unsigned long long* word, uint32_t pass, int report, cudaStream_t st) {
    ANN_CHECK_ARG(nq <= 65535, "pruned scan: %d queries a pass", nq);
    prune_gather_kernel<<<(unsigned)std::min(nq, 2 * kNumSMs), 128, 0, st>>>(q, dpad, list, count, qg, nq, word, pass, report);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace annb
