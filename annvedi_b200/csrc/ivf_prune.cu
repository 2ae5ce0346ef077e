// The exact SQ8 selection of a query batch, its candidates pruned by tensor-core keys.
//
// The batched SQ8 pass (ivf_batched.cu) forms every candidate's SQ8 distance on the FP32 units, of which the best R are
// kept: 1.5 ms of 2.05 for 2,000 queries x 8 of 2,048 lists of 1M x 384 whose sizes follow a power law. As for the linear
// scan (flat_prune.cu), 16-bit keys say which candidates can be among the best R, and only theirs are formed, by the
// batched pass's own arithmetic:
//   * the distance is sum_d (y_d - u_d)^2 with y = scale (code - 127.5) and u = q - offset - 127.5 scale. Codes less 127.5
//     are exact in 16 bits, so the lists' operand has no rounding at all, and the queries' carries the scale:
//     key = |y|^2 - 2 sum_d (code_d - 127.5) f16(scale_d u_d), all of it scaled by powers of two into FP16's range. Centred
//     so, the keys' error does not grow with the data's distance from the origin. FP16 and not BF16: a list of 40,000
//     rows around one centre holds its best 400 so densely that BF16's window (0.0095 at unit norms) kept several
//     thousand more, FP16's (0.0024) a few hundred;
//   * the heads of the probed lists give a sampled bar per query (as the tensor-core form's), the grouped filter pass keeps
//     the keys up to the bar plus the window, and if the R-th smallest kept key is within the bar, the best R by
//     (distance, stream position) are among the keys up to it plus the window.
// A query that this does not settle (bar too low, more survivors than fit, norms out of range) is counted, and the
// caller runs the batched pass. The batch above: sample and filter passes 0.33 ms, bars 0.035, finish 0.19 in place of
// the batched pass's 1.50 and its selection's 0.18.
#include "block_select.cuh"
#include "common.cuh"
#include "ivf_prune.cuh"

namespace annb {

namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kChunk = 64, kStages = 2;  // 41 KB of stages: three blocks per SM at R = 400
__host__ __device__ constexpr int formed_cap(int R) { return 8 * R; }  // distances formed for a query at most
constexpr int kPitch = kChunk + 16;  // bytes per staged piece: 16-byte reads of 8 lanes fall in different banks

__device__ __forceinline__ float u8f(uint32_t word, int byte) {  // the exact float of a byte (2^23 + byte, less 2^23)
    return __fsub_rn(__uint_as_float(__byte_perm(word, 0x4B000000u, 0x7540u | byte)), 8388608.f);
}

// The FP16 value of v, zero where it would be subnormal: nothing below relies on how an MMA takes those.
__device__ __forceinline__ float f16_normal(float v) {
    const float o = __half2float(__float2half_rn(v));
    return fabsf(o) < 6.103515625e-5f ? 0.f : o;
}

// one warp per row
__global__ void __launch_bounds__(256) sq8_max_norm_kernel(IvfView ix, unsigned* max2) {
    const int lane = threadIdx.x & 31;
    unsigned ms = 0;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < ix.n;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        float s = 0.f;
        for (int d = lane; d < ix.dim; d += 32) {
            const float y = __fmul_rn(ix.scale[d], (float)ix.codes[r * ix.dpad8 + d] - 127.5f);
            s = fmaf(y, y, s);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        ms = max(ms, __float_as_uint(s) & 0x7fffffffu);
    }
    if (lane == 0) atomicMax(max2, ms);
}

// One warp per row. HBM-bound: a byte read and two written an element.
__global__ void __launch_bounds__(256) sq8_operand_kernel(IvfView ix, float g, __half* __restrict__ out, int kpad) {
    const int lane = threadIdx.x & 31;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < ix.n;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        float s = 0.f;
        for (int d = lane; d < kpad; d += 32) {
            const float c = d < ix.dim ? (float)ix.codes[r * ix.dpad8 + d] - 127.5f : 0.f;
            const float y = d < ix.dim ? g * __fmul_rn(ix.scale[d], c) : 0.f;
            s = fmaf(y, y, s);
            if (d < ix.dim || d >= ix.dim + 3) out[r * kpad + d] = __float2half_rn(c * 0.0078125f);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {  // the key columns; what the pieces leave is below 2^-14
            s *= 1024.f;
            const float hi = f16_normal(s), mid = f16_normal(s - hi), lo = f16_normal((s - hi) - mid);
            out[r * kpad + ix.dim] = __float2half_rn(hi);
            out[r * kpad + ix.dim + 1] = __float2half_rn(mid);
            out[r * kpad + ix.dim + 2] = __float2half_rn(lo);
        }
    }
}

// One warp per query: its operand row -2^16 g^2 scale u, then 1/4 for the key columns (a key is 256 g^2 times the distance
// less |u|^2), and its window. With y the rows and w^ the weights w as rounded,
//   |sum_d (code_d - 127.5) (w_d - w^_d)| <= |y| |u (w - w^) / w| + 127.5 sum |w_d|,
// the second sum over the weights that became zero. The FP32 accumulation of the dim + 3 products adds acc times their
// absolute sum (as key_window_l2), the roundings of y, u, w and of the pieces a few 2^-24.
__global__ void __launch_bounds__(256) ivf_prune_queries_kernel(IvfPruneArgs a) {
    const int q = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (q >= a.plan.nq) return;
    const int dim = a.ix.dim;
    float s = 0.f, e = 0.f, z = 0.f;
    for (int d = lane; d < a.kpad; d += 32) {
        float o = d < dim + 3 ? 0.25f : 0.f;
        if (d < dim) {
            const float sc = a.ix.scale[d];
            const float u = __fmaf_rn(-127.5f, sc, __fsub_rn(a.q[(int64_t)q * a.ldq + d], a.ix.offset[d]));
            const float w = __fmul_rn(a.g * sc, a.g * u) * -65536.f;
            o = f16_normal(w);
            if (o != 0.f) {
                const float t = u * ((w - o) / w);  // an overflow ends as inf
                e = fmaf(t, t, e);
            } else {
                z += fabsf(w);
            }
            s = fmaf(u, u, s);
        }
        a.qop[(int64_t)q * a.kpad + d] = __float2half_rn(o);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        e += __shfl_xor_sync(0xffffffffu, e, o);
        z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    const float qn = sqrtf(s), cm = a.cmax, g = a.g, D = qn + cm;
    const float acc = (float)(dim + 19) * 4.76837158e-7f;  // (dim + 19) 2^-21
    // in units of the distance; z is in the operand's: a key's 256 g^2, code units of 128
    const float eps = 2.f * cm * sqrtf(e) + acc * (2.f * cm * qn + 1.25f * cm * cm) + 32.f * 5.9604645e-8f * D * D;
    const float S = 256.f * g * g;
    const bool ok = qn <= kPruneNormMax && (qn >= kPruneNormMin || s == 0.f);
    const float w2 = 2.004f * (S * eps + z);
    if (ok && w2 < kInf) {
        if (lane == 0) a.win[q] = make_float2(w2, S * s);
    } else {  // left to the batched pass; keys of zero meanwhile
        if (lane == 0) a.win[q] = make_float2(__int_as_float(0x7fffffff), 0.f);
        for (int d = lane; d < a.kpad; d += 32) a.qop[(int64_t)q * a.kpad + d] = __float2half_rn(0.f);
    }
}

// The key up to which the best candidates lie if the need-th smallest key is T: twice the keys' error (w.x) and the
// rounding of two SQ8 distances, each of at most (dim + 8) 2^-24 of itself, the distance being T + |u|^2 or less.
__device__ __forceinline__ float prune_limit(float T, float2 w, int dim) {
    const float dist = fmaxf(0.f, T + w.y) + w.x;
    return __fadd_ru(T, __fadd_ru(w.x, 2.2f * (float)(dim + 24) * 5.9604645e-8f * dist));
}

__global__ void ivf_prune_bars_kernel(IvfPruneArgs a) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0) *a.fails = 0;
    if (q >= a.plan.nq) return;
    a.tauX[q] = prune_limit(a.tauF[q], a.win[q], a.ix.dim);
    a.rcount[q] = 0;
}

// One block per query: the bar among its survivors' keys, the SQ8 distances of those within the window and the best R
// of them. A warp forms 16 distances at a time: the sums of the low and of the high half of the padded codes are
// independent chains (ivf_batched.cu), so a lane takes one half of one candidate, its codes staged by coalesced
// asynchronous copies 64 at a time.
__global__ void __launch_bounds__(kThreads) ivf_prune_finish_kernel(IvfPruneArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int cap = a.cap, R = a.R, mcap = formed_cap(a.R), dpad8 = a.ix.dpad8, npc = a.plan.npc;
    unsigned char* sX = smem_raw;                                                // [warps][stages][32][kPitch]
    float* sQ = reinterpret_cast<float*>(sX + kWarps * kStages * 32 * kPitch);   // [dpad8] -(q - offset)
    float* sS = sQ + dpad8;                                                      // [dpad8] scale
    unsigned long long* sE = reinterpret_cast<unsigned long long*>(sS + dpad8);  // [mcap] (distance, position)
    uint32_t* sO = reinterpret_cast<uint32_t*>(sE);  // [cap = 2 mcap] keys, before sE is filled
    __shared__ int sHist[256];
    __shared__ int sMisc[12];
    __shared__ int sN;
    __shared__ int64_t sStart[kIvfPruneMaxLists], sPref[kIvfPruneMaxLists + 1];
    const int q = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cnt = a.rcount[q], ns = a.plan.n_seg[q];
    const float2 w = a.win[q];
    const float tauF = a.tauF[q];
    const int gave_up = *a.err;
    const int64_t cands = a.plan.n_cands[q];
    const int need = (int)min((int64_t)R, cands);
    const float* fk = a.fkey + (int64_t)q * cap;
    const int* fr = a.frow + (int64_t)q * cap;
    float* ok = a.keyR + (int64_t)q * R;
    int* oi = a.idR + (int64_t)q * R;
    for (int e = need + tid; e < R; e += kThreads) {
        ok[e] = kInf;
        oi[e] = kNoId;
    }
    if (need == 0) return;  // an empty stream (a query set apart)
    bool fail = ns < 0 || cnt > cap || cnt < need || !(w.x < kInf) || gave_up != 0;
    float T = 0.f;
    if (!fail) {  // the need-th smallest kept key
        for (int i = tid; i < cnt; i += kThreads) sO[i] = ord_f32(fk[i]);
        __syncthreads();
        T = f32_ord(block_kth([&](int i) { return sO[i]; }, cnt, need, sHist, sMisc));
        fail = !(T <= tauF);
    }
    if (fail) {  // uniform
        if (tid == 0) atomicAdd(a.fails, 1);
        return;
    }
    const float lim = prune_limit(T, w, a.ix.dim);
    if (tid == 0) {
        sN = 0;
        sPref[ns] = cands;
    }
    if (tid < ns) {
        sStart[tid] = a.plan.seg_start[(int64_t)q * npc + tid];
        sPref[tid] = a.plan.seg_pref[(int64_t)q * (npc + 1) + tid];
    }
    for (int d = tid; d < dpad8; d += kThreads) {
        const bool in = d < a.ix.dim;
        sQ[d] = in ? -__fsub_rn(a.q[(int64_t)q * a.ldq + d], a.ix.offset[d]) : 0.f;
        sS[d] = in ? a.ix.scale[d] : 0.f;
    }
    __syncthreads();
    for (int i = tid; i < cnt; i += kThreads) {
        if (!(fk[i] <= lim)) continue;
        const int at = atomicAdd(&sN, 1);
        if (at < mcap) sE[at] = (unsigned)fr[i];
    }
    __syncthreads();
    const int m = sN;  // >= need
    if (m > mcap) {
        if (tid == 0) atomicAdd(a.fails, 1);
        return;
    }
    unsigned char* myX = sX + (size_t)warp * kStages * 32 * kPitch;
    const int half = dpad8 / 2, nch = half / kChunk;
    const int cl = lane & 15, hl = lane >> 4;
    for (int g = warp * 16; g < m; g += kWarps * 16) {
        const int row = (int)(unsigned)sE[min(g + cl, m - 1)];
        auto issue = [&](int c) {
            if (c < nch) {
                unsigned char* dst = myX + (c % kStages) * 32 * kPitch;
#pragma unroll
                for (int i = 0; i < 4; ++i) {  // 32 (half, candidate) pieces of 4 x 16 bytes
                    const int p = 8 * i + (lane >> 2);
                    const int rr = __shfl_sync(0xffffffffu, row, p);
                    const unsigned sm = (unsigned)__cvta_generic_to_shared(dst + p * kPitch + (lane & 3) * 16);
                    const uint8_t* src =
                        a.ix.codes + (int64_t)rr * dpad8 + (p >> 4) * half + c * kChunk + (lane & 3) * 16;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sm), "l"(src) : "memory");
                }
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        float acc = 0.f;
        __syncwarp();  // every lane is done with the last group's stages
        issue(0);
        for (int c = 0; c < nch; ++c) {
            issue(c + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncwarp();
            const unsigned char* x = myX + (c % kStages) * 32 * kPitch + lane * kPitch;
            const float* sc = sS + hl * half + c * kChunk;
            const float* qc = sQ + hl * half + c * kChunk;
#pragma unroll
            for (int p = 0; p < kChunk / 16; ++p) {
                const uint4 cw = *reinterpret_cast<const uint4*>(x + p * 16);
                const uint32_t wv[4] = {cw.x, cw.y, cw.z, cw.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 s4 = *reinterpret_cast<const float4*>(sc + p * 16 + 4 * j);
                    const float4 q4 = *reinterpret_cast<const float4*>(qc + p * 16 + 4 * j);
                    const float e0 = __fmaf_rn(u8f(wv[j], 0), s4.x, q4.x), e1 = __fmaf_rn(u8f(wv[j], 1), s4.y, q4.y);
                    const float e2 = __fmaf_rn(u8f(wv[j], 2), s4.z, q4.z), e3 = __fmaf_rn(u8f(wv[j], 3), s4.w, q4.w);
                    acc = __fmaf_rn(e0, e0, acc);
                    acc = __fmaf_rn(e1, e1, acc);
                    acc = __fmaf_rn(e2, e2, acc);
                    acc = __fmaf_rn(e3, e3, acc);
                }
            }
            __syncwarp();  // the stage is free for the copies issued next
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        const float high = __shfl_down_sync(0xffffffffu, acc, 16);
        if (lane < 16 && g + lane < m) {
            int64_t pos = 0;
            for (int j = 0; j < ns; ++j)
                if (row >= sStart[j] && row < sStart[j] + (sPref[j + 1] - sPref[j])) pos = sPref[j] + (row - sStart[j]);
            sE[g + lane] = select_word(__fadd_rn(acc, high), pos);
        }
    }
    __syncthreads();
    const SelectBound bound = block_select_bound<true>([&](int i) { return sE[i]; }, m, need, sHist, sMisc);
    if (tid == 0) sN = 0;
    __syncthreads();
    for (int i = tid; i < m; i += kThreads) {
        if (!bound.in(sE[i])) continue;
        const int at = atomicAdd(&sN, 1);
        ok[at] = f32_ord((uint32_t)(sE[i] >> 32));
        oi[at] = (int)plan_row(a.plan, q, (int64_t)(unsigned)sE[i]);
    }
}

size_t finish_smem(int R, int dpad8) {
    return (size_t)kWarps * kStages * 32 * kPitch + sizeof(float) * 2 * dpad8 + sizeof(unsigned long long) * formed_cap(R);
}

}  // namespace

bool ivf_prune_fits(int R, int npc, int dpad8) {
    return npc <= kIvfPruneMaxLists && dpad8 % 128 == 0 && R <= 1024 && finish_smem(R, dpad8) <= 200 * 1024;
}

int launch_sq8_max_norm(const IvfView& ix, unsigned* max2, cudaStream_t st) {
    ANN_CUDA_TRY(cudaMemsetAsync(max2, 0, sizeof(unsigned), st));
    sq8_max_norm_kernel<<<(unsigned)std::min<int64_t>(ceil_div(ix.n, 8), 16 * kNumSMs), 256, 0, st>>>(ix, max2);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_sq8_operand(const IvfView& ix, float g, __half* out, int kpad, cudaStream_t st) {
    sq8_operand_kernel<<<(unsigned)std::min<int64_t>(ceil_div(ix.n, 8), 16 * kNumSMs), 256, 0, st>>>(ix, g, out, kpad);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_ivf_prune_queries(const IvfPruneArgs& a, cudaStream_t st) {
    ivf_prune_queries_kernel<<<(unsigned)ceil_div(a.plan.nq, 8), 256, 0, st>>>(a);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_ivf_prune_bars(const IvfPruneArgs& a, cudaStream_t st) {
    ivf_prune_bars_kernel<<<(unsigned)ceil_div(a.plan.nq, 256), 256, 0, st>>>(a);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

int launch_ivf_prune_finish(const IvfPruneArgs& a, cudaStream_t st) {
    ANN_CHECK_ARG(a.R <= a.cap && a.cap <= 2 * formed_cap(a.R) && ivf_prune_fits(a.R, a.plan.npc, a.ix.dpad8),
                  "pruned SQ8 selection: R=%d, %d lists, code stride %d", a.R, a.plan.npc, a.ix.dpad8);
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(ivf_prune_finish_kernel)));
    ivf_prune_finish_kernel<<<a.plan.nq, kThreads, finish_smem(a.R, a.ix.dpad8), st>>>(a);
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace annb
