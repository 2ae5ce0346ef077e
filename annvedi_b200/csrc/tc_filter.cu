// Dense filter pass of the tensor-core searches: for every (query, base row) the key of tc_gemm.cuh, and only the keys
// at or below the query's bar kept, appended to the query's own buffer.
//
// The pass is a [M, N] = A B^T GEMM whose output is thrown away but for about 1 key in 1,000. What bounded it as a
// plain 128 x 256 tiling (one CTA a tile, both operands through the ring) on 2,560 queries x 400k, by ncu: with BF16 at
// dim 384 the L2-to-SM path, 15.1 TB/s = 62 of its 64 bytes/clock/SM, the tensor pipe 59% active; with E4M3 at dim 256
// (half the bytes, twice the rate) the epilogue, 11 instructions a key. So here
//   * two CTAs of a cluster share a 256 x 256 tile (cta_group::2): each loads its 128 query rows and half of the
//     tile's base rows, so a base row crosses to an SM pair once, not twice;
//   * the query tile stays in shared memory for a run of base tiles where it fits beside the ring (K up to about
//     570 BF16), so only base rows stream (4.7 TB/s over the L2 path);
//   * runs are cut from L2-sized chunks of the base, all clusters inside one chunk at a time, so that a base row
//     comes from HBM once, whatever the number of query tiles;
//   * the epilogue takes a three-input minimum over 8 keys and looks at single keys only where a lane's minimum
//     passes its bar; survivors are queued per warp and go out 32 at a time (an atomic a survivor as it is met
//     made each wait for the one before: 10,000 clocks a tile). The accumulator is released as soon as it is in
//     registers.
//   * the MMA issuer's loop is kept short (see there): at 66 instructions' latency a k-block it, not the tensor cores,
//     set the rate.
// Measured at 5,120 queries x 1M x 384: 2.48 ms with no survivors (1.65 PFLOP/s; 1.81 at K = 512, cuBLAS's measured burst
// is 1.69), 2.65 ms with 1.2 survivors per 1,000 keys, where the plain tiling took 3.48 ms and grouped its survivors in
// 0.28 ms more; E4M3 at dim 256 1.29 ms (2.04 PFLOP/s; 2.3 ms before, by the 4M-row case). With the first issue loop
// 3.24 ms, and neither ring depth, chunk size nor residency of the query tile changed that by 1%.
// Batches of up to 128 queries are bound by reading the base once and keep one CTA a tile (CG = 1).
//
//   warp 0      base-row producer (TMA, 128-byte swizzle);  warp 18: query-tile producer (resident form)
//   warp 1      TMEM (two 256-column accumulators) and, in the pair's first CTA, the MMA issuer
//   warps 2-17  epilogue: warp w reads TMEM lanes 32 (w % 4), 64 columns
// Every mbarrier wait is bounded (2 s); a timeout raises the device flag and the CTAs wind down together.
#include <algorithm>
#include <mutex>
#include <map>

#include "tc_filter.cuh"
#include "tc_ptx.cuh"

namespace annb {

namespace {

constexpr int kFiEpi = 16;
constexpr int kFiThreads = 32 * (kFiEpi + 3);
constexpr int kFiWarpA = kFiEpi + 2;     // the query-tile producer
constexpr int kFiCols = kBN / (kFiEpi / 4);  // columns of a tile per epilogue warp
constexpr int kFiMaxStages = 12, kFiMaxKt = 12;
constexpr size_t kFiSmemMax = 227 * 1024;
constexpr int kFiQueue = 64, kFiQueueBytes = kFiQueue * 9;  // survivors waiting per epilogue warp
constexpr size_t kFiFixed = 1024 /* alignment */ + 512 /* barriers */ + kFiEpi * kFiQueueBytes;
static_assert(kFiQueueBytes % 16 == 0, "the queues keep the factors 16-byte aligned");

struct FilterShape {
    int mt, nt, kt;     // query tiles, base tiles, k-blocks
    int nb;             // base tiles of a chunk
    int nst;            // ring stages
    int resident;       // the query tile stays in shared memory
    int a_box;          // query rows copied a tile: 128, or the batch rounded up to 8 when smaller
};

__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ uint32_t leader_addr(const void* p) {  // the pair's first CTA's copy of a shared address
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(su32(p)));
    return r;
}
template <int CG>
__device__ __forceinline__ void fi_tma(void* dst, const CUtensorMap* tm, int c0, int c1, uint32_t bar) {
    if (CG == 2)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
            "%3}], [%4];" ::"r"(su32(dst)),
            "l"(tm), "r"(c0), "r"(c1), "r"(bar)
            : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                su32(dst)),
            "l"(tm), "r"(c0), "r"(c1), "r"(bar)
            : "memory");
}
// Arrival on `bar` of every CTA of the tile once the MMAs issued so far are done.
template <int CG>
__device__ __forceinline__ void fi_commit_at(uint32_t bar) {
    if (CG == 2)
        asm volatile(
            "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
            "h"((uint16_t)3)
            : "memory");
    else
        mma_commit_at(bar);
}
template <int CG>
__device__ __forceinline__ void fi_commit(uint64_t* bar) {
    fi_commit_at<CG>(su32(bar));
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive;" ::: "memory");
    asm volatile("barrier.cluster.wait;" ::: "memory");
}

// The work of a cluster, in order: chunks of nb base tiles; in a chunk, items (query tile, base tile), query tile
// major, cut into equal runs, one a cluster. The clusters' places rotate from chunk to chunk so that the runs that
// are one item longer fall on different ones.
struct FilterWork {
    const FilterShape& s;
    int cl, ncl, chunk = 0, c0 = 0, tn = 0;
    int left = 0, r = 0;  // items left of the cluster's run in this chunk; base tile inside the chunk
    int m = 0, n = 0;     // the item's query tile and base tile
    bool first = false;   // the item starts a run of one query tile
    bool last = false;    // the item ends it
    __device__ FilterWork(const FilterShape& sh, int cluster, int nclusters) : s(sh), cl(cluster), ncl(nclusters) {}
    __device__ __forceinline__ bool next() {  // no division but at a chunk's start: every role steps per tile
        first = false;
        if (++r == tn) {
            r = 0;
            ++m;
            first = true;
        }
        while (left == 0) {
            if (chunk > 0) c0 += s.nb;
            if (c0 >= s.nt) return false;
            tn = min(s.nb, s.nt - c0);
            const int64_t total = (int64_t)s.mt * tn;
            const int place = (int)((cl + 29ll * chunk) % ncl);
            const int64_t lo = total * place / ncl;
            left = (int)(total * (place + 1) / ncl - lo);
            m = (int)(lo / tn);
            r = (int)(lo - (int64_t)m * tn);
            ++chunk;
            first = true;
        }
        --left;
        n = c0 + r;
        last = left == 0 || r == tn - 1;
        return true;
    }
};

// A ring position: stage and the parity of its current use.
struct RingPos {
    int s = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void step(int nst) {
        if (++s == nst) {
            s = 0;
            ph ^= 1u;
        }
    }
};

// SAMPLE: no bars and no survivors, the minima of 8 columns are written instead.
template <int KIND, int CG, bool SAMPLE>
__global__ void __launch_bounds__(kFiThreads, 1) tc_filter_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                 const __grid_constant__ CUtensorMap tmB,
                                                                 const TcFilterArgs a, const FilterShape sh) {
    constexpr int kBlockK = KindOf<KIND>::kBlockK, kMmaK = KindOf<KIND>::kMmaK;
    constexpr int kBRows = kBN / CG;
    constexpr int kBSize = kBRows * kRowBytes;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (su32(smem_raw) & 1023)) & 1023);
    const bool resident = sh.resident != 0;
    const int nst = sh.nst, kt = sh.kt;
    unsigned char* sA = smem;                                            // resident: kt blocks, else nst
    unsigned char* sB = sA + (size_t)(resident ? kt : nst) * kABytes;    // nst blocks
    uint64_t* full = reinterpret_cast<uint64_t*>(sB + (size_t)nst * kBSize);
    uint64_t* empty = full + kFiMaxStages;
    uint64_t* afull = empty + kFiMaxStages;
    uint64_t* aempty = afull + kFiMaxKt;
    uint64_t* tfull = aempty + 1;
    uint64_t* tempty = tfull + 2;
    uint64_t* done = tempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    unsigned char* sQueue = reinterpret_cast<unsigned char*>(full) + 512;                  // [warps][kFiQueueBytes]
    float* sFac = reinterpret_cast<float*>(sQueue + kFiEpi * kFiQueueBytes);               // [warps][2][kFiCols]

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp: known uniform
    const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0;  // clusters are pairs of consecutive CTAs
    const int k_last = (a.K - (kt - 1) * kBlockK) / kMmaK;  // MMAs of the last k-block

    if (threadIdx.x == 0) {
        for (int s = 0; s < nst; ++s) {
            bar_init(&full[s], 1);
            bar_init(&empty[s], 1);
        }
        for (int kb = 0; kb < kt && kb < kFiMaxKt; ++kb) bar_init(&afull[kb], 1);
        bar_init(aempty, 1);
        for (int b = 0; b < 2; ++b) {
            bar_init(&tfull[b], 1);
            bar_init(&tempty[b], CG * kFiEpi);
        }
        bar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tmem_slot)),
                         "r"(kTmemCols)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    if (CG == 2) cluster_sync();  // the pair's barriers exist before either CTA signals them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    FilterWork work(sh, (int)blockIdx.x / CG, (int)gridDim.x / CG);

    if (warp == 0) {
        if (lane == 0 && !a.test_no_loads) {  // base rows (and, when not resident, the query rows of the same k-block)
            RingPos pos;
            bool ok = true;
            const uint32_t a_bytes = (uint32_t)sh.a_box * kRowBytes;
            const uint32_t bytes = CG * (kBSize + (resident ? 0u : a_bytes));  // of both CTAs: one barrier counts them
            while (ok && work.next()) {
                const int arow = work.m * CG * kBM + rank * kBM;
                const int brow = work.n * kBN * (SAMPLE ? a.b_tile_stride : 1) + rank * kBRows;
                for (int kb = 0; kb < kt; ++kb, pos.step(nst)) {
                    const int s = pos.s;
                    if (!(ok = bar_wait(&empty[s], pos.ph ^ 1u, a.err, a.wait_ns))) break;
                    if (rank == 0) bar_expect(&full[s], bytes);
                    const uint32_t fb = CG == 2 ? leader_addr(&full[s]) : su32(&full[s]);
                    if (!resident) fi_tma<CG>(sA + (size_t)s * kABytes, &tmA, kb * kBlockK, arow, fb);
                    fi_tma<CG>(sB + (size_t)s * kBSize, &tmB, kb * kBlockK, brow, fb);
                }
            }
        }
    } else if (warp == kFiWarpA) {
        if (lane == 0 && resident && !a.test_no_loads) {  // the query tile of each run
            int run = 0;
            bool ok = true;
            while (ok && work.next()) {
                if (!work.first) continue;
                if (!(ok = bar_wait(aempty, (uint32_t)((run & 1) ^ 1), a.err, a.wait_ns))) break;
                for (int kb = 0; kb < kt; ++kb) {
                    if (rank == 0) bar_expect(&afull[kb], CG * (uint32_t)sh.a_box * kRowBytes);
                    const uint32_t fb = CG == 2 ? leader_addr(&afull[kb]) : su32(&afull[kb]);
                    fi_tma<CG>(sA + (size_t)kb * kABytes, &tmA, kb * kBlockK, work.m * CG * kBM + rank * kBM, fb);
                }
                ++run;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {  // MMA issuer
            // One thread issues 4 MMAs a k-block of 512 clocks between the epilogue warps of its scheduler, so its
            // instructions count: the warp runs the loop as one (uniform registers feed the MMAs), one elected lane
            // issues, and descriptors and barrier addresses are stepped, not made again. (Made again by a lone lane, a
            // k-block took 750 clocks and a tile 1,000 more, whatever the operand kind.)
            int acc = 0, run = -1;
            RingPos pos;
            bool ok = true;
            const bool leader = elect_one();
            const uint64_t da0 = sw128_desc(sA), db0 = sw128_desc(sB);
            const uint32_t full_a = su32(full), empty_a = su32(empty), afull_a = su32(afull), tempty_a = su32(tempty);
            constexpr int kMmas = kBlockK / kMmaK;
            while (ok && work.next()) {
                const int b = acc & 1;
                if (work.first) ++run;
                if (!(ok = bar_wait_warp(tempty_a + 8u * b, (uint32_t)(((acc >> 1) & 1) ^ 1), a.err, a.wait_ns))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (uint32_t)(b * kBN);
                const bool wait_a = resident && work.first;
                uint64_t da = da0;  // resident: steps with kb
                for (int kb = 0; kb < kt; ++kb) {
                    const uint32_t s = (uint32_t)pos.s;
                    if (wait_a && !(ok = bar_wait_warp(afull_a + 8u * kb, (uint32_t)(run & 1), a.err, a.wait_ns))) break;
                    if (!(ok = bar_wait_warp(full_a + 8u * s, pos.ph, a.err, a.wait_ns))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = resident ? da : da0 + s * (uint32_t)(kABytes >> 4);
                    const uint64_t bd = db0 + s * (uint32_t)(kBSize >> 4);
                    if (leader) {
                        if (kb + 1 < kt || k_last == kMmas) {
                            mma_issue<KIND, CG>(d, ad, bd, kb ? 1u : 0u);
#pragma unroll
                            for (int k = 1; k < kMmas; ++k) mma_issue<KIND, CG>(d, ad + 2u * k, bd + 2u * k, 1u);
                        } else {
                            for (int k = 0; k < k_last; ++k)
                                mma_issue<KIND, CG>(d, ad + 2u * k, bd + 2u * k, (kb | k) ? 1u : 0u);
                        }
                        fi_commit_at<CG>(empty_a + 8u * s);
                    }
                    __syncwarp();
                    da += (uint32_t)(kABytes >> 4);
                    pos.step(nst);
                }
                if (!ok) break;
                if (leader) {
                    if (resident && work.last) fi_commit<CG>(aempty);
                    fi_commit<CG>(&tfull[b]);
                }
                __syncwarp();
                ++acc;
            }
            if (leader) fi_commit<CG>(done);
            __syncwarp();
            if (!ok) let_copies_land();  // (a producer may have issued its last copies and left without a wait)
        }
        bar_wait_warp(su32(done), 0, nullptr, 0);  // every MMA issued has completed before TMEM is released
    } else {  // epilogue
        const int lane_base = 32 * (warp & 3), ew = warp - 2;
        const int col0 = kFiCols * (ew >> 2);
        float* sfx = sFac + ew * 2 * kFiCols;
        float* sfy = sfx + kFiCols;
        int acc = 0;
        float tau = 0.f, rfac = 1.f;
        // the warp's survivors wait in shared memory (key, column, lane of the row) until there are 32: then each
        // lane takes one to its row's buffer, the atomics' latency paid once for all. Slots past the capacity are
        // not stored.
        float* qk = reinterpret_cast<float*>(sQueue + ew * kFiQueueBytes);
        int* qc = reinterpret_cast<int*>(qk + kFiQueue);
        unsigned char* ql = reinterpret_cast<unsigned char*>(qc + kFiQueue);
        int nq = 0;    // uniform across the warp
        int row0 = 0;  // row of lane 0
        auto flush = [&](int cnt) {  // the last cnt <= 32 entries
            __syncwarp();
            nq -= cnt;
            if (lane < cnt) {
                const float key = qk[nq + lane];
                const int col = qc[nq + lane];
                const int row = row0 + ql[nq + lane];
                const int slot = atomicAdd(&a.rcount[row], 1);
                if (slot < a.cap) {
                    a.fkey[(int64_t)row * a.cap + slot] = key;
                    a.fcol[(int64_t)row * a.cap + slot] = col;
                }
            }
            __syncwarp();
        };
        while (work.next()) {
            const int b = (int)(acc & 1);
            if (work.first) {
                if (!SAMPLE) flush(nq);
                row0 = work.m * CG * kBM + rank * kBM + lane_base;
                const int rq = row0 + lane;
                const bool valid = rq < a.M;
                if (!SAMPLE) tau = valid ? a.tau[rq] : __int_as_float(0x7fffffff);  // NaN: no key passes
                if (KIND != kTcBF16) rfac = valid ? a.row_fac[rq] : 1.f;
            }
            const int n0 = work.n * kBN + col0;
            if (KIND != kTcBF16) {  // the factors of the warp's columns, zeros past N
                __syncwarp();  // every lane is done with the last tile's
#pragma unroll
                for (int i = 0; i < kFiCols / 32; ++i) {
                    const int c = n0 + 32 * i + lane;
                    const bool in = c < a.N;
                    const int64_t brow = SAMPLE ? (int64_t)work.n * kBN * a.b_tile_stride + (c - work.n * kBN) : c;
                    const float* src = reinterpret_cast<const float*>(a.col_fac + (in ? brow : 0));
                    cp_async4(sfx + 32 * i + lane, src, in);
                    cp_async4(sfy + 32 * i + lane, src + 1, in);
                }
            }
            const bool got = bar_wait(&tfull[b], (uint32_t)((acc >> 1) & 1), a.err, a.wait_ns);
            if (!__all_sync(0xffffffffu, got)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (KIND != kTcBF16) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
            }
            const uint32_t tb = tmem + ((uint32_t)lane_base << 16) + (uint32_t)(b * kBN + col0);
            // 32 columns a trip, and the rare path a loop, not unrolled: the code stays within the instruction
            // cache (with every column's survivor path inlined, warps waited for instructions 20 slots in 33)
#pragma unroll 1
            for (int h = 0; h < kFiCols; h += 32) {
                uint32_t r[32];
                __syncwarp();  // tcgen05.ld is .sync.aligned: the whole warp, converged
                tmem_ld32(tb + h, r);
                tmem_wait(r);
                if (h + 32 == kFiCols) {  // the warp's last load: the accumulator may be written again
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 2)
                            asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(
                                             leader_addr(&tempty[b]))
                                         : "memory");
                        else
                            bar_arrive(&tempty[b]);
                    }
                }
                if (!SAMPLE && n0 + h + 32 > a.N) {  // the ragged last tile: columns past N become NaN keys, which pass no bar
#pragma unroll
                    for (int u = 0; u < 32; ++u)
                        if (n0 + h + u >= a.N) r[u] = 0x7fffffffu;
                }
                float mins[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    float v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) v[u] = __uint_as_float(r[8 * g + u]);
                    if (KIND != kTcBF16) {  // key = f.y + f.x * (row factor * accumulator), two at a time
                        const float2 r2 = make_float2(rfac, rfac);
#pragma unroll
                        for (int u = 0; u < 8; u += 4) {
                            const float4 fx = *reinterpret_cast<const float4*>(sfx + h + 8 * g + u);
                            const float4 fy = *reinterpret_cast<const float4*>(sfy + h + 8 * g + u);
                            const float2 t0 = __fmul2_rn(r2, make_float2(v[u], v[u + 1]));
                            const float2 t1 = __fmul2_rn(r2, make_float2(v[u + 2], v[u + 3]));
                            const float2 k0 = __ffma2_rn(make_float2(fx.x, fx.y), t0, make_float2(fy.x, fy.y));
                            const float2 k1 = __ffma2_rn(make_float2(fx.z, fx.w), t1, make_float2(fy.z, fy.w));
                            v[u] = k0.x;
                            v[u + 1] = k0.y;
                            v[u + 2] = k1.x;
                            v[u + 3] = k1.y;
                        }
                    }
                    const float mn = min3f(min3f(v[0], v[1], v[2]), min3f(v[3], v[4], v[5]), fminf(v[6], v[7]));
                    if (SAMPLE) {
                        mins[g] = mn;
                        continue;
                    }
                    if (!__any_sync(0xffffffffu, mn <= tau)) continue;
                    uint32_t mask = 0;  // the lane's survivors of the 8
#pragma unroll
                    for (int u = 0; u < 8; ++u) mask |= v[u] <= tau ? 1u << u : 0u;
#pragma unroll 1
                    while (true) {  // one survivor a lane each trip
                        const unsigned hit = __ballot_sync(0xffffffffu, mask != 0u);
                        if (hit == 0u) break;
                        if (mask) {
                            const int u = __ffs(mask) - 1;
                            mask &= mask - 1;
                            float s4[4], s2[2];  // v[u] for a run-time u
#pragma unroll
                            for (int z = 0; z < 4; ++z) s4[z] = (u & 4) ? v[z + 4] : v[z];
#pragma unroll
                            for (int z = 0; z < 2; ++z) s2[z] = (u & 2) ? s4[z + 2] : s4[z];
                            const int at = nq + __popc(hit & ((1u << lane) - 1u));
                            qk[at] = (u & 1) ? s2[1] : s2[0];
                            qc[at] = n0 + h + 8 * g + u;
                            ql[at] = (unsigned char)lane;
                        }
                        nq += __popc(hit);
                        if (nq >= 32) flush(32);
                    }
                }
                if (SAMPLE && row0 + lane < a.M)
                    *reinterpret_cast<float4*>(a.out_min + (int64_t)(row0 + lane) * (a.N / 8) + (n0 + h) / 8) =
                        make_float4(mins[0], mins[1], mins[2], mins[3]);
            }
            ++acc;
        }
        if (!SAMPLE) flush(nq);
        if (KIND != kTcBF16) asm volatile("cp.async.wait_all;" ::: "memory");  // (left over where a wait gave up)
    }
    __syncthreads();
    if (CG == 2) cluster_sync();  // neither CTA's barriers or accumulators are in use any more
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 2)
            asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        else
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
    if (CG == 2) cluster_sync();
}

// Clusters of a kernel that are resident at once, asked once per (kernel, device, shared memory).
int resident_clusters(const void* kern, int cg, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, size_t>, int> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return kNumSMs / cg;
    std::lock_guard<std::mutex> lk(mu);
    int& n = known[{kern, dev, smem}];
    if (n == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kNumSMs);
        cfg.blockDim = dim3(kFiThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = cg;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = kNumSMs / cg;
        }
    }
    return n;
}

template <int KIND, int CG, bool SAMPLE>
int run_filter(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st) {
    CUtensorMap tmA, tmB;
    FilterShape sh{};
    // Rows past the batch are not copied (their products, of whatever the shared memory holds, meet NaN bars): a box that
    // is mostly zero fill takes longer than the rows it holds (one query over 1M x 384: 152 us, 117 us for 128 queries).
    sh.a_box = CG == 1 ? (int)std::min<int64_t>(kBM, ceil_div(a.M, 8) * 8) : kBM;
    int rc = tc_make_map(&tmA, A, a.M, a.K, sh.a_box, KIND);
    if (rc) return rc;
    if ((rc = tc_make_map(&tmB, B, SAMPLE ? a.b_rows : a.N, a.K, kBN / CG, KIND))) return rc;
    sh.mt = (int)ceil_div(a.M, CG * kBM);
    sh.nt = (int)ceil_div(a.N, kBN);
    sh.kt = (int)ceil_div(a.K, KindOf<KIND>::kBlockK);
    const size_t fac = KIND == kTcBF16 ? 0 : (size_t)kFiEpi * 2 * kFiCols * 4;
    const size_t room = kFiSmemMax - kFiFixed - fac, bs = (size_t)kBN / CG * kRowBytes;
    // the query tile stays where at least three (32 KB) or four (16 KB) ring stages fit beside it
    sh.resident = sh.kt <= kFiMaxKt && (size_t)sh.kt * kABytes + (CG == 1 ? 3 : 4) * bs <= room;
    const size_t left = sh.resident ? room - (size_t)sh.kt * kABytes : room;
    sh.nst = (int)std::min<size_t>(kFiMaxStages, left / (bs + (sh.resident ? 0 : kABytes)));
    const size_t smem = kFiFixed + fac + (size_t)sh.nst * (bs + (sh.resident ? 0 : kABytes)) +
                        (sh.resident ? (size_t)sh.kt * kABytes : 0);
    auto kern = tc_filter_kernel<KIND, CG, SAMPLE>;
    ANN_CUDA_TRY(smem_optin(reinterpret_cast<const void*>(kern)));
    const int64_t tiles = (int64_t)sh.mt * sh.nt;
    const int ncl = (int)std::min<int64_t>(tiles, resident_clusters(reinterpret_cast<const void*>(kern), CG, smem));
    // chunks of about 24 MB of base rows (L2 holds several), longer where a run would hold fewer than 16 tiles, up
    // to 64 MB; one query tile: no chunks
    const int64_t tile_bytes = (int64_t)kBN * a.K * (KIND == kTcBF16 ? 2 : 1);
    int64_t nb = std::max<int64_t>(((int64_t)24 << 20) / tile_bytes, ceil_div(16 * (int64_t)ncl, sh.mt));
    nb = std::max<int64_t>(1, std::min(nb, ((int64_t)64 << 20) / tile_bytes));
    sh.nb = sh.mt == 1 ? sh.nt : (int)std::min<int64_t>(nb, sh.nt);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ncl * CG);
    cfg.blockDim = dim3(kFiThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = CG;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ANN_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmA, tmB, a, sh));
    ANN_LAUNCH_CHECK();
    return ANN_OK;
}

}  // namespace

static int check_filter(const void* A, const void* B, const TcFilterArgs& a) {
    const int step = a.kind == kTcBF16 ? 16 : 32;
    ANN_CHECK_ARG(a.kind == kTcBF16 || a.kind == kTcE4M3, "tensor-core filter: element kind %d", a.kind);
    ANN_CHECK_ARG(a.K % step == 0 && a.K > 0, "tensor-core filter: K=%d not a positive multiple of %d", a.K, step);
    ANN_CHECK_ARG(a.kind == kTcBF16 || (a.col_fac && a.row_fac), "tensor-core filter: E4M3 operands need their factors");
    ANN_CHECK_ARG((reinterpret_cast<uintptr_t>(A) & 15) == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0,
                  "tensor-core filter: operands must be 16-byte aligned");
    return ANN_OK;
}

// one CTA a tile up to 128 queries: the base is read once either way, and a pair would multiply padding
template <bool SAMPLE>
static int dispatch_filter(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st) {
    if (a.M == 0 || a.N == 0) return ANN_OK;
    if (a.kind == kTcBF16)
        return a.M <= kBM ? run_filter<kTcBF16, 1, SAMPLE>(A, B, a, st) : run_filter<kTcBF16, 2, SAMPLE>(A, B, a, st);
    return a.M <= kBM ? run_filter<kTcE4M3, 1, SAMPLE>(A, B, a, st) : run_filter<kTcE4M3, 2, SAMPLE>(A, B, a, st);
}

int launch_tc_filter(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st) {
    const int rc = check_filter(A, B, a);
    if (rc) return rc;
    ANN_CHECK_ARG(a.tau && a.fkey && a.fcol && a.rcount && a.cap > 0, "tensor-core filter: no buffers");
    return dispatch_filter<false>(A, B, a, st);
}

int launch_tc_sample(const void* A, const void* B, const TcFilterArgs& a, cudaStream_t st) {
    const int rc = check_filter(A, B, a);
    if (rc) return rc;
    ANN_CHECK_ARG(a.out_min && a.N % kBN == 0 && a.b_tile_stride >= 1 &&
                      ((int64_t)a.N / kBN - 1) * kBN * a.b_tile_stride + kBN <= a.b_rows,
                  "tensor-core sample: %d columns, stride %d", a.N, a.b_tile_stride);
    return dispatch_filter<true>(A, B, a, st);
}

}  // namespace annb
