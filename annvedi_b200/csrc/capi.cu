// C ABI: error state, workspaces and the flat (linear) index.
//
// The flat index mirrors linear_ann_cpp.LinearIndex (competitors/linear/src/linear_index.cpp:
// 62-131): fit copies the base into memory the index owns (linear_index.cpp:82 copies into a
// std::vector; here the copy lands in HBM as zero-padded rows), query returns int64 ids and adds
// n to the cumulative distance counter per query (linear_index.cpp:108, 123).
#include <cmath>
#include <cstdarg>
#include <cstring>
#include <algorithm>
#include <atomic>
#include <optional>
#include <vector>

#include "block_select.cuh"
#include "common.cuh"
#include "compat.cuh"
#include "flat_scan.cuh"
#include "runtime.cuh"
#include "flat_internal.cuh"
#include "ivf.cuh"
#include "tc_filter.cuh"
#include "tc_gemm.cuh"
#include "tc_search.cuh"
#include "radix_select.cuh"

namespace annb {

static thread_local char g_err[1024] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}
void clear_error() { g_err[0] = 0; }

int queries_in(float* dev, int64_t dpad, const float* host, int64_t ld, int64_t rows, int cols, cudaStream_t st) {
    if (rows == 0) return ANN_OK;
    ANN_CUDA_TRY(cudaMemcpy2DAsync(dev, sizeof(float) * dpad, host, sizeof(float) * ld, sizeof(float) * cols, rows,
                                   cudaMemcpyHostToDevice, st));
    if (dpad > cols)
        ANN_CUDA_TRY(cudaMemset2DAsync(dev + cols, sizeof(float) * dpad, 0, sizeof(float) * (dpad - cols), rows, st));
    return ANN_OK;
}

static std::atomic<int64_t> g_launches{0};
void count_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

int ws_reserve_device(ann_workspace* ws, size_t bytes) {
    std::lock_guard<std::mutex> lk(ws->mu);
    if (ws->dev_cap >= bytes) return ANN_OK;
    size_t cap = std::max(bytes, ws->dev_cap + ws->dev_cap / 2);
    if (ws->dev) {
        ANN_CUDA_TRY(cudaDeviceSynchronize());
        ANN_CUDA_TRY(cudaFree(ws->dev));
        ws->dev = nullptr;
        ws->dev_cap = 0;
    }
    cudaError_t e = cudaMalloc(&ws->dev, cap);
    if (e != cudaSuccess) {
        cudaGetLastError();
        e = cudaMalloc(&ws->dev, bytes);
        cap = bytes;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        ws->dev = nullptr;
        set_error("workspace: cannot allocate %zu bytes of device scratch (%s)", bytes, cudaGetErrorString(e));
        return ANN_ERR_NOMEM;
    }
    ws->dev_cap = cap;
    return ANN_OK;
}

int ws_pinned(ann_workspace* ws, int64_t** out) {
    std::lock_guard<std::mutex> lk(ws->mu);
    if (!ws->pinned) {
        void* p = nullptr;
        const cudaError_t e = cudaHostAlloc(&p, 8 * sizeof(int64_t), cudaHostAllocDefault);
        if (e != cudaSuccess) {
            cudaGetLastError();
            set_error("workspace: cannot allocate page-locked host words (%s)", cudaGetErrorString(e));
            return ANN_ERR_NOMEM;
        }
        ws->pinned = static_cast<int64_t*>(p);
    }
    *out = ws->pinned;
    return ANN_OK;
}

int ws_reserve_big(ann_workspace* ws, size_t bytes) {
    std::lock_guard<std::mutex> lk(ws->mu);
    if (ws->big_cap >= bytes) return ANN_OK;
    size_t cap = std::max(bytes, ws->big_cap + ws->big_cap / 4);
    if (ws->big) {
        ANN_CUDA_TRY(cudaDeviceSynchronize());
        ANN_CUDA_TRY(cudaFree(ws->big));
        ws->big = nullptr;
        ws->big_cap = 0;
    }
    cudaError_t e = cudaMalloc(&ws->big, cap);
    if (e != cudaSuccess) {
        cudaGetLastError();
        e = cudaMalloc(&ws->big, bytes);
        cap = bytes;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        ws->big = nullptr;
        set_error("workspace: cannot allocate %zu bytes of device scratch (%s)", bytes, cudaGetErrorString(e));
        return ANN_ERR_NOMEM;
    }
    ws->big_cap = cap;
    return ANN_OK;
}

}  // namespace annb

using namespace annb;


// An empty kernel compiled with the library's flags: its attributes are the library's code form.
__global__ void arch_probe_kernel() {}

extern "C" {

const char* ann_version(void) { return "annvedi_b200 0.1 sm_100a"; }

int ann_tc_wait_selftest(int device, int64_t wait_ns, int32_t* flag_out) {
    clear_error();
    ANN_CHECK_ARG(flag_out != nullptr, "ann_tc_wait_selftest: flag_out is NULL");
    ANN_CHECK_ARG(wait_ns >= 1000 && wait_ns <= 2000000000LL, "ann_tc_wait_selftest: wait_ns=%lld outside [1e3, 2e9]",
                  (long long)wait_ns);
    DeviceGuard g(device);
    if (!g.ok) {
        cudaGetLastError();
        set_error("ann_tc_wait_selftest: device %d not usable", device);
        return ANN_ERR_CUDA;
    }
    int flag = -1;
    const int rc = tc_wait_selftest((uint64_t)wait_ns, &flag);
    *flag_out = flag;
    return rc;
}

int ann_kernel_arch(int device, int32_t* out2) {
    clear_error();
    ANN_CHECK_ARG(out2 != nullptr, "ann_kernel_arch: out2 is NULL");
    DeviceGuard g(device);
    if (!g.ok) {
        cudaGetLastError();
        set_error("ann_kernel_arch: device %d not usable", device);
        return ANN_ERR_CUDA;
    }
    cudaFuncAttributes fa{};
    ANN_CUDA_TRY(cudaFuncGetAttributes(&fa, arch_probe_kernel));
    out2[0] = fa.binaryVersion;
    out2[1] = fa.ptxVersion;
    return ANN_OK;
}
const char* ann_last_error(void) { return g_err; }
int64_t ann_kernel_launches(void) { return g_launches.load(); }

int ann_workspace_create(ann_workspace** out, int device) {
    ANN_CHECK_ARG(out != nullptr, "ann_workspace_create: out is NULL");
    ann_workspace* ws = new (std::nothrow) ann_workspace();
    if (!ws) {
        set_error("ann_workspace_create: out of host memory");
        return ANN_ERR_NOMEM;
    }
    ws->device = device;
    *out = ws;
    return ANN_OK;
}

static void ws_release(ann_workspace* ws) {
    DeviceGuard g(ws->device);
    if (ws->dev) cudaFree(ws->dev);
    if (ws->big) cudaFree(ws->big);
    if (ws->pinned) cudaFreeHost(ws->pinned);
    ws->pinned = nullptr;
    ws->dev = nullptr;
    ws->big = nullptr;
    ws->dev_cap = ws->big_cap = 0;
}

int ann_workspace_destroy(ann_workspace* ws) {
    if (!ws) return ANN_OK;
    ws_release(ws);
    delete ws;
    return ANN_OK;
}

int64_t ann_workspace_bytes(const ann_workspace* ws) { return ws ? (int64_t)(ws->dev_cap + ws->big_cap) : 0; }

int ann_flat_create(ann_flat** out, int device) {
    clear_error();
    ANN_CHECK_ARG(out != nullptr, "ann_flat_create: out is NULL");
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device visible (%s)", e == cudaSuccess ? "0 devices" : cudaGetErrorString(e));
        return ANN_ERR_CUDA;
    }
    ANN_CHECK_ARG(device >= 0 && device < ndev, "ann_flat_create: device %d not in [0, %d)", device, ndev);
    ann_flat* h = new (std::nothrow) ann_flat();
    if (!h) {
        set_error("ann_flat_create: out of host memory");
        return ANN_ERR_NOMEM;
    }
    h->device = device;
    h->ws.device = device;
    *out = h;
    return ANN_OK;
}

int ann_flat_destroy(ann_flat* h) {
    if (!h) return ANN_OK;
    {
        DeviceGuard g(h->device);
        if (h->base) cudaFree(h->base);
        if (h->base_bf16) cudaFree(h->base_bf16);
        if (h->base_e4m3) cudaFree(h->base_e4m3);
        if (h->fac_e4m3) cudaFree(h->fac_e4m3);
        if (h->d_err) cudaFree(h->d_err);
        if (h->prune_word) cudaFreeHost(h->prune_word);  // (the frees above have waited for the device)
    }
    ws_release(&h->ws);
    delete h;
    return ANN_OK;
}

int ann_flat_fit(ann_flat* h, const float* data, int64_t n, int32_t dim, int64_t ld, int32_t metric, int32_t mem,
                 void* stream) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr, "ann_flat_fit: null index");
    ANN_CHECK_ARG(n >= 1 && dim >= 1, "ann_flat_fit: need a non-empty 2-D array, got [%lld, %d]", (long long)n, dim);
    ANN_CHECK_ARG(n < INT32_MAX, "ann_flat_fit: n=%lld exceeds 32-bit ids", (long long)n);
    ANN_CHECK_ARG(ld >= dim, "ann_flat_fit: row stride %lld < dim %d", (long long)ld, dim);
    ANN_CHECK_ARG(metric == ANN_METRIC_L2 || metric == ANN_METRIC_IP, "ann_flat_fit: unknown metric %d", metric);
    ANN_CHECK_ARG(data != nullptr, "ann_flat_fit: data is NULL");
    DeviceGuard g(h->device);
    cudaStream_t st = as_stream(stream);
    const int dpad = (int)ceil_div(dim, 32) * 32;
    if (h->base) {
        ANN_CUDA_TRY(cudaDeviceSynchronize());
        ANN_CUDA_TRY(cudaFree(h->base));
        h->base = nullptr;
    }
    if (h->base_bf16) {
        ANN_CUDA_TRY(cudaFree(h->base_bf16));
        h->base_bf16 = nullptr;
    }
    if (h->base_e4m3) {
        ANN_CUDA_TRY(cudaFree(h->base_e4m3));
        ANN_CUDA_TRY(cudaFree(h->fac_e4m3));
        h->base_e4m3 = nullptr;
        h->fac_e4m3 = nullptr;
    }
    h->bounds_known = false;
    h->prune_credit_us = 0.0;
    h->prune_refused = false;
    h->prune_ws_refused = SIZE_MAX;
    h->prune_streak = h->prune_skip = 0;
    if (h->prune_word) {  // (the old base's passes are done: their end is not read)
        h->prune_seen = (uint32_t)(h->prune_word[0] >> 32);
        h->prune_word[1] = 0;
    }
    const size_t bytes = sizeof(float) * (size_t)n * dpad;
    cudaError_t e = cudaMalloc(&h->base, bytes);
    if (e != cudaSuccess) {
        cudaGetLastError();
        h->base = nullptr;
        h->n = 0;
        set_error("ann_flat_fit: cannot allocate %zu bytes for the base (%s)", bytes, cudaGetErrorString(e));
        return ANN_ERR_NOMEM;
    }
    if (dpad != dim) ANN_CUDA_TRY(cudaMemsetAsync(h->base, 0, bytes, st));
    ANN_CUDA_TRY(cudaMemcpy2DAsync(h->base, sizeof(float) * dpad, data, sizeof(float) * ld, sizeof(float) * dim, n,
                                   mem == ANN_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice, st));
    if (mem == ANN_MEM_HOST) ANN_CUDA_TRY(cudaStreamSynchronize(st));
    h->n = n;
    h->dim = dim;
    h->dpad = dpad;
    h->metric = metric;
    return ANN_OK;
}

}  // extern "C"

// Number of row splits for an exact scan of n rows by nq queries in tiles of bq.
int annb::flat_choose_nsplit(int64_t n, int nq, int bq, int64_t* rows_per_split, int ctas_per_sm) {
    // Choose the splits per query tile so that (query tiles x splits) fills whole waves of
    // kNumSMs * ctas_per_sm CTAs, with a small charge per split for the merge.
    const int64_t wave = (int64_t)kNumSMs * std::max(1, ctas_per_sm);
    const int64_t n_qtiles = ceil_div(nq, bq);
    const int64_t tile = 256;
    const int64_t max_split = std::max<int64_t>(1, std::min<int64_t>(ceil_div(n, 2 * tile), 4 * wave));
    int64_t best_s = 1;
    double best = 1e300;
    for (int64_t s = 1; s <= max_split; ++s) {
        const int64_t ctas = n_qtiles * s;
        const int64_t waves = ceil_div(ctas, wave);
        const double cost = (double)waves * wave / (double)ctas * (1.0 + 0.002 * (double)s);
        if (cost < best - 1e-12) {
            best = cost;
            best_s = s;
        }
    }
    int64_t rps = ceil_div(ceil_div(n, best_s), tile) * tile;
    const int64_t nsplit = ceil_div(n, rps);
    *rows_per_split = rps;
    return (int)nsplit;
}

extern "C" {

static int flat_exact_pruned(ann_flat* h, ann_workspace* ws, const float* qdev, int nq, int kk, int64_t* ids_dev,
                             float* dists_dev, cudaStream_t st, bool* done);

int ann_flat_query(ann_flat* h, ann_workspace* ws, const float* queries, int32_t nq, int64_t ldq, int32_t k,
                   int32_t mode, int32_t mem, int64_t* out_ids, float* out_dists, void* stream) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr, "ann_flat_query: null index");
    if (h->base == nullptr || h->n == 0) {
        set_error("index not fitted");
        return ANN_ERR_STATE;
    }
    ANN_CHECK_ARG(nq >= 0, "ann_flat_query: nq=%d < 0", nq);
    ANN_CHECK_ARG(k >= 1, "ann_flat_query: k=%d < 1", k);
    ANN_CHECK_ARG(ldq >= h->dim, "ann_flat_query: query stride %lld < dim %d", (long long)ldq, h->dim);
    ANN_CHECK_ARG(mode == ANN_MODE_EXACT || mode == ANN_MODE_REFERENCE, "ann_flat_query: unknown mode %d", mode);
    ANN_CHECK_ARG(mode == ANN_MODE_EXACT || h->metric == ANN_METRIC_L2,
                  "ann_flat_query: the reference ranking is defined for squared L2 only");
    ANN_CHECK_ARG(nq == 0 || (queries != nullptr && out_ids != nullptr), "ann_flat_query: null pointer");
    if (nq == 0) return ANN_OK;
    const int kk = (int)std::min<int64_t>(k, h->n);
    if (kk > 512) {
        set_error("ann_flat_query: k=%d > 512 is not supported by the fused selection", kk);
        return ANN_ERR_UNSUPPORTED;
    }
    if (!ws) ws = &h->ws;
    DeviceGuard g(h->device);
    cudaStream_t st = as_stream(stream);
    const int dpad = h->dpad;
    const bool host = mem == ANN_MEM_HOST;
    const bool need_pad = host || (mode == ANN_MODE_EXACT && (ldq != dpad || (reinterpret_cast<uintptr_t>(queries) & 15)));

    // ---- plan the scratch: [padded queries][device outputs][search scratch] ----
    int bq = 0, nsplit = 0, qc = 0, ncp = 0, nseg = 0;
    int64_t rps = 0;
    Sizer sz;
    if (need_pad) sz.take<float>((size_t)nq * dpad);
    if (host) {
        sz.take<int64_t>((size_t)nq * kk);
        sz.take<float>((size_t)nq * kk);
    }
    bool radix_merge = false;
    if (mode == ANN_MODE_EXACT) {
        bq = std::min(h->query_tile > 0 ? h->query_tile : flat_scan_bq(nq), flat_scan_max_bq(kk));
        nsplit = flat_choose_nsplit(h->n, nq, bq, &rps, flat_scan_ctas_per_sm(bq, kk, dpad, h->metric));
        sz.take<float>((size_t)nq * nsplit * kk);
        sz.take<int>((size_t)nq * nsplit * kk);
        sz.take<float>((size_t)(nq + 1) / 2 * 2 * dpad);  // the paired query tile
        // many splits per query: select the k best with the radix selection, then sort them
        radix_merge = nsplit >= 16;
        if (radix_merge) {
            sz.take<float>((size_t)nq * kk);
            sz.take<int>((size_t)nq * kk);
        }
    } else {
        ncp = compat_num_checkpoints(h->dim);
        nseg = (int)ceil_div(h->n, select_seg_rows(h->n));
        const size_t per_q = sizeof(float) * (size_t)h->n * (ncp + 2) + (size_t)nseg * (64 * 4 + (size_t)kk * 8);
        const size_t budget = (size_t)1 << 30;
        qc = (int)std::min<size_t>(32768, std::max<size_t>(1, std::min<size_t>((size_t)nq, budget / per_q)));
        sz.take<float>((size_t)qc * h->n);
        sz.take<float>((size_t)qc * h->n * ncp);
        sz.take<float>((size_t)qc * h->n);
        sz.take<float>((size_t)qc * nseg * 64);
        sz.take<unsigned long long>((size_t)qc * nseg * kk);
    }
    int rc = ws_reserve_device(ws, sz.bytes());
    if (rc) return rc;
    Carver cv(ws->dev);
    float* qdev = const_cast<float*>(queries);
    int64_t ldq_dev = ldq;
    if (need_pad) {
        qdev = cv.take<float>((size_t)nq * dpad);
        ldq_dev = dpad;
    }
    int64_t* ids_dev = out_ids;
    float* dists_dev = out_dists;
    if (host) {
        ids_dev = cv.take<int64_t>((size_t)nq * kk);
        dists_dev = cv.take<float>((size_t)nq * kk);
    }

    // ---- queries in ----
    if (host) {
        if ((rc = queries_in(qdev, dpad, queries, ldq, nq, h->dim, st))) return rc;
    } else if (need_pad) {
        rc = launch_pad_rows(queries, nq, h->dim, ldq, qdev, dpad, st);
        if (rc) return rc;
    }

    // ---- search ----
    const int prec = h->prof.begin(st);
    bool pruned = false;
    if (mode == ANN_MODE_EXACT && h->prune) {
        if ((rc = flat_exact_pruned(h, ws, qdev, nq, kk, ids_dev, dists_dev, st, &pruned))) return rc;
    }
    if (pruned) {
        h->prof.mark(prec, st);
        if (prec >= 0) h->prof.launches += 1;
    } else if (mode == ANN_MODE_EXACT) {
        float* skey = cv.take<float>((size_t)nq * nsplit * kk);
        int* sid = cv.take<int>((size_t)nq * nsplit * kk);
        float* qpair = cv.take<float>((size_t)(nq + 1) / 2 * 2 * dpad);
        FlatScanArgs a{h->base, h->n, dpad, qdev, nq, h->metric, kk, rps, nsplit, skey, sid};
        a.qpair = qpair;
        rc = launch_flat_scan(a, bq, st);
        if (rc) return rc;
        h->prof.mark(prec, st);
        if (radix_merge) {
            float* mkey = cv.take<float>((size_t)nq * kk);
            int* mid = cv.take<int>((size_t)nq * kk);
            RadixSelectArgs rs{};
            rs.keys = skey;
            rs.ld = (int64_t)nsplit * kk;
            rs.ids = sid;
            rs.R = kk;
            rs.out_key = mkey;
            rs.out_id = mid;
            if ((rc = launch_radix_select(rs, nq, st))) return rc;
            rc = launch_sort_topk(mkey, mid, nq, kk, h->metric == ANN_METRIC_IP ? 1 : 0, ids_dev, dists_dev, st);
        } else {
            MergeArgs m{skey, sid, nq, nsplit, kk, kk, h->metric == ANN_METRIC_IP ? 1 : 0, ids_dev, dists_dev};
            rc = launch_merge_splits(m, st);
        }
        if (rc) return rc;
        h->prof.mark(prec, st);
        if (prec >= 0) h->prof.launches += 1;
    } else {
        CompatArgs a{};
        a.base = h->base;
        a.n = h->n;
        a.dim = h->dim;
        a.ldb = dpad;
        a.q = qdev;
        a.ldq = ldq_dev;
        a.k = kk;
        a.ncp = ncp;
        a.D = cv.take<float>((size_t)qc * h->n);
        a.P = cv.take<float>((size_t)qc * h->n * ncp);
        a.T = cv.take<float>((size_t)qc * h->n);
        a.seg_heap = cv.take<float>((size_t)qc * nseg * 64);
        a.seg_best = cv.take<unsigned long long>((size_t)qc * nseg * kk);
        a.out_ids = ids_dev;
        a.out_dists = dists_dev;
        for (int q0 = 0; q0 < nq; q0 += qc) {
            rc = launch_compat(a, q0, std::min(qc, nq - q0), st);
            if (rc) return rc;
        }
    }
    h->ndist.fetch_add(h->n * (int64_t)nq);

    // ---- results out ----
    if (host) {
        ANN_CUDA_TRY(cudaMemcpyAsync(out_ids, ids_dev, sizeof(int64_t) * (size_t)nq * kk, cudaMemcpyDeviceToHost, st));
        if (out_dists)
            ANN_CUDA_TRY(cudaMemcpyAsync(out_dists, dists_dev, sizeof(float) * (size_t)nq * kk, cudaMemcpyDeviceToHost, st));
        ANN_CUDA_TRY(cudaStreamSynchronize(st));
    }
    return ANN_OK;
}

int ann_flat_set_profiling(ann_flat* h, int32_t enable) {
    ANN_CHECK_ARG(h != nullptr, "null index");
    h->prof.enabled = enable != 0;
    return ANN_OK;
}

int ann_flat_profile(ann_flat* h, double* out4) {
    ANN_CHECK_ARG(h != nullptr && out4 != nullptr, "null argument");
    DeviceGuard g(h->device);
    h->prof.collect();
    out4[0] = h->prof.total_ms[0];
    out4[1] = h->prof.total_ms[1];
    out4[2] = (double)h->prof.launches;
    out4[3] = (double)h->prof.calls;
    return ANN_OK;
}

int ann_flat_profile_stages(ann_flat* h, double* out10) {
    ANN_CHECK_ARG(h != nullptr && out10 != nullptr, "null argument");
    DeviceGuard g(h->device);
    h->prof.collect();
    for (int i = 0; i < 6; ++i) out10[i] = h->prof.total_ms[i];
    out10[6] = (double)h->prof.launches;
    out10[7] = (double)h->prof.tc_launches;
    out10[8] = (double)h->prof.filter_launches;
    out10[9] = (double)h->prof.calls;
    return ANN_OK;
}

int ann_flat_reset_profile(ann_flat* h) {
    ANN_CHECK_ARG(h != nullptr, "null index");
    DeviceGuard g(h->device);
    h->prof.reset();
    return ANN_OK;
}

// BF16 operand form of the base for the tensor-core scan (key columns included, rows in the Weyl
// order of tc_row_mult), built once.
static int flat_ensure_bf16(ann_flat* h, cudaStream_t st) {
    if (h->base_bf16) return ANN_OK;
    const int kpad = tc_kpad(h->dim, h->metric);
    __nv_bfloat16* b = nullptr;
    int* err = nullptr;
    cudaError_t e = cudaMalloc(&b, sizeof(__nv_bfloat16) * (size_t)h->n * kpad);
    if (e == cudaSuccess && !h->d_err) e = cudaMalloc(&err, sizeof(int));
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (b) cudaFree(b);
        if (err) cudaFree(err);
        set_error("tensor-core scan: cannot allocate the BF16 copy of the base (%s)", cudaGetErrorString(e));
        return ANN_ERR_NOMEM;
    }
    if (err) {
        ANN_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), st));
        h->d_err = err;
    }
    const int64_t mult = tc_row_mult(h->n);
    int rc = launch_tc_operand(h->base, h->n, h->dim, h->dpad, b, kpad, kTcBase, h->metric, mult, st);
    if (rc) {
        cudaFree(b);
        return rc;
    }
    ANN_CUDA_TRY(cudaStreamSynchronize(st));
    h->base_bf16 = b;
    h->row_mult = mult;
    h->kpad = kpad;
    return ANN_OK;
}

// E4M3 operand form of the base (per-row scales, same Weyl order), built once.
static int flat_ensure_e4m3(ann_flat* h, cudaStream_t st) {
    if (h->base_e4m3) return ANN_OK;
    int rc = flat_ensure_bf16(h, st);  // the row order and the error flag
    if (rc) return rc;
    const int kpad8 = (int)ceil_div(h->dim, 32) * 32;
    uint8_t* b = nullptr;
    float2* f = nullptr;
    cudaError_t e = cudaMalloc(&b, (size_t)h->n * kpad8);
    if (e == cudaSuccess) e = cudaMalloc(&f, sizeof(float2) * (size_t)h->n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        if (b) cudaFree(b);
        set_error("tensor-core scan: cannot allocate the E4M3 copy of the base (%s)", cudaGetErrorString(e));
        return ANN_ERR_NOMEM;
    }
    rc = launch_tc_operand_e4m3(h->base, h->n, h->dim, h->dpad, b, kpad8, kTcBase, h->metric, h->row_mult, nullptr, f,
                                st);
    if (rc) {
        cudaFree(b);
        cudaFree(f);
        return rc;
    }
    ANN_CUDA_TRY(cudaStreamSynchronize(st));
    h->base_e4m3 = b;
    h->fac_e4m3 = f;
    h->kpad8 = kpad8;
    return ANN_OK;
}

// The tensor-core operands of the index's current element kind.
struct FlatTc {
    int kind, kpad;
    size_t es;  // bytes per element
    const void* base;
    const float2* cfac;
};
static int flat_ensure_tc(ann_flat* h, cudaStream_t st, FlatTc* t) {
    std::lock_guard<std::mutex> lk(h->tc_mu);
    int rc = h->tc_kind == kTcE4M3 ? flat_ensure_e4m3(h, st) : flat_ensure_bf16(h, st);
    if (rc) return rc;
    t->kind = h->tc_kind;
    t->kpad = t->kind == kTcE4M3 ? h->kpad8 : h->kpad;
    t->es = t->kind == kTcE4M3 ? 1 : 2;
    t->base = t->kind == kTcE4M3 ? (const void*)h->base_e4m3 : (const void*)h->base_bf16;
    t->cfac = t->kind == kTcE4M3 ? h->fac_e4m3 : nullptr;
    return ANN_OK;
}
// Queries to the operand form: E4M3 rows with their scales into rfac, or BF16 rows.
static int flat_tc_queries(const ann_flat* h, const FlatTc& t, const float* q, int nq, int64_t ldq, void* out,
                           float* rfac, cudaStream_t st) {
    if (t.kind == kTcE4M3)
        return launch_tc_operand_e4m3(q, nq, h->dim, ldq, static_cast<uint8_t*>(out), t.kpad, kTcQuery, h->metric, 0,
                                      rfac, nullptr, st);
    return launch_tc_operand(q, nq, h->dim, ldq, static_cast<__nv_bfloat16*>(out), t.kpad, kTcQuery, h->metric, 0, st);
}

static int flat_check_err(ann_flat* h) {
    int v = 0;
    if (!h->d_err) return ANN_OK;
    ANN_CUDA_TRY(cudaMemcpy(&v, h->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (v) {
        ANN_CUDA_TRY(cudaMemset(h->d_err, 0, sizeof(int)));
        set_error("a device-side wait gave up after its time limit; the results are invalid");
        return ANN_ERR_TIMEOUT;
    }
    return ANN_OK;
}

// The BF16 copy and its keys' bounds for the pruned exact scan. Laying them out costs about 0.5 ms + 3.1e-6 us an
// element (1.7 ms at 1M x 384), a pruned call saves 40 us and up, so a base that is searched only once or twice
// should not pay: the calls' estimated savings add up (prune_credit_us), and the copy is laid out by the call
// that brings them to its cost -- at once for a large batch, after a dozen single queries otherwise. Measured, scan
// / pruned, us a call: 1M x 384: 376 / 194 (1 query), 1121 / 213 (8), 45342 / 873 (1,000); 32768 x 64: 105 / 68
// (1), 2550 / 130 (1,000). *ok = false (and no error) where the search keeps to the plain scan: not yet laid out,
// a copy that would take more than half of the free memory (asked once a fit), or rows that the bounds do not cover.
static bool flat_prune_open(ann_flat* h, bool capturing);
static int flat_ensure_pruned(ann_flat* h, int nq, cudaStream_t st, bool capturing, bool* ok) {
    *ok = false;
    std::lock_guard<std::mutex> lk(h->tc_mu);
    if (!h->bounds_known) {
        const double elems = (double)h->n * h->dim;
        h->prune_credit_us += 40.0 + elems * (nq <= 4 ? 0.25e-6 + 0.2e-6 * (nq - 1) : 1.0e-7 * nq);
        if (!h->base_bf16 && h->prune_credit_us < 500.0 + 3.1e-6 * elems) return ANN_OK;
        if (capturing || (h->prune_refused && !h->base_bf16)) return ANN_OK;
        CaptureRelax relax;
        // the norms first: rows that the bounds do not cover need no copy
        unsigned *d2 = nullptr, h2[2] = {0, 0};
        if (cudaMalloc(&d2, sizeof(h2)) != cudaSuccess) {
            cudaGetLastError();
            h->prune_refused = true;
            return ANN_OK;
        }
        int rc = launch_base_norms(h->base, h->n, h->dim, h->dpad, d2, st);
        cudaError_t e = cudaSuccess;
        if (!rc) e = cudaMemcpyAsync(h2, d2, sizeof(h2), cudaMemcpyDeviceToHost, st);
        if (!rc && e == cudaSuccess) e = cudaStreamSynchronize(st);
        cudaFree(d2);
        if (rc) return rc;
        ANN_CUDA_TRY(e);
        float s2, e2;
        memcpy(&s2, &h2[0], 4);
        memcpy(&e2, &h2[1], 4);
        const float c = std::sqrt(s2), r = std::sqrt(e2);
        const bool covered = c >= kPruneNormMin && c <= kPruneNormMax && r <= c;
        if (covered && !h->base_bf16) {
            size_t mfree = 0, mtotal = 0;
            ANN_CUDA_TRY(cudaMemGetInfo(&mfree, &mtotal));
            const bool fits = sizeof(__nv_bfloat16) * (size_t)h->n * tc_kpad(h->dim, h->metric) <= mfree / 2;
            if (fits) rc = flat_ensure_bf16(h, st);
            if (!fits || rc == ANN_ERR_NOMEM) {  // not asked for again: the query for free memory alone can stall a server
                clear_error();
                h->prune_refused = true;
                return ANN_OK;
            }
            if (rc) return rc;
        }
        h->bounds = covered ? PruneBounds{c * 1.001f, r * 1.001f} : PruneBounds{};
        h->bounds_known = true;
        if (!h->prune_word) {
            void* w = nullptr;
            if (cudaHostAlloc(&w, 2 * sizeof(*h->prune_word), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
                h->prune_word = static_cast<unsigned long long*>(w);
                h->prune_word[0] = (unsigned long long)h->prune_seen << 32;
                h->prune_word[1] = 0;
            } else {
                cudaGetLastError();  // no back-off then
            }
        }
    }
    *ok = h->bounds.cmax > 0.f && flat_prune_open(h, capturing);
    return ANN_OK;
}

// Whether this call tries the pruned form (under tc_mu). The window grows with |x| |q|, not with the rows' spread: over data
// far from the origin, or with more copies of a row than survivors fit, the pass leaves the queries to the scan and was
// for nothing (N(50, 0.01), 37 queries over 131,725 x 33, inner product: 328 us scanned, 902 with the pass). A pass that
// left more than a quarter of its query tiles (any query, in batches of a tile) is followed by 4 calls of the scan alone,
// then 8, up to 1,024, until one does not.
// The device writes the count; it is read here without a wait, so by a later call than the next where calls are queued.
// A captured call keeps the form for every replay, and one bad pass may have been its queries' doing (a warm-up on zeros):
// it is the scan from the second such pass on.
static bool flat_prune_open(ann_flat* h, bool capturing) {
    if (h->prune_word) {
        const unsigned long long w = __atomic_load_n(h->prune_word, __ATOMIC_RELAXED);
        if ((uint32_t)(w >> 32) != h->prune_seen) {
            h->prune_seen = (uint32_t)(w >> 32);
            const int n = (int)((w >> 16) & 0xffffu), left = (int)(w & 0xffffu);
            // the scan reads the base once per query tile, however few of a tile's queries are left
            const int bq = h->query_tile > 0 ? h->query_tile : flat_scan_bq(n);
            if (4 * ceil_div(left, bq) > ceil_div(n, bq)) {
                h->prune_skip = 4 << std::min(h->prune_streak, 8);
                ++h->prune_streak;
            } else {
                h->prune_streak = h->prune_skip = 0;
            }
        }
    }
    if (capturing) return h->prune_streak < 2;
    if (h->prune_skip > 0) {
        --h->prune_skip;
        return false;
    }
    return true;
}

// The pruned form of the exact scan (flat_prune.cu) for queries qdev [nq, dpad]; *done = false, and nothing
// written, where the plain scan answers the call.
static int flat_exact_pruned(ann_flat* h, ann_workspace* ws, const float* qdev, int nq, int kk, int64_t* ids_dev,
                             float* dists_dev, cudaStream_t st, bool* done) {
    *done = false;
    const int64_t n = h->n;
    const int dpad = h->dpad;
    if (!prune_rows(n, nq, kk) || n < 64 * (int64_t)kk || !prune_fits(kk, dpad)) return ANN_OK;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    ANN_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    bool ok = false;
    int rc = flat_ensure_pruned(h, nq, st, capturing, &ok);
    if (rc || !ok) return rc;
    std::optional<CaptureRelax> relax;  // the first pass loads its kernels
    if (!capturing && h->prune_pass == 0) relax.emplace();
    const int bq = std::min(h->query_tile > 0 ? h->query_tile : flat_scan_bq(nq), flat_scan_max_bq(kk));
    const bool stream_form = flat_stream_eligible(bq, kk, dpad);
    // a sample of about 64 tiles of 256 rows, an eighth of a small base
    const int64_t full_tiles = n / 256;
    const int64_t want_tiles = std::min<int64_t>(64, full_tiles / 8);
    const int stride = (int)(full_tiles / want_tiles);
    const int64_t S = full_tiles / stride * 256;
    const int rF = prune_bar_rank(kk, S, n), cap = prune_cap(kk);
    const int kpad = h->kpad;
    constexpr int kChunk = 10240;  // queries at a time: 0.4 GB of sampled minima and survivors (k <= 128)
    const int nchunks = (int)ceil_div(nq, kChunk);
    const int qc = nchunks == 1 ? nq : (int)std::min<int64_t>(kChunk, ceil_div(ceil_div(nq, nchunks), 128) * 128);
    // the scan of the queries left over: up to one split per SM, its lists bounded to 256 MB
    int64_t rps = 0;
    const int ns_plain = flat_choose_nsplit(n, qc, bq, &rps, flat_scan_ctas_per_sm(bq, kk, dpad, h->metric));
    int nsplit = (int)std::max<int64_t>(ns_plain, std::min<int64_t>(kNumSMs, ((int64_t)256 << 20) / ((int64_t)qc * kk * 8)));
    rps = ceil_div(ceil_div(n, nsplit), 256) * 256;
    nsplit = (int)ceil_div(n, rps);
    Sizer sz;
    sz.take<__nv_bfloat16>((size_t)qc * kpad);
    sz.take<float>((size_t)qc * (S / 8));
    for (int i = 0; i < 3; ++i) sz.take<float>((size_t)qc);
    sz.take<float>((size_t)qc * cap);
    sz.take<int>((size_t)qc * cap);
    for (int i = 0; i < 2; ++i) sz.take<int>((size_t)qc);
    for (int i = 0; i < 2; ++i) sz.take<int>(1);
    sz.take<float>((size_t)qc * dpad);
    sz.take<float>((size_t)(qc + 1) / 2 * 2 * dpad);
    sz.take<float>((size_t)qc * nsplit * kk);
    sz.take<int>((size_t)qc * nsplit * kk);
    if (prune_split(qc)) {
        sz.take<unsigned long long>((size_t)qc * cap);
        sz.take<int2>((size_t)qc);
    }
    if (ws->big_cap < sz.bytes()) {
        if (capturing) return ANN_OK;  // the scan's own scratch is there
        std::lock_guard<std::mutex> lk(h->tc_mu);
        if (sz.bytes() >= h->prune_ws_refused) return ANN_OK;
        CaptureRelax allow;
        if ((rc = ws_reserve_big(ws, sz.bytes()))) {
            if (rc != ANN_ERR_NOMEM) return rc;
            clear_error();
            h->prune_ws_refused = std::min(h->prune_ws_refused, sz.bytes());
            return ANN_OK;
        }
    }
    Carver cv(ws->big);
    __nv_bfloat16* qb = cv.take<__nv_bfloat16>((size_t)qc * kpad);
    float* kA = cv.take<float>((size_t)qc * (S / 8));
    float* win = cv.take<float>((size_t)qc);
    float* tauF = cv.take<float>((size_t)qc);
    float* tauX = cv.take<float>((size_t)qc);
    float* fkey = cv.take<float>((size_t)qc * cap);
    int* fcol = cv.take<int>((size_t)qc * cap);
    int* rcount = cv.take<int>((size_t)qc);
    int* list = cv.take<int>((size_t)qc);
    int* count = cv.take<int>(1);
    int* err = cv.take<int>(1);
    float* qg = cv.take<float>((size_t)qc * dpad);
    float* qpair = cv.take<float>((size_t)(qc + 1) / 2 * 2 * dpad);
    float* skey = cv.take<float>((size_t)qc * nsplit * kk);
    int* sid = cv.take<int>((size_t)qc * nsplit * kk);
    unsigned long long* words = prune_split(qc) ? cv.take<unsigned long long>((size_t)qc * cap) : nullptr;
    int2* joined = prune_split(qc) ? cv.take<int2>((size_t)qc) : nullptr;
    for (int q0 = 0; q0 < nq; q0 += qc) {
        const int nc = std::min(qc, nq - q0);
        const float* q = qdev + (size_t)q0 * dpad;
        PruneArgs p{};
        p.base = h->base;
        p.n = n;
        p.dim = h->dim;
        p.dpad = dpad;
        p.mult = h->row_mult;
        p.q = q;
        p.nq = nc;
        p.k = kk;
        p.metric = h->metric;
        p.stream_form = stream_form;
        p.b = h->bounds;
        p.win = win;
        p.tauF = tauF;
        p.cap = cap;
        p.fkey = fkey;
        p.fcol = fcol;
        p.rcount = rcount;
        p.list = list;
        p.count = count;
        p.err = err;
        // (a captured call is replayed on queries to come)
        const bool shared = capturing || !h->prune_word || __atomic_load_n(&h->prune_word[1], __ATOMIC_RELAXED) != 0;
        p.words = shared ? words : nullptr;
        p.joined = shared ? joined : nullptr;
        p.wide = words && !shared ? h->prune_word + 1 : nullptr;
        p.out_ids = ids_dev + (size_t)q0 * kk;
        p.out_dists = dists_dev ? dists_dev + (size_t)q0 * kk : nullptr;
        if ((rc = launch_prune_queries(p, qb, kpad, st))) return rc;
        TcFilterArgs sa{nc, (int)S, kpad, kTcBF16};
        sa.err = err;
        sa.out_min = kA;
        sa.b_tile_stride = stride;
        sa.b_rows = n;
        sa.wait_ns = h->wait_ns;
        sa.test_no_loads = h->wait_ns > 0;
        if ((rc = launch_tc_sample(qb, h->base_bf16, sa, st))) return rc;
        if ((rc = launch_bars(kA, nullptr, nullptr, nc, rF, rF, tauF, tauX, st, S / 8, win))) return rc;
        const TcFilterArgs fa{nc, (int)n, kpad, kTcBF16, tauX, fkey, fcol, cap, rcount, nullptr, nullptr, err, h->wait_ns,
                              h->wait_ns > 0};
        if ((rc = launch_tc_filter(qb, h->base_bf16, fa, st))) return rc;
        if ((rc = launch_prune_finish(p, st))) return rc;
        // the queries on the list, by the plain scan (none, nearly always: the kernels read the count and return)
        uint32_t pass;
        int report;
        {
            std::lock_guard<std::mutex> lk(h->tc_mu);
            pass = ++h->prune_pass;
            h->prune_nq = nc;
            report = h->prune_streak > 0;
        }
        if ((rc = launch_prune_gather(q, dpad, list, count, nc, qg, h->prune_word, pass, report, st))) return rc;
        FlatScanArgs a{h->base, n, dpad, qg, nc, h->metric, kk, rps, nsplit, skey, sid};
        a.qpair = qpair;
        a.nq_dev = count;
        if ((rc = launch_flat_scan(a, bq, st))) return rc;
        MergeArgs m{skey, sid, nc, nsplit, kk, kk, h->metric == ANN_METRIC_IP ? 1 : 0, p.out_ids, p.out_dists};
        m.nq_dev = count;
        m.out_rows = list;
        if ((rc = launch_merge_splits(m, st))) return rc;
    }
    *done = true;
    return ANN_OK;
}

int ann_flat_scores_tc(ann_flat* h, const float* queries, int32_t nq, int64_t ldq, float* out_keys, void* stream) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr && h->base != nullptr, "ann_flat_scores_tc: index not fitted");
    ANN_CHECK_ARG(nq >= 0 && ldq >= h->dim && (nq == 0 || (queries && out_keys)), "ann_flat_scores_tc: bad arguments");
    if (nq == 0) return ANN_OK;
    DeviceGuard g(h->device);
    cudaStream_t st = as_stream(stream);
    FlatTc t;
    int rc = flat_ensure_tc(h, st, &t);
    if (rc) return rc;
    Sizer sz;
    sz.take<unsigned char>((size_t)nq * t.kpad * t.es);
    sz.take<float>((size_t)nq);
    if ((rc = ws_reserve_device(&h->ws, sz.bytes()))) return rc;
    if ((rc = ws_reserve_big(&h->ws, sizeof(float) * (size_t)nq * h->n))) return rc;
    Carver cv(h->ws.dev);
    unsigned char* qb = cv.take<unsigned char>((size_t)nq * t.kpad * t.es);
    float* rfac = cv.take<float>((size_t)nq);
    float* tmp = reinterpret_cast<float*>(h->ws.big);
    if ((rc = flat_tc_queries(h, t, queries, nq, ldq, qb, rfac, st))) return rc;
    TcGemmArgs a{nq, (int)h->n, t.kpad, tmp, h->n, h->d_err};
    a.wait_ns = h->wait_ns;
    a.test_no_loads = h->wait_ns > 0;
    a.kind = t.kind;
    a.col_fac = t.cfac;
    a.row_fac = t.kind == kTcE4M3 ? rfac : nullptr;
    if ((rc = launch_tc_gemm(qb, t.base, a, st))) return rc;
    if ((rc = launch_tc_unpermute(tmp, nq, h->n, h->row_mult, out_keys, st))) return rc;
    ANN_CUDA_TRY(cudaStreamSynchronize(st));
    return flat_check_err(h);
}

int ann_flat_set_option(ann_flat* h, int32_t option, int64_t value) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr, "ann_flat_set_option: null index");
    switch (option) {
        case ANN_FLAT_OPT_QUERY_TILE:
            ANN_CHECK_ARG(value == 0 || value == 8 || value == 16 || value == 32,
                          "ann_flat_set_option: query tile %lld (0, 8, 16 or 32)", (long long)value);
            h->query_tile = (int)value;
            return ANN_OK;
        case ANN_FLAT_OPT_PRUNE:
            ANN_CHECK_ARG(value == 0 || value == 1, "ann_flat_set_option: pruning %lld (0 or 1)", (long long)value);
            h->prune = value != 0;
            return ANN_OK;
        case ANN_FLAT_OPT_WAIT_SELFTEST:
            ANN_CHECK_ARG(value == 0 || (value >= 1000 && value <= 2000000000LL), "ann_flat_set_option: wait limit %lld ns",
                          (long long)value);
            h->wait_ns = (uint64_t)value;
            return ANN_OK;
        default:
            set_error("ann_flat_set_option: unknown option %d", option);
            return ANN_ERR_INVALID;
    }
}

int ann_flat_prune_stats(ann_flat* h, int64_t* out4) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr && out4 != nullptr, "ann_flat_prune_stats: null argument");
    std::lock_guard<std::mutex> lk(h->tc_mu);
    const unsigned long long w = h->prune_word ? __atomic_load_n(&h->prune_word[0], __ATOMIC_RELAXED) : 0;
    out4[0] = h->prune_pass;
    out4[1] = h->prune_nq;
    out4[2] = (uint32_t)(w >> 32) == h->prune_pass ? (int64_t)w & 0xffff : 0;  // (a pass that settled all need not write)
    out4[3] = h->prune_skip;
    return ANN_OK;
}

int ann_flat_set_tc_precision(ann_flat* h, int32_t precision) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr, "ann_flat_set_tc_precision: null index");
    ANN_CHECK_ARG(precision == ANN_TC_BF16 || precision == ANN_TC_E4M3, "ann_flat_set_tc_precision: %d", precision);
    h->tc_kind = precision == ANN_TC_E4M3 ? kTcE4M3 : kTcBF16;
    return ANN_OK;
}

int ann_flat_query_tc(ann_flat* h, ann_workspace* ws, const float* queries, int32_t nq, int64_t ldq, int32_t k,
                      int32_t refine_r, int32_t mem, int64_t* out_ids, float* out_dists, void* stream) {
    clear_error();
    ANN_CHECK_ARG(h != nullptr, "ann_flat_query_tc: null index");
    if (h->base == nullptr || h->n == 0) {
        set_error("index not fitted");
        return ANN_ERR_STATE;
    }
    ANN_CHECK_ARG(nq >= 0 && k >= 1, "ann_flat_query_tc: nq=%d, k=%d", nq, k);
    ANN_CHECK_ARG(ldq >= h->dim, "ann_flat_query_tc: query stride < dim");
    ANN_CHECK_ARG(nq == 0 || (queries && out_ids), "ann_flat_query_tc: null pointer");
    if (nq == 0) return ANN_OK;
    const int kk = (int)std::min<int64_t>(k, h->n);
    const int R = (int)std::min<int64_t>(std::max(kk, refine_r > 0 ? refine_r : 4 * kk), h->n);
    ANN_CHECK_ARG(kk <= 1024 && R <= 8192, "ann_flat_query_tc: k=%d, refine %d too large", kk, R);
    if (!ws) ws = &h->ws;
    DeviceGuard g(h->device);
    cudaStream_t st = as_stream(stream);
    FlatTc t;
    int rc = flat_ensure_tc(h, st, &t);
    if (rc) return rc;
    const int dpad = h->dpad, kpad = t.kpad;
    const size_t rowb = (size_t)kpad * t.es;  // bytes of an operand row
    const bool e4 = t.kind == kTcE4M3;
    const bool host = mem == ANN_MEM_HOST;
    Sizer sz;
    sz.take<float>((size_t)nq * dpad);
    sz.take<unsigned char>((size_t)nq * rowb);
    sz.take<float>((size_t)nq);
    sz.take<float>((size_t)nq * R);
    sz.take<int>((size_t)nq * R);
    if (host) {
        sz.take<int64_t>((size_t)nq * kk);
        sz.take<float>((size_t)nq * kk);
    }
    if ((rc = ws_reserve_device(ws, sz.bytes()))) return rc;
    Carver cv(ws->dev);
    float* qdev = cv.take<float>((size_t)nq * dpad);
    unsigned char* qb = cv.take<unsigned char>((size_t)nq * rowb);
    float* rfac = cv.take<float>((size_t)nq);
    float* keyR = cv.take<float>((size_t)nq * R);
    int* idR = cv.take<int>((size_t)nq * R);
    int64_t* ids_dev = out_ids;
    float* dists_dev = out_dists;
    if (host) {
        ids_dev = cv.take<int64_t>((size_t)nq * kk);
        dists_dev = cv.take<float>((size_t)nq * kk);
        if ((rc = queries_in(qdev, dpad, queries, ldq, nq, h->dim, st))) return rc;
    } else {
        if ((rc = launch_pad_rows(queries, nq, h->dim, ldq, qdev, dpad, st))) return rc;
    }
    if ((rc = flat_tc_queries(h, t, qdev, nq, dpad, qb, rfac, st))) return rc;
    // Sampled bars: keys over a strided sample of S positions of the operand copy (an even sample of the
    // base, by its row order), of which the smallest of every 8 are kept, give each query two bars. The safe
    // bar, the R-th smallest of them, is at or above its R-th best key over all rows (a little more than
    // n R / S keys pass it). The fast bar, the rF-th, lets n rF / S keys pass, rF just past the number of the
    // R best that a sample holds: fewer than R survivors, about 1 query in 10^7. The full pass keeps the keys
    // under the fast bar; a query with fewer than R survivors (the count is exact) is re-run under its
    // safe bar, so every query ends with its best R keys among its survivors. A query with more survivors than its
    // buffer holds (thousands of copies of a row) is re-run under its fast bar with room for all of them: with the
    // chunk's full key matrix in its place, 5 queries over 191,343 x 9, a third of the rows zero, took 1,145 us, 338 now.
    // Small bases use the full key matrix. (With every sampled key written and binned, a tenth of
    // a 10,000-query call went to the bars: sample and bars 1.59 ms, 0.31 ms from the minima.)
    const int64_t n = h->n;
    const int64_t full_tiles = n / 256;
    const int64_t want_tiles = std::max(std::max<int64_t>(128, ceil_div(16 * (int64_t)R, 256)), full_tiles / 64);
    const bool sampled = full_tiles >= 4 * want_tiles;
    const int stride = sampled ? (int)(full_tiles / want_tiles) : 1;
    const int64_t S = sampled ? (full_tiles / stride) * 256 : 0;
    const int rF = sampled ? prune_bar_rank(R, S, n) : 0;
    constexpr int kRerunBatch = 128;
    // queries per chunk: 1 GB of survivors, or ~4 GB of full key matrix
    const int64_t qfull64 = std::max<int64_t>(128, ((int64_t)4 << 30) / (int64_t)(sizeof(float) * n) / 128 * 128);
    const int qfull = (int)std::min<int64_t>(qfull64, 65535);
    const int64_t cap64 = std::min<int64_t>(n, 16 * (int64_t)R);
    const int qmax = sampled ? (int)std::clamp<int64_t>(((int64_t)1 << 30) / (8 * cap64) / 128 * 128, 128, 16384) : qfull;
    const int nchunks = (int)ceil_div(nq, qmax);
    const int qc = (int)std::min<int64_t>(qmax, ceil_div(ceil_div(nq, nchunks), 128) * 128);
    for (int q0 = 0; q0 < nq; q0 += qc) {
        const int nc = std::min(qc, nq - q0);
        const unsigned char* qbc = qb + (size_t)q0 * rowb;
        const float* rfc = e4 ? rfac + q0 : nullptr;
        float* keyRc = keyR + (size_t)q0 * R;
        int* idRc = idR + (size_t)q0 * R;
        bool done = false;
        if (sampled) {
            // survivors kept per query: about 3 R pass the fast bar (9 R were met over 5,000 queries of a 4M-row
            // mixture), n R / S the safe bar of a re-run
            const int cap = (int)cap64;
            const int cap2 = (int)std::min<int64_t>(n, 2 * ceil_div((int64_t)R * n, S) + 1024);
            const size_t ent = std::max(std::max((size_t)nc * cap, (size_t)std::min(nc, kRerunBatch) * cap2),
                                        (size_t)std::min<int64_t>(n, 1 << 24));  // one query's every row at least
            Sizer s2;
            s2.take<float>((size_t)nc * (S / 8));      // minima of 8 sampled keys
            s2.take<float>(ent);                       // survivors: key, position
            s2.take<int>(ent);
            for (int i = 0; i < 3; ++i) s2.take<float>((size_t)nc);  // fast, safe, gathered bars
            for (int i = 0; i < 3; ++i) s2.take<int>((size_t)nc);    // row counts, re-run lists
            s2.take<int>(4);                           // flags
            s2.take<unsigned char>((size_t)kRerunBatch * rowb);
            s2.take<float>((size_t)kRerunBatch);
            if ((rc = ws_reserve_big(ws, s2.bytes()))) return rc;
            Carver cb(ws->big);
            float* kA = cb.take<float>((size_t)nc * (S / 8));
            float* fkey = cb.take<float>(ent);
            int* fcol = cb.take<int>(ent);
            float* tauF = cb.take<float>((size_t)nc);
            float* tauS = cb.take<float>((size_t)nc);
            float* tau2 = cb.take<float>((size_t)nc);
            int* rowcnt = cb.take<int>((size_t)nc);
            int* list = cb.take<int>((size_t)nc);
            int* over = cb.take<int>((size_t)nc);
            int* flags = cb.take<int>(4);  // queries in list and in over, most survivors of a query
            unsigned char* A2 = cb.take<unsigned char>((size_t)kRerunBatch * rowb);
            float* rfac2 = cb.take<float>((size_t)kRerunBatch);

            // stages 2: sample pass and bars, 3: filter pass, 4: grouping, selections and re-runs
            const int prec = h->prof.begin(st, 2);
            TcFilterArgs sa{nc, (int)S, kpad, t.kind};
            sa.col_fac = t.cfac;
            sa.row_fac = rfc;
            sa.err = h->d_err;
            sa.out_min = kA;
            sa.b_tile_stride = stride;
            sa.b_rows = n;
            sa.wait_ns = h->wait_ns;
            sa.test_no_loads = h->wait_ns > 0;
            if ((rc = launch_tc_sample(qbc, t.base, sa, st))) return rc;
            const int S8 = (int)(S / 8);
            if ((rc = launch_bars(kA, nullptr, nullptr, nc, rF, R, tauF, tauS, st, S8))) return rc;
            h->prof.mark(prec, st);
            auto filter = [&](const void* A, int M, const float* tau, const float* rf, int rcap) -> int {
                ANN_CUDA_TRY(cudaMemsetAsync(rowcnt, 0, sizeof(int) * (size_t)M, st));
                const TcFilterArgs fa{M,    (int)n, kpad,   t.kind, tau, fkey,     fcol,
                                      rcap, rowcnt, t.cfac, rf,     h->d_err, h->wait_ns, h->wait_ns > 0};
                int r = launch_tc_filter(A, t.base, fa, st);
                if (r) return r;
                return launch_max_int(rowcnt, M, flags + 2, st);
            };
            if ((rc = filter(qbc, nc, tauF, rfc, cap))) return rc;
            h->prof.mark(prec, st);
            if (prec >= 0) h->prof.filter_launches += 1;
            ANN_CUDA_TRY(cudaMemsetAsync(flags, 0, 2 * sizeof(int), st));
            if ((rc = launch_tc_bar_check(rowcnt, nc, R, list, flags, st, nullptr, nullptr, cap, over))) return rc;
            int hf[3] = {0, 0, 0};
            ANN_CUDA_TRY(cudaMemcpyAsync(hf, flags, sizeof(hf), cudaMemcpyDeviceToHost, st));
            ANN_CUDA_TRY(cudaStreamSynchronize(st));
            int ngemm = 2;
            RadixSelectArgs sv{};
            sv.keys = fkey;
            sv.ld = cap;
            sv.lens32 = rowcnt;
            sv.ids = fcol;
            sv.R = R;
            sv.out_key = keyRc;
            sv.out_id = idRc;
            if ((rc = launch_radix_select(sv, nc, st))) return rc;
            done = true;
            // queries rows[0..count) again under the bars tau, room for rcap survivors each, or for as many as one turns out
            // to have; done = false where those exceed the buffer
            auto redo = [&](const int* rows, int count, const float* tau, int rcap) -> int {
                for (int j0 = 0; j0 < count && done;) {
                    if ((size_t)rcap > ent) {
                        done = false;
                        break;
                    }
                    const int nb = (int)std::min<size_t>(std::min(kRerunBatch, count - j0), ent / rcap);
                    int r = launch_tc_gather(qbc, (int)rowb, rows + j0, nb, tau, A2, tau2, rfc, rfac2, st);
                    if (r || (r = filter(A2, nb, tau2, e4 ? rfac2 : nullptr, rcap))) return r;
                    ++ngemm;
                    int hmax = 0;
                    ANN_CUDA_TRY(cudaMemcpyAsync(&hmax, flags + 2, sizeof(int), cudaMemcpyDeviceToHost, st));
                    ANN_CUDA_TRY(cudaStreamSynchronize(st));
                    if (hmax > rcap) {
                        rcap = hmax;
                        continue;
                    }
                    RadixSelectArgs sv2 = sv;
                    sv2.ld = rcap;
                    sv2.out_rows = rows + j0;
                    if ((r = launch_radix_select(sv2, nb, st))) return r;
                    j0 += nb;
                }
                return ANN_OK;
            };
            if ((rc = redo(list, hf[0], tauS, cap2))) return rc;
            // Measured: a pass of its own 0.2 ms, its survivors 0.17 ns each; the full matrix 1 ms (its selection of whole
            // rows) and 0.02 ns a key. 1,000 queries over 1M x 384 with 200,000 copies each: 33 ms by passes, 20 by the
            // matrix; 70 of 184 over 184,924 x 70 with 74,000 copies, three to a pass: 4.8, 2.1.
            const int64_t per_pass = std::max<int64_t>(1, std::min<int64_t>(kRerunBatch, (int64_t)ent / std::max(1, hf[2])));
            const double passes_us = 200.0 * (double)ceil_div(hf[1], per_pass) + 1.7e-4 * (double)hf[1] * hf[2];
            if (passes_us > 1000.0 + 2e-5 * (double)nc * (double)n)
                done = false;
            else if ((rc = redo(over, hf[1], tauF, hf[2])))
                return rc;
            // positions of the operand copy -> rows
            if (done && (rc = launch_tc_map_ids(idRc, (int64_t)nc * R, n, h->row_mult, st))) return rc;
            h->prof.mark(prec, st);
            if (prec >= 0) h->prof.tc_launches += ngemm;
        }
        for (int f0 = 0; !done && f0 < nc; f0 += qfull) {  // the full key matrix, qfull queries at a time
            const int nf = std::min(qfull, nc - f0);
            if ((rc = ws_reserve_big(ws, sizeof(float) * (size_t)nf * n))) return rc;
            float* keys = reinterpret_cast<float*>(ws->big);
            const int prec = h->prof.begin(st, 3);  // stage 3: the full key matrix, 4: its selection
            TcGemmArgs a{nf, (int)n, kpad, keys, n, h->d_err};
            a.wait_ns = h->wait_ns;
            a.test_no_loads = h->wait_ns > 0;
            a.kind = t.kind;
            a.col_fac = t.cfac;
            a.row_fac = e4 ? rfc + f0 : nullptr;
            if ((rc = launch_tc_gemm(qbc + (size_t)f0 * rowb, t.base, a, st))) return rc;
            h->prof.mark(prec, st);
            RadixSelectArgs fs{};
            fs.keys = keys;
            fs.ld = n;
            fs.R = R;
            fs.out_key = keyRc + (size_t)f0 * R;
            fs.out_id = idRc + (size_t)f0 * R;
            if ((rc = launch_radix_select(fs, nf, st))) return rc;
            if ((rc = launch_tc_map_ids(fs.out_id, (int64_t)nf * R, n, h->row_mult, st))) return rc;
            h->prof.mark(prec, st);
            if (prec >= 0) h->prof.tc_launches += 1;
        }
    }
    const int prec = h->prof.begin(st, 5);  // stage 5: re-rank
    IvfQueryArgs ra{};
    ra.ix.n = h->n;
    ra.ix.dim = h->dim;
    ra.ix.dpad = dpad;
    ra.ix.original = h->base;
    ra.ix.r2o = nullptr;
    ra.plan.nq = nq;
    ra.q = qdev;
    ra.ldq = dpad;
    ra.k = kk;
    ra.R = R;
    ra.metric = h->metric;
    ra.out_ids = ids_dev;
    ra.out_dists = dists_dev;
    if ((rc = launch_ivf_rerank(ra, keyR, idR, 0, st))) return rc;
    h->prof.mark(prec, st);
    h->ndist.fetch_add(h->n * (int64_t)nq);
    if (host) {
        ANN_CUDA_TRY(cudaMemcpyAsync(out_ids, ids_dev, sizeof(int64_t) * (size_t)nq * kk, cudaMemcpyDeviceToHost, st));
        if (out_dists)
            ANN_CUDA_TRY(cudaMemcpyAsync(out_dists, dists_dev, sizeof(float) * (size_t)nq * kk, cudaMemcpyDeviceToHost, st));
        ANN_CUDA_TRY(cudaStreamSynchronize(st));
        return flat_check_err(h);
    }
    return ANN_OK;
}

int ann_flat_device_status(ann_flat* h) {
    ANN_CHECK_ARG(h != nullptr, "null index");
    DeviceGuard g(h->device);
    return flat_check_err(h);
}

int ann_merge_topk(const float* dists, const int64_t* ids, int32_t nq, int32_t parts, int32_t k, int32_t metric,
                   int64_t* out_ids, float* out_dists, void* stream) {
    clear_error();
    ANN_CHECK_ARG(nq >= 0 && (nq == 0 || (dists && ids && out_ids)), "ann_merge_topk: null pointer");
    ANN_CHECK_ARG(metric == ANN_METRIC_L2 || metric == ANN_METRIC_IP, "ann_merge_topk: metric %d", metric);
    return launch_merge_parts(dists, ids, nq, parts, k, metric == ANN_METRIC_IP ? 1 : 0, out_ids, out_dists,
                              as_stream(stream));
}

int ann_select_smallest(const float* keys, int64_t ld, const int64_t* lens, int32_t nq, int32_t r, float* out_keys,
                        int32_t* out_pos, void* stream) {
    clear_error();
    ANN_CHECK_ARG(nq >= 0 && r >= 1 && ld >= 0 && ld < INT32_MAX, "ann_select_smallest: nq=%d r=%d ld=%lld", nq, r,
                  (long long)ld);
    ANN_CHECK_ARG(nq == 0 || (keys && out_keys && out_pos), "ann_select_smallest: null pointer");
    RadixSelectArgs a{};
    a.keys = keys;
    a.ld = ld;
    a.lens = lens;
    a.R = r;
    a.out_key = out_keys;
    a.out_id = out_pos;
    return launch_radix_select(a, nq, as_stream(stream));
}

int64_t ann_flat_total_distances(const ann_flat* h) { return h ? h->ndist.load() : 0; }
int32_t ann_flat_dim(const ann_flat* h) { return h ? h->dim : 0; }
int64_t ann_flat_size(const ann_flat* h) { return h ? h->n : 0; }

}  // extern "C"
