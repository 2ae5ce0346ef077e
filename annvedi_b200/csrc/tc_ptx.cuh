// Device primitives of the tcgen05 GEMM kernels (sm_100a): bounded mbarrier waits, TMA loads, MMA issue, TMEM loads.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace annb {

// The 128-byte-swizzle tensor map of a row-major [rows, cols] operand of `kind`, in boxes of box_rows rows of 128 bytes.
int tc_make_map(CUtensorMap* tm, const void* base, int64_t rows, int cols, int box_rows, int kind);

namespace {

// A k-block is one 128-byte row per operand row: 64 BF16 / FP16 or 128 E4M3 elements.
constexpr int kBM = 128, kBN = 256, kBK = 64;
constexpr int kRowBytes = 128;
constexpr int kABytes = kBM * kRowBytes;  // 16 KB
constexpr int kBBytes = kBN * kRowBytes;  // 32 KB
template <int KIND>
struct KindOf {
    static constexpr int kBlockK = tc_16bit(KIND) ? 64 : 128;  // elements per k-block
    static constexpr int kMmaK = tc_16bit(KIND) ? 16 : 32;     // elements per MMA
};
constexpr int kTmemCols = 512;

__device__ __forceinline__ uint32_t su32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 4 bytes from global src to shared dst, asynchronously (zeros when !valid: no bytes are read)
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(su32(dst)), "l"(src), "r"(valid ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(b)), "r"(n) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(su32(b)), "r"(parity)
                 : "memory");
    return ok != 0;
}
// try_wait that may suspend the thread for up to 0.1 ms (woken early when the phase completes), so a
// waiting warp takes few issue slots from the epilogue warps that share its scheduler
__device__ __forceinline__ bool bar_try_sleep(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(su32(b)), "r"(parity), "r"(100000u)
        : "memory");
    return ok != 0;
}
// bar_wait by shared-memory address (for loops that step it).
__device__ __forceinline__ bool bar_try_at(uint32_t b, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(b), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Waits for the phase; gives up after `limit_ns` (2 s when 0), sets *err = 2 and returns false.
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, int* err, uint64_t limit_ns = 0) {
    if (bar_try(b, parity)) return true;
    const uint64_t limit = limit_ns ? limit_ns : 2000000000ull;
    const uint64_t t0 = gtimer();
    while (!bar_try_sleep(b, parity))
        if (gtimer() - t0 > limit) {
            if (err) atomicExch(err, 2);
            return false;
        }
    return true;
}
// The whole (converged) warp waits; every lane gets the same answer.
__device__ __forceinline__ bool bar_wait_warp(uint32_t b, uint32_t parity, int* err, uint64_t limit_ns) {
    if (__all_sync(0xffffffffu, bar_try_at(b, parity))) return true;
    const uint64_t limit = limit_ns ? limit_ns : 2000000000ull;
    const uint64_t t0 = gtimer();
    while (!__all_sync(0xffffffffu, bar_try_at(b, parity)))
        if (__any_sync(0xffffffffu, gtimer() - t0 > limit)) {
            if (err) atomicExch(err, 2);
            return false;
        }
    return true;
}
// A warp that gave up holds its CTA (and with it the pair) for 5 ms before the CTA may end: copies in flight into its shared
// memory take microseconds, and once the MMA issuer has given up nothing else waits for them.
__device__ __forceinline__ void let_copies_land() {
    const uint64_t t0 = gtimer();
    while (gtimer() - t0 < 5000000ull) {
    }
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}" ::"r"(su32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(su32(b)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* tm, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            su32(dst)),
        "l"(tm), "r"(c0), "r"(c1), "r"(su32(bar))
        : "memory");
}
// Shared-memory matrix descriptor for a K-major tile in the 128-byte swizzle layout (rows of 128 B,
// 8-row groups 1024 B apart): start address >> 4, leading offset 1 (unused with swizzle), stride
// offset 1024 >> 4, descriptor version 1, layout type 2 (128-byte swizzle).
__device__ __forceinline__ uint64_t sw128_desc(const void* p) {
    const uint64_t addr = (su32(p) >> 4) & 0x3FFFull;
    return addr | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptors: FP32 accumulator (bits 4-5 = 1), A and B K-major, N = 256 (bits 17-22 = N / 8),
// M = 128 (bits 24-28 = M / 16); A and B types in bits 7-9 and 10-12: BF16 = 1 and FP16 = 0 under kind::f16,
// E4M3 = 0 under kind::f8f6f4.
// (CG = 2, two CTAs a tile: M = 256)
template <int CG>
constexpr uint32_t kIdescShape = (1u << 4) | ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(CG * kBM >> 4) << 24);
template <int CG>
constexpr uint32_t kIdescBF16 = kIdescShape<CG> | (1u << 7) | (1u << 10);
template <int CG>
constexpr uint32_t kIdescE4M3 = kIdescShape<CG>;
constexpr uint32_t kIdescF16 = kIdescShape<1>;
// kind::i8: S32 accumulator (bits 4-5 = 2), A signed (bits 7-9 = 1), B unsigned (bits 10-12 = 0)
constexpr uint32_t kIdescI8 = (2u << 4) | ((uint32_t)(kBN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24) | (1u << 7);

// One MMA of the 32 bytes of K that follow each descriptor's start: 16 BF16 or 32 E4M3 elements. CG = 2: both CTAs of
// the pair take part, each with its 128 rows of A, its half of B's rows and the accumulator rows of its A.
#define ANN_MMA(cg, kind, idesc)                                                  \
    asm volatile(                                                                 \
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"                             \
        " tcgen05.mma.cta_group::" cg ".kind::" kind " [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d), \
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)                             \
        : "memory")
template <int KIND, int CG = 1>
__device__ __forceinline__ void mma_issue(uint32_t tmem_d, uint64_t ad, uint64_t bd, uint32_t accumulate) {
    static_assert((KIND != kTcI8 && KIND != kTcF16) || CG == 1, "int8 and FP16 operands: one CTA");
    if constexpr (KIND == kTcBF16 && CG == 1)
        ANN_MMA("1", "f16", kIdescBF16<1>);
    else if constexpr (KIND == kTcBF16)
        ANN_MMA("2", "f16", kIdescBF16<2>);
    else if constexpr (KIND == kTcE4M3 && CG == 1)
        ANN_MMA("1", "f8f6f4", kIdescE4M3<1>);
    else if constexpr (KIND == kTcE4M3)
        ANN_MMA("2", "f8f6f4", kIdescE4M3<2>);
    else if constexpr (KIND == kTcF16)
        ANN_MMA("1", "f16", kIdescF16);
    else
        ANN_MMA("1", "i8", kIdescI8);
}
#undef ANN_MMA
// One lane of the (converged) warp, the same at every call.
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(ok));
    return ok != 0;
}
// An accumulator read from TMEM as a float: FP32 bits, or (kind::i8) an int32 converted (exact below 2^24).
template <int KIND>
__device__ __forceinline__ float acc_value(uint32_t r) {
    return KIND == kTcI8 ? __int2float_rn((int)r) : __uint_as_float(r);
}
__device__ __forceinline__ void mma_commit_at(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) { mma_commit_at(su32(bar)); }
// tcgen05.ld of 32 consecutive columns of the warp's 32 lanes; the registers are valid only after
// tmem_wait (which names them, so no use is scheduled before the wait).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
// Orders a second register set after the wait already issued for the first.
__device__ __forceinline__ void tmem_after_wait(uint32_t (&r)[32]) {
    asm volatile(""
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

}  // namespace
}  // namespace annb
