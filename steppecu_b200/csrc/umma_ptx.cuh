// steppecu_b200/csrc/umma_ptx.cuh
//
// Inline-PTX building blocks shared by the tcgen05 contraction kernels (f2_umma.cu,
// f2_fx.cu): mbarriers with bounded waits, plain bulk copies (no tensor maps, no
// multicast), tcgen05 MMA issue / commit / TMEM loads, and the K-major swizzled
// shared-memory descriptor. sm_100a only.
#pragma once

#include <cstdint>

namespace stpf2 {
namespace ptx {

// Default bound of every spin-wait in the contraction kernels (ns of %globaltimer).
constexpr unsigned long long kTimeoutNs = 4000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(unsigned long long* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(b))
                 : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, uint32_t bytes) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                     smem_u32(b)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait on an mbarrier phase: false on timeout (which raises the CTA's abort flag
// and the global error flag) or, with honour_abort, once another role of the CTA has
// aborted.
__device__ __forceinline__ bool wait_bounded(unsigned long long* b, uint32_t parity, volatile int* abort_flag,
                                             int* err, unsigned long long timeout_ns, bool honour_abort = true) {
    if (mbar_try_wait(b, parity)) return true;
    const unsigned long long t0 = globaltimer();
    for (uint32_t it = 1;; ++it) {
        if (mbar_try_wait(b, parity)) return true;
        if ((it & 63u) == 0) {
            if (honour_abort && *abort_flag) return false;
            if (globaltimer() - t0 > timeout_ns) {
                *abort_flag = 1;
                atomicExch(err, 1);
                return false;
            }
        }
    }
}

// ---- warp-uniform issue ----
//
// tcgen05.mma, tcgen05.commit and cp.async.bulk take their operands from uniform registers. A
// role that runs as one lane of a divergent branch computes them in vector registers and
// moves each over per instruction. So a whole warp runs an issuing role, every value that
// reaches those instructions made uniform where it enters (uni), and one elected lane executes
// them, with descriptors that differ by constants from one per slot. Against single-lane roles:
// f2 at 100 populations x 1.15M SNPs 269 -> 254 us, at 603 ragged ones 1,341 -> 1,283; their
// counts 133 -> 114; the split form at 300 x 400,000 832 -> 809. At 1,000 populations, where the
// tensor and shared-memory pipes bound f2, 8.76 -> 8.48 ms (the fastest launches; 9.4 -> 9.0 in
// the median, under the power cap), and the counts 0.81 -> 0.72.
__device__ __forceinline__ int uni(int x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ uint32_t uni(uint32_t x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ int64_t uni(int64_t x) { return __shfl_sync(0xffffffffu, x, 0); }
template <class T>
__device__ __forceinline__ const T* uni(const T* p) {
    return reinterpret_cast<const T*>(uni(static_cast<int64_t>(reinterpret_cast<uintptr_t>(p))));
}

__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

// wait_bounded for a whole warp: the answer is the same for every lane.
__device__ __forceinline__ bool wait_warp(unsigned long long* b, uint32_t parity, volatile int* abort_flag, int* err,
                                          unsigned long long timeout_ns, int lane) {
    if (__all_sync(0xffffffffu, mbar_try_wait(b, parity))) return true;
    int ok = 1;
    if (lane == 0) ok = wait_bounded(b, parity, abort_flag, err, timeout_ns);
    ok = uni(ok);
    __syncwarp();
    return ok != 0;
}

// Plain bulk copy global -> shared, completing on an mbarrier (no tensor map, no
// multicast): size and both addresses multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// kind::i8 with the A operand kept in the MMA's collector buffer: kFill reads A from shared
// memory and keeps it, kUse / kLastUse take it from the buffer (the descriptor must name the
// same A; kLastUse releases it), kDiscard is the plain form.
enum class CollectorA { kDiscard, kFill, kUse, kLastUse };

template <CollectorA kC>
__device__ __forceinline__ void mma_i8_c(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    if constexpr (kC == CollectorA::kFill) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8.collector::a::fill [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc)
            : "memory");
    } else if constexpr (kC == CollectorA::kUse) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8.collector::a::use [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc)
            : "memory");
    } else if constexpr (kC == CollectorA::kLastUse) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::i8.collector::a::lastuse [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc)
            : "memory");
    } else {
        mma_i8(d, a, b, idesc, acc);
    }
}

__device__ __forceinline__ void mma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x N consecutive 32-bit TMEM columns -> N registers per thread.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}

// UMMA shared-memory descriptor, K-major, swizzled: start address, LBO (unused for a
// single swizzle atom along K, encoded 1), SBO = byte distance between 8-row groups,
// descriptor version 1 (sm_100), layout type (4 = 64B swizzle, 6 = 32B swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t sbo_bytes, uint64_t layout) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (1ull << 16) |
           (static_cast<uint64_t>(sbo_bytes >> 4) << 32) | (1ull << 46) | (layout << 61);
}

}  // namespace ptx
}  // namespace stpf2
