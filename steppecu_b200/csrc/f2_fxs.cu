// steppecu_b200/csrc/f2_fxs.cu
//
// The fixed-point f2 contraction of f2_fx.cu for requests of at most 64 populations: the same
// digits and exact integer sums (f2_fx.cu's header has the arithmetic), with the digit planes
// stacked into the MMA's rows and columns. A block's sum is one int64 here and rounded once; the
// general kernel rounds and adds in FP64 per 16,384 SNPs. So the results are the same bit for
// bit for blocks of up to 16,384 SNPs, and within a few FP64 roundings beyond.
//
// With P <= 64 populations a 128-row tile of one plane is mostly padding, and an MMA of N <=
// 64 columns costs as much as one of 64 (about 44 cycles whatever its columns), so the
// general kernel spends ~800 cycles per 32 SNPs on 12 narrow MMAs and another kernel on the
// counts. Here R = P rounded up to 8, and one chunk's image is nine R-row planes
// [X0 X1 X2 X3 E6 M E3 E4 E5] (kFxsImage), so that
//     D1 = [X2; X3] (2R rows)  x  [X0; X1; X2; X3] (4R columns)
//     D2 = [E6; M]  (2R rows)  x  [M; E3; E4; E5]  (4R columns)
// hold, between them, every product the pair (i, j) needs or its mirror at (j, i) - there is
// one tile, so both are in it - and the both-present counts M M. Two MMAs of N = 4R per
// chunk: 64 to 256 cycles. Rows 2R.. of A are whatever follows in shared memory; their
// accumulator lanes are never read.
//
// From lane R + i (rows X3 / M) and lane i (rows X2 / E6), with T = 2 (what appears once) +
// (what is symmetric by itself), every sum exact:
//     T_hi(i, j) = 2 [X3X0 + M E3 + 2^8 (X3X1 + M E4) + 2^16 (X3X2 + M E5)] + 2^24 X3X3
//     T_lo(i, j) = 2 [X2X1 + 2^24 E6 M] + 2^8 X2X2
//     W(i, j)    = (T(i, j) + T(j, i)) / 2,   T = T_hi + T_lo
// and W is f2_fx_kernel's W, over the whole block: |T| < 2^39.6 per SNP, so int64 holds a block
// of 2^22 SNPs (longer blocks take the general kernels). An accumulator entry is one digit product per SNP, at
// most 2^14, so int32 holds 131,040 SNPs; longer blocks run in segments.
//
// One persistent launch, one CTA per SM: warp 0 copies (several chunks per bulk copy: the
// images of consecutive chunks are contiguous), warp 1 issues the MMAs, eight epilogue warps
// read the accumulators, exchange T through shared memory and write whole slabs of f2 and
// vpair as contiguous runs. Up to 32 rows per plane two accumulators alternate; above, one.
// Measured (f2 and counts together): 20 populations x 50,000 SNPs in 40 blocks 32.4 -> 10.3 us; the
// sixteen requests of 4 to 64 populations in a batch over 400,000 SNPs 1,612 -> 366 us. The line at
// 64 is where the planes fill the accumulators; up to it the stacked form is the faster one alone
// too (whole passes over 200,000 SNPs in 140 blocks, general and stacked: 33 populations 151 and
// 58 us, 48 163 and 68, 64 164 and 80; over one block 5.8 ms and 0.9 to 1.3; 10,000 blocks of 10
// SNPs 1.03 ms and 0.32 to 0.57), while 65 populations take the general one (122 us).
#include <algorithm>

#include "stpf2_internal.cuh"
#include "umma_ptx.cuh"

namespace stpf2 {

namespace {

using namespace ptx;

constexpr int kItemRing = 4;
constexpr int kStages = 3;
constexpr uint32_t kStageBytes = 128 * kFxsPlanes * 32;  // 36 KiB: 128 / R chunks
constexpr int kEpiWarps = 8;
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr int kSegChunks = 4095;  // 131,040 SNPs: 2^14 per SNP stays below 2^31
static_assert(16384ll * 32 * kSegChunks < (1ll << 31), "segment bound");
constexpr int kPitch = kFxsMaxPops + 1;
constexpr uint32_t kTmemCols = 512;

struct FxsArgs {
    const uint8_t* images;  // chunk c's image at c * kFxsPlanes * 32 * R
    const BlockInfo* work;  // one item per block, costliest first
    int n_work;
    int P;
    double* f2;
    double* vpair;
    const double* rcp;  // rcp[k] = 1/k
    int rcp_max;
    int* err;
    int* next;  // work counter, zero at launch and left zero
    int b_base;
    unsigned long long timeout_ns;
    long long withhold;  // test hook: the producer stops before its stage of this index
    const GroupInfo* groups;
    int* grp_done;
    unsigned long long* grp_ns;
    const int* grp_items;
};

struct FxsCtl {
    unsigned long long item_full[kItemRing], item_empty[kItemRing];
    BlockInfo item[kItemRing];  // k < 0: no more work
    unsigned long long full[kStages], empty[kStages];
    unsigned long long acc_full[2], acc_empty[2];
    unsigned long long drain;
    uint32_t tmem_base;
    volatile int abort;
};

__device__ __forceinline__ bool waitb(unsigned long long* b, uint32_t parity, FxsCtl* ctl, const FxsArgs& a,
                                      bool honour_abort = true) {
    return wait_bounded(b, parity, &ctl->abort, a.err, a.timeout_ns, honour_abort);
}

__device__ __forceinline__ bool waitw(unsigned long long* b, uint32_t parity, FxsCtl* ctl, const FxsArgs& a, int lane) {
    return wait_warp(b, parity, &ctl->abort, a.err, a.timeout_ns, lane);
}

template <bool kGrouped>
__device__ __forceinline__ int pops_of(const FxsArgs& a, const BlockInfo& bi) {
    return kGrouped ? bi.P : a.P;
}

__device__ __forceinline__ int chunks_of(const BlockInfo& bi) { return (bi.k + 31) / 32; }

// Which accumulator slots the items use, in the issuer's and the epilogue's step: a plane of
// up to 32 rows takes one 256-column slot, alternating; a longer one takes both. uses[s]
// counts the times slot s has been handed over.
struct AccRing {
    uint32_t uses[2] = {0, 0};
    int turn = 0;
    __device__ __forceinline__ int slot(int R) {
        if (R > 32) return 0;
        const int s = turn;
        turn ^= 1;
        return s;
    }
};

// The whole of warp 0.
template <bool kGrouped>
__device__ void fxs_producer(const FxsArgs& a, uint8_t* smem, FxsCtl* ctl, int lane) {
    uint32_t g = 0;
    // A CTA's first item is its own number, read while the kernels before still run (the work
    // list is older than they are); the counter deals out the rest. Its answer and the next
    // item's record arrive while the current item streams (lane 0 holds them). Against a claim
    // from the counter first the pass over 20 populations x 50,000 SNPs took 25.4 us, now 24.6.
    int it = a.n_work;
    BlockInfo cur{}, nxt{};
    cur.k = nxt.k = -1;
    if (lane == 0) cur = a.work[blockIdx.x];
    pdl_wait();  // the decode's images, and the counter
    if (lane == 0) it = static_cast<int>(gridDim.x) + atomicAdd(a.next, 1);
    bool stopped = false;
    for (uint32_t gi = 0; !stopped; ++gi) {
        const int slot = static_cast<int>(gi % kItemRing);
        if (!waitw(&ctl->item_empty[slot], ((gi / kItemRing) & 1u) ^ 1u, ctl, a, lane)) {
            stopped = true;
            break;
        }
        if (lane == 0) {
            ctl->item[slot] = cur;
            mbar_arrive(&ctl->item_full[slot]);
        }
        const int k = uni(cur.k);
        if (k < 0) return;
        nxt.k = -1;
        if (lane == 0 && it < a.n_work) {
            nxt = a.work[it];
            it = static_cast<int>(gridDim.x) + atomicAdd(a.next, 1);
        }
        const int grp = uni(cur.grp);
        const int R = uni(fxs_rows(kGrouped ? uni(cur.P) : a.P));
        const uint32_t chunk = static_cast<uint32_t>(kFxsPlanes * 32 * R);
        const int per = 128 / R;
        const uint8_t* src = uni((kGrouped ? a.groups[grp].images : a.images) + uni(cur.col) / 32 * chunk);
        const int nch = (k + 31) / 32;
        for (int p0 = 0; p0 < nch && !stopped; p0 += kSegChunks) {
            const int p1 = min(nch, p0 + kSegChunks);
            for (int c0 = p0; c0 < p1; c0 += per, ++g) {
                if (static_cast<long long>(g) == a.withhold) return;  // test hook: stop feeding
                const int st = static_cast<int>(g % kStages);
                if (!waitw(&ctl->empty[st], ((g / kStages) & 1u) ^ 1u, ctl, a, lane)) {
                    stopped = true;
                    break;
                }
                const uint32_t bytes = static_cast<uint32_t>(min(per, p1 - c0)) * chunk;
                if (elect_one()) {
                    mbar_expect_tx(&ctl->full[st], bytes);
                    bulk_load(smem + st * kStageBytes, src + static_cast<int64_t>(c0) * chunk, bytes, &ctl->full[st]);
                }
                __syncwarp();
            }
        }
        cur = nxt;
    }
    // After an abort, let the copies already issued land before the CTA's shared memory goes away.
    if (lane == 0)
        for (uint32_t k = (g >= kStages ? g - kStages : 0); k < g; ++k)
            waitb(&ctl->full[k % kStages], (k / kStages) & 1u, ctl, a, false);
    __syncwarp();
}

// The whole of warp 1.
template <bool kGrouped>
__device__ void fxs_issuer(const FxsArgs& a, uint8_t* smem, FxsCtl* ctl, uint32_t tmem_base, int lane) {
    uint32_t g = 0;
    const uint32_t tmem = uni(tmem_base);
    const uint64_t d0 = smem_desc(smem_u32(smem), 256, 6);
    AccRing acc;
    for (uint32_t gi = 0;; ++gi) {
        const int slot = static_cast<int>(gi % kItemRing);
        if (!waitw(&ctl->item_full[slot], (gi / kItemRing) & 1u, ctl, a, lane)) goto done;
        {
            const BlockInfo bi = ctl->item[slot];
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctl->item_empty[slot]);
            const int k = uni(bi.k);
            if (k < 0) break;
            const int R = uni(fxs_rows(pops_of<kGrouped>(a, bi)));
            const uint64_t plane = static_cast<uint64_t>(2 * R);  // 32 R bytes, in 16-byte units
            const int per = 128 / R;
            // D = s32, A = B = s8, K-major, N = 4R, M = 128.
            const uint32_t id = (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(4 * R) >> 3 << 17) | (8u << 24);
            const int nch = (k + 31) / 32;
            for (int p0 = 0; p0 < nch; p0 += kSegChunks) {
                const int p1 = min(nch, p0 + kSegChunks);
                const int s = acc.slot(R);
                if (!waitw(&ctl->acc_empty[s], (acc.uses[s] & 1u) ^ 1u, ctl, a, lane)) goto done;
                ++acc.uses[s];
                if (R > 32) {
                    if (!waitw(&ctl->acc_empty[1], (acc.uses[1] & 1u) ^ 1u, ctl, a, lane)) goto done;
                    ++acc.uses[1];
                }
                tc_fence_after();
                const uint32_t d1 = tmem + static_cast<uint32_t>(s) * 256u, d2 = d1 + static_cast<uint32_t>(4 * R);
                for (int c0 = p0; c0 < p1; c0 += per, ++g) {
                    const int st = static_cast<int>(g % kStages);
                    if (!waitw(&ctl->full[st], (g / kStages) & 1u, ctl, a, lane)) goto done;
                    tc_fence_after();
                    const int n = min(per, p1 - c0);
                    if (elect_one()) {
                        uint64_t da = d0 + static_cast<uint64_t>(st) * (kStageBytes / 16);
                        for (int j = 0; j < n; ++j, da += kFxsPlanes * plane) {
                            const uint32_t f = c0 + j > p0 ? 1u : 0u;
                            mma_i8(d1, da + 2 * plane, da, id, f);
                            mma_i8(d2, da + 4 * plane, da + 5 * plane, id, f);
                        }
                        mma_commit(&ctl->empty[st]);
                        if (c0 + per >= p1) mma_commit(&ctl->acc_full[s]);
                    }
                    __syncwarp();
                }
            }
        }
    }
done:
    // Every MMA this warp issued completes before TMEM is released.
    if (elect_one()) {
        mma_commit(&ctl->drain);
        waitb(&ctl->drain, 0u, ctl, a, false);
    }
    __syncwarp();
}

// A barrier of the eight epilogue warps that also tells whether any of them has seen a wait
// run out: they share barriers, so they leave together.
__device__ __forceinline__ bool epi_any(bool stop) {
    int any;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.popc.u32 %0, 1, %2, p;\n\t}"
                 : "=r"(any)
                 : "r"(stop ? 1 : 0), "n"(kEpiThreads)
                 : "memory");
    return any != 0;
}

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory"); }

__device__ __forceinline__ int64_t wide(uint32_t v) { return static_cast<int64_t>(static_cast<int32_t>(v)); }

// One item, or one segment of it, out of the accumulators into this thread's entries of T and
// the counts: lane l < R is row l of X2 / E6, lane R <= l < 2R row l - R of X3 / M. The eight
// columns of a step are the same population columns of all eight stacked planes.
__device__ __forceinline__ void fxs_read(uint32_t d1, int R, int l, int h, bool add, int64_t* t_hi, int64_t* t_lo,
                                         int32_t* s_vp) {
    for (int j8 = h; j8 < R / 8; j8 += 2) {
        __syncwarp();
        uint32_t x[4][8], e[4][8];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            tmem_ld8(d1 + static_cast<uint32_t>(p * R + 8 * j8), x[p]);
            tmem_ld8(d1 + static_cast<uint32_t>(4 * R + p * R + 8 * j8), e[p]);
        }
        tmem_wait_ld();
        if (l >= 2 * R) continue;
        const bool hi = l >= R;
        int64_t* row = (hi ? t_hi + (l - R) * kPitch : t_lo + l * kPitch) + 8 * j8;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int64_t t_3 = 2 * ((wide(x[0][c]) + wide(e[1][c])) + ((wide(x[1][c]) + wide(e[2][c])) << 8) +
                                     ((wide(x[2][c]) + wide(e[3][c])) << 16)) +
                                (wide(x[3][c]) << 24);
            const int64_t t_2 = 2 * (wide(x[1][c]) + (wide(e[0][c]) << 24)) + (wide(x[2][c]) << 8);
            const int64_t t = hi ? t_3 : t_2;
            row[c] = add ? row[c] + t : t;
        }
        if (hi) {
            int32_t* vp = s_vp + (l - R) * kPitch + 8 * j8;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const int32_t n = static_cast<int32_t>(e[0][c]) >> 12;  // 64 * 64 per both-present SNP
                vp[c] = add ? vp[c] + n : n;
            }
        }
    }
}

template <bool kGrouped>
__device__ void fxs_epilogue(const FxsArgs& a, FxsCtl* ctl, uint32_t tmem, int64_t* t_hi, int64_t* t_lo, int32_t* s_vp,
                             int warp, int lane) {
    const int q = warp & 3;         // TMEM lane quarter this warp may access
    const int h = (warp - 2) >> 2;  // which half of the column steps
    const int l = q * 32 + lane;
    const int tid = (warp - 2) * 32 + lane;
    const uint32_t base = tmem + (static_cast<uint32_t>(q * 32) << 16);
    AccRing acc;
    BlockInfo bi;
    for (uint32_t gi = 0;; ++gi) {
        int ok = 1;
        if (lane == 0) ok = waitb(&ctl->item_full[gi % kItemRing], (gi / kItemRing) & 1u, ctl, a);
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (epi_any(ok == 0)) return;
        bi = ctl->item[gi % kItemRing];  // published to every lane by the barrier above
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->item_empty[gi % kItemRing]);
        if (bi.k < 0) return;
        const int P = pops_of<kGrouped>(a, bi);
        double* f2 = kGrouped ? a.groups[bi.grp].f2 : a.f2;
        double* vp = kGrouped ? a.groups[bi.grp].vpair : a.vpair;
        const int64_t slab = static_cast<int64_t>(P) * P * (bi.b - a.b_base);
        const int R = fxs_rows(P), nch = chunks_of(bi);
        for (int p0 = 0; p0 < nch; p0 += kSegChunks) {
            const int s = acc.slot(R);
            if (lane == 0) ok = waitb(&ctl->acc_full[s], acc.uses[s] & 1u, ctl, a);
            ++acc.uses[s];
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (epi_any(ok == 0)) return;
            tc_fence_after();
            if (q * 32 < 2 * R) fxs_read(base + static_cast<uint32_t>(s) * 256u, R, l, h, p0 > 0, t_hi, t_lo, s_vp);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&ctl->acc_empty[s]);
                if (R > 32) mbar_arrive(&ctl->acc_empty[1]);
            }
        }
        epi_sync();  // T and the counts of the item are complete
        for (int e = tid; e < P * P; e += kEpiThreads) {
            const int j = e / P, i = e - j * P;
            double f = 0.0, v = 0.0;
            if (nch > 0) {  // an empty block id: zeros (cpu_backend.cpp:234)
                const int64_t w = (t_hi[i * kPitch + j] + t_lo[i * kPitch + j] + t_hi[j * kPitch + i] + t_lo[j * kPitch + i]) >> 1;
                const int32_t n = s_vp[i * kPitch + j];
                const int32_t vk = n < a.rcp_max ? n : a.rcp_max;
                f = vk > 0 ? i64_to_f64(w) * kFxNumScale * __ldg(a.rcp + vk) : 0.0;
                v = static_cast<double>(n);
            }
            __stcs(f2 + slab + e, f);
            __stcs(vp + slab + e, v);
        }
        if (kGrouped && a.grp_done) {
            __syncwarp();
            if (lane == 0) {
                __threadfence();
                if (atomicAdd(a.grp_done + bi.grp, 1) == a.grp_items[bi.grp] * kEpiWarps - 1) a.grp_ns[bi.grp] = globaltimer();
            }
        }
        epi_sync();  // the exchange buffers are free again
    }
}

constexpr size_t kExchangeBytes = size_t(kFxsMaxPops) * kPitch * (2 * sizeof(int64_t) + sizeof(int32_t));
constexpr size_t kFxsSmemBytes = kStages * kStageBytes + kExchangeBytes + sizeof(FxsCtl) + 1024 + 64;
// A of a last chunk reads 128 rows from its fifth plane: past the stages, but inside the block's memory.
static_assert(kExchangeBytes >= 128 * 32, "A rows past the stages");

template <bool kGrouped>
__global__ void __launch_bounds__(kThreads, 1) f2_fxs_kernel(const __grid_constant__ FxsArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    int64_t* t_hi = reinterpret_cast<int64_t*>(smem + kStages * kStageBytes);
    int64_t* t_lo = t_hi + kFxsMaxPops * kPitch;
    int32_t* s_vp = reinterpret_cast<int32_t*>(t_lo + kFxsMaxPops * kPitch);
    FxsCtl* ctl = reinterpret_cast<FxsCtl*>(smem + ((kStages * kStageBytes + kExchangeBytes + 15) & ~size_t(15)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kItemRing; ++s) {
            mbar_init(&ctl->item_full[s], 1);
            mbar_init(&ctl->item_empty[s], 1 + kEpiWarps);
        }
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&ctl->acc_full[s], 1);
            mbar_init(&ctl->acc_empty[s], kEpiWarps);
        }
        mbar_init(&ctl->drain, 1);
        ctl->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(&ctl->tmem_base, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = ctl->tmem_base;
    if (warp < 2) {
        if (warp == 0) {
            fxs_producer<kGrouped>(a, smem, ctl, lane);
        } else {
            pdl_wait();
            fxs_issuer<kGrouped>(a, smem, ctl, tmem, lane);
        }
    } else {
        pdl_wait();
        fxs_epilogue<kGrouped>(a, ctl, tmem, t_hi, t_lo, s_vp, warp, lane);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem, kTmemCols);
    if (threadIdx.x == 0) reset_counter(a.next);
}

}  // namespace

void fxs_prepare() {
    const int b = static_cast<int>(kFxsSmemBytes);
    STPF2_CUDA(cudaFuncSetAttribute(f2_fxs_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
    STPF2_CUDA(cudaFuncSetAttribute(f2_fxs_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, b));
}

void launch_fxs(Ctx& c, const FxsLaunch& L, cudaStream_t s) {
    if (L.n_work <= 0) return;
    FxsArgs a{};
    a.images = L.images;
    a.work = L.work;
    a.n_work = L.n_work;
    a.P = L.P;
    a.f2 = L.f2;
    a.vpair = L.vpair;
    a.rcp = L.rcp;
    a.rcp_max = L.rcp_max;
    a.err = L.err;
    a.next = L.counter;
    a.b_base = L.b_base;
    a.timeout_ns = c.fx_tuning.timeout_ns;
    a.withhold = c.fx_tuning.withhold_stage;  // test hook: starves the issuer
    a.groups = L.groups;
    a.grp_done = L.grp_done;
    a.grp_ns = L.grp_ns;
    a.grp_items = L.grp_items;
    const int grid = std::min(c.sm_count, L.n_work);
    launch_kernel_on(L.groups ? f2_fxs_kernel<true> : f2_fxs_kernel<false>, static_cast<unsigned>(grid), kThreads,
                     kFxsSmemBytes, s, L.early, a);
    c.launches++;
}

}  // namespace stpf2
