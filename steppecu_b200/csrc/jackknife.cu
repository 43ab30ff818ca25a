// steppecu_b200/csrc/jackknife.cu
//
// FP64 block jackknife over per-block values: the block-size-weighted total, leave-one-out
// values, their weighted mean and the AT2 jackknife variance of cpu_backend.cpp:2674-2720
// (compute_loo_and_total) and :2273-2306 (jackknife_diag). The reference sums in long
// double; the device has no wider type, so every sum here is a compensated (two-sum) FP64
// sum, whose error stays at the level of one FP64 rounding of the result.
#include <algorithm>

#include "stpf2_internal.cuh"

namespace stpf2 {

namespace {

struct CSum {  // Neumaier compensated sum
    double s = 0.0, c = 0.0;
    __device__ void add(double x) {
        const double t = s + x;
        c += (fabs(s) >= fabs(x)) ? ((s - t) + x) : ((x - t) + s);
        s = t;
    }
    __device__ double value() const { return s + c; }
};

// 32 items (a lane each, so every load is 256 contiguous bytes) per kWarps warps, which take
// the blocks round robin; each sum is combined over the warps through shared memory, the
// compensations included. What depends on the block alone (its weight, n / bl, the root and the
// reciprocals of what the items divide by) is computed once per warp and block, one block per
// lane, and shuffled; an item's quotient is the product with the reciprocal and one correction
// by the exact remainder (Markstein's division, 1990: with a reciprocal rounded to nearest the
// corrected quotient is the rounded one for all but extreme exponents).
//
// 16 warps where items alone leave the chip idle: 5,000 items x 714 blocks are 157 CTAs instead of
// 40 and a 16th of the serial chain of compensated adds (a thread per item 785 us at 700 blocks, a
// warp per 32 items 295, 16 warps 74; 32 warps, one CTA to an SM and so a wave and a bit, 98). One
// warp, with no barrier and no shared memory and kJkGroups such to a CTA, where there are items
// enough or few blocks: 1,000,000 items x 24 blocks 187 us (16 warps 828, a thread per item 273),
// x 2 blocks 33 (541, 31), 20 items x 12 blocks 8 each way. See jk_single_warp for the line.
constexpr int kJkWarps = 16, kJkGroups = 4;

struct JkBlock {
    double bl, rel, w, rw;   // bl, bl / n, 1 - bl / n, 1 / w
    double h, root, rroot;   // n / bl, sqrt(n / bl - 1), 1 / root
};

template <int kWarps>
using JkParts = double[2][kWarps][32];  // (sum, compensation) of each warp and item

__device__ __forceinline__ double jk_div(double a, double b, double rb) {
    const double q = a * rb;
    return fma(fma(-q, b, a), rb, q);
}

// N sums over the warps, in warp order, warp k adding sum k for all: every warp adding them
// for itself filled the FP64 pipe with the same compensated additions once per warp (144 us with
// 32 warps, 98 us without).
template <int kWarps, int N>
__device__ __forceinline__ void jk_totals(const CSum (&v)[N], double (&tot)[N], JkParts<kWarps>* p, int warp, int lane) {
    if constexpr (kWarps == 1) {
#pragma unroll
        for (int k = 0; k < N; ++k) tot[k] = v[k].value();
        return;
    }
    __syncthreads();  // the previous totals have been read
#pragma unroll
    for (int k = 0; k < N; ++k) {
        p[k][0][warp][lane] = v[k].s;
        p[k][1][warp][lane] = v[k].c;
    }
    __syncthreads();
    if (warp < N) {
        CSum t;
#pragma unroll 4
        for (int w = 0; w < kWarps; ++w) {
            t.add(p[warp][0][w][lane]);
            t.add(p[warp][1][w][lane]);
        }
        p[warp][0][0][lane] = t.value();
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < N; ++k) tot[k] = p[k][0][0][lane];
}

// f(block, value) for every block of this warp, in block order.
template <bool kRoot, int kWarps, class F>
__device__ __forceinline__ void jk_blocks(const double* __restrict__ x, const int32_t* __restrict__ bl, int64_t m, int nb,
                                          double n, int64_t k, bool real, int warp, int lane, F&& f) {
    for (int b0 = warp; b0 < nb; b0 += 32 * kWarps) {
        JkBlock mine{1.0, 0.0, 1.0, 1.0, 0.0, 0.0, 0.0};
        const int bm = b0 + lane * kWarps;
        if (bm < nb) {
            mine.bl = static_cast<double>(bl[bm]);
            mine.rel = mine.bl / n;
            mine.w = 1.0 - mine.rel;
            mine.rw = 1.0 / mine.w;
            if constexpr (kRoot) {
                mine.h = n / mine.bl;
                mine.root = sqrt(mine.h - 1.0);
                mine.rroot = 1.0 / mine.root;
            }
        }
        const int cnt = min(32, (nb - b0 + kWarps - 1) / kWarps);
#pragma unroll 4
        for (int j = 0; j < cnt; ++j) {
            JkBlock t;
            t.bl = __shfl_sync(0xffffffffu, mine.bl, j);
            t.rel = __shfl_sync(0xffffffffu, mine.rel, j);
            t.w = __shfl_sync(0xffffffffu, mine.w, j);
            t.rw = __shfl_sync(0xffffffffu, mine.rw, j);
            if constexpr (kRoot) {
                t.h = __shfl_sync(0xffffffffu, mine.h, j);
                t.root = __shfl_sync(0xffffffffu, mine.root, j);
                t.rroot = __shfl_sync(0xffffffffu, mine.rroot, j);
            }
            f(t, real ? x[k + m * (b0 + j * kWarps)] : 0.0);
        }
    }
}

template <int kWarps>
__global__ void __launch_bounds__(kWarps == 1 ? 32 * kJkGroups : 32 * kWarps)
jackknife_kernel(const double* __restrict__ x, const int32_t* __restrict__ bl, int64_t m, int nb, double n, double* est,
                 double* var) {
    __shared__ JkParts<kWarps> parts[kWarps == 1 ? 1 : 3];
    double total[1], totals[3];
    const int lane = threadIdx.x & 31;
    // A single warp's 32 items are its own: kJkGroups of them to a CTA, with no barrier.
    const int warp = kWarps == 1 ? 0 : threadIdx.x >> 5;
    const int64_t group = kWarps == 1 ? static_cast<int64_t>(blockIdx.x) * kJkGroups + (threadIdx.x >> 5) : blockIdx.x;
    const int64_t k = group * 32 + lane;
    const bool real = k < m;
    if (kWarps == 1 && group * 32 >= m) return;
    CSum num[1];
    jk_blocks<false, kWarps>(x, bl, m, nb, n, k, real, warp, lane, [&](const JkBlock& t, double v) { num[0].add(v * t.bl); });
    jk_totals<kWarps>(num, total, parts, warp, lane);
    const double tot = total[0] / n;
    // Weighted mean of the leave-one-out values (weights 1 - bl/n).
    CSum w3[3];
    jk_blocks<false, kWarps>(x, bl, m, nb, n, k, real, warp, lane, [&](const JkBlock& t, double v) {
        const double loo = jk_div(tot - v * t.rel, t.w, t.rw);
        w3[0].add(loo * t.w);
        w3[1].add(t.w);
        w3[2].add(loo * t.bl);
    });
    jk_totals<kWarps>(w3, totals, parts, warp, lane);
    const double totline = totals[0] / totals[1];
    const double wbl_n = totals[2] / n;
    CSum diff[1];
    jk_blocks<false, kWarps>(x, bl, m, nb, n, k, real, warp, lane, [&](const JkBlock& t, double v) {
        diff[0].add(totline - jk_div(tot - v * t.rel, t.w, t.rw));
    });
    jk_totals<kWarps>(diff, total, parts, warp, lane);
    const double term1 = (total[0] / nb) * nb;
    const double e = term1 + wbl_n;
    CSum acc[1];
    jk_blocks<true, kWarps>(x, bl, m, nb, n, k, real, warp, lane, [&](const JkBlock& t, double v) {
        const double loo = jk_div(tot - v * t.rel, t.w, t.rw);
        const double xtau = jk_div(e * t.h - loo * (t.h - 1.0) - totline, t.root, t.rroot);
        acc[0].add(xtau * xtau);
    });
    jk_totals<kWarps>(acc, total, parts, warp, lane);
    if (real && warp == 0) {
        est[k] = e;
        var[k] = total[0] / nb;
    }
}

// survivor_blocks (cpu_backend.cpp:124-151): one CTA per block; keep[b] = 0 when block b
// has a missing pair (vpair not > 0, f2_estimator.hpp:49-51) and a present one.
__global__ void survivor_kernel(const double* __restrict__ vpair, int64_t slab, int32_t* __restrict__ keep) {
    const int64_t b = blockIdx.x;
    const double* v = vpair + slab * b;
    int missing = 0, present = 0;
    // Four independent loads per thread in flight: the pass streams every slab once.
    for (int64_t e = threadIdx.x; e < slab; e += 4 * static_cast<int64_t>(blockDim.x)) {
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t k = e + static_cast<int64_t>(u) * blockDim.x;
            x[u] = k < slab ? __ldg(v + k) : 0.0;  // not loaded, and not counted, past the slab
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t k = e + static_cast<int64_t>(u) * blockDim.x;
            if (k < slab) {
                const bool p = x[u] > 0.0;
                present |= p;
                missing |= !p;
            }
        }
    }
    missing = __syncthreads_or(missing);
    present = __syncthreads_or(present);
    if (threadIdx.x == 0) keep[b] = !(missing && present);
}

// assemble_f4_quartets / assemble_f3_triples / assemble_f4 (cpu_backend.cpp:2064-2216):
// x[k + m*bs] for statistic k over surviving block bs (block surv[bs]), each sum in the
// reference's operation order.
__global__ void fstat_assemble_kernel(const double* __restrict__ f2, int64_t P, const int32_t* __restrict__ surv,
                                      int ns, int kind, const int32_t* __restrict__ idx, int64_t n_stat,
                                      int64_t m, int64_t nr, double* __restrict__ x) {
    const int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= m * ns) return;
    const int64_t k = t % m, bs = t / m;
    const double* f = f2 + P * P * surv[bs];
    auto at = [&](int i, int j) { return f[i + P * j]; };
    double v;
    if (kind == 0) {
        const int p1 = idx[4 * k], p2 = idx[4 * k + 1], p3 = idx[4 * k + 2], p4 = idx[4 * k + 3];
        v = 0.5 * (at(p2, p3) + at(p1, p4) - at(p1, p3) - at(p2, p4));
    } else if (kind == 1) {
        const int pc = idx[3 * k], pa = idx[3 * k + 1], pb = idx[3 * k + 2];
        v = 0.5 * (at(pc, pa) + at(pc, pb) - at(pa, pb));
    } else {
        const int64_t i = k / nr, j = k % nr;  // k = j + nr*i
        const int L0 = idx[0], R0 = idx[n_stat], Li = idx[1 + i], Rj = idx[n_stat + 1 + j];
        v = 0.5 * (at(Li, R0) + at(L0, Rj) - at(L0, R0) - at(Li, Rj));
    }
    x[t] = v;
}

}  // namespace

// Up to 12 blocks 16 warps have nothing to share (1 to 5,000 items: 8.3 us or less against 8.3 to
// 10.4). Beyond, the line between the forms is at about 250 items per block, measured on both
// sides: 5,000 items 10.3 and 10.4 us at 16 blocks, 12.4 and 10.8 at 24; 20,000 items 29.6 and 30.8
// at 64, 59.5 and 43.2 at 128; 50,000 items 107 and 127 at 200, 646 and 448 at 700; from 100,000
// items on one warp is the faster for any number of blocks (759 and 847 at 700).
static bool jk_single_warp(int64_t m, int nb) { return nb <= 12 || m >= 250 * static_cast<int64_t>(std::min(nb, 400)); }

void launch_jackknife(Ctx& c, const double* x, const int32_t* block_sizes, const std::vector<int32_t>& sizes,
                      int64_t m, double* est, double* var, cudaStream_t s) {
    const int nb = static_cast<int>(sizes.size());
    if (m <= 0 || nb <= 0) return;
    // n = sum of block sizes (exact in FP64 for any realistic SNP count).
    double n = 0.0;
    for (int32_t v : sizes) n += static_cast<double>(v);
    if (jk_single_warp(m, nb))
        jackknife_kernel<1><<<static_cast<unsigned>((m + 32 * kJkGroups - 1) / (32 * kJkGroups)), 32 * kJkGroups, 0, s>>>(
            x, block_sizes, m, nb, n, est, var);
    else
        jackknife_kernel<kJkWarps><<<static_cast<unsigned>((m + 31) / 32), 32 * kJkWarps, 0, s>>>(x, block_sizes, m, nb, n,
                                                                                                est, var);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

void launch_survivors(Ctx& c, const double* vpair, int P, int nb, int32_t* keep, cudaStream_t s) {
    if (nb <= 0) return;
    survivor_kernel<<<nb, 256, 0, s>>>(vpair, static_cast<int64_t>(P) * P, keep);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

void launch_fstat_assemble(Ctx& c, const double* f2, int P, const int32_t* surv, int ns, int kind,
                           const int32_t* idx, int64_t n_stat, int64_t m, int64_t nr, double* x, cudaStream_t s) {
    if (m <= 0 || ns <= 0) return;
    const int64_t n = m * ns;
    fstat_assemble_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(f2, P, surv, ns, kind, idx, n_stat, m, nr, x);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

}  // namespace stpf2
