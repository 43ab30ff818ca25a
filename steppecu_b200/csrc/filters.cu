// steppecu_b200/csrc/filters.cu
//
// extract-f2's per-SNP keep mask on the device (the regime-B decision of
// decode_compact_kernel.cu:39-68 in the reference): one thread per SNP reduces the
// populations in order p = 0..P-1 into the pooled summary of
// snp_summary_reduce.hpp:38-59 (q = ac / n by IEEE division, the product q * n rounded
// before it is added: no fused multiply-add, so the sum is the host's bit for bit), then
// applies keep_decision_pooled (snp_summary_reduce.hpp:64-79) and the population-coverage
// bound: drop a SNP when more than `maxmiss` of the populations have no call
// (extract_f2_core.cpp:245-259). The pooled missing-fraction test runs with its bound at 1,
// as extract-f2 sets it (cuda_backend_decode.cu:512-513), so it never drops anything.
//
// Two inputs: the packed exact counts of the SNP-major decode (population-major, ac2 | n <<
// 16), and FP64 q / n planes [P x M] (i + P * s), the layout of ComputeBackend::decode_af.
#include "stpf2_internal.cuh"

namespace stpf2 {

namespace {

// Allele-pair predicates of filter_decision.hpp:43-87, restated: A/C/G/T in either case,
// anything else is "no allele".
__device__ __forceinline__ char norm_allele(char a) {
    const char u = (a >= 'a' && a <= 'z') ? static_cast<char>(a - 0x20) : a;
    return (u == 'A' || u == 'C' || u == 'G' || u == 'T') ? u : '\0';
}
__device__ __forceinline__ char complement_of(char a) {
    switch (a) {
        case 'A': return 'T';
        case 'T': return 'A';
        case 'C': return 'G';
        case 'G': return 'C';
    }
    return '\0';
}
__device__ __forceinline__ bool purine(char a) { return a == 'A' || a == 'G'; }

struct Summary {
    double pooled_ref_count = 0.0, allele_count = 0.0, nonmissing = 0.0;
    int missing_pops = 0;
    // One population's q and n (n = 0: no call, q = 0), in population order.
    __device__ __forceinline__ void add(double q, double nd) {
        pooled_ref_count = __dadd_rn(pooled_ref_count, __dmul_rn(q, nd));
        allele_count = __dadd_rn(allele_count, nd);
        nonmissing = __dadd_rn(nonmissing, __ddiv_rn(nd, 2.0));  // called alleles / ploidy 2
        if (!(nd > 0.0)) ++missing_pops;
    }
};

__device__ __forceinline__ uint8_t decide(const Summary& sm, char ref, char alt, int chrom, const stp_snp_filter& f,
                                          int P, double total_indiv, double* out4, int64_t s, int64_t M) {
    const double ref_af = sm.allele_count > 0.0 ? __ddiv_rn(sm.pooled_ref_count, sm.allele_count) : 0.0;
    const double minor = (ref_af < 1.0 - ref_af) ? ref_af : 1.0 - ref_af;
    const double missing_frac = total_indiv > 0.0 ? 1.0 - __ddiv_rn(sm.nonmissing, total_indiv) : 1.0;
    if (out4) {
        out4[s] = ref_af;
        out4[M + s] = minor;
        out4[2 * M + s] = missing_frac;
        out4[3 * M + s] = sm.allele_count;
    }
    const char a = norm_allele(ref), b = norm_allele(alt);
    const bool multi = a == '\0' || b == '\0' || a == b;
    if (multi) return 0;
    if (f.strand_mode == STP_STRAND_DROP && a == complement_of(b)) return 0;
    if (!(minor >= f.maf_min)) return 0;
    if (!(missing_frac <= 1.0)) return 0;
    if (f.drop_monomorphic && minor == 0.0) return 0;
    if (f.transversions_only && purine(a) == purine(b)) return 0;  // a transition
    if (f.autosomes_only && !(chrom >= 1 && chrom <= 22)) return 0;
    if (f.maxmiss < 1.0 && static_cast<double>(sm.missing_pops) / static_cast<double>(P) > f.maxmiss) return 0;
    return 1;
}

// q * n of one population as the reference rounds it: q = ac / n by an IEEE division, then
// the product. The quotient comes from rn = 1 / n (itself an IEEE division, from a table):
// with q0 = ac * rn within 1.5 ulp of ac / n, the remainder ac - q0 n is exact (n < 2^16),
// and q0 + remainder * rn misses the true quotient by under 2^-52 ulp before its one rounding,
// while ac / n (ac a multiple of 1/2) is at least 2^-17 ulp from any rounding boundary: the
// correctly rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990).
__device__ __forceinline__ double pooled_term(double ac, double nd, double rn) {
    const double q0 = __dmul_rn(ac, rn);
    return __dmul_rn(__fma_rn(__fma_rn(-q0, nd, ac), rn, q0), nd);
}

// One thread per SNP, eight populations' counts in flight. The sum of q * n is taken in
// population order (its roundings are the reference's); the called alleles and missing
// populations are whole numbers, summed as such (the FP64 sums of them are exact). The pass
// was bound by two FP64 divisions per count and one load at a time: 604 -> 200 us for 200
// populations x 600,000 SNPs. kTable: the terms of every (n, a2) come from shared memory, one
// FP64 operation per count instead of eight (200 -> 97 us).
template <bool kTable>
__global__ void __launch_bounds__(256)
keep_mask_counts_kernel(const uint32_t* __restrict__ cnt, int64_t ld, int P, int64_t M, const double* __restrict__ rec_n,
                        int n_max, const char* __restrict__ ref, const char* __restrict__ alt,
                        const int32_t* __restrict__ chrom, stp_snp_filter f, double total_indiv,
                        uint8_t* __restrict__ keep, double* __restrict__ out4) {
    extern __shared__ double s_term[];  // kTable: n * t_ld + a2
    const uint32_t t_ld = static_cast<uint32_t>(2 * n_max + 1);
    auto term = [&](uint32_t n, uint32_t a2) {
        // Whole numbers below 2^16 to FP64 through the mantissa of 2^52, exactly.
        const double nd = __hiloint2double(0x43300000, static_cast<int>(n)) - 4503599627370496.0;
        const double a2d = __hiloint2double(0x43300000, static_cast<int>(a2)) - 4503599627370496.0;
        // n = 0: rn = 0 and ac = 0, a term of zero.
        return pooled_term(0.5 * a2d, nd, __ldg(rec_n + n));
    };
    if constexpr (kTable) {
        for (uint32_t k = threadIdx.x; k < static_cast<uint32_t>(n_max + 1) * t_ld; k += blockDim.x)
            s_term[k] = term(k / t_ld, k % t_ld);
        __syncthreads();
    }
    const int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= M) return;
    Summary sm;
    int64_t called = 0;
    const uint32_t* p = cnt + s;
    auto add = [&](uint32_t v) {
        const uint32_t n = v >> 16, a2 = v & 0xFFFFu;
        double t;
        if constexpr (kTable) t = s_term[n * t_ld + a2];
        else t = term(n, a2);
        sm.pooled_ref_count = __dadd_rn(sm.pooled_ref_count, t);
        called += n;
        sm.missing_pops += n == 0 ? 1 : 0;
    };
    constexpr int kAhead = 8;
    int i = 0;
    for (; i + kAhead <= P; i += kAhead, p += kAhead * ld) {
        uint32_t v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = __ldcs(p + u * ld);
#pragma unroll
        for (int u = 0; u < kAhead; ++u) add(v[u]);
    }
    for (; i < P; ++i, p += ld) add(__ldcs(p));
    sm.allele_count = static_cast<double>(called);
    sm.nonmissing = 0.5 * static_cast<double>(called);  // called alleles / ploidy 2
    keep[s] = decide(sm, ref[s], alt[s], chrom[s], f, P, total_indiv, out4, s, M);
}

__global__ void keep_mask_qn_kernel(const double* __restrict__ Q, const double* __restrict__ N, int P, int64_t M,
                                    const char* __restrict__ ref, const char* __restrict__ alt,
                                    const int32_t* __restrict__ chrom, stp_snp_filter f, double total_indiv,
                                    uint8_t* __restrict__ keep, double* __restrict__ out4) {
    const int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (s >= M) return;
    Summary sm;
    for (int i = 0; i < P; ++i) {
        const int64_t o = static_cast<int64_t>(i) + static_cast<int64_t>(P) * s;
        sm.add(Q[o], N[o]);
    }
    keep[s] = decide(sm, ref[s], alt[s], chrom[s], f, P, total_indiv, out4, s, M);
}

// Compaction of FP64 [P x M] planes to the kept columns: out column keep_idx[s] <- column s.
__global__ void compact_columns_kernel(const double* __restrict__ in, int P, int64_t M,
                                       const int64_t* __restrict__ dst_col, double* __restrict__ out) {
    const int64_t s = static_cast<int64_t>(blockIdx.x) * blockDim.y + threadIdx.y;
    if (s >= M) return;
    const int64_t d = dst_col[s];
    if (d < 0) return;
    for (int i = threadIdx.x; i < P; i += blockDim.x)
        out[static_cast<int64_t>(i) + static_cast<int64_t>(P) * d] = in[static_cast<int64_t>(i) + static_cast<int64_t>(P) * s];
}

}  // namespace

void launch_keep_mask_counts(Ctx& c, const uint32_t* cnt, int64_t ld, int P, int64_t M, const double* rec_n, int64_t n_max,
                             const char* ref, const char* alt, const int32_t* chrom, const stp_snp_filter& f,
                             double total_indiv, uint8_t* keep, double* out4, cudaStream_t s) {
    if (M <= 0) return;
    const unsigned grid = static_cast<unsigned>((M + 255) / 256);
    // The terms of populations of up to 15 samples are 16 KB at most: eight CTAs of 256
    // threads still fit an SM. A thread computes entries / 256 of them and saves a division per
    // population, so the table pays from about one population per 128 entries on (600,000 SNPs,
    // on the fly and table, us: 15 samples 16.1 and 18.2 at 12 populations, 19.2 and 20.1 at 16, 34.0
    // and 28.9 at 32; 10 samples 13.2 and 13.5 at 8, 16.2 and 15.6 at 12; 5 samples 10.0 and 10.0
    // at 4, 12.0 and 11.3 at 6; one sample 11.0 and 11.2 at 1, 11.5 and 10.9 at 4).
    const int64_t entries = n_max <= 31 ? (n_max + 1) * (2 * n_max + 1) : 0;
    if (entries > 0 && P >= 3 + entries / 128)
        keep_mask_counts_kernel<true><<<grid, 256, static_cast<size_t>(entries) * sizeof(double), s>>>(
            cnt, ld, P, M, rec_n, static_cast<int>(n_max), ref, alt, chrom, f, total_indiv, keep, out4);
    else
        keep_mask_counts_kernel<false><<<grid, 256, 0, s>>>(cnt, ld, P, M, rec_n, 0, ref, alt, chrom, f, total_indiv, keep, out4);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

void launch_keep_mask_qn(Ctx& c, const double* Q, const double* N, int P, int64_t M, const char* ref, const char* alt,
                         const int32_t* chrom, const stp_snp_filter& f, double total_indiv, uint8_t* keep,
                         double* out4, cudaStream_t s) {
    if (M <= 0) return;
    keep_mask_qn_kernel<<<static_cast<unsigned>((M + 255) / 256), 256, 0, s>>>(Q, N, P, M, ref, alt, chrom, f,
                                                                               total_indiv, keep, out4);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

void launch_compact_columns(Ctx& c, const double* in, int P, int64_t M, const int64_t* dst_col, double* out,
                            cudaStream_t s) {
    if (M <= 0 || P <= 0) return;
    const dim3 block(32, 8);
    compact_columns_kernel<<<static_cast<unsigned>((M + 7) / 8), block, 0, s>>>(in, P, M, dst_col, out);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

}  // namespace stpf2
