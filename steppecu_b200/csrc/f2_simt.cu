// steppecu_b200/csrc/f2_simt.cu
//
// The plain FP32 SIMT contraction (no tensor cores): the comparison form of the f2
// extraction. For every (block, 64x64 tile pair ti <= tj) one CTA accumulates, over the
// block's SNP columns,
//     acc(i,j)   = sum_s (Ah_i M_j + M_i Ah_j - Pt_i Pt_j)     (FP32, drained to FP64 every
//                                                              16 SNPs)
//     vpair(i,j) = sum_s M_i M_j                                (exact: whole numbers)
// and writes f2 = 2*acc/vpair (0 when vpair = 0) and vpair into both (i,j) and (j,i) of
// the block's slab: the per-block work of compute_f2_blocks (cpu_backend.cpp:217-264;
// f2_estimator.hpp:38-46 for the numerator and the divide).
#include "stpf2_internal.cuh"

namespace stpf2 {

namespace {

constexpr int kT = 64;        // tile edge (populations)
constexpr int kKc = 16;       // SNP columns per shared-memory chunk
constexpr int kThreads = 256; // 16 x 16 threads, 4 x 4 outputs each
constexpr int kPitch = kT + 4;

struct SimtOps {
    const float* pt;
    const float* ah;
    const uint8_t* m;
    int64_t ld;
    int P;
};

// Two FP32 multiply-adds of one instruction, each rounded as fmaf.
__device__ __forceinline__ void ffma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}

// What one thread stages of a chunk: four columns of one row.
struct Staged {
    float4 p, a;
    uint32_t m;
};

__device__ __forceinline__ Staged stage_load(const SimtOps& op, int row, int64_t col) {
    Staged s{make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f), 0u};
    if (row < op.P) {
        const int64_t o = static_cast<int64_t>(row) * op.ld + col;
        s.p = __ldg(reinterpret_cast<const float4*>(op.pt + o));
        s.a = __ldg(reinterpret_cast<const float4*>(op.ah + o));
        s.m = __ldg(reinterpret_cast<const uint32_t*>(op.m + o));
    }
    return s;
}

// Bound by shared-memory loads (six 16-byte loads per SNP for the 48 multiply-adds of a
// thread's 4 x 4 outputs): 3 multiply-adds per SNP and pair, as f32x2 pairs over two columns,
// the row operands paired with themselves in registers (held twice in shared memory, at nine
// loads per SNP, the kernel took 573 us instead). The counts are whole numbers and go through
// byte dot products on the integer pipe instead of a fourth multiply-add. The next chunk's
// loads are in flight while one is computed. Warps whose eight rows lie past the last
// population do nothing, and the tile side with fewer populations is the row side. 631 ->
// 492 us for 100 populations x 200,000 SNPs.
__global__ void __launch_bounds__(kThreads, 2)
f2_simt_kernel(const WorkItem* __restrict__ items, const BlockInfo* __restrict__ blocks,
               SimtOps op, double* __restrict__ f2, double* __restrict__ vpair) {
    __shared__ __align__(16) float rP[kKc][kPitch], rA[kKc][kPitch], rM[kKc][kPitch];
    __shared__ __align__(16) float cP[kKc][kPitch], cA[kKc][kPitch], cM[kKc][kPitch];
    __shared__ __align__(16) uint32_t rB[kKc / 4][kT], cB[kKc / 4][kT];  // M bytes of four SNPs

    const WorkItem it = items[blockIdx.x];
    const BlockInfo bi = blocks[it.blk];
    const int P = op.P;
    const bool swapped = min(kT, P - it.tj * kT) < min(kT, P - it.ti * kT);
    const int row0 = (swapped ? it.tj : it.ti) * kT, col0 = (swapped ? it.ti : it.tj) * kT;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const bool active = row0 + (ty & ~1) * 4 < P;  // the same for a warp
    // The sums keep the order Ah_i M_j, M_i Ah_j, Pt_i Pt_j with i of row tile ti.
    float(*const r1)[kPitch] = swapped ? rM : rA;
    float(*const r2)[kPitch] = swapped ? rA : rM;
    float(*const c1)[kPitch] = swapped ? cA : cM;
    float(*const c2)[kPitch] = swapped ? cM : cA;

    double dacc[4][4];
    uint32_t vp[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            dacc[r][c] = 0.0;
            vp[r][c] = 0u;
        }

    const int sr = threadIdx.x >> 2, k4 = threadIdx.x & 3;
    const int kpad = (bi.k + kKc - 1) / kKc * kKc;
    Staged nr{}, nc{};
    if (kpad > 0) {
        nr = stage_load(op, row0 + sr, bi.col + 4 * k4);
        nc = stage_load(op, col0 + sr, bi.col + 4 * k4);
    }
    for (int k0 = 0; k0 < kpad; k0 += kKc) {
        {
            const float rp[4] = {nr.p.x, nr.p.y, nr.p.z, nr.p.w}, ra[4] = {nr.a.x, nr.a.y, nr.a.z, nr.a.w};
            const float cp[4] = {nc.p.x, nc.p.y, nc.p.z, nc.p.w}, ca[4] = {nc.a.x, nc.a.y, nc.a.z, nc.a.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = 4 * k4 + q;
                const float rm = static_cast<float>((nr.m >> (8 * q)) & 0xffu), cm = static_cast<float>((nc.m >> (8 * q)) & 0xffu);
                rP[k][sr] = -rp[q];
                rA[k][sr] = ra[q];
                rM[k][sr] = rm;
                cP[k][sr] = cp[q];
                cA[k][sr] = ca[q];
                cM[k][sr] = cm;
            }
            rB[k4][sr] = nr.m;
            cB[k4][sr] = nc.m;
        }
        __syncthreads();
        if (k0 + kKc < kpad) {
            nr = stage_load(op, row0 + sr, bi.col + k0 + kKc + 4 * k4);
            nc = stage_load(op, col0 + sr, bi.col + k0 + kKc + 4 * k4);
        }
        if (active) {
            unsigned long long acc[4][2];
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[r][0] = acc[r][1] = 0ull;
#pragma unroll 4
            for (int k = 0; k < kKc; ++k) {
                const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&c1[k][tx * 4]);
                const ulonglong2 b2 = *reinterpret_cast<const ulonglong2*>(&c2[k][tx * 4]);
                const ulonglong2 bp = *reinterpret_cast<const ulonglong2*>(&cP[k][tx * 4]);
                const float4 a1 = *reinterpret_cast<const float4*>(&r1[k][ty * 4]);
                const float4 a2 = *reinterpret_cast<const float4*>(&r2[k][ty * 4]);
                const float4 ap = *reinterpret_cast<const float4*>(&rP[k][ty * 4]);
                const float A1[4] = {a1.x, a1.y, a1.z, a1.w}, A2[4] = {a2.x, a2.y, a2.z, a2.w};
                const float AP[4] = {ap.x, ap.y, ap.z, ap.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const unsigned long long x1 = twice(A1[r]), x2 = twice(A2[r]), xp = twice(AP[r]);
                    ffma2(acc[r][0], x1, b1.x);
                    ffma2(acc[r][1], x1, b1.y);
                    ffma2(acc[r][0], x2, b2.x);
                    ffma2(acc[r][1], x2, b2.y);
                    ffma2(acc[r][0], xp, bp.x);
                    ffma2(acc[r][1], xp, bp.y);
                }
            }
#pragma unroll
            for (int w = 0; w < kKc / 4; ++w) {
                const uint4 am = *reinterpret_cast<const uint4*>(&rB[w][ty * 4]);
                const uint4 bm = *reinterpret_cast<const uint4*>(&cB[w][tx * 4]);
                const uint32_t AM[4] = {am.x, am.y, am.z, am.w}, BM[4] = {bm.x, bm.y, bm.z, bm.w};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) vp[r][c] = __dp4a(AM[r], BM[c], vp[r][c]);
            }
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    dacc[r][2 * h] += static_cast<double>(__uint_as_float(static_cast<uint32_t>(acc[r][h])));
                    dacc[r][2 * h + 1] += static_cast<double>(__uint_as_float(static_cast<uint32_t>(acc[r][h] >> 32)));
                }
        }
        __syncthreads();
    }

    // Epilogue: finalize_f2 (f2_estimator.hpp:42-46) into both triangles of slab b.
    const int64_t slab = static_cast<int64_t>(P) * P * bi.b;
    const bool diag = it.ti == it.tj;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = swapped ? col0 + tx * 4 + c : row0 + ty * 4 + r;
            const int j = swapped ? row0 + ty * 4 + r : col0 + tx * 4 + c;
            if (i >= P || j >= P) continue;
            if (diag && i > j) continue;
            const double v = static_cast<double>(vp[r][c]);
            const double val = (v > 0.0) ? (2.0 * dacc[r][c]) / v : 0.0;
            const int64_t ij = slab + i + static_cast<int64_t>(P) * j;
            const int64_t ji = slab + j + static_cast<int64_t>(P) * i;
            f2[ij] = val;
            vpair[ij] = v;
            f2[ji] = val;
            vpair[ji] = v;
        }
    }
}

}  // namespace

void launch_f2_simt(Ctx& c, const WorkItem* items, int n_items, const BlockInfo* blocks,
                    const OperandPlanes& op, double* f2, double* vpair, cudaStream_t s) {
    if (n_items <= 0) return;
    if (op.fmt != OpFmt::F32) fail(STP_INVALID_ARGUMENT, "f2_simt: needs FP32 operand planes");
    SimtOps o;
    o.pt = static_cast<const float*>(op.planes);
    o.ah = o.pt + static_cast<int64_t>(op.P) * op.ld;
    o.m = op.m_u8;
    o.ld = op.ld;
    o.P = op.P;
    f2_simt_kernel<<<static_cast<unsigned>(n_items), kThreads, 0, s>>>(items, blocks, o, f2, vpair);
    STPF2_CUDA(cudaGetLastError());
    c.launches++;
}

int simt_tile() { return kT; }

}  // namespace stpf2
