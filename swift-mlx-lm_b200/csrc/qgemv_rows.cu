// Q4 group-64 products of 2..16 activation rows for sm_100a (decode steps of small batches, `gemm_q4_g64` for few sequence
// positions, Generator/MetalSourceGenerator+Quantized.swift:88-156, which re-reads the weights once per position).
//
// What bounds it: the 0.5625 bytes per weight that cross HBM once, and behind that the instructions per weight: at the copy peak
// an SM takes in 41 weights per clock, so a 16 x 64 tile may cost about 100 warp instructions. Hence
//   * activations in registers: a warp owns one stage (four 64-column groups) of K for the whole launch, loads its B fragments
//     once (32 bytes per lane: two halves would fetch every sector twice) and then only streams weights; the sums of the groups,
//     which the zero points multiply, come out of a product with ones;
//   * the warps of a group cover K side by side, a row tile (16 rows) is one round: each warp contracts its stage, the parts meet
//     in shared memory behind one named barrier per round (two buffers), so nothing of a row tile goes through global memory;
//   * K beyond 16 stages (4096 columns) is cut over the CTAs of a cluster, which send their parts to the CTA that finishes a
//     column through distributed shared memory; the cluster barrier of a round is waited for behind the next round's products;
//   * row tiles are dealt cyclically, so that the GPU reads one contiguous window of the matrix per round, through a cp.async ring
//     per warp that is filled before the preceding kernel has finished.
// fp16 mma.m16n8k16 runs at 970 of the nominal 1024 FMA per clock and SM here; 16 rows at the copy peak need 656.
// Measured, 14336 x 4096 at 16 rows back to back: 20.2 us with the kernel that staged, converted and read the activations in shared
// memory (0.21 instructions per weight), 17.2 us (1.9 TB/s of weights); 28672 x 4096 with the norm in front 74 us in one launch of
// that kernel (every CTA read and normed all rows), about 31 us as norm and product. What is left is the start of a launch (128 KB of
// activations per SM through L2) and issue slots, half of them empty.
//
// Arithmetic: a nibble becomes the fp16 number q - 8 (exact; sums of 1024 + q, which save one instruction per register, lose seven
// bits to the cancellation), activations are converted bf16 -> fp16 times a power of two per warp and row (exact unless an element
// is 2^-24 below the largest of its 256), a group's sum is scale * acc + (zero + 8 scale) * sum(x) in fp32.
#include <algorithm>

#include <cooperative_groups.h>

#include "swlm_internal.h"

namespace cg = cooperative_groups;

namespace swlm {
namespace {

constexpr int kRowsWarps = 16;                 // per CTA
constexpr int kRowsStages = 4;                 // ring depth per warp
constexpr int kRowsStageBytes = 4 * 512 + 256; // four tiles and their scale / zero pairs
constexpr int kRowsPitch = 20;                 // floats per column of a part (16 rows): writes of a fragment meet no bank twice
constexpr int kRowsMaxCluster = 8;
constexpr int kRowsSMs = 148;

struct QRowsParams {
    const uint4* tiles;
    const uint4* sb;
    int row_tiles, kt4;
    const __nv_bfloat16* x;
    int x_stride, k, m;
    __nv_bfloat16* y[3];
    int y_stride[3], seg_end[3];
    int gated_act;
    bool wide;                    // every row of x starts on 32 bytes
    int kc, groups, sk, rounds;   // stages per CTA at most, groups of warps, CTAs along K, rounds of every group
};

__device__ __forceinline__ void rows_cp16(unsigned dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ uint4 rows_lds128(unsigned sa) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(sa));
    return v;
}
__device__ __forceinline__ void rows_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void rows_mma_first(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// q - 8 of the low (high) nibbles of a byte pair as fp16, exact: 1024 + q less 1032; (1024 + 16 q) / 16 less 72
__device__ __forceinline__ unsigned rows_low(unsigned w) {
    const unsigned v = (w & 0x000F000Fu) | 0x64006400u, c = 0x64086408u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&c));
    return *reinterpret_cast<const unsigned*>(&h);
}
__device__ __forceinline__ unsigned rows_high(unsigned w) {
    const unsigned v = (w & 0x00F000F0u) | 0x64006400u, f = 0x2C002C00u, c = 0xD480D480u;
    const __half2 h = __hfma2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&f), *reinterpret_cast<const __half2*>(&c));
    return *reinterpret_cast<const unsigned*>(&h);
}
// 16 bf16 of a row: one 32-byte load where every row starts on 32 bytes (two halves fetch each sector twice)
__device__ __forceinline__ void rows_load32(const __nv_bfloat16* src, bool wide, unsigned (&v)[8]) {
    if (wide) {
        asm volatile("ld.global.cg.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(src) : "memory");
    } else {
        const uint4 a = __ldcg(reinterpret_cast<const uint4*>(src)), b = __ldcg(reinterpret_cast<const uint4*>(src) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}
template <bool F16SB>
__device__ __forceinline__ float rows_scale(unsigned pair) { return F16SB ? __half2float(__ushort_as_half((unsigned short)(pair & 0xFFFFu))) : __uint_as_float(pair << 16); }
template <bool F16SB>
__device__ __forceinline__ float rows_zero(unsigned pair) { return F16SB ? __half2float(__ushort_as_half((unsigned short)(pair >> 16))) : __uint_as_float(pair & 0xFFFF0000u); }

// one finished pair of sums: EPI_STORE: rows r and r + 8 of a tile; EPI_SWIGLU: a gate row and its up row
template <int EPI>
__device__ __forceinline__ void rows_finish(const QRowsParams& p, int rt, int r, int col, float lo, float hi) {
    if (col >= p.m) return;
    if (EPI == QGEMV_EPI_STORE) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = rt * 16 + r + 8 * h;
            const __nv_bfloat16 v = __float2bfloat16_rn(h ? hi : lo);
            if (row < p.seg_end[0]) p.y[0][(size_t)col * p.y_stride[0] + row] = v;
            else if (row < p.seg_end[1]) p.y[1][(size_t)col * p.y_stride[1] + (row - p.seg_end[0])] = v;
            else if (row < p.seg_end[2]) p.y[2][(size_t)col * p.y_stride[2] + (row - p.seg_end[1])] = v;
        }
    } else {
        // both are rounded to bf16 first because the reference stores them to bf16 scratch before `swiglu` reads them
        // (Primitives/ElementwiseFragment.swift:49-54)
        const int row = rt * 8 + r;
        if (row < p.seg_end[0]) {
            const float gate = __bfloat162float(__float2bfloat16_rn(lo)), up = __bfloat162float(__float2bfloat16_rn(hi));
            p.y[0][(size_t)col * p.y_stride[0] + row] = __float2bfloat16_rn(gated_activation(gate, up, p.gated_act));
        }
    }
}

// shared memory: ring | group sums of the activations [warp][4][COLS] | parts [2][warp][COLS][pitch] | received [2][groups, at most 8][sk][COLS / sk][16]
template <int NT>
constexpr size_t rows_smem_bytes() {
    return (size_t)kRowsWarps * (kRowsStages * kRowsStageBytes + 4 * 8 * NT * 4 + 2 * 8 * NT * kRowsPitch * 4) + (size_t)2 * (kRowsWarps / 2) * 8 * NT * 16 * 4;
}

template <int NT, int EPI, bool F16SB>
__global__ void __launch_bounds__(kRowsWarps * 32, 1) qgemv_rows_kernel(const QRowsParams p) {
    constexpr int COLS = 8 * NT;
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int rank = p.sk > 1 ? (int)blockIdx.x % p.sk : 0, cluster_id = (int)blockIdx.x / p.sk, clusters = (int)gridDim.x / p.sk;
    const int grp = warp / p.kc, wk = warp - grp * p.kc;
    const int k_lo = (int)((long long)rank * p.kt4 / p.sk), kc = (int)((long long)(rank + 1) * p.kt4 / p.sk) - k_lo;   // this CTA's stages
    const bool in_group = grp < p.groups, works = in_group && wk < kc;
    const int stage = k_lo + wk;
    const int vb = grp * clusters + cluster_id, vgrid = clusters * p.groups;

    const unsigned ring = (unsigned)__cvta_generic_to_shared(smem) + warp * (kRowsStages * kRowsStageBytes);
    float* const xs = reinterpret_cast<float*>(smem + kRowsWarps * kRowsStages * kRowsStageBytes) + warp * (4 * COLS);
    float* const parts = reinterpret_cast<float*>(smem + kRowsWarps * (kRowsStages * kRowsStageBytes + 4 * COLS * 4));
    float* const recv = parts + 2 * kRowsWarps * COLS * kRowsPitch;

    // the issue side runs kRowsStages - 1 rounds ahead; a round's stage lies one row tile stride behind the last one's
    const uint4* w_src = p.tiles + ((size_t)vb * p.kt4 + stage) * 128 + lane;
    const uint4* s_src = p.sb + ((size_t)vb * p.kt4 + stage) * 16 + lane;
    const size_t w_step = (size_t)vgrid * p.kt4 * 128, s_step = (size_t)vgrid * p.kt4 * 16;
    int i_rt = works ? vb : p.row_tiles;
    auto issue = [&](int slot) {
        if (i_rt < p.row_tiles) {
            const unsigned dst = ring + slot * kRowsStageBytes + lane * 16;
#pragma unroll
            for (int q = 0; q < 4; ++q) rows_cp16(dst + q * 512, w_src + q * 32);
            if (lane < 16) rows_cp16(dst + 2048, s_src);
            w_src += w_step; s_src += s_step; i_rt += vgrid;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    pdl_launch_dependents();
    // weights do not depend on the preceding kernel
#pragma unroll
    for (int i = 0; i < kRowsStages - 1; ++i) issue(i);
    pdl_wait();

    // ---- B fragments of this warp's four groups: lane (g, t) holds columns 16 t .. 16 t + 15 of rows 8 nt + g ----------
    unsigned xb[4][NT][8];
    float inv[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int b = 8 * nt + g;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k0 = (stage * 4 + q) * 64 + 16 * t;
#pragma unroll
            for (int i = 0; i < 8; ++i) xb[q][nt][i] = 0u;
            if (works && b < p.m && k0 < p.k) rows_load32(p.x + (size_t)b * p.x_stride + k0, p.wide, xb[q][nt]);
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        unsigned m2 = 0;   // bf16 magnitudes order like their bits
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 8; ++i) m2 = __vmaxu2(m2, xb[q][nt][i] & 0x7FFF7FFFu);
        m2 = __vmaxu2(m2, __shfl_xor_sync(0xffffffffu, m2, 1));
        m2 = __vmaxu2(m2, __shfl_xor_sync(0xffffffffu, m2, 2));
        // the largest exponent goes to 2^13: fp16 keeps every bf16 mantissa bit
        const int e = (int)(max(m2 & 0xFFFFu, m2 >> 16) >> 7);
        const int sh = (e == 0 || e == 255) ? 0 : max(-120, min(120, 140 - e));
        const float mul = __uint_as_float((unsigned)(127 + sh) << 23);
        inv[nt] = __uint_as_float((unsigned)(127 - sh) << 23);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned w = xb[q][nt][i];
                const __half2 h = __floats2half2_rn(__uint_as_float(w << 16) * mul, __uint_as_float(w & 0xFFFF0000u) * mul);
                xb[q][nt][i] = *reinterpret_cast<const unsigned*>(&h);
            }
            // the group's sums come out of a product with ones, in the lanes and columns that need them
            float sum[4];
            rows_mma_first(sum, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, xb[q][nt][0], xb[q][nt][1]);
#pragma unroll
            for (int j = 1; j < 4; ++j) rows_mma(sum, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, xb[q][nt][2 * j], xb[q][nt][2 * j + 1]);
            if (g == 0) *reinterpret_cast<float2*>(xs + q * COLS + 8 * nt + 2 * t) = make_float2(sum[0], sum[1]);
        }
    }
    __syncwarp();
    float cs[NT][2];   // undoes the scaling of this lane's accumulator columns 8 nt + 2 t, + 1
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        cs[nt][0] = __shfl_sync(0xffffffffu, inv[nt], 8 * t);
        cs[nt][1] = __shfl_sync(0xffffffffu, inv[nt], 8 * t + 4);
    }
    const unsigned xs_sa = (unsigned)__cvta_generic_to_shared(xs) + 8 * t;

    const int gtid = tid - grp * p.kc * 32, gthreads = p.kc * 32;
    const int cols_own = COLS / p.sk;   // columns that this CTA of the cluster finishes
    const cg::cluster_group cluster = cg::this_cluster();
    if (p.sk > 1) cluster.sync();       // every CTA of the cluster runs before anything is sent to it
    // sums what the cluster sent for round `round`
    auto finish_received = [&](int round) {
        const int rt = vb + round * vgrid;
        if (!in_group || rt >= p.row_tiles) return;
        const float* src = recv + ((round & 1) * p.groups + grp) * (16 * COLS);
        for (int o = gtid; o < 8 * cols_own; o += gthreads) {
            const int r = o & 7, c = o >> 3;
            float lo = 0.f, hi = 0.f;
            for (int z = 0; z < p.sk; ++z) { lo += src[(z * cols_own + c) * 16 + r]; hi += src[(z * cols_own + c) * 16 + r + 8]; }
            rows_finish<EPI>(p, rt, r, rank * cols_own + c, lo, hi);
        }
    };

    int slot = 0, islot = kRowsStages - 1;
    for (int round = 0, rt = vb; round < p.rounds; ++round, rt += vgrid) {
        issue(islot);
        islot = islot + 1 == kRowsStages ? 0 : islot + 1;
        if (in_group && rt < p.row_tiles) {   // the same for every warp of a group
            if (works) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kRowsStages - 1) : "memory");
                __syncwarp();
                const unsigned st = ring + slot * kRowsStageBytes;
                float tot[NT][4];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) tot[nt][0] = tot[nt][1] = tot[nt][2] = tot[nt][3] = 0.f;
                const uint4 sA = rows_lds128(st + 2048 + g * 16), sB = rows_lds128(st + 2048 + (g + 8) * 16);
                const unsigned sAw[4] = {sA.x, sA.y, sA.z, sA.w}, sBw[4] = {sB.x, sB.y, sB.z, sB.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint4 wv = rows_lds128(st + q * 512 + lane * 16);
                    const unsigned wr[4] = {wv.x, wv.y, wv.z, wv.w};
                    float acc[NT][4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        // the low nibble of each byte pair is row g, the high one row g + 8
                        const unsigned r0 = wr[j], r8 = r0 >> 8;
                        const unsigned a0 = rows_low(r0), a1 = rows_high(r0), a2 = rows_low(r8), a3 = rows_high(r8);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            if (j == 0) rows_mma_first(acc[nt], a0, a1, a2, a3, xb[q][nt][0], xb[q][nt][1]);
                            else rows_mma(acc[nt], a0, a1, a2, a3, xb[q][nt][2 * j], xb[q][nt][2 * j + 1]);
                        }
                    }
                    const float s_lo = rows_scale<F16SB>(sAw[q]), s_hi = rows_scale<F16SB>(sBw[q]);
                    const float z_lo = fmaf(8.f, s_lo, rows_zero<F16SB>(sAw[q])), z_hi = fmaf(8.f, s_hi, rows_zero<F16SB>(sBw[q]));
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt) {
                        float2 x2;
                        asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(x2.x), "=f"(x2.y) : "r"(xs_sa + (q * COLS + 8 * nt) * 4));
                        tot[nt][0] = fmaf(s_lo, acc[nt][0], fmaf(z_lo, x2.x, tot[nt][0]));
                        tot[nt][1] = fmaf(s_lo, acc[nt][1], fmaf(z_lo, x2.y, tot[nt][1]));
                        tot[nt][2] = fmaf(s_hi, acc[nt][2], fmaf(z_hi, x2.x, tot[nt][2]));
                        tot[nt][3] = fmaf(s_hi, acc[nt][3], fmaf(z_hi, x2.y, tot[nt][3]));
                    }
                }
                float* dst = parts + ((round & 1) * kRowsWarps + warp) * (COLS * kRowsPitch);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[(8 * nt + 2 * t + (i & 1)) * kRowsPitch + g + 8 * (i >> 1)] = tot[nt][i] * cs[nt][i & 1];
            }
            asm volatile("bar.sync %0, %1;" ::"r"(grp), "r"(gthreads) : "memory");
        }
        if (p.sk > 1 && round > 0) {
            // the parts of the round before have arrived; nobody sends to the other buffer again before this
            __syncwarp();
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            finish_received(round - 1);
        }
        if (in_group && rt < p.row_tiles) {
            const float* src = parts + ((round & 1) * kRowsWarps + grp * p.kc) * (COLS * kRowsPitch);
            for (int o = gtid; o < 8 * COLS; o += gthreads) {
                const int r = o & 7, c = o >> 3;
                float lo = 0.f, hi = 0.f;
#pragma unroll 4
                for (int w = 0; w < kc; ++w) {
                    lo += src[w * (COLS * kRowsPitch) + c * kRowsPitch + r];
                    hi += src[w * (COLS * kRowsPitch) + c * kRowsPitch + r + 8];
                }
                if (p.sk == 1) {
                    rows_finish<EPI>(p, rt, r, c, lo, hi);
                } else {
                    const int owner = c / cols_own;
                    float* dst = cluster.map_shared_rank(recv, owner) + ((round & 1) * p.groups + grp) * (16 * COLS) + (rank * cols_own + (c - owner * cols_own)) * 16;
                    dst[r] = lo; dst[r + 8] = hi;
                }
            }
        }
        if (p.sk > 1) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        }
        slot = slot + 1 == kRowsStages ? 0 : slot + 1;
    }
    if (p.sk > 1) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        finish_received(p.rounds - 1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

int g_rows_clusters[4] = {kRowsSMs, 0, 0, 0};   // clusters of 1, 2, 4, 8 CTAs that run at once (the fewest over the instantiations)

template <int NT, int EPI, bool F16SB>
int rows_init_one() {
    SWLM_CUDA(cudaFuncSetAttribute(qgemv_rows_kernel<NT, EPI, F16SB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem_bytes<NT>()));
    for (int i = 1; i < 4; ++i) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1u << i; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(kRowsSMs >> i) << i); cfg.blockDim = dim3(kRowsWarps * 32); cfg.dynamicSmemBytes = rows_smem_bytes<NT>();
        cfg.attrs = attr; cfg.numAttrs = 1;
        int n = 0;
        SWLM_CUDA(cudaOccupancyMaxActiveClusters(&n, qgemv_rows_kernel<NT, EPI, F16SB>, &cfg));
        if (n < 1) { set_error("qgemv rows: no cluster of %d CTAs fits this device", 1 << i); return SWLM_ERR_UNSUPPORTED; }
        n = std::min(n, kRowsSMs >> i);
        g_rows_clusters[i] = g_rows_clusters[i] ? std::min(g_rows_clusters[i], n) : n;
    }
    return SWLM_OK;
}

template <int NT, int EPI, bool F16SB>
int rows_launch(const QRowsParams& p, int clusters, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * p.sk)); cfg.blockDim = dim3(kRowsWarps * 32); cfg.dynamicSmemBytes = rows_smem_bytes<NT>(); cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)p.sk; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, qgemv_rows_kernel<NT, EPI, F16SB>, p);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "qgemv rows launch");
}

}  // namespace

int qgemv_rows_init() {
    int rc;
    if ((rc = rows_init_one<1, 0, false>()) || (rc = rows_init_one<1, 0, true>()) || (rc = rows_init_one<1, 1, false>()) || (rc = rows_init_one<1, 1, true>()) ||
        (rc = rows_init_one<2, 0, false>()) || (rc = rows_init_one<2, 0, true>()) || (rc = rows_init_one<2, 1, false>()) || (rc = rows_init_one<2, 1, true>())) return rc;
    return SWLM_OK;
}

bool qgemv_rows_takes(const Q4Tiled& w, int m) { return m >= 2 && m <= kQGemvMaxRows && w.kt_pad / 4 <= kRowsWarps * kRowsMaxCluster; }

int launch_qgemv_rows(const QGemvLaunch& a, cudaStream_t s) {
    const Q4Tiled& w = *a.w;
    if ((a.x_stride & 7) || (reinterpret_cast<uintptr_t>(a.x) & 15)) {
        set_error("qgemv: x must be 16-byte aligned with a stride that is a multiple of 8 elements");
        return SWLM_ERR_INVALID;
    }
    QRowsParams p{};
    p.tiles = w.tiles; p.sb = w.sb; p.row_tiles = w.row_tiles; p.kt4 = w.kt_pad / 4;
    p.x = a.x; p.x_stride = a.x_stride; p.k = w.k; p.m = a.m; p.gated_act = a.gated_act;
    p.wide = !(a.x_stride & 15) && !(reinterpret_cast<uintptr_t>(a.x) & 31);
    for (int i = 0; i < 3; ++i) {
        p.y[i] = a.y[i]; p.y_stride[i] = a.y_stride[i];
        p.seg_end[i] = a.seg_end[i] > 0 ? a.seg_end[i] : (i ? p.seg_end[i - 1] : 0);
    }
    // The fewest CTAs along K that keep (nearly) all warps at work: kt4 * groups / sk of the 16 warps have a stage. Going to twice
    // the CTAs costs an exchange per round, so it has to bring a quarter more warps (K = 2304: 9 stages, 9 warps against 13.5).
    double best = 0.0;
    int log_sk = 0;
    for (int i = 0; i < 4; ++i) {
        const int sk = 1 << i, kc = (p.kt4 + sk - 1) / sk;
        if (kc > kRowsWarps || sk > p.kt4) continue;
        const int groups = kRowsWarps / kc;
        const double at_work = (double)p.kt4 * groups / sk;
        if (at_work <= 1.25 * best) continue;
        best = at_work; log_sk = i; p.sk = sk; p.kc = kc; p.groups = groups;
    }
    if (p.sk == 0 || (p.sk > 1 && p.groups > kRowsWarps / 2)) { set_error("qgemv rows: k=%d", w.k); return SWLM_ERR_INVALID; }
    const int clusters = std::min(g_rows_clusters[log_sk], (p.row_tiles + p.groups - 1) / p.groups);
    p.rounds = (p.row_tiles + clusters * p.groups - 1) / (clusters * p.groups);
    const bool gated = a.epilogue == QGEMV_EPI_SWIGLU;
    if (a.m <= 8) {
        if (gated) return w.sb_f16 ? rows_launch<1, 1, true>(p, clusters, s) : rows_launch<1, 1, false>(p, clusters, s);
        return w.sb_f16 ? rows_launch<1, 0, true>(p, clusters, s) : rows_launch<1, 0, false>(p, clusters, s);
    }
    if (gated) return w.sb_f16 ? rows_launch<2, 1, true>(p, clusters, s) : rows_launch<2, 1, false>(p, clusters, s);
    return w.sb_f16 ? rows_launch<2, 0, true>(p, clusters, s) : rows_launch<2, 0, false>(p, clusters, s);
}

}  // namespace swlm
