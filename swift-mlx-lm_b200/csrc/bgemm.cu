// Dense products of fp32-stream plans: Y[m][n] = X[m][k] . W[n][k]^T with bf16 weights and fp32 accumulation.
//
//   bgemv_kernel     1..kGemvRows activation rows: the weights are streamed once from HBM with 16-byte loads, four weight
//                    rows per warp and K cut across the warps of a CTA; the norm in front of the product can run in the
//                    prologue, gate and up in one launch with the gated activation in the epilogue. Activations bf16 or fp32
//                    (with fp32 ones the product is a true fp32 product: a bf16 weight is exact in fp32).
//   bgemm_tc_kernel  more rows, bf16 activations: tcgen05.mma with both operands staged by TMA (128-byte swizzle), one SM or a pair of
//                    them per tile, gate and up side by side in tensor memory, K cut over the CTAs of a cluster when there are few
//                    tiles. Grouped form: activation rows sorted by expert, a device table names the expert and the rows of every
//                    tile.
//   sgemm_kernel     more rows, fp32 activations: fp32 FMAs on 64 x 64 tiles.
#include <algorithm>
#include <cstdlib>
#include <mutex>

#include <cooperative_groups.h>

#include "swlm_internal.h"
#include "tc_device.cuh"

namespace cg = cooperative_groups;

namespace swlm {
namespace {

__device__ __forceinline__ float b_lo(unsigned w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float b_hi(unsigned w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Where the results of one weight row go: that of activation row m is m * stride bytes behind y.
struct ProductRow { unsigned char* y; size_t stride; bool f32; float bias; };
template <bool BIASED>
__device__ __forceinline__ ProductRow product_row(const ProductOut& o, int row) {
    void* y = o.y[0];
    const __nv_bfloat16* bias = BIASED ? o.bias[0] : nullptr;
    int first = 0, stride = o.stride[0], f32 = o.f32[0];
#pragma unroll
    for (int q = 1; q < kMaxProductSegs; ++q)
        if (q < o.count && row >= o.end[q - 1]) { y = o.y[q]; first = o.end[q - 1]; stride = o.stride[q]; f32 = o.f32[q]; if (BIASED) bias = o.bias[q]; }
    const int size = f32 ? 4 : 2;
    return ProductRow{static_cast<unsigned char*>(y) + (ptrdiff_t)(row - first) * size, (size_t)stride * size, f32 != 0,
                      BIASED && bias && row < o.end[o.count - 1] ? __bfloat162float(bias[row - first]) : 0.f};
}
template <bool BIASED>
__device__ __forceinline__ void product_store(const ProductOut& o, int m, int row, float val) {
    const ProductRow r = product_row<BIASED>(o, row);
    if (BIASED) val += r.bias;
    if (o.softcap > 0.f) val = o.softcap * tanhf(val / o.softcap);
    if (o.gelu) val = gelu_erf(val);
    if (r.f32) *reinterpret_cast<float*>(r.y + m * r.stride) = val;
    else *reinterpret_cast<__nv_bfloat16*>(r.y + m * r.stride) = __float2bfloat16_rn(val);
}

// ---- few rows ---------------------------------------------------------------------------------------------------------
constexpr int kGemvRows = 4;
constexpr int kGemvThreads = 256, kGemvWarps = kGemvThreads / 32;
constexpr int kGemvUnroll = 4;                       // 16-byte loads in flight per weight row and lane
constexpr size_t kGemvMaxSmem = 200 * 1024;

struct GemvParams {
    const __nv_bfloat16* w; const __nv_bfloat16* w2;
    int ld, n, k, m;
    GatedAct act;
    const void* x; int x_stride;
    const void* x2; int x2_stride, split;        // rows from `split` on (a multiple of four) meet a second input
    StreamNorm norm;
    ProductOut out;
};

__device__ __forceinline__ float cta_sum(float v, float* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < kGemvWarps; ++i) total += red[i];
    __syncthreads();
    return total;
}
__device__ __forceinline__ void put_x(float* p, float v) { *p = v; }
__device__ __forceinline__ void put_x(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }
// eight consecutive activations
__device__ __forceinline__ void get_x8(const float* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void get_x8(const __nv_bfloat16* p, float (&f)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    f[0] = b_lo(v.x); f[1] = b_hi(v.x); f[2] = b_lo(v.y); f[3] = b_hi(v.y); f[4] = b_lo(v.z); f[5] = b_hi(v.z); f[6] = b_lo(v.w); f[7] = b_hi(v.w);
}

// A warp takes groups of four weight rows (GATED: two of gate and the same two of up); WK warps share a group and cut K. MORE: biases
// and a second input are possible (others do without that code: its instructions have to be fetched, too).
template <typename T, int MR, int WK, bool GATED, bool MORE>
__global__ void __launch_bounds__(kGemvThreads, 2) bgemv_kernel(const GemvParams p) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) unsigned char gemv_raw[];
    __shared__ float red[kGemvWarps];
    __shared__ float part[kGemvWarps][4 * MR];
    T* xs = reinterpret_cast<T*>(gemv_raw);                    // [MR][ld]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kw = warp % WK, rg = warp / WK;
    constexpr int ROWS = GATED ? 2 : 4;                         // output rows of a group
    const int groups = (p.n + ROWS - 1) / ROWS, per_cta = kGemvWarps / WK;
    const int chunks = p.ld >> 3;                               // 16-byte chunks per weight row
    constexpr int STEP = 32 * WK;

    auto row_ptr = [&](int group, int i) -> const __nv_bfloat16* {
        const int r = min(group * ROWS + (GATED ? (i & 1) : i), p.n - 1);
        return (GATED && i >= 2 ? p.w2 : p.w) + (size_t)r * p.ld;
    };
    uint4 wv[4][kGemvUnroll];
    auto load = [&](int group, int c0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const __nv_bfloat16* row = row_ptr(group, i);
#pragma unroll
            for (int u = 0; u < kGemvUnroll; ++u) {
                const int c = c0 + u * STEP;
                wv[i][u] = c < chunks ? ldg_stream(row + 8 * c) : make_uint4(0, 0, 0, 0);
            }
        }
    };
    const int first_chunk = kw * 32 + lane;
    int group = blockIdx.x * per_cta + rg;
    // the first weights (and a norm's) do not depend on the preceding kernel
    if (group < groups) load(group, first_chunk);
    // a norm over at most 4096 entries keeps its row in registers: entries 4 tid + 1024 j
    const bool norm_regs = p.norm.mode && p.k <= 16 * kGemvThreads && (p.k & 3) == 0;
    uint2 nw[4], npw[4];
    if (norm_regs) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = 4 * tid + 4 * kGemvThreads * j;
            nw[j] = i < p.k ? __ldg(reinterpret_cast<const uint2*>(p.norm.w + i)) : make_uint2(0, 0);
            npw[j] = i < p.k && p.norm.w_post ? __ldg(reinterpret_cast<const uint2*>(p.norm.w_post + i)) : make_uint2(0, 0);
        }
    }
    pdl_wait();

    // ---- activations to shared memory: plain rows, or the norm in front of the product (every CTA computes it; CTA 0 stores
    // the new residual) ----
    if (norm_regs) {
        for (int m = 0; m < MR; ++m) {
            T* xr = xs + (size_t)m * p.ld;
            const float* in = p.norm.in + (size_t)m * p.norm.in_stride;
            const float* res = p.norm.res_in ? p.norm.res_in + (size_t)m * p.norm.res_stride : nullptr;
            const __nv_bfloat16* joins = p.norm.table ? p.norm.table_row(m, p.k) : nullptr;
            float h[4][4], rv[4][4];
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = 4 * tid + 4 * kGemvThreads * j;
                const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                const float4 a = i < p.k ? __ldcg(reinterpret_cast<const float4*>(in + i)) : z, b = i < p.k && res ? __ldcg(reinterpret_cast<const float4*>(res + i)) : z;
                h[j][0] = a.x; h[j][1] = a.y; h[j][2] = a.z; h[j][3] = a.w;
                rv[j][0] = b.x; rv[j][1] = b.y; rv[j][2] = b.z; rv[j][3] = b.w;
                if (joins && i < p.k) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(joins + i));
                    rv[j][0] += b_lo(v.x) * p.norm.table_scale; rv[j][1] += b_hi(v.x) * p.norm.table_scale;
                    rv[j][2] += b_lo(v.y) * p.norm.table_scale; rv[j][3] += b_hi(v.y) * p.norm.table_scale;
                }
            }
            if (p.norm.w_post) {
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) ss = fmaf(h[j][e], h[j][e], ss);
                const float sc = 1.0f / sqrtf(cta_sum(ss, red) / (float)p.k + p.norm.eps);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float wf[4] = {b_lo(npw[j].x), b_hi(npw[j].x), b_lo(npw[j].y), b_hi(npw[j].y)};
#pragma unroll
                    for (int e = 0; e < 4; ++e) h[j][e] = h[j][e] * sc * (wf[e] + p.norm.weight_bias);
                }
            }
            ss = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) { h[j][e] += rv[j][e]; ss = fmaf(h[j][e], h[j][e], ss); }
            // (entries past k: zero input, zero residual)
            const float sc = 1.0f / sqrtf(cta_sum(ss, red) / (float)p.k + p.norm.eps);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = 4 * tid + 4 * kGemvThreads * j;
                const float wf[4] = {b_lo(nw[j].x), b_hi(nw[j].x), b_lo(nw[j].y), b_hi(nw[j].y)};
                if (i < p.k) {
                    if (p.norm.res_out && blockIdx.x == 0)
                        *reinterpret_cast<float4*>(p.norm.res_out + (size_t)m * p.norm.res_stride + i) = make_float4(h[j][0], h[j][1], h[j][2], h[j][3]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) put_x(xr + i + e, h[j][e] * sc * (wf[e] + p.norm.weight_bias));
                } else if (i < p.ld) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) put_x(xr + i + e, 0.f);
                }
            }
        }
    } else if (p.norm.mode) {
        for (int m = 0; m < MR; ++m) {
            T* xr = xs + (size_t)m * p.ld;
            float* rowf = reinterpret_cast<float*>(gemv_raw + (size_t)MR * p.ld * sizeof(T));
            const float* in = p.norm.in + (size_t)m * p.norm.in_stride;
            const float* res = p.norm.res_in ? p.norm.res_in + (size_t)m * p.norm.res_stride : nullptr;
            const __nv_bfloat16* joins = p.norm.table ? p.norm.table_row(m, p.k) : nullptr;
            float post_scale = 1.f;
            float ss = 0.f;
            for (int i = tid; i < p.k; i += kGemvThreads) { const float v = in[i]; rowf[i] = v; ss = fmaf(v, v, ss); }
            if (p.norm.w_post) post_scale = 1.0f / sqrtf(cta_sum(ss, red) / (float)p.k + p.norm.eps);
            ss = 0.f;
            for (int i = tid; i < p.k; i += kGemvThreads) {
                float h = rowf[i];
                if (p.norm.w_post) h = h * post_scale * (__bfloat162float(p.norm.w_post[i]) + p.norm.weight_bias);
                if (res) h += res[i];
                if (joins) h += __bfloat162float(joins[i]) * p.norm.table_scale;
                if (p.norm.res_out && blockIdx.x == 0) p.norm.res_out[(size_t)m * p.norm.res_stride + i] = h;
                rowf[i] = h;
                ss = fmaf(h, h, ss);
            }
            const float sc = 1.0f / sqrtf(cta_sum(ss, red) / (float)p.k + p.norm.eps);
            for (int i = tid; i < p.ld; i += kGemvThreads)
                put_x(xr + i, i < p.k ? rowf[i] * sc * (__bfloat162float(p.norm.w[i]) + p.norm.weight_bias) : 0.f);
        }
    } else {
        for (int m = 0; m < MR; ++m) {
            const T* src = static_cast<const T*>(p.x) + (size_t)m * p.x_stride;
            for (int i = tid; i < p.ld; i += kGemvThreads) { T v = T(0.0f); if (i < p.k) v = src[i]; xs[(size_t)m * p.ld + i] = v; }
        }
        if (MORE && p.x2)
            for (int m = 0; m < MR; ++m) {
                const T* src = static_cast<const T*>(p.x2) + (size_t)m * p.x2_stride;
                for (int i = tid; i < p.ld; i += kGemvThreads) { T v = T(0.0f); if (i < p.k) v = src[i]; xs[(size_t)(MR + m) * p.ld + i] = v; }
            }
    }
    __syncthreads();

    const int rounds = (groups + gridDim.x * per_cta - 1) / (gridDim.x * per_cta);
    for (int it = 0; it < rounds; ++it) {
        float acc[4][MR];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int m = 0; m < MR; ++m) acc[i][m] = 0.f;
        const bool live = group < groups;
        const T* xg = xs + (MORE && p.x2 && group * ROWS >= p.split ? (size_t)MR * p.ld : 0);
        if (live) {
            for (int c0 = first_chunk; c0 < chunks; c0 += STEP * kGemvUnroll) {
                if (it > 0 || c0 != first_chunk) load(group, c0);
#pragma unroll
                for (int u = 0; u < kGemvUnroll; ++u) {
                    const int c = c0 + u * STEP;
                    if (c < chunks) {
                        float wf[4][8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 v = wv[i][u];
                            wf[i][0] = b_lo(v.x); wf[i][1] = b_hi(v.x); wf[i][2] = b_lo(v.y); wf[i][3] = b_hi(v.y);
                            wf[i][4] = b_lo(v.z); wf[i][5] = b_hi(v.z); wf[i][6] = b_lo(v.w); wf[i][7] = b_hi(v.w);
                        }
#pragma unroll
                        for (int m = 0; m < MR; ++m) {
                            float xf[8];
                            get_x8(xg + (size_t)m * p.ld + 8 * c, xf);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int e = 0; e < 8; ++e) acc[i][m] = fmaf(wf[i][e], xf[e], acc[i][m]);
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int m = 0; m < MR; ++m)
                for (int o = 16; o > 0; o >>= 1) acc[i][m] += __shfl_xor_sync(0xffffffffu, acc[i][m], o);
        if (WK > 1) {
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int m = 0; m < MR; ++m) part[warp][i * MR + m] = acc[i][m];
            }
            __syncthreads();
            if (kw == 0) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int m = 0; m < MR; ++m) {
                        float v = 0.f;
#pragma unroll
                        for (int q = 0; q < WK; ++q) v += part[rg * WK + q][i * MR + m];
                        acc[i][m] = v;
                    }
            }
            __syncthreads();
        }
        if (live && kw == 0) {
            // lane (i * MR + m) stores one value
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                if (GATED) {
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const int row = group * 2 + i;
                        if (lane == i * MR + m && row < p.n) product_store<false>(p.out, m, row, gated_activation(acc[i][m], acc[2 + i][m], p.act));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int row = group * 4 + i;
                        if (lane == i * MR + m && row < p.n) product_store<MORE>(p.out, m, row, acc[i][m]);
                    }
                }
            }
        }
        group += gridDim.x * per_cta;
    }
}

// ---- many rows, bf16: tcgen05, K over the CTAs of a cluster ---------------------------------------------------------------
// CTA groups of CG = 1 or 2 take a tile of 128 CG weight rows x BN activation rows over one K range; `ranges` groups side by side in a
// cluster take the K ranges and meet through distributed shared memory (the ring's, which is free by then): each sums the ranges of
// BN / ranges activation rows, in order, and stores them.
// What bounds it: what an SM takes in from L2 (about 38 bytes per clock with all of them reading). A pair of SMs holds 256 x BN results
// with half of the activations in either's shared memory: 512 rows through 2048 x 16384 (gate and up) move 201 MB instead of the 268 MB
// of one SM per tile.
constexpr int kTileRows = 128;       // weight rows of a CTA = its lanes of tensor memory
constexpr int kTcK = 64;             // columns per stage = one 128-byte swizzle row
constexpr int kTcEpilogueWarps = 8;
constexpr int kTcWarps = 2 + kTcEpilogueWarps;   // TMA, MMA, epilogue
constexpr int kTcBlock = kTcWarps * 32;

struct TcParams {
    int n, m, steps;                 // weight rows, activation rows, 64-column steps of K
    int ranges;                      // K ranges = CTA groups of a cluster
    int split;                       // weight rows from here on (a multiple of 256) meet the activations of wmap2's place
    GatedAct act;
    const int4* tiles;               // grouped form: (expert, first row, rows, 0) of tile blockIdx.y; n = rows of one expert's matrix
    ProductOut out;
    int* status;
};

__device__ __forceinline__ unsigned cluster_place(unsigned addr, int rank) {   // the same shared-memory place in another CTA of the cluster
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_cluster_v4(unsigned addr, unsigned a, unsigned b, unsigned c, unsigned d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// kind::f16: D fp32, A = B = bf16, both K-major
__host__ __device__ constexpr unsigned tc_idesc(int m, int bn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(bn >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
// (descriptors by their low words)
template <int CG>
__device__ __forceinline__ void umma_bf16(unsigned d_tmem, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned accumulate) {
    if (CG == 1)
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}"
            ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "mov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}"
            ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(accumulate) : "memory");
}
// arrival at the same barrier of both CTAs of the pair when the MMAs issued so far are done; `pair`: the bits of their cluster ranks
__device__ __forceinline__ void umma_commit_to(unsigned long long* bar, unsigned short pair) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"(pair) : "memory");
}

__device__ __forceinline__ void tmem_ld16(unsigned (&v)[16], unsigned at) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(at) : "memory");
}

// `count` (at most 16) results of one weight row, activation rows `token` on. No branch between the values of a batch: their
// exponentials and stores overlap.
__device__ __forceinline__ void tc_emit(const TcParams& p, const ProductRow& dst, float (&val)[16], int token, int count) {
    if (p.out.biased) {
#pragma unroll
        for (int i = 0; i < 16; ++i) val[i] += dst.bias;
    }
    if (p.out.softcap > 0.f) {
#pragma unroll
        for (int i = 0; i < 16; ++i) val[i] = p.out.softcap * tanhf(val[i] / p.out.softcap);
    }
    if (p.out.gelu) {
#pragma unroll
        for (int i = 0; i < 16; ++i) val[i] = gelu_erf(val[i]);
    }
    unsigned char* y = dst.y + (size_t)token * dst.stride;
    if (dst.f32) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < count) *reinterpret_cast<float*>(y + i * dst.stride) = val[i];
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (i < count) *reinterpret_cast<__nv_bfloat16*>(y + i * dst.stride) = __float2bfloat16_rn(val[i]);
    }
}
// gated_activation without a branch between values: tanh-GELU as g / (1 + e^-2u), the same function
__device__ __forceinline__ float tc_gated(float g, float up, const GatedAct& act) {
    const bool clamped = act.kind == GATED_ACT_CLAMPED;
    if (clamped) { g = fminf(g, act.limit); up = fminf(fmaxf(up, -act.limit), act.limit) + 1.0f; }
    const float u = act.kind == GATED_ACT_GELU_TANH ? 1.5957691216f * (g + 0.044715f * g * g * g) : clamped ? act.alpha * g : g;
    return 0.25f * g * four_over(1.0f + expf(-u)) * up;
}

template <int CG, int BN, int STAGES, bool GATED>
__global__ void __launch_bounds__(kTcBlock) bgemm_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap xmap,
                                                            const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap wmap2) {
    extern __shared__ __align__(1024) unsigned char tc_raw[];
    unsigned char* smem = tc_raw + ((1024 - (smem_u32(tc_raw) & 1023)) & 1023);   // swizzle atoms
    constexpr int NACC = GATED ? 2 : 1;
    constexpr int A_BYTES = kTileRows * 128, B_BYTES = BN / CG * 128, STAGE = NACC * A_BYTES + B_BYTES;
    constexpr unsigned kCols = NACC * BN;
    static_assert(kCols >= 32 && kCols <= 512, "tensor memory");
    static_assert((GATED && BN == 256) || STAGES * STAGE >= NACC * (BN + 4 * 8 / CG) * kTileRows * 4, "the ring takes what the cluster sends");
    __shared__ __align__(8) unsigned long long full_bar[STAGES], empty_bar[STAGES], done_bar;
    __shared__ unsigned tmem_base;
    __shared__ int failed_word;
    volatile int* const failed = &failed_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int crank = (int)blockIdx.x, rank = crank % CG, range = crank / CG;   // place in the cluster, in the group; K range
    int tok0 = blockIdx.y * BN, tok_end = p.m, wrow0 = 0;      // wrow0: first row of the expert's matrix
    if (p.tiles) {
        pdl_wait();   // (the table is the preceding kernel's)
        const int4 tile = p.tiles[blockIdx.y];
        if (tile.z == 0) { pdl_launch_dependents(); return; }   // (the same for all CTAs of a cluster)
        wrow0 = tile.x * p.n;
        tok0 = tile.y;
        tok_end = tile.y + tile.z;
    }
    const int row0 = (int)blockIdx.z * (kTileRows * CG) + rank * kTileRows;
    const int step0 = p.steps * range / p.ranges, steps = p.steps * (range + 1) / p.ranges - step0;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(&done_bar, 1);
        failed_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        __syncwarp();
        if (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(kCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)), "r"(kCols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    const cg::cluster_group cluster = cg::this_cluster();
    if (CG == 2) cluster.sync();   // both CTAs' barriers are ready
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem = tmem_base;
    pdl_launch_dependents();   // behind the allocation: a successor that wants tensor memory cannot get in between

    if (warp == 0) {
        // The warp runs its loop as a whole, one lane issues. The weights of the first stages do not depend on the preceding kernel; the
        // activations do. Of a pair both CTAs' copies count on the barrier of the CTA that issues the MMAs; the other's may get there
        // before the bytes are announced: the phase ends with the announcement at the earliest.
        const bool el = elect_one();
        const CUtensorMap* const x = !GATED && row0 - rank * kTileRows >= p.split ? &wmap2 : &xmap;
        const unsigned full0 = CG == 1 ? smem_u32(&full_bar[0]) : cluster_place(smem_u32(&full_bar[0]), crank - rank), ring = smem_u32(smem);
        auto load = [&](unsigned dst, const CUtensorMap* map, int col, int row, int s) {
            if (CG == 1) tma_load_2d(dst, map, col, row, full0 + 8u * s);
            else tma_load_2d_pair(dst, map, col, row, full0 + 8u * s);
        };
        auto weights = [&](int kt, int s) {
            if (rank == 0) mbar_expect(full0 + 8u * s, (unsigned)(CG * STAGE));
            load(ring + s * STAGE, &wmap, (step0 + kt) * kTcK, wrow0 + row0, s);
            if (GATED) load(ring + s * STAGE + A_BYTES, &wmap2, (step0 + kt) * kTcK, wrow0 + row0, s);
        };
        auto activations = [&](int kt, int s) { load(ring + s * STAGE + NACC * A_BYTES, x, (step0 + kt) * kTcK, tok0 + rank * (BN / CG), s); };
        const int ahead = min(STAGES, steps);
        if (el)
            for (int kt = 0; kt < ahead; ++kt) weights(kt, kt);
        __syncwarp();
        pdl_wait();
        if (el)
            for (int kt = 0; kt < ahead; ++kt) activations(kt, kt);
        __syncwarp();
        int s = 0, kt = ahead;
        unsigned par = 0;
        bool ok = true;
        for (; kt < steps; ++kt) {
            if (!mbar_wait_warp(&empty_bar[s], par)) { ok = false; break; }
            if (el) { weights(kt, s); activations(kt, s); }
            __syncwarp();
            if (++s == STAGES) { s = 0; par ^= 1u; }
        }
        if (!ok) {   // copies already requested still write shared memory (in a pair's second CTA, whose barrier this is not, the limit of the wait is the time they get)
            if (el) { atomicExch(p.status, 31); *failed = 1; }
            for (int i = kt > STAGES ? kt - STAGES : 0; i < kt; ++i) mbar_wait_warp(&full_bar[i % STAGES], (unsigned)((i / STAGES) & 1));
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0) {
            // the warp runs its loop as a whole, one lane issues (a lone lane's loop took longer over its eight MMAs than a step of 128
            // activation rows takes to multiply)
            constexpr unsigned idesc = tc_idesc(kTileRows * CG, BN);
            const unsigned short pair = (unsigned short)(3u << crank);
            const bool el = elect_one();
            int s = 0;
            unsigned par = 0;
            for (int kt = 0; kt < steps; ++kt) {
                const bool ok = CG == 1 ? mbar_wait_warp(&full_bar[s], par) : mbar_wait_cluster_warp(&full_bar[s], par);
                if (!ok) { if (el) { atomicExch(p.status, 32); *failed = 1; } break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (el) {
                    const unsigned a = umma_desc_lo(smem_u32(smem + s * STAGE)), b = a + NACC * A_BYTES / 16;
#pragma unroll
                    for (int j = 0; j < kTcK / 16; ++j) {
                        const unsigned acc = j > 0 ? 1u : kt > 0 ? 1u : 0u;
                        umma_bf16<CG>(tmem, a + 2 * j, b + 2 * j, idesc, acc);
                        if (GATED) umma_bf16<CG>(tmem + BN, a + A_BYTES / 16 + 2 * j, b + 2 * j, idesc, acc);
                    }
                    if (CG == 1) umma_commit(&empty_bar[s]);
                    else umma_commit_to(&empty_bar[s], pair);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; par ^= 1u; }
            }
            if (el) {   // also behind whatever was issued before a failure
                if (CG == 1) umma_commit(&done_bar);
                else umma_commit_to(&done_bar, pair);
            }
        }
        __syncwarp();
    }
    // ---- results: a warp reads the 32 accumulator lanes of its quarter (warp & 3), lane = weight row; the two warps of a quarter
    // take turns with the activation rows ----
    const int epi = warp - 2, quarter = warp & 3, row = row0 + quarter * 32 + lane;
    const unsigned lanes = tmem + ((unsigned)(quarter * 32) << 16);
    bool ok = true;
    if (epi >= 0) {
        pdl_wait();   // the outputs may still be read by the kernel before this one
        ok = mbar_wait_warp(&done_bar, 0u);
        if (!ok && lane == 0) { atomicExch(p.status, 33); *failed = 1; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (p.ranges == 1) {
        if (epi >= 0 && ok && !*failed) {
            const ProductRow dst = product_row<true>(p.out, row);
#pragma unroll 1
            for (int c0 = 16 * (epi >> 2); c0 < BN; c0 += 16 * (kTcEpilogueWarps / 4)) {
                const int token = tok0 + c0;
                if (token >= tok_end) break;   // uniform across the warp
                unsigned v[16], u[16];
                tmem_ld16(v, lanes + (unsigned)c0);
                if (GATED) tmem_ld16(u, lanes + (unsigned)(BN + c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float val[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) val[i] = GATED ? tc_gated(__uint_as_float(v[i]), __uint_as_float(u[i]), p.act) : __uint_as_float(v[i]);
                if (row < p.n) tc_emit(p, dst, val, token, min(16, tok_end - token));
                __syncwarp();
            }
        }
    } else {
        // part (accumulator a, range z, column c of the receiver's) at [((a ranges + z) 128 + weight row) pitch + c], four columns at a time
        const int own = BN / p.ranges, pitch = own + 4;   // (a multiple of four; eight lanes' pieces meet no bank twice)
        cluster.sync();   // every ring of the cluster is free
        if (epi >= 0 && ok) {
#pragma unroll 1
            for (int c0 = 16 * (epi >> 2); c0 < BN; c0 += 16 * (kTcEpilogueWarps / 4)) {
                if (tok0 + c0 >= tok_end) break;
#pragma unroll
                for (int a = 0; a < NACC; ++a) {
                    unsigned v[16];
                    tmem_ld16(v, lanes + (unsigned)(a * BN + c0));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const int owner = (c0 + i) / own, c = c0 + i - owner * own;
                        st_cluster_v4(cluster_place(smem_u32(smem), owner * CG + rank) + (unsigned)(((a * p.ranges + range) * kTileRows + quarter * 32 + lane) * pitch + c) * 4u, v[i], v[i + 1], v[i + 2], v[i + 3]);
                    }
                }
            }
        }
        cluster.sync();
        if (epi >= 0 && ok && !*failed) {
            const float* got = reinterpret_cast<const float*>(smem) + (quarter * 32 + lane) * pitch;
            const ProductRow dst = product_row<true>(p.out, row);
#pragma unroll 1
            for (int first = 8 * (epi >> 2); first < own; first += 8 * (kTcEpilogueWarps / 4)) {
                const int token = tok0 + range * own + first, count = min(min(8, own - first), tok_end - token);
                if (count <= 0) break;
                float val[16] = {}, up[16] = {};
#pragma unroll 1
                for (int z = 0; z < p.ranges; ++z)
#pragma unroll
                    for (int i = 0; i < 8; i += 4)
                        if (first + i < own) {
                            const float4 g = *reinterpret_cast<const float4*>(got + z * (kTileRows * pitch) + first + i);
                            val[i] += g.x; val[i + 1] += g.y; val[i + 2] += g.z; val[i + 3] += g.w;
                            if (GATED) {
                                const float4 u = *reinterpret_cast<const float4*>(got + (p.ranges + z) * (kTileRows * pitch) + first + i);
                                up[i] += u.x; up[i + 1] += u.y; up[i + 2] += u.z; up[i + 3] += u.w;
                            }
                        }
                if (GATED) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) val[i] = tc_gated(val[i], up[i], p.act);
                }
                if (row < p.n) tc_emit(p, dst, val, token, count);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (CG == 2) cluster.sync();   // no MMA of the pair reads tensor memory or arrives at a barrier of a CTA that has left
    if (warp == 1) {
        if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
    }
}

// ---- many rows, fp32 --------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) sgemm_kernel(const __nv_bfloat16* w, int ld, int n, int k, int m, const float* x, int x_stride, const ProductOut out) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float ws[16][68], xsm[16][68];
    const int n0 = blockIdx.x * 64, m0 = blockIdx.y * 64, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < k; k0 += 16) {
        for (int i = threadIdx.x; i < 64 * 16; i += 256) {
            const int r = i >> 4, c = i & 15;
            ws[c][r] = n0 + r < n && k0 + c < k ? __bfloat162float(w[(size_t)(n0 + r) * ld + k0 + c]) : 0.f;
            xsm[c][r] = m0 + r < m && k0 + c < k ? x[(size_t)(m0 + r) * x_stride + k0 + c] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 16; ++c) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { a[i] = xsm[c][ty * 4 + i]; b[i] = ws[c][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
    for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) {
            const int mm = m0 + ty * 4 + i, nn = n0 + tx * 4 + j;
            if (mm < m && nn < n) product_store<true>(out, mm, nn, acc[i][j]);
        }
}

// ---- launches ---------------------------------------------------------------------------------------------------------
template <typename T, int MR, int WK, bool GATED, bool MORE = false>
int gemv_launch(const GemvParams& p, size_t smem, unsigned grid, cudaStream_t s) {
    static const cudaError_t attr = cudaFuncSetAttribute(bgemv_kernel<T, MR, WK, GATED, MORE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemvMaxSmem);
    if (attr != cudaSuccess) return cuda_fail(attr, "bgemv attributes");
    const cudaError_t e = launch_k(bgemv_kernel<T, MR, WK, GATED, MORE>, dim3(grid), dim3(kGemvThreads), smem, s, p);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "bgemv launch");
}
template <typename T, int MR>
int gemv_pick(const GemvParams& p, bool gated, size_t smem, cudaStream_t s) {
    const int groups = (p.n + (gated ? 1 : 3)) / (gated ? 2 : 4);
    // warps that share a group: the fewest passes over the loop of 16-byte loads, a round of groups costing a little by itself
    const int max_grid = 148 * (smem > 100 * 1024 ? 1 : 2), chunks = p.ld >> 3;
    int wk = 1;
    float best = 0.f;
    for (int q = 1; q <= 8; q *= 2) {
        const int ctas = max_grid * (kGemvWarps / q), rounds = (groups + ctas - 1) / ctas, passes = (chunks + 32 * q * kGemvUnroll - 1) / (32 * q * kGemvUnroll);
        const float cost = rounds * (passes + 0.3f);
        if (q == 1 || cost < best) { best = cost; wk = q; }
    }
    const int per_cta = kGemvWarps / wk;
    const unsigned grid = (unsigned)std::min((groups + per_cta - 1) / per_cta, max_grid);
    if (gated) {
        switch (wk) {
        case 1: return gemv_launch<T, MR, 1, true>(p, smem, grid, s);
        case 2: return gemv_launch<T, MR, 2, true>(p, smem, grid, s);
        case 4: return gemv_launch<T, MR, 4, true>(p, smem, grid, s);
        default: return gemv_launch<T, MR, 8, true>(p, smem, grid, s);
        }
    }
    if (p.x2 || p.out.biased) {
        switch (wk) {
        case 1: return gemv_launch<T, MR, 1, false, true>(p, smem, grid, s);
        case 2: return gemv_launch<T, MR, 2, false, true>(p, smem, grid, s);
        case 4: return gemv_launch<T, MR, 4, false, true>(p, smem, grid, s);
        default: return gemv_launch<T, MR, 8, false, true>(p, smem, grid, s);
        }
    }
    switch (wk) {
    case 1: return gemv_launch<T, MR, 1, false>(p, smem, grid, s);
    case 2: return gemv_launch<T, MR, 2, false>(p, smem, grid, s);
    case 4: return gemv_launch<T, MR, 4, false>(p, smem, grid, s);
    default: return gemv_launch<T, MR, 8, false>(p, smem, grid, s);
    }
}
template <typename T>
int gemv_rows(const GemvParams& p, bool gated, size_t smem, cudaStream_t s) {
    switch (p.m) {
    case 1: return gemv_pick<T, 1>(p, gated, smem, s);
    case 2: return gemv_pick<T, 2>(p, gated, smem, s);
    case 3: return gemv_pick<T, 3>(p, gated, smem, s);
    default: return gemv_pick<T, 4>(p, gated, smem, s);
    }
}
size_t gemv_smem(int m, int ld, bool x_f32, bool norm) { return (size_t)m * ld * (x_f32 ? 4 : 2) + (norm ? (size_t)ld * 4 : 0); }

// bf16 matrix [rows][ld] as a 2-D tensor, k columns valid (beyond: zeros); box = 64 columns x box_rows, 128-byte swizzle
int bf16_map(const __nv_bfloat16* p, int ld, int rows, int k, int box_rows, CUtensorMap* map) {
    TensorMapEncodeFn fn = tensor_map_encode_fn();
    if (!fn) { set_error("dense product: cuTensorMapEncodeTiled is not available"); return SWLM_ERR_CUDA; }
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kTcK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(p), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("dense product: cuTensorMapEncodeTiled failed (%d)", (int)r); return SWLM_ERR_CUDA; }
    return SWLM_OK;
}

struct TcShape { int cg, bn, per_sm, ranges, tiles_m, tiles_n; };
constexpr int kTcSMs = 148;
template <int BN, int PER_SM, bool GATED>
constexpr int tc_stages() {
    return BN == 32 ? (GATED ? 6 : 10) / PER_SM : BN == 64 ? (GATED ? 5 : 8 / PER_SM) : BN == 128 ? (GATED ? 5 : 8) : (GATED ? 4 : 7);
}
template <int CG, int BN, int PER_SM, bool GATED>
constexpr size_t tc_smem() { return (size_t)tc_stages<BN, PER_SM, GATED>() * ((GATED ? 2 : 1) * kTileRows * 128 + BN / CG * 128) + 1024; }

// Clusters of 1, 2, 4, 8 CTAs that run at once on a device, one CTA per SM; 0: it takes none of that size, and products do without. Filled
// when the device's first context is made, before any launch on it.
struct TcClusters { std::once_flag once; int at[4] = {kTcSMs, kTcSMs / 2, 0, 0}; };
constexpr int kTcDevices = 64;
TcClusters g_tc_clusters[kTcDevices + 1];   // (the last one: devices beyond, without clusters of 4 and 8)
TcClusters& tc_clusters() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) { cudaGetLastError(); return g_tc_clusters[kTcDevices]; }
    return g_tc_clusters[std::min(device, kTcDevices)];
}

// How a product runs: the form with the least time by what was measured for n = 2048 .. 32768, K = 512 .. 8192, 16 .. 1024 rows (us;
// graphs of launches, weights from memory). A step of 64 columns takes 0.21 (the round trip of a stage over the ring's depth; 0.25 with
// half the depth, two CTAs per SM; 0.3 with 256 rows, 0.7 with gate and up of 256), or what L2 gives all CTAs together (12 TB/s). A launch
// starts and ends in 3, tanh-GELU of 256 rows takes 4 more. The exchange between K ranges costs 2 (32 rows) to 5 (128): 2048 x 8192 at
// 512 rows 27.3 / 21.0 for 1 and 2 ranges, at 16 rows 28.3 / 16.7 / 11.2 / 10.7 for 1, 2, 4, 8. Clusters of eight do not fill the GPU at
// one CTA per SM (128 CTAs in eights: 16.9 instead of 10.7). Against one SM per 256 x 128 tile with the ranges' sums in memory and added by a
// second launch: 3664 x 2048 at 512 rows 28.9 -> 11.3, 2048 x 8192 31.3 -> 21.0, gate and up of 8192 x 2048 59.5 -> 31.5; at 16 rows
// 8.7 -> 6.7, 12.6 -> 10.7, 21.3 -> 15.0.
TcShape tc_shape(int n, int k, int m, bool gated, const int* clusters) {
    TcShape best{};
    const int steps = (k + kTcK - 1) / kTcK;
    double least = 1e30;
    for (int bn = 32; bn <= 256; bn *= 2)
        for (int per_sm = 1; per_sm <= (bn == 32 || (bn == 64 && !gated) ? 2 : 1); ++per_sm) {
            const int cg = bn <= 64 ? 1 : 2, tiles_m = (m + bn - 1) / bn, tiles_n = (n + kTileRows * cg - 1) / (kTileRows * cg);
            const double bytes = (gated ? 2 : 1) * kTileRows * 128 + bn / cg * 128, ends = 3 + (gated ? bn / 64 : bn / 128);
            const double alone = bn == 256 ? (gated ? 0.7 : 0.3) : per_sm == 2 ? 0.25 : 0.21;
            for (int i = 0; i < 4; ++i) {
                const int z = (1 << i) / cg;   // clusters of 1, 2, 4, 8 CTAs
                if (z < 1 || z > steps || clusters[i] < 1 || (gated && bn == 256 && z > 1)) continue;
                const long long groups = (long long)tiles_m * tiles_n, slots = (long long)clusters[i] * per_sm;
                const double waves = (double)((groups + slots - 1) / slots);
                const double step = std::max(alone, bytes * (double)(std::min(groups, slots) << i) / 12e6);
                const double cost = waves * (step * ((steps + z - 1) / z) + ends) + (z > 1 ? 1.5 + bn / 40.0 + 0.2 * z : 0.0);
                if (cost < least) { least = cost; best = {cg, bn, per_sm, z, tiles_m, tiles_n}; }
            }
        }
    return best;
}

template <int CG, int BN, int PER_SM, bool GATED>
int tc_attr() {
    SWLM_CUDA(cudaFuncSetAttribute(bgemm_tc_kernel<CG, BN, tc_stages<BN, PER_SM, GATED>(), GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc_smem<CG, BN, PER_SM, GATED>()));
    return SWLM_OK;
}
template <int CG, int BN, int PER_SM, bool GATED>
int tc_launch(const ProductLaunch& a, const TcShape& t, cudaStream_t s) {
    TcParams p{};
    p.n = a.experts ? a.w->n / a.experts : a.w->n; p.tiles = a.tiles; p.m = a.m; p.steps = (a.w->k + kTcK - 1) / kTcK; p.ranges = t.ranges; p.act = a.act; p.out = a.out; p.status = a.status;
    CUtensorMap xmap, wmap, wmap2;
    int rc = bf16_map(static_cast<const __nv_bfloat16*>(a.x), a.x_stride, a.m, a.w->k, BN / CG, &xmap);
    if (!rc) rc = bf16_map(a.w->data, a.w->ld, a.w->n, a.w->k, kTileRows, &wmap);
    wmap2 = wmap;
    p.split = a.x2 ? a.split : p.n;
    if (!rc && a.x2) rc = bf16_map(static_cast<const __nv_bfloat16*>(a.x2), a.x2_stride, a.m, a.w->k, BN / CG, &wmap2);
    if (!rc && GATED) rc = bf16_map(a.w2->data, a.w2->ld, a.w2->n, a.w2->k, kTileRows, &wmap2);
    if (rc) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(CG * t.ranges), (unsigned)t.tiles_m, (unsigned)t.tiles_n); cfg.blockDim = dim3(kTcBlock); cfg.dynamicSmemBytes = tc_smem<CG, BN, PER_SM, GATED>(); cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(CG * t.ranges); attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, bgemm_tc_kernel<CG, BN, tc_stages<BN, PER_SM, GATED>(), GATED>, p, xmap, wmap, wmap2);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "bgemm launch");
}
template <bool GATED>
int tc_pick(const ProductLaunch& a, const TcShape& t, cudaStream_t s) {
    switch (t.bn) {
    case 32: return t.per_sm == 2 ? tc_launch<1, 32, 2, GATED>(a, t, s) : tc_launch<1, 32, 1, GATED>(a, t, s);
    case 64: return t.per_sm == 2 && !GATED ? tc_launch<1, 64, GATED ? 1 : 2, GATED>(a, t, s) : tc_launch<1, 64, 1, GATED>(a, t, s);
    case 128: return tc_launch<2, 128, 1, GATED>(a, t, s);
    default: return tc_launch<2, 256, 1, GATED>(a, t, s);
    }
}

TcShape grouped_shape(const ProductLaunch& a) {
    TcShape t;
    const int n = a.w->n / a.experts;
    t.bn = a.group_bn; t.cg = t.bn <= 64 ? 1 : 2; t.per_sm = t.bn <= 64 ? 2 : 1; t.ranges = 1;
    t.tiles_m = a.max_tiles; t.tiles_n = (n + kTileRows * t.cg - 1) / (kTileRows * t.cg);
    return t;
}

bool gemv_fits(int m, int k, bool x_f32, bool norm) {
    const int ld = (k + 7) / 8 * 8;
    return m <= kGemvRows && gemv_smem(m, ld, x_f32, norm) <= kGemvMaxSmem;
}

}  // namespace

int bgemm_init() {
    int rc;
    if ((rc = tc_attr<1, 32, 1, false>()) || (rc = tc_attr<1, 32, 2, false>()) || (rc = tc_attr<1, 32, 1, true>()) || (rc = tc_attr<1, 32, 2, true>()) ||
        (rc = tc_attr<1, 64, 1, false>()) || (rc = tc_attr<1, 64, 2, false>()) || (rc = tc_attr<1, 64, 1, true>()) || (rc = tc_attr<2, 128, 1, false>()) ||
        (rc = tc_attr<2, 128, 1, true>()) || (rc = tc_attr<2, 256, 1, false>()) || (rc = tc_attr<2, 256, 1, true>())) return rc;
    TcClusters& of = tc_clusters();
    if (&of == &g_tc_clusters[kTcDevices]) return SWLM_OK;
    std::call_once(of.once, [&] {
        for (int i = 2; i < 4; ++i) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1u << i; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(1u << i, 1, 64); cfg.blockDim = dim3(kTcBlock); cfg.dynamicSmemBytes = tc_smem<1, 32, 1, false>(); cfg.attrs = attr; cfg.numAttrs = 1;
            int fit = 0;
            if (cudaOccupancyMaxActiveClusters(&fit, bgemm_tc_kernel<1, 32, tc_stages<32, 1, false>(), false>, &cfg) != cudaSuccess) { cudaGetLastError(); fit = 0; }
            of.at[i] = fit;
        }
    });
    return SWLM_OK;
}

bool product_takes_norm(int m, int k) { return m <= 2 && k <= 16384 && gemv_fits(m, k, true, true); }
// gate and up in one launch: always, except as true fp32 products over many rows
bool product_takes_gate(int m, int k, bool x_f32) { return !x_f32 || gemv_fits(m, k, true, false); }

bool product_takes_two(int m, int k, int split, bool x_f32) {
    if (gemv_fits(m, k, x_f32, false)) return !(split & 3) && gemv_smem(2 * m, (k + 7) / 8 * 8, x_f32, false) <= kGemvMaxSmem;
    return !x_f32 && split % (2 * kTileRows) == 0;   // no tile has rows of both
}

// tiles about as tall as an expert has rows on average
int grouped_bn(int rows, int experts) {
    const int avg = rows / std::max(1, experts);
    return avg > 160 ? 256 : avg > 64 ? 128 : avg > 24 ? 64 : 32;
}
int grouped_max_tiles(int rows, int experts) { return std::min(rows, experts) + rows / grouped_bn(rows, experts); }

int launch_product(const ProductLaunch& a, cudaStream_t s) {
    if (a.m <= 0) return SWLM_OK;
    const bool gated = a.w2 != nullptr;
    if (gated && (a.w2->n != a.w->n || a.w2->k != a.w->k)) { set_error("gated product: the two matrices differ in shape"); return SWLM_ERR_INVALID; }
    if (a.experts && (a.x_f32 || a.norm.mode || !a.tiles)) { set_error("a grouped product takes plain bf16 rows"); return SWLM_ERR_INVALID; }
    if (!a.experts && gemv_fits(a.m, a.w->k, a.x_f32, a.norm.mode != 0)) {
        GemvParams p{};
        p.w = a.w->data; p.w2 = gated ? a.w2->data : nullptr; p.ld = a.w->ld; p.n = a.w->n; p.k = a.w->k; p.m = a.m; p.act = a.act;
        p.x = a.x; p.x_stride = a.x_stride; p.norm = a.norm; p.out = a.out;
        if (a.x2 && (gated || a.norm.mode || !product_takes_two(a.m, a.w->k, a.split, a.x_f32))) { set_error("two inputs of a product over %d rows run one after the other", a.m); return SWLM_ERR_INVALID; }
        p.x2 = a.x2; p.x2_stride = a.x2_stride; p.split = a.split;
        const size_t smem = gemv_smem(a.x2 ? 2 * a.m : a.m, a.w->ld, a.x_f32, a.norm.mode != 0);
        return a.x_f32 ? gemv_rows<float>(p, gated, smem, s) : gemv_rows<__nv_bfloat16>(p, gated, smem, s);
    }
    if (a.x2 && (gated || a.experts || !product_takes_two(a.m, a.w->k, a.split, a.x_f32))) { set_error("two inputs of a product over %d rows run one after the other", a.m); return SWLM_ERR_INVALID; }
    if (a.norm.mode) { set_error("a norm in front of a product over %d rows runs on its own", a.m); return SWLM_ERR_INVALID; }
    if (a.x_f32) {
        if (gated) { set_error("gate and up of fp32 rows run one after the other"); return SWLM_ERR_INVALID; }
        const cudaError_t e = launch_k(sgemm_kernel, dim3((a.w->n + 63) / 64, (a.m + 63) / 64), dim3(256), 0, s, (const __nv_bfloat16*)a.w->data,
                                       a.w->ld, a.w->n, a.w->k, a.m, static_cast<const float*>(a.x), a.x_stride, a.out);
        return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "sgemm launch");
    }
    if (((a.x_stride | a.x2_stride) & 7) || ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.x2)) & 15)) { set_error("dense product: activation rows must be 16-byte aligned"); return SWLM_ERR_INVALID; }
    const TcShape t = a.experts ? grouped_shape(a) : tc_shape(a.w->n, a.w->k, a.m, gated, tc_clusters().at);
    return gated ? tc_pick<true>(a, t, s) : tc_pick<false>(a, t, s);
}

}  // namespace swlm

extern "C" int swlm_op_dense_form(int m, int n, int k, int gated, const int* clusters, int* form) {
    using namespace swlm;
    if (m <= 0 || n <= 0 || k <= 0 || !form || (clusters && (clusters[0] < 1 || clusters[1] < 1))) { set_error("bad argument"); return SWLM_ERR_INVALID; }
    const TcShape t = tc_shape(n, k, m, gated != 0, clusters ? clusters : tc_clusters().at);
    form[0] = t.cg; form[1] = t.bn; form[2] = t.per_sm; form[3] = t.ranges;
    return SWLM_OK;
}
