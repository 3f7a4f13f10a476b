// Flash-decode GQA attention over a bf16 KV cache for sm_100a.
//
// Replaces `rope_flash_attn_decode` (Generator/MetalSourceGenerator+Attention.swift:551-930): the
// reference runs one 32-thread group per query head that walks the context sequentially and re-reads
// the K/V rows of a GQA group once per query head. Here
//   * the KV range is split across CTAs (flash-decode); the last CTA of a (sequence, KV head) to finish
//     merges the partial (max, sum, output) triples, so the whole step is one launch;
//   * one CTA serves all query heads of a KV head, so K/V are read once per group;
//   * QK^T and PV run on the tensor cores (mma.m16n8k16, bf16 in, fp32 accumulate) with the head
//     dimension permuted so that every lane fetches K and V with 128-bit loads and no shared memory:
//     the contraction over d is order-independent, and for PV two tokens' values of one dimension are
//     paired into a B-fragment register with one PRMT;
//   * q is rotated (RoPE) in fp32 and fed to the tensor core as a bf16 hi + lo pair, so it keeps
//     ~16 bits of mantissa (the reference keeps the rotated q in fp32);
//   * the current token is not read back from the cache: the merging CTA adds its term in fp32 from
//     the unrounded rotated k and v, exactly as the reference does (:866-868, :905-907), while the
//     bf16-rounded copy is appended to the cache for later steps (:761-805).
//   * blocks of 64 tokens are dealt to the splits round-robin, so a split's first block does not depend on the
//     context length: in a decode step it is requested before the device-resident position has arrived, and
//     the split's later blocks are asked into L2 as soon as it has; q, k and v of the new token are requested
//     before any of that, and each RoPE pair is rotated once in shared memory.
// Prompt chunks take the tensor-core kernel of attn_prompt.cu.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cmath>

#include "swlm_internal.h"

namespace swlm {
namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kSplitWarps = 4;
constexpr int kSplitThreads = kSplitWarps * 32;
constexpr int kMaxGroup = 8;  // query heads per KV head served by one CTA

struct AttnParams {
    int heads, kv_heads, rope_dim, max_seq, splits;
    float scale_log2;  // attention scale * log2(e)
    const float* inv_freq;
    const __nv_bfloat16* q; int q_stride;
    const __nv_bfloat16* k; int k_stride;
    const __nv_bfloat16* v; int v_stride;
    __nv_bfloat16* kcache;
    __nv_bfloat16* vcache;
    size_t cache_seq_stride;   // elements between sequences
    size_t cache_head_stride;  // elements between KV heads
    const int32_t* position;   // decode: device array, one entry per sequence; plain: nullptr
    int ctx_len;               // plain: number of cached tokens
    int pos_base;              // prompt ingestion: position of the chunk's first token
    int chunk_tokens;          // prompt ingestion: tokens in the chunk
    int window;                // sliding window (0 = none): a token attends itself and the window - 1 rows before it
    int kv_bits, kv_group;     // quantized cache: bits per value (8 or 4) and values per block (32, 64 or 128)
    int q_first;               // 1: the first K/V rows are requested only after q, k, v have arrived
    __nv_bfloat16* out; int out_stride;
    float* part_o;   // [m][heads][splits][HD]
    float* part_ml;  // [m][heads][splits][2]
    unsigned* counters;  // [m][kv_heads], zero between launches
    PrefetchTarget prefetch;  // weights of a later product, requested into L2 while this kernel runs
    unsigned long long* trace;  // SWLM_TRACE=1: [cta][4] = entry, predecessor complete, loop done, partials published
    // rotated cache schemes: this layer's rotors [kv_heads][ceil(HD / 3)][4] fp16, the projection matrix
    // [HD][qjl_dim] fp16 and this layer's projected K residuals [m][kv_heads][max_seq][qjl_dim] fp16 (qjl_dim 0: none)
    const __half* rotors;
    const __half* qjl_matrix;
    __half* qjl_res;
    int qjl_dim;
};
// With the per-head RMS norm of q and the new k before the rotation (MODE 3 below). A block of its own: 24 bytes more of parameters made
// every launch of the other modes dearer (flash-decode of 24 x 519 tokens, calls back to back on three streams: 5.31 us against 4.93).
struct AttnNormParams : AttnParams {
    const __nv_bfloat16* q_norm; const __nv_bfloat16* k_norm;
    float qk_eps, qk_bias;
};
template <int MODE> struct AttnArgs { typedef AttnParams type; };
template <> struct AttnArgs<3> { typedef AttnNormParams type; };

__device__ __forceinline__ unsigned long long attn_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ uint4 ldg128(const void* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }

// MODE 0: plain flash-decode over an existing cache (q already rotated, context length from the host).
// MODE 1: decode step: sequence b at the device-resident position; rotates q and the new k, appends k/v to the
//         cache and adds the new token's own term from the unrounded values.
// MODE 3: the same behind a per-head RMS norm of q and the new k (a form of its own: plans without that norm keep their code).
// MODE 2: prompt ingestion: "sequence" b is prompt token b of ONE sequence at position pos_base + b; all of the
//         chunk's k/v rows are already in the cache (rope_append_kernel), token b attends rows 0..pos_base+b.
// MODE 4: as MODE 0 over a grid of CTAs that fill the GPU once: all blocks of 64 cached rows of all (sequence, KV head) pairs lie one after
//         the other and every CTA takes the same number of them, of one pair or several. What a CTA has of a pair goes to one of its two
//         places for partial results (pairs that began in an earlier CTA to the first), and the last CTA of a pair to arrive merges them.
template <int HD, int MODE>
__global__ void __launch_bounds__(kSplitThreads) attn_split_kernel(const typename AttnArgs<MODE>::type p) {
    constexpr bool DECODE = MODE == 1 || MODE == 3;
    constexpr bool QK_NORM = MODE == 3;
    constexpr bool PREFILL = MODE == 2;
    constexpr bool STREAM = MODE == 4;
    const int cta_linear = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
    if (p.trace && threadIdx.x == 0) p.trace[cta_linear * 4] = attn_timer_ns();
    pdl_launch_dependents();
    if (DECODE)
        prefetch_target_slice(p.prefetch, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x,
                              gridDim.x * gridDim.y * gridDim.z, threadIdx.x, kSplitThreads);
    constexpr int NCH = HD / 32;  // 16-byte K chunks per lane per token
    constexpr int VH = HD / 64;   // 64-dimension halves of V
    constexpr int VPR = HD / 8;   // 16-byte vectors per head row
    constexpr int PITCH = HD + 2; // row pitch of q in shared memory: the 8-byte fragment reads below hit 16 different bank pairs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int G = p.heads / p.kv_heads;
    const bool rotate = (DECODE || PREFILL) && p.rope_dim > 0;
    // rotation: this thread owns the pairs (i, i + rope_dim/2) of rows tid / (HD/2), + kSplitThreads / (HD/2), ...;
    // its frequency is a constant of the model and is fetched before the predecessor has finished
    const int pairs = p.rope_dim >> 1;
    const int rot_i = tid & (HD / 2 - 1);
    float inv_f = 0.f;
    if (rotate && rot_i < pairs) inv_f = __ldg(p.inv_freq + rot_i);
    pdl_wait();
    if (p.trace && threadIdx.x == 0) p.trace[cta_linear * 4 + 1] = attn_timer_ns();

    constexpr int kBlock = kSplitWarps * 16;
    // blocks of a pair and of all, this CTA's share
    const int nb = STREAM ? (p.ctx_len + kBlock - 1) / kBlock : 0;
    const unsigned total = STREAM ? (unsigned)(p.splits * nb) : 1u;
    unsigned unit = 0, unit_end = 1;
    if constexpr (STREAM) {
        unit = (unsigned)((unsigned long long)blockIdx.x * total / gridDim.x);
        unit_end = (unsigned)((unsigned long long)(blockIdx.x + 1) * total / gridDim.x);
    }

    __shared__ __align__(16) float qk[kMaxGroup + 1][PITCH];  // rows 0..G-1: q of the group, row G: the new k
    __shared__ float vraw[HD];                                // new v
    __shared__ float self_score[kMaxGroup];                   // q . k of the new token, log2 domain
    __shared__ float osm[kSplitWarps][kMaxGroup][HD + 4];
    __shared__ float msm[kSplitWarps][kMaxGroup], lsm[kSplitWarps][kMaxGroup];

    do {
    int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;   // STREAM: split 0 has the pair's first blocks
    int nsplit = p.splits, blk0 = 0, blk1 = 0, cta_first = 0;   // blk0, blk1: this CTA's blocks of the pair; the CTA that has its first one
    if constexpr (STREAM) {
        const unsigned pair = unit / (unsigned)nb, first = pair * nb;
        b = (int)(pair / (unsigned)p.kv_heads);
        kvh = (int)pair - b * p.kv_heads;
        blk0 = (int)(unit - first);
        blk1 = min(nb, blk0 + (int)(unit_end - unit));
        // the CTA of block x of all: the last one that starts at or before it
        auto cta_of = [&](unsigned x) { return (int)((((unsigned long long)x + 1) * gridDim.x - 1) / total); };
        cta_first = cta_of(first);
        nsplit = cta_of(first + nb - 1) - cta_first + 1;
        split = blk0 == 0 ? 0 : 1;
        unit += (unsigned)(blk1 - blk0);
    }
    // a partial result's place: split `z` of the pair, head r of the group
    auto slot_of = [&](int z, int r) {
        if (STREAM) return (size_t)(2 * (cta_first + z) + (z == 0 ? 1 : 0)) * G + r;
        return ((size_t)b * p.heads + (size_t)kvh * G + r) * p.splits + z;
    };
    auto hop = [&](int z) { return STREAM ? (slot_of(z, 0) - slot_of(0, 0)) * HD : (size_t)z * HD; };   // from split 0's result to z's
    // ---- q and the new k and v are requested first: they do not depend on the position --------------------
    uint4 qv = make_uint4(0, 0, 0, 0), kv = qv, vv = qv;
    const bool has_q = tid < G * VPR;
    const bool has_k = DECODE && tid >= 64 && tid < 64 + VPR;
    const bool has_v = DECODE && tid >= 96 && tid < 96 + VPR;
    if (has_q) qv = *reinterpret_cast<const uint4*>(p.q + (size_t)b * p.q_stride + (size_t)kvh * G * HD + (size_t)tid * 8);
    if (has_k) kv = *reinterpret_cast<const uint4*>(p.k + (size_t)b * p.k_stride + (size_t)kvh * HD + (size_t)(tid - 64) * 8);
    if (has_v) vv = *reinterpret_cast<const uint4*>(p.v + (size_t)b * p.v_stride + (size_t)kvh * HD + (size_t)(tid - 96) * 8);

    // cached tokens to attend (in a decode step the new token is not among them)
    const int n_ctx = DECODE ? p.position[b] : PREFILL ? p.pos_base + b + 1 : p.ctx_len;
    const int rope_pos = PREFILL ? p.pos_base + b : n_ctx;

    const __nv_bfloat16* kbase = p.kcache + (PREFILL ? 0 : (size_t)b * p.cache_seq_stride) + (size_t)kvh * p.cache_head_stride;
    const __nv_bfloat16* vbase = p.vcache + (PREFILL ? 0 : (size_t)b * p.cache_seq_stride) + (size_t)kvh * p.cache_head_stride;

    // ---- tokens of this split: blocks of 64 tokens, block j belongs to split j % splits. A split's first block
    // does not depend on the context length, so in a decode step it is requested before the position has arrived
    // (rows are clamped to the cache's last row there; what lies beyond the context is masked below).
    const int t_begin = STREAM ? blk0 * kBlock : split * kBlock;
    const int t_end = STREAM ? min(n_ctx, blk1 * kBlock) : n_ctx;
    const int t_stride = STREAM ? kBlock : p.splits * kBlock;

    // K and V of 16 tokens per warp live in registers; the first batch is requested before the rest of the
    // prologue so that its trip to HBM overlaps it
    uint4 kreg[2][NCH];
    uint4 va[VH], vb[VH], vc[VH], vd[VH];
    auto load_k = [&](int tok0, int last) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const __nv_bfloat16* rowp = kbase + (size_t)min(tok0 + 8 * nt + g, last) * HD;
#pragma unroll
            for (int i = 0; i < NCH; ++i) kreg[nt][i] = ldg128(rowp + (4 * i + t) * 8);
        }
    };
    auto load_v = [&](int tok0, int last) {
        const __nv_bfloat16* ra = vbase + (size_t)min(tok0 + 2 * t, last) * HD + 8 * g;
        const __nv_bfloat16* rb = vbase + (size_t)min(tok0 + 2 * t + 1, last) * HD + 8 * g;
        const __nv_bfloat16* rc = vbase + (size_t)min(tok0 + 2 * t + 8, last) * HD + 8 * g;
        const __nv_bfloat16* rd = vbase + (size_t)min(tok0 + 2 * t + 9, last) * HD + 8 * g;
#pragma unroll
        for (int hh = 0; hh < VH; ++hh) {
            va[hh] = ldg128(ra + 64 * hh); vb[hh] = ldg128(rb + 64 * hh);
            vc[hh] = ldg128(rc + 64 * hh); vd[hh] = ldg128(rd + 64 * hh);
        }
    };
    int tok0 = t_begin + warp * 16;
    if (p.q_first) { /* requested below, once q, k and v are in shared memory */ }
    else if (DECODE) { load_k(tok0, p.max_seq - 1); load_v(tok0, p.max_seq - 1); }
    else if (tok0 < t_end) { load_k(tok0, t_end - 1); load_v(tok0, t_end - 1); }
    // sliding window (Generator/MetalSourceGenerator+Attention.swift:851-853): cached rows below t_lo are left out.
    // A split whose first blocks lie wholly below the window starts at its first block that reaches into it.
    const int t_lo = p.window > 0 ? max(0, n_ctx + (DECODE ? 1 : 0) - p.window) : 0;
    if (!STREAM && t_lo / kBlock > split) {
        const int skip = (t_lo / kBlock - split + p.splits - 1) / p.splits;
        tok0 = (split + skip * p.splits) * kBlock + warp * 16;
        if (!p.q_first && tok0 < t_end) { load_k(tok0, t_end - 1); load_v(tok0, t_end - 1); }
    }
    // the split's later blocks are asked into L2 (two ahead; the loop keeps that distance): the register loads
    // of the loop then find them there
    constexpr int kAhead = 2;
    auto prefetch_block = [&](int blk_tok) {
        if (blk_tok >= t_end) return;
        const unsigned bytes = (unsigned)(min(kBlock, t_end - blk_tok) * HD * 2);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(kbase + (size_t)blk_tok * HD), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(vbase + (size_t)blk_tok * HD), "r"(bytes) : "memory");
    };
    if (tid < kAhead) prefetch_block(t_begin + (tid + 1) * t_stride);

    // ---- prologue: q, k, v to shared memory as floats; then every pair is rotated once, in place ----------
    float rot_s = 0.f, rot_c = 1.f;
    if (rotate && rot_i < pairs) sincosf((float)rope_pos * inv_f, &rot_s, &rot_c);
    {
        auto spill8 = [](float* dst, const uint4& w) {  // dst is 8-byte aligned
            const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<float2*>(dst + 2 * j) = make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
        };
        if (has_q) spill8(&qk[tid / VPR][(tid % VPR) * 8], qv);
        if (has_k) spill8(&qk[G][(tid - 64) * 8], kv);
        if (has_v) {
            const unsigned u[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { vraw[(tid - 96) * 8 + 2 * j] = __uint_as_float(u[j] << 16); vraw[(tid - 96) * 8 + 2 * j + 1] = __uint_as_float(u[j] & 0xffff0000u); }
            if (split == 0 && n_ctx < p.max_seq)  // the new v row goes to the cache as it is
                *reinterpret_cast<uint4*>(p.vcache + (size_t)b * p.cache_seq_stride + (size_t)kvh * p.cache_head_stride + (size_t)n_ctx * HD + (size_t)(tid - 96) * 8) = vv;
        }
    }
    __syncthreads();
    // 8 MB of K/V requests from all CTAs at once delay the 4 KB of q, k, v that the whole prologue waits for (the
    // memory system serves requests in arrival order): in this mode the rows are requested behind them
    if (p.q_first && tok0 < t_end) { load_k(tok0, t_end - 1); load_v(tok0, t_end - 1); }
    const int n_ctas = gridDim.x * gridDim.y * gridDim.z;
    const bool stamp0 = p.trace && cta_linear == 0 && threadIdx.x == 0;  // finer stamps of the first CTA only
    if (stamp0) p.trace[n_ctas * 4 + 1] = attn_timer_ns();
    if constexpr (QK_NORM) {
        // batched_qk_rms_norm_2 (Generator/MetalSourceGenerator+Batched.swift:681-760) of the G rows of q and of the new k, a warp
        // per row, with the bf16 rounding that a launch of its own leaves; every split repeats it (0.2 us instead of a launch)
        for (int r = warp; r <= G; r += kSplitWarps) {
            const __nv_bfloat16* w = r < G ? p.q_norm : p.k_norm;
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < HD / 32; ++i) { const float v = qk[r][lane + 32 * i]; ss = fmaf(v, v, ss); }
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float rs = rsqrtf(ss / (float)HD + p.qk_eps);
#pragma unroll
            for (int i = 0; i < HD / 32; ++i)
                qk[r][lane + 32 * i] = __bfloat162float(__float2bfloat16_rn(qk[r][lane + 32 * i] * rs * (__bfloat162float(w[lane + 32 * i]) + p.qk_bias)));
        }
        __syncthreads();
    }
    if (rotate) {
        // rotate-half RoPE (Generator/MetalSourceGenerator+Attention.swift:596-617): pairs (i, i + rope_dim/2)
        if (rot_i < pairs)
            for (int r = tid / (HD / 2); r < G + (DECODE ? 1 : 0); r += kSplitThreads / (HD / 2)) {
                const float lo = qk[r][rot_i], hi = qk[r][rot_i + pairs];
                qk[r][rot_i] = lo * rot_c - hi * rot_s;
                qk[r][rot_i + pairs] = lo * rot_s + hi * rot_c;
            }
        __syncthreads();
    }
    if (stamp0) p.trace[(n_ctas + 1) * 4 + 1] = attn_timer_ns();
    if (DECODE) {
        if (split == 0 && n_ctx < p.max_seq) {  // the rotated new k row, rounded, for later steps
            __nv_bfloat16* kw = p.kcache + (size_t)b * p.cache_seq_stride + (size_t)kvh * p.cache_head_stride + (size_t)n_ctx * HD;
            for (int d = tid; d < HD; d += kSplitThreads) kw[d] = __float2bfloat16_rn(qk[G][d]);
        }
        // score of the new token against itself, in fp32 from the unrounded rotated q and k
        // (Generator/MetalSourceGenerator+Attention.swift:866-868)
        for (int r = warp; r < G; r += kSplitWarps) {
            float prod = 0.f;
#pragma unroll
            for (int i = 0; i < HD / 32; ++i) prod = fmaf(qk[r][lane + 32 * i], qk[G][lane + 32 * i], prod);
            for (int o = 16; o > 0; o >>= 1) prod += __shfl_xor_sync(0xffffffffu, prod, o);
            if (lane == 0) self_score[r] = prod * p.scale_log2;
        }
    }

    if (stamp0) p.trace[(n_ctas + 1) * 4 + 2] = attn_timer_ns();
    // A fragments of the rotated q: lane (g, t) holds q[g][32*i + 8*t + 0..7]; hi + lo bf16 split
    unsigned qhi[NCH][4], qlo[NCH][4];
#pragma unroll
    for (int i = 0; i < NCH; ++i)
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            float2 ac = make_float2(0.f, 0.f);
            if (g < G) ac = *reinterpret_cast<const float2*>(&qk[g][32 * i + 8 * t + 2 * w]);
            const float ah = __bfloat162float(__float2bfloat16_rn(ac.x)), ch = __bfloat162float(__float2bfloat16_rn(ac.y));
            qhi[i][w] = pack_bf16(ah, ch);
            qlo[i][w] = pack_bf16(ac.x - ah, ac.y - ch);
        }

    if (stamp0) p.trace[n_ctas * 4 + 2] = attn_timer_ns();
    float m_run = -INFINITY, l_run = 0.f;
    float oacc[VH][8][4];
#pragma unroll
    for (int hh = 0; hh < VH; ++hh)
#pragma unroll
        for (int u = 0; u < 8; ++u) oacc[hh][u][0] = oacc[hh][u][1] = oacc[hh][u][2] = oacc[hh][u][3] = 0.f;

    if (DECODE && tok0 < t_end && tok0 + 16 > t_end) {
        // first batch, requested before the context length was known: rows beyond the context may hold anything;
        // their probabilities are zero, their values must be finite
        const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int hh = 0; hh < VH; ++hh) {
            if (tok0 + 2 * t >= t_end) va[hh] = z;
            if (tok0 + 2 * t + 1 >= t_end) vb[hh] = z;
            if (tok0 + 2 * t + 8 >= t_end) vc[hh] = z;
            if (tok0 + 2 * t + 9 >= t_end) vd[hh] = z;
        }
    }
    for (; tok0 < t_end; tok0 += t_stride) {
        const int nxt = tok0 + t_stride;
        if (tid == 0) prefetch_block(tok0 + (kAhead + 1) * t_stride);
        // S = q . K^T for 16 tokens
        float sacc[2][4];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            sacc[nt][0] = sacc[nt][1] = sacc[nt][2] = sacc[nt][3] = 0.f;
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
                const uint4 kk = kreg[nt][i];
                // rows g carry the high parts of q, rows g + 8 the low parts: one instruction forms both
                // products, and their sum is taken in-lane below
                mma_bf16(sacc[nt], qhi[i][0], qlo[i][0], qhi[i][1], qlo[i][1], kk.x, kk.y);
                mma_bf16(sacc[nt], qhi[i][2], qlo[i][2], qhi[i][3], qlo[i][3], kk.z, kk.w);
            }
        }
        if (nxt < t_end) load_k(nxt, t_end - 1);  // the K registers are free again
        // online softmax in the log2 domain; row g lives in the four lanes t = 0..3
        float sv[2][2];
        float rmax = -INFINITY;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tok = tok0 + 8 * nt + 2 * t + e;
                sv[nt][e] = tok < t_end && tok >= t_lo ? (sacc[nt][e] + sacc[nt][2 + e]) * p.scale_log2 : -INFINITY;
                rmax = fmaxf(rmax, sv[nt][e]);
            }
        rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 1));
        rmax = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, 2));
        const float m_new = fmaxf(m_run, rmax);
        const float m_ref = m_new == -INFINITY ? 0.f : m_new;  // 16 rows wholly below a sliding window: all weights 0
        const float corr = exp2f(m_run - m_ref);
        float pv[2][2];
        float psum = 0.f;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) { pv[nt][e] = exp2f(sv[nt][e] - m_ref); psum += pv[nt][e]; }
        l_run = l_run * corr + psum;
        m_run = m_new;
        if (__any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll
            for (int hh = 0; hh < VH; ++hh)
#pragma unroll
                for (int u = 0; u < 8; ++u) { oacc[hh][u][0] *= corr; oacc[hh][u][1] *= corr; oacc[hh][u][2] *= corr; oacc[hh][u][3] *= corr; }
        }
        // O += P . V ; dimension 64*hh + 8*col + u sits in n-tile (hh, u), column col. P is fed as a bf16
        // hi + lo pair: a single bf16 P (8 mantissa bits) costs ~2 bf16 ulps of the output at short contexts.
        float ph[2][2];
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) ph[nt][e] = __bfloat162float(__float2bfloat16_rn(pv[nt][e]));
        const unsigned pa0 = pack_bf16(ph[0][0], ph[0][1]);
        const unsigned pa2 = pack_bf16(ph[1][0], ph[1][1]);
        const unsigned pl0 = pack_bf16(pv[0][0] - ph[0][0], pv[0][1] - ph[0][1]);
        const unsigned pl2 = pack_bf16(pv[1][0] - ph[1][0], pv[1][1] - ph[1][1]);
#pragma unroll
        for (int hh = 0; hh < VH; ++hh) {
            const unsigned aw[4] = {va[hh].x, va[hh].y, va[hh].z, va[hh].w};
            const unsigned bw[4] = {vb[hh].x, vb[hh].y, vb[hh].z, vb[hh].w};
            const unsigned cw[4] = {vc[hh].x, vc[hh].y, vc[hh].z, vc[hh].w};
            const unsigned dw[4] = {vd[hh].x, vd[hh].y, vd[hh].z, vd[hh].w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const unsigned b0e = __byte_perm(aw[w], bw[w], 0x5410), b1e = __byte_perm(cw[w], dw[w], 0x5410);
                const unsigned b0o = __byte_perm(aw[w], bw[w], 0x7632), b1o = __byte_perm(cw[w], dw[w], 0x7632);
                // rows g: high part of P, rows g + 8: low part; added when the accumulators are read out
                mma_bf16(oacc[hh][2 * w], pa0, pl0, pa2, pl2, b0e, b1e);
                mma_bf16(oacc[hh][2 * w + 1], pa0, pl0, pa2, pl2, b0o, b1o);
            }
        }
        if (nxt < t_end) load_v(nxt, t_end - 1);
        if (stamp0 && tok0 == t_begin) p.trace[n_ctas * 4 + 3] = attn_timer_ns();
    }

    if (p.trace && threadIdx.x == 0) p.trace[cta_linear * 4 + 2] = attn_timer_ns();
    // ---- merge the warps of this CTA ---------------------------------------------------------------
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (g < G) {
#pragma unroll
        for (int hh = 0; hh < VH; ++hh)
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                osm[warp][g][64 * hh + 8 * (2 * t) + u] = oacc[hh][u][0] + oacc[hh][u][2];
                osm[warp][g][64 * hh + 8 * (2 * t + 1) + u] = oacc[hh][u][1] + oacc[hh][u][3];
            }
        if (t == 0) { msm[warp][g] = m_run; lsm[warp][g] = l_run; }
    }
    __syncthreads();
    for (int idx = tid; idx < G * HD; idx += kSplitThreads) {
        const int r = idx / HD, d = idx - r * HD;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < kSplitWarps; ++w) mx = fmaxf(mx, msm[w][r]);
        float o = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < kSplitWarps; ++w) {
            const float wgt = msm[w][r] == -INFINITY ? 0.f : exp2f(msm[w][r] - mx);
            o = fmaf(wgt, osm[w][r][d], o);
            l = fmaf(wgt, lsm[w][r], l);
        }
        const size_t slot = STREAM ? (size_t)(2 * blockIdx.x + (blk0 == 0 ? 1 : 0)) * G + r : slot_of(split, r);
        __stcg(p.part_o + slot * HD + d, o);
        if (d == 0) { __stcg(p.part_ml + slot * 2, mx); __stcg(p.part_ml + slot * 2 + 1, l); }
    }

    // ---- the last CTA of this (sequence, KV head) to arrive merges the splits and writes the output ----
    __shared__ int is_last;
    __syncthreads();
    if (tid == 0) {
        // release: cumulative over the partials every thread of this CTA wrote before the barrier; acquire: the
        // last arriver sees the partials of all the others
        unsigned* ctr = p.counters + (size_t)b * p.kv_heads + kvh;
        unsigned prev;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(prev) : "l"(ctr) : "memory");
        is_last = prev == (unsigned)nsplit - 1u;
        if (is_last) *ctr = 0u;  // ready for the next launch
    }
    __syncthreads();
    if (p.trace && threadIdx.x == 0) p.trace[cta_linear * 4 + 3] = attn_timer_ns();
    if (is_last) {

    // Everything that does not depend on the split weights is requested first: the (max, sum) pairs and the
    // first 16 partial outputs of this thread's four dimensions travel together.
    // (a pair of MODE 4 has eight parts at most. With heads of 64 room for more costs the third CTA per SM; with heads of 128 room for eight
    // only gives a loop that is 5 to 13 % slower in long caches: 41 x 5000 rows 160 us, with sixteen 143)
    constexpr int kPre = !STREAM ? 32 : HD == 128 ? 16 : 8;
    const int n_out4 = G * HD / 4;  // float4 outputs of the group
    float* wsm = &osm[1][0][0];     // [G][splits] weights (splits <= 64: fits the reused buffer)
    float* msm2 = &osm[2][0][0];    // [G][splits] split maxima
    float* lsm2 = &osm[3][0][0];    // [G][splits] split sums
    float2 ml[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int idx = tid + j * kSplitThreads;
        if (idx < G * nsplit) {
            const int r = idx / nsplit, sidx = idx - r * nsplit;
            const size_t slot = slot_of(sidx, r);
            ml[j] = __ldcg(reinterpret_cast<const float2*>(p.part_ml + slot * 2));
        }
    }
    float4 pre[kPre];
    const float* po0 = nullptr;
    if (tid < n_out4) {
        const int r = tid / (HD / 4), d4 = tid - r * (HD / 4);
        po0 = p.part_o + slot_of(0, r) * HD + d4 * 4;
#pragma unroll
        for (int sidx = 0; sidx < kPre; ++sidx)
            if (sidx < nsplit) pre[sidx] = __ldcg(reinterpret_cast<const float4*>(po0 + hop(sidx)));
    }
    for (int j = 0; j < 2; ++j) {
        const int idx = tid + j * kSplitThreads;
        if (idx < G * nsplit) { msm2[idx] = ml[j].x; lsm2[idx] = ml[j].y; }
    }
    for (int idx = tid + 2 * kSplitThreads; idx < G * nsplit; idx += kSplitThreads) {
        const int r = idx / nsplit, sidx = idx - r * nsplit;
        const size_t slot = slot_of(sidx, r);
        msm2[idx] = __ldcg(p.part_ml + slot * 2);
        lsm2[idx] = __ldcg(p.part_ml + slot * 2 + 1);
    }
    __syncthreads();
    // weights of the splits: w = 2^(m_s - max), normalised by the total mass; the new token enters with its
    // own score and its unrounded v (Generator/MetalSourceGenerator+Attention.swift:905-907)
    float* inv_den = msm[0];  // reuse: G floats
    float* w_self = msm[1];
    for (int r = warp; r < G; r += kSplitWarps) {
        const float m_self = DECODE ? self_score[r] : -INFINITY;
        float mx = m_self;
        for (int sidx = lane; sidx < nsplit; sidx += 32) mx = fmaxf(mx, msm2[r * nsplit + sidx]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float den = 0.f;
        for (int sidx = lane; sidx < nsplit; sidx += 32) {
            const float ms = msm2[r * nsplit + sidx];
            const float w = ms == -INFINITY ? 0.f : exp2f(ms - mx);
            wsm[r * nsplit + sidx] = w;
            den = fmaf(w, lsm2[r * nsplit + sidx], den);
        }
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        const float ws = DECODE ? exp2f(m_self - mx) : 0.f;
        den += ws;
        if (lane == 0) { inv_den[r] = den > 0.f ? 1.0f / den : 0.f; w_self[r] = ws; }
    }
    __syncthreads();
    for (int idx = tid; idx < n_out4; idx += kSplitThreads) {
        const int r = idx / (HD / 4), d4 = idx - r * (HD / 4);
        const float* po = p.part_o + slot_of(0, r) * HD + d4 * 4;
        const float* wr = wsm + r * nsplit;
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
        if (DECODE) {
            const float ws = w_self[r];
            num = make_float4(ws * vraw[d4 * 4], ws * vraw[d4 * 4 + 1], ws * vraw[d4 * 4 + 2], ws * vraw[d4 * 4 + 3]);
        }
        int s0 = 0;
        if (idx == tid) {  // this thread's first output: its first partials are already in registers
#pragma unroll
            for (int sidx = 0; sidx < kPre; ++sidx)
                if (sidx < nsplit) {
                    const float w = wr[sidx];
                    num.x = fmaf(w, pre[sidx].x, num.x); num.y = fmaf(w, pre[sidx].y, num.y);
                    num.z = fmaf(w, pre[sidx].z, num.z); num.w = fmaf(w, pre[sidx].w, num.w);
                }
            s0 = min(kPre, nsplit);
        }
#pragma unroll 16
        for (int sidx = s0; sidx < nsplit; ++sidx) {
            const float4 v4 = __ldcg(reinterpret_cast<const float4*>(po + hop(sidx)));
            const float w = wr[sidx];
            num.x = fmaf(w, v4.x, num.x); num.y = fmaf(w, v4.y, num.y);
            num.z = fmaf(w, v4.z, num.z); num.w = fmaf(w, v4.w, num.w);
        }
        const float inv = inv_den[r];
        uint2 packed;
        packed.x = pack_bf16(num.x * inv, num.y * inv);
        packed.y = pack_bf16(num.z * inv, num.w * inv);
        *reinterpret_cast<uint2*>(p.out + (size_t)b * p.out_stride + (size_t)(kvh * G + r) * HD + d4 * 4) = packed;
    }
    if (p.trace) {
        __syncthreads();
        if (threadIdx.x == 0) p.trace[(gridDim.x * gridDim.y * gridDim.z + (blockIdx.z * gridDim.y + blockIdx.y)) * 4] = attn_timer_ns();  // merged
    }
    }   // is_last
    if (STREAM) __syncthreads();   // (shared memory is written again for the next pair)
    } while (STREAM && unit < unit_end);
}

// Prompt ingestion: rotate the chunk's k rows (token b at position pos_base + b) and append them and the v rows to
// the cache of sequence 0, rounded to bf16 (Generator/MetalSourceGenerator+Attention.swift:761-805 does the same
// per decode step). A warp takes one to four KV heads of a token at a time: their angles are worked out once, and their keys and values are
// requested before any is stored (the cache may overlap its inputs for all the compiler knows: with each head's stores in front of the next
// one's loads 40 tokens x 8 heads of 128 took 14.8 us under ncu, 2048 14.7). 40 tokens 4.5 us, 512 4.8, 1024 5.8, 2048 7.5; with a CTA per
// token and head, each with angles of its own, 4.1, 7.2, 11.2 and 19.9.
constexpr int kRopeWarps = 4, kRopeAhead = 4;
__global__ void __launch_bounds__(kRopeWarps * 32) rope_append_kernel(const AttnParams p, int hd, int heads_each) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.x * kRopeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int pos = p.pos_base + b, pairs = p.rope_dim >> 1, h_end = min(p.kv_heads, ((int)blockIdx.y + 1) * heads_each);
    if (b >= p.chunk_tokens || pos >= p.max_seq) return;
    const bool wide = ((hd | p.v_stride) & 7) == 0 && ((reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.vcache)) & 15) == 0 && (p.cache_head_stride & 7) == 0;
    const __nv_bfloat16* const k_row = p.k + (size_t)b * p.k_stride;
    const __nv_bfloat16* const v_row = p.v + (size_t)b * p.v_stride;
    const size_t to_pos = (size_t)pos * hd;
    const int vecs = hd >> 3;   // (at most 16)
    float cs[2], sn[2];         // (at most 64 pairs)
#pragma unroll
    for (int j = 0; j < 2; ++j)
        if (lane + 32 * j < pairs) sincosf((float)pos * p.inv_freq[lane + 32 * j], &sn[j], &cs[j]);
    for (int h0 = (int)blockIdx.y * heads_each; h0 < h_end; h0 += kRopeAhead) {
        const int heads = min(kRopeAhead, h_end - h0);
        __nv_bfloat16 lo[kRopeAhead][2], hi[kRopeAhead][2];
        uint4 v[kRopeAhead / 2];
#pragma unroll
        for (int u = 0; u < kRopeAhead; ++u)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (u < heads && lane + 32 * j < pairs) {
                    const __nv_bfloat16* k = k_row + (h0 + u) * hd + lane + 32 * j;
                    lo[u][j] = k[0]; hi[u][j] = k[pairs];
                }
        if (wide) {
#pragma unroll
            for (int j = 0; j < kRopeAhead / 2; ++j)
                if (lane + 32 * j < heads * vecs) v[j] = *reinterpret_cast<const uint4*>(v_row + h0 * hd + 8 * (lane + 32 * j));
        }
#pragma unroll
        for (int u = 0; u < kRopeAhead; ++u)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (u < heads && lane + 32 * j < pairs) {
                    __nv_bfloat16* at = p.kcache + (size_t)(h0 + u) * p.cache_head_stride + to_pos + lane + 32 * j;
                    const float x = __bfloat162float(lo[u][j]), y = __bfloat162float(hi[u][j]);
                    at[0] = __float2bfloat16_rn(x * cs[j] - y * sn[j]);
                    at[pairs] = __float2bfloat16_rn(x * sn[j] + y * cs[j]);
                }
        if (wide) {
#pragma unroll
            for (int j = 0; j < kRopeAhead / 2; ++j)
                if (lane + 32 * j < heads * vecs) {
                    const int u = (lane + 32 * j) / vecs, i = lane + 32 * j - u * vecs;
                    reinterpret_cast<uint4*>(p.vcache + (size_t)(h0 + u) * p.cache_head_stride + to_pos)[i] = v[j];
                }
        }
        for (int u = 0; u < heads; ++u) {
            const size_t row = (size_t)(h0 + u) * p.cache_head_stride + to_pos;
            for (int d = p.rope_dim + lane; d < hd; d += 32) p.kcache[row + d] = k_row[(h0 + u) * hd + d];
            if (!wide)
                for (int d = lane; d < hd; d += 32) p.vcache[row + d] = v_row[(h0 + u) * hd + d];
        }
    }
}

int check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, what);
    return SWLM_OK;
}


// ---- decode attention over a quantized cache (8-bit groups of 32 / 64 / 128, 4-bit groups of 64 / 128) ----------------
// Rows are head_dim / group blocks of fp16 scale | fp16 zero | payload (36 bytes for 8-bit groups of 32), value = scale * q + zero
// (read_kv_element, Generator/MetalSourceGenerator+Attention.swift:1923-1956). Half the bytes of the bf16 cache cross
// HBM. One CTA per (split, KV head, sequence) as in the bf16 kernel; a warp takes one token at a time, every lane
// dequantises its head_dim / 32 consecutive elements of the K row and of the V row and the dot products of the GQA
// group's q rows are reduced across the warp; online softmax in fp32. The new token enters with its unrounded rotated k
// and its v (:866-868, :905-907); split 0 quantises both into the cache (write_kv_quantized_q8, :2057-2101: scale =
// (max - min) / 255 per group, q = round((x - min) / scale), fp16 scale and min stored). The last CTA of a
// (sequence, KV head) to arrive merges the splits.
constexpr int kQ8Warps = 8, kQ8Threads = kQ8Warps * 32;

// One row of head_dim floats into blocks of `group` values with `bits` bits each: a warp per group, a lane takes
// group / 32 consecutive values (write_kv_quantized_q8 / _q4, Generator/MetalSourceGenerator+Attention.swift:2057-2150).
// RESID: resid[i] = src[i] - the value the stored block gives back for it (fp16 scale and zero), the residual that
// qjl_compute_residual (:1983-2013) projects.
template <bool RESID = false>
__device__ __forceinline__ void q8_quantise_row(const float* src, unsigned char* row, int hd, int bits, int group, int warp, int lane, float* resid = nullptr) {
    const int epg = group / 32, bb = 4 + group * bits / 8;
    const float levels = bits == 8 ? 255.0f : 15.0f;
    for (int g = warp; g * group < hd; g += kQ8Warps) {
        float x[4];
        float lo = HUGE_VALF, hi = -HUGE_VALF;
        for (int j = 0; j < epg; ++j) { x[j] = src[g * group + lane * epg + j]; lo = fminf(lo, x[j]); hi = fmaxf(hi, x[j]); }
        for (int o = 16; o > 0; o >>= 1) { lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o)); hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o)); }
        float scale = (hi - lo) / levels;
        if (scale < 1e-10f) scale = 1e-10f;
        unsigned char* blk = row + (size_t)g * bb;
        if (lane == 0) {
            const __half2 hdr = __floats2half2_rn(scale, lo);
            *reinterpret_cast<__half2*>(blk) = hdr;
        }
        int q[4];
        for (int j = 0; j < epg; ++j) q[j] = min(max((int)roundf((x[j] - lo) / scale), 0), (int)levels);
        if (RESID) {
            const float sh = __half2float(__float2half_rn(scale)), zh = __half2float(__float2half_rn(lo));
            for (int j = 0; j < epg; ++j) resid[g * group + lane * epg + j] = x[j] - fmaf(sh, (float)q[j], zh);
        }
        if (bits == 8) {
            for (int j = 0; j < epg; ++j) blk[4 + lane * epg + j] = (unsigned char)q[j];
        } else {   // two values per byte, the even one in the low nibble (epg is 2 or 4)
            for (int j = 0; j < epg; j += 2) blk[4 + (lane * epg + j) / 2] = (unsigned char)(q[j] | (q[j + 1] << 4));
        }
    }
}

// Sandwich product of Cl(3,0) (rotor_sandwich / rotor_sandwich_inverse, Generator/MetalSourceGenerator+Attention.swift:
// 1807-1821): the rotor R = (s, b12, b13, b23) turns (x, y, z) like the unit quaternion (s, b23, -b13, b12), in the
// cross-product form v + s t + p x t with t = 2 p x v; INV uses the conjugate.
template <bool INV>
__device__ __forceinline__ void rotor_turn(const __half* R, float& x, float& y, float& z) {
    const float s = __half2float(R[0]);
    float px = __half2float(R[3]), py = -__half2float(R[2]), pz = __half2float(R[1]);
    if (INV) { px = -px; py = -py; pz = -pz; }
    const float tx = 2.0f * (py * z - pz * y), ty = 2.0f * (pz * x - px * z), tz = 2.0f * (px * y - py * x);
    const float rx = x + s * tx + (py * tz - pz * ty);
    const float ry = y + s * ty + (pz * tx - px * tz);
    const float rz = z + s * tz + (px * ty - py * tx);
    x = rx; y = ry; z = rz;
}
// group g = values 3g .. 3g + 2 of a row of hd floats, in place; values past the row's end enter as zeros and are not
// stored (rotor_apply_forward / _inverse, :1827-1884)
template <bool INV>
__device__ __forceinline__ void rotor_turn_group(float* row, int hd, const __half* rotors, int g) {
    const int base = 3 * g;
    float x = row[base], y = base + 1 < hd ? row[base + 1] : 0.0f, z = base + 2 < hd ? row[base + 2] : 0.0f;
    rotor_turn<INV>(rotors + 4 * g, x, y, z);
    row[base] = x;
    if (base + 1 < hd) row[base + 1] = y;
    if (base + 2 < hd) row[base + 2] = z;
}

// G (query heads per KV head) is a template argument: the per-head dot products, warp reductions and softmax updates of
// a row are then one basic block whose four or eight independent chains the compiler interleaves.
//
// ROTOR (the rotated schemes, :694-930): q, the new k (both after RoPE) and the new v are turned by the KV head's rotors
// before anything else, so the cache holds turned rows and q . k is unchanged; the merged output is turned back. With
// qjl_dim > 0 split 0 also stores Phi . (k - its dequantised row) for the new row, and the score of a cached row gains
// (Phi . q) . (that row's stored values): lane l carries columns l and l + 32 of both into the warp reduction.
// (Up to four query heads per KV head the rotated form is held to 128 registers so that two CTAs share an SM like the
// plain form's, which fits by itself: the kernel is bound by instruction issue and needs both. The plain form states no
// minimum - a minimum of one would let the compiler spread it over 150 registers and halve its occupancy.)
template <int HD, int G, int BITS, bool ROTOR>
__global__ void __launch_bounds__(kQ8Threads, ROTOR && G <= 4 ? 2 : 0) attn_q8_split_kernel(const AttnParams p) {
    constexpr int EPL = HD / 32;           // elements per lane
    constexpr int NG = (HD + 2) / 3;       // rotors per KV head
    const int GROUP = p.kv_group, BB = 4 + GROUP * BITS / 8;   // values and bytes per block (BITS per value)
    const int ROW_BYTES = HD / GROUP * BB;
    pdl_launch_dependents();
    const int split = blockIdx.x, kvh = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ float qs[G][HD];
    __shared__ float kcur[HD], vcur[HD];
    __shared__ float osm[kQ8Warps][kMaxGroup][HD];   // (sized for the merge scratch below whatever G is)
    __shared__ float msm[kQ8Warps][kMaxGroup], lsm[kQ8Warps][kMaxGroup];
    __shared__ __align__(16) float weights[kQ8Warps][8 * G];   // of a batch of eight rows
    __shared__ int is_last;
    __shared__ float kres[ROTOR ? HD : 1];          // the new k row minus its dequantised blocks
    __shared__ float qp[ROTOR ? G : 1][64];         // Phi . q of every head of the group
    const __half* const head_rotors = ROTOR ? p.rotors + (size_t)kvh * NG * 4 : nullptr;
    const int qjl = ROTOR ? p.qjl_dim : 0;
    pdl_wait();
    const int n_ctx = p.position[b];
    const size_t head_bytes = (size_t)p.max_seq * ROW_BYTES;
    unsigned char* kbase = reinterpret_cast<unsigned char*>(p.kcache) + ((size_t)b * p.kv_heads + kvh) * head_bytes;
    unsigned char* vbase = reinterpret_cast<unsigned char*>(p.vcache) + ((size_t)b * p.kv_heads + kvh) * head_bytes;
    // the split's share of the cached rows [t_lo, n_ctx): contiguous; a warp takes every eighth row of it. All of it is asked into L2
    // before q is staged and rotated
    const int t_lo = p.window > 0 ? max(0, n_ctx + 1 - p.window) : 0;
    const int per = (n_ctx - t_lo + p.splits - 1) / p.splits;
    const int t0 = t_lo + split * per, t1 = min(n_ctx, t0 + per);
    for (int off = tid * 128; off < (t1 - t0) * ROW_BYTES; off += kQ8Threads * 128) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(kbase + (size_t)t0 * ROW_BYTES + off));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(vbase + (size_t)t0 * ROW_BYTES + off));
    }
    for (int idx = tid; idx < G * HD; idx += kQ8Threads)
        qs[idx / HD][idx % HD] = __bfloat162float(p.q[(size_t)b * p.q_stride + (size_t)kvh * G * HD + idx]);
    for (int d = tid; d < HD; d += kQ8Threads) {
        kcur[d] = __bfloat162float(p.k[(size_t)b * p.k_stride + (size_t)kvh * HD + d]);
        vcur[d] = __bfloat162float(p.v[(size_t)b * p.v_stride + (size_t)kvh * HD + d]);
    }
    __syncthreads();
    if (p.rope_dim > 0) {
        // rotate-half RoPE (Generator/MetalSourceGenerator+Attention.swift:596-617): pairs (i, i + rope_dim/2)
        const int pairs = p.rope_dim >> 1;
        for (int idx = tid; idx < (G + 1) * pairs; idx += kQ8Threads) {
            const int r = idx / pairs, i = idx - r * pairs;
            float sn, cs;
            sincosf((float)n_ctx * p.inv_freq[i], &sn, &cs);
            float* row = r < G ? qs[r] : kcur;
            const float lo = row[i], hi = row[i + pairs];
            row[i] = lo * cs - hi * sn;
            row[i + pairs] = lo * sn + hi * cs;
        }
        __syncthreads();
    }
    if (ROTOR) {
        for (int idx = tid; idx < (G + 2) * NG; idx += kQ8Threads) {
            const int r = idx / NG, g = idx - r * NG;
            rotor_turn_group<false>(r < G ? qs[r] : r == G ? kcur : vcur, HD, head_rotors, g);
        }
        __syncthreads();
    }
    const __half* const res_base = ROTOR && qjl > 0 ? p.qjl_res + ((size_t)b * p.kv_heads + kvh) * p.max_seq * qjl : nullptr;
    if (split == 0 && n_ctx < p.max_seq) {
        q8_quantise_row<ROTOR>(kcur, kbase + (size_t)n_ctx * ROW_BYTES, HD, BITS, GROUP, warp, lane, kres);
        q8_quantise_row(vcur, vbase + (size_t)n_ctx * ROW_BYTES, HD, BITS, GROUP, warp, lane);
        if (ROTOR && qjl > 0) {   // (the branch is uniform over the CTA)
            __syncthreads();
            __half* res = p.qjl_res + (((size_t)b * p.kv_heads + kvh) * p.max_seq + n_ctx) * qjl;
            for (int j = warp; j < qjl; j += kQ8Warps) {
                float a = 0.f;
                for (int d = lane; d < HD; d += 32) a = fmaf(kres[d], __half2float(__ldg(p.qjl_matrix + (size_t)d * qjl + j)), a);
                for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (lane == 0) res[j] = __float2half_rn(a);
            }
        }
    }
    float qpr[G][2];   // this lane's two columns of Phi . q (zero past qjl_dim)
#pragma unroll
    for (int r = 0; r < G; ++r) qpr[r][0] = qpr[r][1] = 0.f;
    if (ROTOR && qjl > 0) {
        const int cols = ROTOR ? qjl : 1;   // (the plain instantiation never gets here; keeps its dead code free of a constant zero divisor)
        for (int idx = tid; idx < G * qjl; idx += kQ8Threads) {
            const int r = idx / cols, j = idx - r * cols;
            float a = 0.f;
            for (int d = 0; d < HD; ++d) a = fmaf(qs[r][d], __half2float(__ldg(p.qjl_matrix + (size_t)d * qjl + j)), a);
            qp[r][j] = a;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < G; ++r) {
            if (lane < qjl) qpr[r][0] = qp[r][lane];
            if (lane + 32 < qjl) qpr[r][1] = qp[r][lane + 32];
        }
    }
    // this lane's elements e0 .. e0 + EPL - 1 lie in one block; its payload is EPL * BITS / 8 bytes (4, 2 or 1),
    // naturally aligned
    const int e0 = lane * EPL, blk_off = (e0 / GROUP) * BB, pay_off = blk_off + 4 + (e0 % GROUP) * BITS / 8;
    constexpr int pay_bytes = EPL * BITS / 8;
    constexpr unsigned qmask = BITS == 8 ? 0xffu : 0xfu;
    auto load_payload = [&](const unsigned char* ptr) -> unsigned {
        if (pay_bytes == 4) return __ldg(reinterpret_cast<const unsigned*>(ptr));
        if (pay_bytes == 2) return __ldg(reinterpret_cast<const unsigned short*>(ptr));
        return __ldg(ptr);
    };
    float qr[G][EPL];
#pragma unroll
    for (int r = 0; r < G; ++r)
#pragma unroll
        for (int j = 0; j < EPL; ++j) qr[r][j] = qs[r][e0 + j];
    float m_run[G], l_run[G], acc[G][EPL];
#pragma unroll
    for (int r = 0; r < G; ++r) {
        m_run[r] = -INFINITY; l_run[r] = 0.f;
#pragma unroll
        for (int j = 0; j < EPL; ++j) acc[r][j] = 0.f;
    }
    // one row's scores (already reduced over the warp, unscaled) and values enter the running softmax of every head
    auto update = [&](const float (&sc)[G], const float (&vf)[EPL]) {
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const float s = sc[r] * p.scale_log2;
            const float m_new = fmaxf(m_run[r], s);
            const float corr = exp2f(m_run[r] - m_new), w = exp2f(s - m_new);
            l_run[r] = l_run[r] * corr + w;
            m_run[r] = m_new;
#pragma unroll
            for (int j = 0; j < EPL; ++j) acc[r][j] = fmaf(w, vf[j], acc[r][j] * corr);
        }
    };
    // eight rows per warp are requested before the first is used: one trip to memory per eight rows instead of one per row
    constexpr int UN = 8;
    constexpr int NV = UN * G, VPL = NV > 32 ? NV / 32 : 1, REP = NV < 32 ? 32 / NV : 1;   // values of a batch, per lane, lanes per value
    float m_l[VPL], l_l[VPL];   // running maximum and sum (of this lane's rows) of the heads this lane's values belong to
#pragma unroll
    for (int e = 0; e < VPL; ++e) { m_l[e] = -INFINITY; l_l[e] = 0.f; }
    for (int tb = t0 + warp; tb < t1; tb += kQ8Warps * UN) {
        unsigned kw[UN], vw[UN], khd[UN], vhd[UN];
        unsigned short rz0[ROTOR ? UN : 1], rz1[ROTOR ? UN : 1];   // the row's projected residual, columns lane and lane + 32
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const int t = min(tb + u * kQ8Warps, t1 - 1);   // rows past the end repeat the last one and are not absorbed
            const unsigned char* kr = kbase + (size_t)t * ROW_BYTES;
            const unsigned char* vr = vbase + (size_t)t * ROW_BYTES;
            khd[u] = __ldg(reinterpret_cast<const unsigned*>(kr + blk_off));
            vhd[u] = __ldg(reinterpret_cast<const unsigned*>(vr + blk_off));
            kw[u] = load_payload(kr + pay_off);
            vw[u] = load_payload(vr + pay_off);
            if (ROTOR) {
                rz0[u] = rz1[u] = 0;
                if (qjl > 0) {
                    const unsigned short* rr = reinterpret_cast<const unsigned short*>(res_base) + (size_t)t * qjl;
                    if (lane < qjl) rz0[u] = __ldg(rr + lane);
                    if (lane + 32 < qjl) rz1[u] = __ldg(rr + lane + 32);
                }
            }
        }
        // the scores of the eight rows for all heads, value u * G + r: partial sums of this lane's elements
        float sc[NV];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const __half2 kh = *reinterpret_cast<const __half2*>(&khd[u]);
            const float ks = __low2float(kh), kz = __high2float(kh);
            float kf[EPL];
#pragma unroll
            for (int j = 0; j < EPL; ++j) kf[j] = fmaf(ks, (float)((kw[u] >> (BITS * j)) & qmask), kz);
#pragma unroll
            for (int r = 0; r < G; ++r) {
                float a = 0.f;
#pragma unroll
                for (int j = 0; j < EPL; ++j) a = fmaf(qr[r][j], kf[j], a);
                sc[u * G + r] = a;
            }
            if (ROTOR) {
                const float r0 = __half2float(__ushort_as_half(rz0[u])), r1 = __half2float(__ushort_as_half(rz1[u]));
#pragma unroll
                for (int r = 0; r < G; ++r) sc[u * G + r] = fmaf(qpr[r][1], r1, fmaf(qpr[r][0], r0, sc[u * G + r]));
            }
        }
        // summed over the warp so that every lane ends with values of its own: at each exchange a lane keeps one half of what it has
        // and gives the other away (31 exchanges for 32 values instead of 160), and one lane works out a value's weight instead of all
#pragma unroll
        for (int st = 0; st < 5; ++st) {
            const int o = 16 >> st, have = NV >> st;
            if (have > 1) {
                const bool up = lane & o;
#pragma unroll
                for (int i = 0; i < (have > 1 ? have / 2 : 1); ++i) {
                    const float keep = up ? sc[have / 2 + i] : sc[i], give = up ? sc[i] : sc[have / 2 + i];
                    sc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            } else {
                sc[0] += __shfl_xor_sync(0xffffffffu, sc[0], o);
            }
        }
        float corr_l[VPL];
#pragma unroll
        for (int e = 0; e < VPL; ++e) {
            const int idx = lane * VPL / REP + e, u = idx / G;   // rows past the end get weight 0
            const float s = tb + u * kQ8Warps < t1 ? sc[e] * p.scale_log2 : -INFINITY;
            float top = s;   // over the rows of the same head
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            const float m_new = fmaxf(m_l[e], top);              // finite: the batch's first row is inside the range
            corr_l[e] = exp2f(m_l[e] - m_new);
            const float w = exp2f(s - m_new);
            l_l[e] = l_l[e] * corr_l[e] + w;
            m_l[e] = m_new;
            if (lane % REP == 0) weights[warp][idx] = w;
        }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < G; ++r) {
            const float corr = __shfl_sync(0xffffffffu, corr_l[r % VPL], r * REP / VPL);
#pragma unroll
            for (int j = 0; j < EPL; ++j) acc[r][j] *= corr;
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
            const __half2 vh = *reinterpret_cast<const __half2*>(&vhd[u]);
            const float vs = __low2float(vh), vz = __high2float(vh);
            float vf[EPL];
#pragma unroll
            for (int j = 0; j < EPL; ++j) vf[j] = fmaf(vs, (float)((vw[u] >> (BITS * j)) & qmask), vz);
#pragma unroll
            for (int r = 0; r < G; ++r) {
                const float w = weights[warp][u * G + r];
#pragma unroll
                for (int j = 0; j < EPL; ++j) acc[r][j] = fmaf(w, vf[j], acc[r][j]);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int e = 0; e < VPL; ++e)
        for (int o = 4; o < 32; o <<= 1) l_l[e] += __shfl_xor_sync(0xffffffffu, l_l[e], o);
#pragma unroll
    for (int r = 0; r < G; ++r) {
        m_run[r] = __shfl_sync(0xffffffffu, m_l[r % VPL], r * REP / VPL);
        l_run[r] = __shfl_sync(0xffffffffu, l_l[r % VPL], r * REP / VPL);
    }
    if (split == 0 && warp == 0) {   // the new token: unrounded rotated k, v as given
        float vf[EPL], sc[G];
#pragma unroll
        for (int j = 0; j < EPL; ++j) vf[j] = vcur[e0 + j];
#pragma unroll
        for (int r = 0; r < G; ++r) {
            sc[r] = 0.f;
#pragma unroll
            for (int j = 0; j < EPL; ++j) sc[r] = fmaf(qr[r][j], kcur[e0 + j], sc[r]);
            for (int o = 16; o > 0; o >>= 1) sc[r] += __shfl_xor_sync(0xffffffffu, sc[r], o);
        }
        update(sc, vf);
    }
    // ---- merge the warps, publish the split's partial ----------------------------------------------------
#pragma unroll
    for (int r = 0; r < G; ++r) {
#pragma unroll
        for (int j = 0; j < EPL; ++j) osm[warp][r][e0 + j] = acc[r][j];
        if (lane == 0) { msm[warp][r] = m_run[r]; lsm[warp][r] = l_run[r]; }
    }
    __syncthreads();
    for (int idx = tid; idx < G * HD; idx += kQ8Threads) {
        const int r = idx / HD, d = idx - r * HD;
        float mx = -INFINITY;
        for (int w = 0; w < kQ8Warps; ++w) mx = fmaxf(mx, msm[w][r]);
        float o = 0.f, l = 0.f;
        for (int w = 0; w < kQ8Warps; ++w) {
            const float wgt = msm[w][r] == -INFINITY ? 0.f : exp2f(msm[w][r] - mx);
            o = fmaf(wgt, osm[w][r][d], o);
            l = fmaf(wgt, lsm[w][r], l);
        }
        const size_t slot = ((size_t)b * p.heads + (size_t)kvh * G + r) * p.splits + split;
        __stcg(p.part_o + slot * HD + d, o);
        if (d == 0) { __stcg(p.part_ml + slot * 2, mx); __stcg(p.part_ml + slot * 2 + 1, l); }
    }
    __syncthreads();
    if (tid == 0) {
        unsigned* ctr = p.counters + (size_t)b * p.kv_heads + kvh;
        unsigned prev;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(prev) : "l"(ctr) : "memory");
        is_last = prev == (unsigned)p.splits - 1u;
        if (is_last) *ctr = 0u;
    }
    __syncthreads();
    if (!is_last) return;
    // the merge: all (max, sum) pairs travel together, then every thread adds up one float4 of one head's output over
    // the splits with the loads of eight splits in flight at a time (rolled loops of dependent L2 round trips made this
    // the longest part of the kernel)
    float* wsm = &osm[0][0][0];              // [G][splits] weights (splits <= 64)
    float* lsm2 = &osm[1][0][0];             // [G][splits] sums
    __shared__ float inv_den[kMaxGroup];
    for (int idx = tid; idx < G * p.splits; idx += kQ8Threads) {
        const int r = idx / p.splits, sidx = idx - r * p.splits;
        const size_t slot = ((size_t)b * p.heads + (size_t)kvh * G + r) * p.splits + sidx;
        const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + slot * 2));
        wsm[idx] = ml.x; lsm2[idx] = ml.y;
    }
    __syncthreads();
    for (int r = warp; r < G; r += kQ8Warps) {
        float mx = -INFINITY;
        for (int sidx = lane; sidx < p.splits; sidx += 32) mx = fmaxf(mx, wsm[r * p.splits + sidx]);
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float den = 0.f;
        for (int sidx = lane; sidx < p.splits; sidx += 32) {
            const float ms = wsm[r * p.splits + sidx];
            const float w = ms == -INFINITY ? 0.f : exp2f(ms - mx);
            wsm[r * p.splits + sidx] = w;
            den = fmaf(w, lsm2[r * p.splits + sidx], den);
        }
        for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
        if (lane == 0) inv_den[r] = den > 0.f ? 1.0f / den : 0.f;
    }
    __syncthreads();
    for (int idx = tid; idx < G * HD / 4; idx += kQ8Threads) {
        const int r = idx / (HD / 4), d4 = idx - r * (HD / 4);
        const float* po = p.part_o + (((size_t)b * p.heads + (size_t)kvh * G + r) * p.splits) * HD + d4 * 4;
        const float* wr = wsm + r * p.splits;
        float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int sidx = 0; sidx < p.splits; ++sidx) {
            const float4 v4 = __ldcg(reinterpret_cast<const float4*>(po + (size_t)sidx * HD));
            const float w = wr[sidx];
            num.x = fmaf(w, v4.x, num.x); num.y = fmaf(w, v4.y, num.y); num.z = fmaf(w, v4.z, num.z); num.w = fmaf(w, v4.w, num.w);
        }
        const float inv = inv_den[r];
        if (ROTOR) {   // normalised, still in the turned basis
            qs[r][d4 * 4 + 0] = num.x * inv; qs[r][d4 * 4 + 1] = num.y * inv;
            qs[r][d4 * 4 + 2] = num.z * inv; qs[r][d4 * 4 + 3] = num.w * inv;
            continue;
        }
        __nv_bfloat16* o = p.out + (size_t)b * p.out_stride + (size_t)(kvh * G + r) * HD + d4 * 4;
        o[0] = __float2bfloat16_rn(num.x * inv); o[1] = __float2bfloat16_rn(num.y * inv);
        o[2] = __float2bfloat16_rn(num.z * inv); o[3] = __float2bfloat16_rn(num.w * inv);
    }
    if (ROTOR) {
        __syncthreads();
        for (int idx = tid; idx < G * NG; idx += kQ8Threads) rotor_turn_group<true>(qs[idx / NG], HD, head_rotors, idx % NG);
        __syncthreads();
        for (int idx = tid; idx < G * HD; idx += kQ8Threads)
            p.out[(size_t)b * p.out_stride + (size_t)kvh * G * HD + idx] = __float2bfloat16_rn(qs[idx / HD][idx % HD]);
    }
}

// MODE 4's CTAs: what the GPU holds at once, three per SM with heads of 64 and two with heads of 128. Every one of them needs a block (they do
// not look whether they have one), and the merge has room for 64 partial results of a pair. 100 pairs of 8 blocks and more give both: with
// 444 CTAs each takes a fifth of a pair's blocks at least, rounded down to one, so that a pair has eight partial results at most.
constexpr int stream_ctas(int hd) { return hd == 64 ? 444 : 296; }
constexpr int kStreamPairs = 100, kStreamRows = 512;
static_assert(kStreamPairs * (kStreamRows / 64) >= stream_ctas(64) && 5 * kStreamPairs >= stream_ctas(64), "a block, a fifth of a pair");
// Flash-decode over sequences of equal length: MODE 4 where the splits of all pairs leave a fifth of their rounds of the GPU empty (a quarter
// with heads of 64) and that is worth more than what a CTA pays for the pairs it meets: 5.5 blocks of 64 rows per CTA, ten of heads of 64.
// Over 13 .. 200 sequences of 512 .. 5000 rows and 1 .. 32 KV heads that is never slower than splits by more than the runs differ. us with
// splits / so; heads of 128: 13 sequences x 5000 rows x 8 KV heads (rounds 0.70 full) 58.6 / 53.4, 24 x 2048 (0.65) 47.4 / 42.6, 41 x 3000
// (0.55) 125 / 89, 41 x 512 28.8 / 25.0; not worth it: 13 x 512 12.0 / 14.8, 24 x 600 18.2 / 19.2; too full: 32 x 5000 (0.86) 106 / 108.
// Heads of 64: 20 x 1024 (0.36) 17.7 / 15.4, 20 x 5000 69 / 41, 41 x 5000 (0.74) 75 / 72; not worth it: 32 x 512 12.8 / 15.2, 41 x 1024
// 20.6 / 21.9; too full: 13 x 512 x 32 KV heads (0.94) 12.8 / 17.1, 56 x 600 x 32 (0.81) 67.0 / 67.8. Decode steps, where each pair's start
// is longer, lost in every batch (41 ragged sequences, 4 layers: 1053 / 1100 a step).
bool attn_streams(int m, int kv_heads, int hd, int ctx_len) {
    const long long pairs = (long long)m * kv_heads, blocks = pairs * ((ctx_len + 63) / 64), ctas = pairs * attn_pick_splits(m, kv_heads, ctx_len);
    if (pairs < kStreamPairs || ctx_len < kStreamRows || blocks >= (1ll << 31)) return false;
    const int slots = stream_ctas(hd);
    const double full = (double)ctas / (double)((ctas + slots - 1) / slots * slots), saved = (double)blocks / slots * (1.0 / full - 1.0);
    return hd == 64 ? full < 0.75 && saved >= 10.0 : full < 0.8 && saved >= 5.5;
}
template <int MODE>
int launch_both(const typename AttnArgs<MODE>::type& p, const dim3& grid, int hd, cudaStream_t s) {
    if (hd == 128) {
        launch_k(attn_split_kernel<128, MODE>, grid, dim3(kSplitThreads), 0, s, p);
    } else if (hd == 64) {
        launch_k(attn_split_kernel<64, MODE>, grid, dim3(kSplitThreads), 0, s, p);
    } else {
        set_error("attention: head_dim %d not supported (64 or 128)", hd);
        return SWLM_ERR_UNSUPPORTED;
    }
    return check_launch("attention launch");
}

}  // namespace

int attn_init() { return attn_prompt_init(); }

int attn_pick_splits(int m, int kv_heads, int max_ctx, bool ragged) {
    static const int forced = [] { const char* v = getenv("SWLM_ATTN_SPLITS"); return v ? atoi(v) : 0; }();
    if (forced >= 1 && forced <= 64) return forced;
    if (m <= 0 || kv_heads <= 0) return 1;
    // Two CTAs fit an SM. Below 300 (sequence, KV head) pairs the splits fill the GPU once. From 150 pairs on that leaves every pair to
    // one CTA, and the longest sequence of a ragged batch, or a second round that is nearly empty, holds up the step. In a long cache at
    // least 450 CTAs then, one and a half rounds. Steps of a model of four layers, 8 KV heads of 128, against one split; sequences of
    // equal length / down to a quarter of it:
    //   pairs  splits   2200 tokens      4000 tokens      two splits at 4000
    //    152      3     -2.3 / -7.6 %    -3.5 / -12.5 %   +1.9 / -10.6 %
    //    192      3     -0.5 / -5.0      -0.3 /  -8.5     +4.4 /  -8.7
    //    240      2                      -4.1 /  -8.3
    //    296      2     -0.8 / -3.0      -4.0 /  -7.3
    //    328      2                      -8.5 /  -5.8
    //    384      2     -4.1 / +0.8      -9.1 /  -4.6
    //    512      2                      -2.2 /  +0.2
    // Short caches lose (192 pairs: +1.4 % at 1000 tokens, 240 pairs at 600 ragged: +1.6), the more pairs the longer: hence ten rows per
    // pair, and from 450 pairs on one split. (A short batch in a long cache pays 1 to 2 % for what it gains when it is long.)
    const int pairs = m * kv_heads;
    int s = 300 / pairs;
    if (ragged && s <= 1 && pairs < 450 && max_ctx >= 10 * pairs) s = (450 + pairs - 1) / pairs;
    const int cap = max_ctx / 128;
    if (s > 32) s = 32;
    if (s > cap) s = cap;
    if (s < 1) s = 1;
    return s;
}

size_t attn_scratch_floats(int m, int heads, int head_dim, int splits) {
    return (size_t)m * heads * splits * (head_dim + 2);
}
// What either form needs from 100 pairs on: scratch taken for a longer context or for more sequences serves what it served without MODE 4.
size_t flash_scratch_floats(int m, int heads, int kv_heads, int hd, int ctx_len) {
    const size_t apart = attn_scratch_floats(m, heads, hd, attn_pick_splits(m, kv_heads, ctx_len));
    return (long long)m * kv_heads >= kStreamPairs ? std::max(apart, (size_t)2 * stream_ctas(hd) * (heads / kv_heads) * (hd + 2)) : apart;
}

static int check_group(int heads, int kv_heads) {
    if (kv_heads <= 0 || heads % kv_heads || heads / kv_heads > kMaxGroup) {
        set_error("attention: %d query heads per KV head not supported (max %d)", kv_heads ? heads / kv_heads : 0, kMaxGroup);
        return SWLM_ERR_UNSUPPORTED;
    }
    return SWLM_OK;
}

int launch_attn_decode(const AttnLaunch& a, cudaStream_t s) {
    int rc = check_group(a.heads, a.kv_heads);
    if (rc) return rc;
    if (a.rope_dim > a.head_dim || (a.rope_dim & 1)) { set_error("attention: bad rope_dim"); return SWLM_ERR_INVALID; }
    if (((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v) | reinterpret_cast<uintptr_t>(a.out)) & 15) ||
        ((a.q_stride | a.k_stride | a.v_stride | a.out_stride) & 7)) {
        set_error("attention: q, k, v and out rows must be 16-byte aligned");
        return SWLM_ERR_INVALID;
    }
    AttnParams p{};
    p.heads = a.heads; p.kv_heads = a.kv_heads; p.rope_dim = a.rope_dim; p.max_seq = a.max_seq; p.splits = a.splits;
    p.scale_log2 = a.scale * kLog2e;
    p.inv_freq = a.inv_freq;
    p.q = a.q; p.q_stride = a.q_stride; p.k = a.k; p.k_stride = a.k_stride; p.v = a.v; p.v_stride = a.v_stride;
    p.kcache = a.kcache; p.vcache = a.vcache;
    p.cache_head_stride = (size_t)a.max_seq * a.head_dim;
    p.cache_seq_stride = p.cache_head_stride * a.kv_heads;
    p.position = a.position; p.ctx_len = 0; p.window = a.window > 0 ? a.window : 0;
    static const int q_first = [] { const char* v = getenv("SWLM_ATTN_QFIRST"); return v ? atoi(v) : 0; }();
    p.q_first = q_first;
    p.out = a.out; p.out_stride = a.out_stride;
    p.part_o = a.scratch;
    p.part_ml = a.scratch + (size_t)a.m * a.heads * a.splits * a.head_dim;
    p.counters = a.counters;
    p.prefetch = a.prefetch;
    if (a.pos_base < 0 && a.m * a.kv_heads * a.splits + a.m * a.kv_heads <= 512)
        p.trace = qgemv_trace_slot(a.m * a.kv_heads * a.splits, -a.kv_heads * a.m, a.splits, 9, 0);
    if (swlm_kv_bits(a.kv_scheme)) {
        if (a.pos_base >= 0) { set_error("attention: prompt chunks over a quantized cache are not supported"); return SWLM_ERR_UNSUPPORTED; }
        p.kv_bits = swlm_kv_bits(a.kv_scheme); p.kv_group = swlm_kv_group(a.kv_scheme);
        if (p.kv_group > a.head_dim) { set_error("attention: cache groups of %d values exceed head_dim %d", p.kv_group, a.head_dim); return SWLM_ERR_UNSUPPORTED; }
        const dim3 grid(p.splits, p.kv_heads, a.m);
        const int G = a.heads / a.kv_heads;
        if (a.head_dim != 64 && a.head_dim != 128) { set_error("attention: head_dim %d not supported over an 8-bit cache (64 or 128)", a.head_dim); return SWLM_ERR_UNSUPPORTED; }
        if (G != 1 && G != 2 && G != 4 && G != 8) { set_error("attention over an 8-bit cache: %d query heads per KV head (1, 2, 4 or 8)", G); return SWLM_ERR_UNSUPPORTED; }
        const bool rotor = swlm_kv_is_rotor(a.kv_scheme);
        if (rotor) {
            if (!a.rotors || a.qjl_dim < 0 || a.qjl_dim > 64 || (a.qjl_dim > 0 && (!a.qjl_matrix || !a.qjl_res))) {
                set_error("attention over a rotated cache: rotors, projection matrix or residual rows missing (qjl_dim %d)", a.qjl_dim);
                return SWLM_ERR_INVALID;
            }
            p.rotors = a.rotors; p.qjl_matrix = a.qjl_matrix; p.qjl_res = a.qjl_res; p.qjl_dim = a.qjl_dim;
        }
#define SWLM_Q8_CASE(HDV, GV) if (a.head_dim == HDV && G == GV) { \
            if (rotor) { \
                if (p.kv_bits == 8) launch_k(attn_q8_split_kernel<HDV, GV, 8, true>, grid, dim3(kQ8Threads), 0, s, p); \
                else launch_k(attn_q8_split_kernel<HDV, GV, 4, true>, grid, dim3(kQ8Threads), 0, s, p); \
            } else if (p.kv_bits == 8) launch_k(attn_q8_split_kernel<HDV, GV, 8, false>, grid, dim3(kQ8Threads), 0, s, p); \
            else launch_k(attn_q8_split_kernel<HDV, GV, 4, false>, grid, dim3(kQ8Threads), 0, s, p); }
        SWLM_Q8_CASE(128, 1); SWLM_Q8_CASE(128, 2); SWLM_Q8_CASE(128, 4); SWLM_Q8_CASE(128, 8);
        SWLM_Q8_CASE(64, 1); SWLM_Q8_CASE(64, 2); SWLM_Q8_CASE(64, 4); SWLM_Q8_CASE(64, 8);
#undef SWLM_Q8_CASE
        return check_launch("attention (8-bit cache) launch");
    }
    if (a.pos_base >= 0) {
        // prompt ingestion: rows of q/k/v are consecutive tokens of sequence 0
        if (a.head_dim > 128) { set_error("attention: head_dim %d not supported", a.head_dim); return SWLM_ERR_UNSUPPORTED; }
        p.pos_base = a.pos_base;
        p.chunk_tokens = a.m;
        // (warps that take one KV head, two or four, us under ncu: 512 tokens of eight heads of 128 5.2 / 5.1 / 5.4, 1024 7.2 / 5.8 / 5.9, 2048
        // 10.8 / 8.1 / 7.4)
        const long long each = (long long)a.m * a.kv_heads;
        const int heads_each = each <= 4096 ? 1 : each <= 8192 ? 2 : 4;
        const dim3 grid((a.m + kRopeWarps - 1) / kRopeWarps, (a.kv_heads + heads_each - 1) / heads_each);
        cudaError_t e = launch_k(rope_append_kernel, grid, dim3(kRopeWarps * 32), 0, s, p, a.head_dim, heads_each);
        if (e != cudaSuccess) return cuda_fail(e, "rope_append launch");
        // tensor cores when the query heads of a KV head fill the 128 rows of a tile evenly; else a token at a time
        if (attn_prompt_takes(a)) return launch_attn_prompt(a, s);
        return launch_both<2>(p, dim3(p.splits, p.kv_heads, a.m), a.head_dim, s);
    }
    if (!a.q_norm) return launch_both<1>(p, dim3(p.splits, p.kv_heads, a.m), a.head_dim, s);
    AttnNormParams n{};
    static_cast<AttnParams&>(n) = p;
    n.q_norm = a.q_norm; n.k_norm = a.k_norm; n.qk_eps = a.qk_eps; n.qk_bias = a.qk_bias;
    return launch_both<3>(n, dim3(n.splits, n.kv_heads, a.m), a.head_dim, s);
}

int launch_flash_decode_plain(int m, int heads, int kv_heads, int hd, int ctx_len, int ctx_stride, float scale,
                              const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v,
                              __nv_bfloat16* out, float* scratch, unsigned* counters, int splits, cudaStream_t s) {
    int rc = check_group(heads, kv_heads);
    if (rc) return rc;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 15) { set_error("flash-decode: q and out must be 16-byte aligned"); return SWLM_ERR_INVALID; }
    AttnParams p{};
    p.heads = heads; p.kv_heads = kv_heads; p.rope_dim = 0; p.max_seq = ctx_stride; p.splits = splits;
    p.scale_log2 = scale * kLog2e;
    p.q = q; p.q_stride = heads * hd;
    p.kcache = const_cast<__nv_bfloat16*>(k); p.vcache = const_cast<__nv_bfloat16*>(v);
    p.cache_head_stride = (size_t)ctx_stride * hd;
    p.cache_seq_stride = p.cache_head_stride * kv_heads;
    p.position = nullptr; p.ctx_len = ctx_len;
    p.out = out; p.out_stride = heads * hd;
    p.part_o = scratch;
    const bool stream = attn_streams(m, kv_heads, hd, ctx_len);
    if (stream) p.splits = m * kv_heads;   // (MODE 4: pairs)
    p.part_ml = scratch + (stream ? (size_t)2 * stream_ctas(hd) * (heads / kv_heads) : (size_t)m * heads * splits) * hd;
    p.counters = counters;
    return stream ? launch_both<4>(p, dim3((unsigned)stream_ctas(hd)), hd, s) : launch_both<0>(p, dim3(splits, kv_heads, m), hd, s);
}

// ---- allocation-free flash-decode ---------------------------------------------------------------------
// Some embedders may not allocate device memory once they are running: a serving loop that reserved its
// whole memory budget at start-up and treats any later cudaMalloc as a bug (it synchronises the device and
// can fail under memory pressure), or a host runtime that owns the allocator and hands this library no
// pool of its own. For them the partial results and arrival counters of the split kernel live in a fixed
// array that is part of the loaded module instead of in caller- or library-allocated scratch.
//
// The array is 8 MiB on every GPU that loads the library, for the life of the process. All calls share it
// and it keeps the previous call's contents: the counters are cleared (asynchronously, on the call's
// stream) before every launch, the partials are overwritten before they are read. Two calls that overlap
// on the GPU (different streams, no ordering between them) would race on it; serialise them.
constexpr size_t kStaticScratchBytes = 8u << 20;
static __device__ __align__(256) unsigned char g_flash_static_scratch[kStaticScratchBytes];
// device address of the array, per device ordinal. Written by whichever thread calls first on a device; every writer
// stores the same value, and the slot is an atomic so that concurrent first calls are a defined program.
static std::atomic<void*> g_flash_static_addr[64];

size_t flash_decode_static_capacity() { return kStaticScratchBytes; }

int launch_flash_decode_static(int device, int m, int heads, int kv_heads, int hd, int ctx_len, int ctx_stride, float scale,
                               const __nv_bfloat16* q, const __nv_bfloat16* k, const __nv_bfloat16* v, __nv_bfloat16* out,
                               cudaStream_t s) {
    if (device < 0 || device >= 64) { set_error("flash-decode (static scratch): device ordinal %d out of range", device); return SWLM_ERR_INVALID; }
    if (!g_flash_static_addr[device].load(std::memory_order_acquire)) {
        // In host code the array's name is only a handle; the kernel needs the device address, which the
        // runtime resolves for the device that is current now. Done once per device, on the first call.
        void* addr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&addr, g_flash_static_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(flash-decode static scratch)");
        g_flash_static_addr[device].store(addr, std::memory_order_release);
    }
    const int splits = attn_pick_splits(m, kv_heads, ctx_len);
    const size_t counter_bytes = (((size_t)m * kv_heads * sizeof(unsigned)) + 255) / 256 * 256;
    const size_t need = counter_bytes + flash_scratch_floats(m, heads, kv_heads, hd, ctx_len) * sizeof(float);
    if (need > kStaticScratchBytes) {
        set_error("flash-decode (static scratch): batch %d x %d heads x %d splits needs %zu bytes, the built-in scratch holds %zu",
                  m, heads, splits, need, kStaticScratchBytes);
        return SWLM_ERR_INVALID;
    }
    unsigned char* base = static_cast<unsigned char*>(g_flash_static_addr[device].load(std::memory_order_acquire));
    SWLM_CUDA(cudaMemsetAsync(base, 0, counter_bytes, s));  // arrival counters must start at zero
    return launch_flash_decode_plain(m, heads, kv_heads, hd, ctx_len, ctx_stride, scale, q, k, v, out,
                                     reinterpret_cast<float*>(base + counter_bytes), reinterpret_cast<unsigned*>(base), splits, s);
}

}  // namespace swlm
