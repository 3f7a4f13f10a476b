// Causal attention of a prompt chunk over the bf16 cache, on the 5th-generation tensor cores (tcgen05 / TMEM).
//
// The chunk's k/v rows are already in the cache (rope_append_kernel); token b of the chunk attends rows 0..pos_base+b (the
// reference's prefill attention walks the context once per query head and position,
// Generator/MetalSourceGenerator+Attention.swift:551-930). One CTA serves 128 query rows = (128 / G) consecutive tokens x the G
// query heads of a KV head, lane r of tensor memory = row r. Precision as in the decode kernel: q is rotated in fp32 and enters as a
// bf16 hi + lo pair, so do the probabilities; scores, softmax and the output accumulate in fp32.
//
// What bounds it: 4 x 128 x 64 x HD multiplications per key tile of 64 (hi and lo, scores and values; 1024 clocks of the tensor pipe at
// HD = 128) against 8192 exponentials and some 60 thousand softmax instructions; two CTAs share an SM, so that one multiplies while
// the other is in its softmax. The mma.sync form this one replaced fetched every key and value from shared memory once per eight
// rows (0.48 of its 1.12 ms for 4096 tokens x 32 heads) and ran at the 540 TFLOP/s of the legacy pipe: 1117 us, now 397 us under ncu.
//
// Roles: a TMA thread brings key and value tiles (one slot each; 128-byte swizzle), a thread issues the MMAs (S = Q K^T for tile
// j + 1 while tile j is in its softmax: two score regions), four warps do the softmax, a thread per row. Probabilities take the place
// of their scores in tensor memory and are read there as the A operand. The reference maximum of a row moves only when it would grow
// by more than 2^8 (probabilities stay below 256, exactly undone by the sum at the end), so that the output is rarely rescaled.
// Every mbarrier wait is bounded (see qgemm_tc.cu).
#include "swlm_internal.h"
#include "tc_device.cuh"

namespace swlm {
namespace {

constexpr int kPaRows = 128, kPaKeys = 64, kPaThreads = 192;
constexpr float kPaLog2e = 1.4426950408889634f;
constexpr float kPaSlack = 8.f;   // log2 of what a row's probabilities may exceed 1 by

struct PromptAttnParams {
    int G, kv_heads, max_seq, rope_dim, pos_base, chunk_tokens, window;
    float scale_log2;
    const float* inv_freq;
    const __nv_bfloat16* q; int q_stride;
    __nv_bfloat16* out; int out_stride;
    int* status;
};

// (descriptors by their low words; `b_hi`: the high word of B's)
__device__ __forceinline__ void pa_mma_ss(unsigned d, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned acc) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}"
                 ::"r"(d), "r"(a_lo), "r"(b_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void pa_mma_ts(unsigned d, unsigned a, unsigned b_lo, unsigned idesc, unsigned acc) {
    asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 b, {%2, %3};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}"
                 ::"r"(d), "r"(a), "r"(b_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(acc) : "memory");
}
// D fp32, A = B = bf16, M = 128, N = n; `b_mn`: B's rows lie along K (its N index is the contiguous one)
__host__ __device__ constexpr unsigned pa_idesc(int n, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? 1u << 16 : 0u) | ((unsigned)(n >> 3) << 17) | ((unsigned)(kPaRows >> 4) << 24);
}
// Descriptor (low word) of a tile whose contiguous index is N: blocks of 64 elements (128 bytes) `block` bytes apart, eight rows of K
// per 1024 bytes
__device__ __forceinline__ unsigned pa_desc_mn_lo(unsigned addr, unsigned block) { return umma_desc_lo(addr) | (block >> 4) << 16; }
#define PA_R8(v, o) "=r"(v[o]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7])
#define PA_I8(v, o) "r"(v[o]), "r"(v[o + 1]), "r"(v[o + 2]), "r"(v[o + 3]), "r"(v[o + 4]), "r"(v[o + 5]), "r"(v[o + 6]), "r"(v[o + 7])
__device__ __forceinline__ void pa_ld32(unsigned addr, unsigned* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : PA_R8(v, 0), PA_R8(v, 8), PA_R8(v, 16), PA_R8(v, 24) : "r"(addr) : "memory");
}
__device__ __forceinline__ void pa_st32(unsigned addr, const unsigned* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(addr), PA_I8(v, 0), PA_I8(v, 8), PA_I8(v, 16), PA_I8(v, 24) : "memory");
}
__device__ __forceinline__ void pa_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pa_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pa_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pa_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pa_arrive(unsigned long long* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ float pa_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ unsigned pa_pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned*>(&v);
}
// (a, b) as bf16 pairs hi + lo
__device__ __forceinline__ void pa_split(float a, float b, unsigned& hi, unsigned& lo) {
    hi = pa_pack(a, b);
    lo = pa_pack(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xFFFF0000u));
}

// A wait by parity cannot tell a phase from the one two before it, so the phase before the awaited one has to be known to be over:
//   q_ready, o_done  have one phase;
//   k_full, p_ready  are waited for phase by phase (MMA warp);
//   v_full           phase by phase by the MMA warp; by a softmax warp for tile j behind pv_done(j - 1), whose product read tile j - 1;
//   s_full[j & 1]    phase by phase by the softmax warps and the TMA thread;
//   pv_done          phase by phase by the TMA thread; for tile j - 1 by the MMA warp, which has waited for tile j - 2 in the round before,
//                    and by a softmax warp behind s_full(j): the scores of tile j are issued behind pv_done(j - 2). Behind the last tile no
//                    scores follow that would imply the tile before it, so that its products' end has a barrier of its own, o_done.
struct PaBars {
    unsigned long long q_ready, k_full, v_full, s_full[2], p_ready[2], pv_done, o_done;   // o_done: every MMA issued is done
    unsigned tmem;
    int failed;
};

template <int HD>
constexpr size_t pa_smem_bytes() { return (size_t)2 * kPaRows * HD * 2 + 2 * kPaKeys * HD * 2 + 1024; }

template <int HD>
__global__ void __launch_bounds__(kPaThreads, 2) attn_prompt_kernel(const PromptAttnParams p, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
    constexpr int HALVES = HD / 64;                        // 128-byte halves of a row
    constexpr unsigned Q_HALF = kPaRows * 128, Q_BYTES = HALVES * Q_HALF, KV_HALF = kPaKeys * 128, KV_BYTES = HALVES * KV_HALF;
    constexpr unsigned kTmemCols = 256, O_COL = 128;       // scores / probabilities 0..63 and 64..127, output from 128 on
    extern __shared__ __align__(1024) unsigned char pa_raw[];
    unsigned char* const sm = pa_raw + ((1024 - (smem_u32(pa_raw) & 1023)) & 1023);
    unsigned char *const q_hi = sm, *const q_lo = sm + Q_BYTES, *const k_sm = sm + 2 * Q_BYTES, *const v_sm = k_sm + KV_BYTES;
    __shared__ __align__(8) PaBars bars;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.G, TQ = kPaRows / G;                   // tokens per CTA
    const int qt = gridDim.x - 1 - blockIdx.x, kvh = blockIdx.y;   // the longest rows first
    const int tok0 = qt * TQ, n_tok = min(TQ, p.chunk_tokens - tok0);
    const int last_pos = p.pos_base + tok0 + n_tok - 1;            // of this CTA's tokens
    const int last_row = p.pos_base + p.chunk_tokens - 1;          // last cache row that holds data
    const int tile_lo = p.window > 0 ? max(0, p.pos_base + tok0 - p.window + 1) / kPaKeys : 0;   // the first token reaches back furthest
    const int n_tiles = last_pos / kPaKeys + 1 - tile_lo;
    volatile int* const failed = &bars.failed;
    auto fail = [&](int code) { atomicExch(p.status, code); *failed = 1; };

    if (tid == 0) {
        mbar_init(&bars.q_ready, 4); mbar_init(&bars.k_full, 1); mbar_init(&bars.v_full, 1); mbar_init(&bars.pv_done, 1); mbar_init(&bars.o_done, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&bars.s_full[i], 1); mbar_init(&bars.p_ready[i], 4); }
        bars.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pa_before();
    __syncthreads();
    pa_after();
    const unsigned tm = bars.tmem;
    pdl_launch_dependents();
    pdl_wait();

    if (warp == 5) {
        if (lane == 0) {
            const int y0 = kvh * p.max_seq + tile_lo * kPaKeys;
            bool ok = true;
            int k_issued = 0, v_issued = 0;
            for (int j = 0; j < n_tiles && ok; ++j) {
                // the key tile before has been multiplied, the value tile before too
                if (*failed || (j > 0 && !mbar_wait(&bars.s_full[(j - 1) & 1], (unsigned)(((j - 1) >> 1) & 1)))) { ok = false; break; }
                mbar_expect(smem_u32(&bars.k_full), KV_BYTES);
                for (int h = 0; h < HALVES; ++h) tma_load_2d(smem_u32(k_sm) + h * KV_HALF, &kmap, 64 * h, y0 + j * kPaKeys, smem_u32(&bars.k_full));
                ++k_issued;
                // (the first value tile takes the place of the rotation table)
                if (!(j > 0 ? mbar_wait(&bars.pv_done, (unsigned)((j - 1) & 1)) : mbar_wait(&bars.q_ready, 0u))) { ok = false; break; }
                mbar_expect(smem_u32(&bars.v_full), KV_BYTES);
                for (int h = 0; h < HALVES; ++h) tma_load_2d(smem_u32(v_sm) + h * KV_HALF, &vmap, 64 * h, y0 + j * kPaKeys, smem_u32(&bars.v_full));
                ++v_issued;
            }
            if (!ok) fail(6);
            if (k_issued) mbar_wait(&bars.k_full, (unsigned)((k_issued - 1) & 1));   // no copy is in flight when the CTA leaves
            if (v_issued) mbar_wait(&bars.v_full, (unsigned)((v_issued - 1) & 1));
        }
        __syncwarp();
    } else if (warp == 4) {
        const bool el = elect_one();
        const unsigned qh = umma_desc_lo(smem_u32(q_hi)), ql = umma_desc_lo(smem_u32(q_lo)), kd = umma_desc_lo(smem_u32(k_sm)), vd = pa_desc_mn_lo(smem_u32(v_sm), KV_HALF);
        auto scores = [&](int j) {
            if (el) {
                const unsigned d = tm + (unsigned)(j & 1) * 64u;
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int kk = 0; kk < HD / 16; ++kk)
                        pa_mma_ss(d, (part ? ql : qh) + (kk >> 2) * (Q_HALF / 16) + 2 * (kk & 3), kd + (kk >> 2) * (KV_HALF / 16) + 2 * (kk & 3),
                                  pa_idesc(kPaKeys, false), part > 0 || kk > 0 ? 1u : 0u);
                umma_commit(&bars.s_full[j & 1]);
            }
            __syncwarp();
        };
        bool ok = mbar_wait_warp(&bars.q_ready, 0u) && mbar_wait_warp(&bars.k_full, 0u);
        if (ok) { pa_after(); scores(0); }
        for (int j = 0; j < n_tiles && ok; ++j) {
            if (j + 1 < n_tiles) {
                // the region of tile j + 1 held the probabilities of tile j - 1
                if (!mbar_wait_warp(&bars.k_full, (unsigned)((j + 1) & 1)) || (j > 0 && !mbar_wait_warp(&bars.pv_done, (unsigned)((j - 1) & 1)))) { ok = false; break; }
                pa_after();
                scores(j + 1);
            }
            if (!mbar_wait_warp(&bars.p_ready[j & 1], (unsigned)((j >> 1) & 1)) || !mbar_wait_warp(&bars.v_full, (unsigned)(j & 1))) { ok = false; break; }
            pa_after();
            if (el) {
#pragma unroll
                for (int part = 0; part < 2; ++part)
#pragma unroll
                    for (int kk = 0; kk < kPaKeys / 16; ++kk)
                        pa_mma_ts(tm + O_COL, tm + (unsigned)(j & 1) * 64u + part * 32u + 8u * kk, vd + kk * (2048 / 16), pa_idesc(HD, true),
                                  part > 0 || kk > 0 ? 1u : j > 0 ? 1u : 0u);
                umma_commit(&bars.pv_done);
            }
            __syncwarp();
        }
        if (el) {
            if (!ok) fail(7);
            umma_commit(&bars.o_done);   // also behind whatever was issued before a failure
        }
        __syncwarp();
        if (!mbar_wait_warp(&bars.o_done, 0u) && el) fail(7);   // tensor memory is not freed under MMAs in flight
    } else {
        const int r = tid, tl = r / G, head = r - tl * G;
        const bool row_ok = tl < n_tok;
        const int pairs = p.rope_dim >> 1;
        // ---- q: this thread's row, rotated (rotate-half, :596-617) and split; rows past the chunk are zeros -----------------------
        {
            // cos / sin of a token are shared by its G rows through the value slot when they fit (G >= 4)
            float2* const table = reinterpret_cast<float2*>(v_sm);
            const bool shared_table = TQ * pairs * 8 <= (int)KV_BYTES;
            if (shared_table)
                for (int idx = tid; idx < n_tok * pairs; idx += 128) {
                    float sn, cs;
                    sincosf((float)(p.pos_base + tok0 + idx / pairs) * p.inv_freq[idx % pairs], &sn, &cs);
                    table[idx] = make_float2(cs, sn);
                }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const __nv_bfloat16* src = p.q + (size_t)(tok0 + (row_ok ? tl : 0)) * p.q_stride + (size_t)(kvh * G + head) * HD;
            auto angle = [&](int i) {
                if (shared_table) return table[tl * pairs + i];
                float sn, cs;
                sincosf((float)(p.pos_base + tok0 + tl) * p.inv_freq[i], &sn, &cs);
                return make_float2(cs, sn);
            };
            auto value = [&](int d) { return __bfloat162float(src[d]); };
            auto put = [&](int c8, const float (&x)[8]) {   // eight columns from 8 c8 on
                unsigned h[4], l[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) pa_split(x[2 * i], x[2 * i + 1], h[i], l[i]);
                const unsigned off = (c8 >> 3) * Q_HALF + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
                *reinterpret_cast<uint4*>(q_hi + off) = make_uint4(h[0], h[1], h[2], h[3]);
                *reinterpret_cast<uint4*>(q_lo + off) = make_uint4(l[0], l[1], l[2], l[3]);
            };
            auto load8 = [&](int c8, float (&x)[8]) {
                uint4 v = make_uint4(0, 0, 0, 0);
                if (row_ok) v = *reinterpret_cast<const uint4*>(src + c8 * 8);
                const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { x[2 * i] = __uint_as_float(u[i] << 16); x[2 * i + 1] = __uint_as_float(u[i] & 0xFFFF0000u); }
            };
            if ((pairs & 7) == 0) {
                for (int c = 0; c < pairs / 8; ++c) {
                    float lo[8], hi[8];
                    load8(c, lo);
                    load8(c + pairs / 8, hi);
                    if (row_ok)
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float2 a = angle(8 * c + i);
                            const float x = lo[i], y = hi[i];
                            lo[i] = x * a.x - y * a.y;
                            hi[i] = x * a.y + y * a.x;
                        }
                    put(c, lo);
                    put(c + pairs / 8, hi);
                }
                for (int c = pairs / 4; c < HD / 8; ++c) {
                    float x[8];
                    load8(c, x);
                    put(c, x);
                }
            } else {
                for (int c = 0; c < HD / 8; ++c) {
                    float x[8];
                    for (int i = 0; i < 8; ++i) {
                        const int d = 8 * c + i;
                        if (!row_ok) { x[i] = 0.f; continue; }
                        if (d < pairs) { const float2 a = angle(d); x[i] = value(d) * a.x - value(d + pairs) * a.y; }
                        else if (d < 2 * pairs) { const float2 a = angle(d - pairs); x[i] = value(d - pairs) * a.y + value(d) * a.x; }
                        else x[i] = value(d);
                    }
                    put(c, x);
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // what the MMAs read, and the slot that the copies write
            __syncwarp();
            if (lane == 0) pa_arrive(&bars.q_ready);
        }
        // ---- softmax, a thread per row -------------------------------------------------------------------------------------------
        const int pos_row = p.pos_base + tok0 + min(tl, n_tok - 1);   // rows past the chunk's end repeat the last token (not stored)
        const int row_lo = p.window > 0 ? pos_row - p.window + 1 : 0;
        const unsigned lanes = (unsigned)(warp * 32) << 16;
        float m_ref = -INFINITY, l_run = 0.f;
        bool ok = true;
        for (int j = 0; j < n_tiles; ++j) {
            const unsigned region = tm + lanes + (unsigned)(j & 1) * 64u;
            if (!mbar_wait_warp(&bars.s_full[j & 1], (unsigned)((j >> 1) & 1))) { ok = false; break; }
            pa_after();
            unsigned v[64];
            pa_ld32(region, v);
            pa_ld32(region + 32u, v + 32);
            pa_wait_ld();
            const int key0 = (tile_lo + j) * kPaKeys;
            float top = -INFINITY;
            if (__all_sync(0xffffffffu, key0 + kPaKeys - 1 <= pos_row && key0 >= row_lo)) {
#pragma unroll
                for (int i = 0; i < 64; ++i) top = fmaxf(top, __uint_as_float(v[i]));
            } else {
#pragma unroll
                for (int i = 0; i < 64; ++i) {
                    if (key0 + i > pos_row || key0 + i < row_lo) v[i] = 0xFF800000u;   // -inf
                    top = fmaxf(top, __uint_as_float(v[i]));
                }
            }
            top *= p.scale_log2;   // (scale > 0: the largest score stays the largest)
            const bool moves = top > m_ref + kPaSlack;
            if (__any_sync(0xffffffffu, moves)) {
                const float corr = moves ? pa_exp2(m_ref - top) : 1.f;   // 0 for a row's first keys
                if (moves) { m_ref = top; l_run *= corr; }
                if (j > 0) {   // the output so far: complete, and the next product waits for this warp
                    if (!mbar_wait_warp(&bars.pv_done, (unsigned)((j - 1) & 1))) { ok = false; break; }
                    pa_after();
#pragma unroll 1
                    for (int c = 0; c < HD; c += 32) {
                        unsigned o[32];
                        pa_ld32(tm + lanes + O_COL + c, o);
                        pa_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        pa_st32(tm + lanes + O_COL + c, o);
                    }
                    pa_wait_st();
                }
            }
            const float base = m_ref == -INFINITY ? 0.f : m_ref;   // nothing attended so far: all probabilities 0
            float sum = 0.f;
            unsigned lo[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float a = pa_exp2(fmaf(__uint_as_float(v[2 * i]), p.scale_log2, -base)), b = pa_exp2(fmaf(__uint_as_float(v[2 * i + 1]), p.scale_log2, -base));
                sum += a + b;
                pa_split(a, b, v[i], lo[i]);
            }
            l_run += sum;
            pa_st32(region, v);
            pa_st32(region + 32u, lo);
            pa_wait_st();
            if (key0 + kPaKeys - 1 > last_row) {   // value rows that nobody wrote get weight 0: they must not hold NaN or infinity
                // (tile j - 1 of the values may still be on its way into the slot: first its product)
                if ((j > 0 && !mbar_wait_warp(&bars.pv_done, (unsigned)((j - 1) & 1))) || !mbar_wait_warp(&bars.v_full, (unsigned)(j & 1))) { ok = false; break; }
                const int first = last_row + 1 - key0;
                for (int idx = tid; idx < (kPaKeys - first) * HALVES * 8; idx += 128) {
                    const int row = first + idx / (HALVES * 8), c = idx % (HALVES * 8);
                    *reinterpret_cast<uint4*>(v_sm + (c >> 3) * KV_HALF + row * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            pa_before();
            __syncwarp();
            if (lane == 0) pa_arrive(&bars.p_ready[j & 1]);
        }
        if (ok && (!mbar_wait_warp(&bars.o_done, 0u) || *failed)) ok = false;
        if (!ok) fail(8);
        __syncwarp();
        pa_after();
        if (ok) {
            const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
            __nv_bfloat16* dst = p.out + (size_t)(tok0 + tl) * p.out_stride + (size_t)(kvh * G + head) * HD;
#pragma unroll 1
            for (int c = 0; c < HD; c += 32) {
                unsigned o[32];
                pa_ld32(tm + lanes + O_COL + c, o);
                pa_wait_ld();
                if (row_ok)
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        unsigned w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) w[e] = pa_pack(__uint_as_float(o[i + 2 * e]) * inv, __uint_as_float(o[i + 2 * e + 1]) * inv);
                        *reinterpret_cast<uint4*>(dst + c + i) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
            }
        }
    }
    pa_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tm), "r"(kTmemCols) : "memory");
}

// cache rows [kv_heads * max_seq][hd] as a 2-D tensor; box = 64 columns x 64 rows, 128-byte swizzle
int pa_map(const __nv_bfloat16* base, int hd, long long rows, CUtensorMap* map) {
    TensorMapEncodeFn fn = tensor_map_encode_fn();
    if (!fn) { set_error("prompt attention: cuTensorMapEncodeTiled is not available"); return SWLM_ERR_CUDA; }
    const cuuint64_t dims[2] = {(cuuint64_t)hd, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)hd * 2};
    const cuuint32_t box[2] = {64, kPaKeys};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("prompt attention: cuTensorMapEncodeTiled failed (%d)", (int)r); return SWLM_ERR_CUDA; }
    return SWLM_OK;
}

template <int HD>
int pa_launch(const PromptAttnParams& p, const __nv_bfloat16* k, const __nv_bfloat16* v, cudaStream_t s) {
    CUtensorMap kmap, vmap;
    int rc = pa_map(k, HD, (long long)p.kv_heads * p.max_seq, &kmap);
    if (rc || (rc = pa_map(v, HD, (long long)p.kv_heads * p.max_seq, &vmap))) return rc;
    const int TQ = kPaRows / p.G;
    const cudaError_t e = launch_k(attn_prompt_kernel<HD>, dim3((unsigned)((p.chunk_tokens + TQ - 1) / TQ), (unsigned)p.kv_heads), dim3(kPaThreads), pa_smem_bytes<HD>(), s, p, kmap, vmap);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "prompt attention launch");
}

}  // namespace

int attn_prompt_init() {
    SWLM_CUDA(cudaFuncSetAttribute(attn_prompt_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pa_smem_bytes<128>()));
    SWLM_CUDA(cudaFuncSetAttribute(attn_prompt_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pa_smem_bytes<64>()));
    return SWLM_OK;
}

bool attn_prompt_takes(const AttnLaunch& a) {
    const int G = a.kv_heads > 0 ? a.heads / a.kv_heads : 0;
    return (G == 1 || G == 2 || G == 4 || G == 8) && (a.head_dim == 64 || a.head_dim == 128) && a.scale > 0.f && a.status &&
           !((reinterpret_cast<uintptr_t>(a.kcache) | reinterpret_cast<uintptr_t>(a.vcache)) & 15);
}

int launch_attn_prompt(const AttnLaunch& a, cudaStream_t s) {
    PromptAttnParams p{};
    p.G = a.heads / a.kv_heads; p.kv_heads = a.kv_heads; p.max_seq = a.max_seq; p.rope_dim = a.rope_dim;
    p.pos_base = a.pos_base; p.chunk_tokens = a.m; p.window = a.window > 0 ? a.window : 0;
    p.scale_log2 = a.scale * kPaLog2e; p.inv_freq = a.inv_freq;
    p.q = a.q; p.q_stride = a.q_stride; p.out = a.out; p.out_stride = a.out_stride; p.status = a.status;
    return a.head_dim == 128 ? pa_launch<128>(p, a.kcache, a.vcache, s) : pa_launch<64>(p, a.kcache, a.vcache, s);
}

}  // namespace swlm
