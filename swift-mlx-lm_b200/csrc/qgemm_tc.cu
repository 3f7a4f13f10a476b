// Q4 group-64 products of 17 and more activation rows for sm_100a on the 5th-generation tensor cores (tcgen05 / TMEM).
//
// Replaces the reference's `gemm_q4_g64` (Generator/MetalSourceGenerator+Quantized.swift:88-156, which repeats the per-row dot
// product for every sequence position and so re-reads the weights M times) with a real contraction whose result equals the
// fp32-weight product up to the order of the fp32 sums. The weight is split as scale*q + zero = scale*(q - 8) + (zero + 8*scale):
// |q - 8| <= 8 has at most three significant bits (or is a power of two) and a bf16 scale at most eight (an fp16 one eleven), so
// scale*(q - 8) is EXACT in fp16 for bf16 scales and is the A operand; the second term is constant over a group of 64 and
// multiplies the group's sum of activations, which becomes three extra K-columns per group appended after the real ones
// (c_hi x sum_hi, c_lo x sum_hi, c_hi x sum_lo, fp16 pairs that carry 22 bits). Both operands of tcgen05.mma kind::f16 have the
// same type, so a small kernel first copies the activations to fp16, every row times a power of two that puts its largest
// magnitude at 2^14 (exact for every element within 2^-28 of the row's largest, immune to fp16's range, undone in the epilogue),
// and appends the per-group sums. (A dequantised weight rounded to 16 bits, the reference's dequantise-then-matmul route of
// +Quantized.swift:361-416, does not hold 1e-2 per output against `gemm_q4_g64`.)
//
// A step of the pipeline is 128 columns of K (two groups). Roles:
//   * a TMA thread keeps a ring of stages full of activations (128 fp16 per row, two 128-byte-swizzled halves);
//   * 16 warps dequantise, each one 16 x 64 tile of the streaming layout per step, through a cp.async ring of its own; nibble pairs to fp16 with LOP3 (1024 + q or 1024 + 16 q), one subtraction and one multiplication of
//     fp16 pairs; what falls out is the A fragment of mma.m16n8k16, which tcgen05.st.16x256b puts into tensor memory as it is:
//     the copy of the activations has its columns in the same order. The A operand is read from TMEM;
//   * one thread issues eight tcgen05.mma (K = 16) per step; tcgen05.commit frees stage and weight tile;
//   * epilogue: tcgen05.ld, undo the row's power of two, round once to bf16, Y[token][row]; or gate and up rows of the interleaved
//     layout together, activated.
// The long form (many rows) pairs two SMs: 256 weight rows x 256 activation rows per tile, each CTA dequantises its 128 weight
// rows and fetches half of the activations.
//
// What bounded the kernel this one replaced (one group per step, weights by TMA as 128 rows of 32 bytes, one tile per CTA): the L2
// traffic of 256 activation rows per 128 weight rows (with seven of eight MMAs left out 2048 x 28672 x 4096 still took 411 of
// 509 us, 10.7 TB/s), 512 arrivals per group, eight MMAs issued by a lone lane (470 to 850 clocks), and two waves of CTAs, the second
// half empty. What bounds it now: the MMAs of the long form (about 0.7 of their rate under the power cap, one and a half waves of tiles at
// 512 rows), dequantising in the short one. 17 to 64 rows have a kernel of their own (qgemm_slab_kernel).
// Measured: 14336 x 4096 at 512 rows 88 -> 65 us, with results stored by rows and appended columns in blocks 57 (1050 TFLOP/s; a test in front
// of every wait makes no difference to the forms here); 28672 x 4096 at 2048 rows 705 us under ncu -> 442 us with pairs of SMs.
//
// Every mbarrier wait is bounded: on expiry an error word is set, the CTA stops issuing, waits (bounded) for the copies and MMAs
// it has in flight, frees its TMEM and returns.
#include <algorithm>
#include <cstdlib>

#include <cooperative_groups.h>
#include <cuda.h>

#include "swlm_internal.h"
#include "tc_device.cuh"

namespace cg = cooperative_groups;

namespace swlm {
namespace {

constexpr int kTcRows = 128;             // weight rows per CTA = lanes of tensor memory
constexpr int kTcStep = 128;             // columns of K per pipeline step
constexpr int kTcDeqWarps = 16;
constexpr int kTcMaxA = 4;               // dequantised weight tiles in flight at most, 64 columns of TMEM each
constexpr int kTcSet = kTcDeqWarps / 2;  // they take turns: half of them dequantise the even steps, the others the odd ones
constexpr int kTcAhead = 3;              // ring of a dequantising warp: steps of its own whose weights it has requested
constexpr int kTcSlotBytes = 1024 + 128; // two 16 x 64 tiles and their 16 times two scale / zero pairs
constexpr int kTcRingBytes = kTcDeqWarps * kTcAhead * kTcSlotBytes;
constexpr int kTcEpiWarps = 8;           // long form: warps that only store results

struct QGemmTcParams {
    const uint4* tiles;       // [row tile][k-tile][32 lanes], see Q4Tiled
    const unsigned* sb;       // [row tile][k-tile / 4][16 rows][4] pairs
    int row_tiles, kt;        // row tiles, k-tiles (groups of 64, a multiple of four)
    const float* rscale;      // [m]: the inverse of each row's power of two
    int m;
    int real_steps, steps;    // steps over the weights; those over the appended columns follow
    int tok_tiles, n_tiles;   // long form: tiles of 256 rows, all tiles
    int splits;               // short form: CTAs of a cluster along K
    int whole, left;          // few rows: passes of eight row tiles per CTA; row tiles of the last one
    int gated, gated_act;     // rows 0-7 of a row tile are gate rows, rows 8-15 the up rows that belong to them
    TcSegments out;           // weight rows [end[q-1], end[q]) go to out.y[q][token][row - end[q-1]]
    int* status;              // set non-zero when a bounded wait expired
};

// Instruction descriptor for kind::f16: D = fp32, A = B = fp16 (format 0), both K-major, M rows, N = BN.
__host__ __device__ constexpr unsigned umma_idesc(int m, int bn) {
    return (1u << 4) | (0u << 7) | (0u << 10) | ((unsigned)(bn >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
// D[tmem] (+)= A[tmem] x B[shared memory]; CG = 2: the rows of A and D and those of B lie half in either CTA of the pair
template <int CG>
__device__ __forceinline__ void umma_f16_ta(unsigned d_tmem, unsigned a_tmem, unsigned b_desc_lo, unsigned idesc, unsigned accumulate) {
    if (CG == 1)
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 d;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 d, {%2, %3};\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n\t}"
                     ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t.reg .b64 d;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 d, {%2, %3};\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], d, %4, p;\n\t}"
                     ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc_lo), "r"(kUmmaDescHi), "r"(idesc), "r"(accumulate) : "memory");
}
// arrival at the same barrier of both CTAs of a pair when the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((unsigned short)3) : "memory");
}
// A row's factor, by a thread that has waited for the kernel in front (pdl_wait), which writes it: what that kernel wrote is visible to
// plain loads then, not to the non-coherent ones. (From L2 for every lane and column: 2 % to 5 % of a product.)
__device__ __forceinline__ float tc_rscale(const QGemmTcParams& p, int token) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p.rscale + token));
    return v;
}
// One result, rounded once to bf16, to the output its weight row belongs to.
__device__ __forceinline__ void tc_store(const TcSegments& o, int token, int row, float val) {
    const __nv_bfloat16 v = __float2bfloat16_rn(val);
    if (row < o.end[0]) o.y[0][(size_t)token * o.stride[0] + row] = v;
    else if (row < o.end[1]) o.y[1][(size_t)token * o.stride[1] + (row - o.end[0])] = v;
    else if (row < o.end[2]) o.y[2][(size_t)token * o.stride[2] + (row - o.end[1])] = v;
}
// A gate row's and its up row's result: both are rounded to bf16 first because the reference stores them to bf16 scratch before
// `swiglu` reads them (Primitives/ElementwiseFragment.swift:49-54).
__device__ __forceinline__ void tc_store_gated(const QGemmTcParams& p, int token, int row, float gate, float up) {
    if (row < p.out.end[0])
        p.out.y[0][(size_t)token * p.out.stride[0] + row] = __float2bfloat16_rn(gated_activation(
            __bfloat162float(__float2bfloat16_rn(gate)), __bfloat162float(__float2bfloat16_rn(up)), p.gated_act));
}
__device__ __forceinline__ void tmem_ld16(unsigned addr, unsigned (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(addr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// 16 lanes x 32 columns in the order of four m16n8 accumulator fragments: lane (g, t), register 4 i + r: row g + 8 (r >> 1),
// column 8 i + 2 t + (r & 1)
__device__ __forceinline__ void tmem_st_frag(unsigned addr, const unsigned (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]),
                   "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ unsigned pair_leader(unsigned addr) {   // the same shared-memory place in the cluster's first CTA
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
// Arrivals at the barriers that an MMA warp waits at.
// Within a CTA: hands over whatever the arriving warp has done or waited for.
__device__ __forceinline__ void tc_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// From either CTA of a pair (`bar`: a cluster address), for what was done to tensor memory: tcgen05 operations are ordered by the waits
// and fences of their own on either side and by the arrival being seen. A release of cluster scope would order nothing more that the
// MMAs read, and waits for the weights that the arriving warp has requested ahead (1200 clocks).
__device__ __forceinline__ void tc_arrive_tmem(unsigned bar) { asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }

// A ring position and the parity of its phase.
template <int N>
struct RingPos {
    int s = 0; unsigned par = 0;
    __device__ __forceinline__ void next() { if (++s == N) { s = 0; par ^= 1u; } }
    __device__ __forceinline__ void skip2() { s += 2; if (s >= N) { s -= N; par ^= 1u; } }
    __device__ __forceinline__ void skip3() { s += 3; if (s >= N) { s -= N; par ^= 1u; } }
};

template <int STAGES>
struct TcBars {
    unsigned long long full[STAGES], empty[STAGES];   // a stage has landed; its MMAs are done
    unsigned long long ready[kTcMaxA];                 // a weight tile is in tensor memory (one arrival per dequantising warp)
    unsigned long long acc_full, acc_empty;           // accumulator complete; read (long kernel)
    unsigned tmem;
    int failed;
};

// Common start: barriers and tensor memory. Ends with all threads (of the pair) synchronised.
template <int STAGES, unsigned COLS, int CG>
__device__ __forceinline__ unsigned tc_setup(TcBars<STAGES>& b) {
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < STAGES; ++s) { mbar_init(&b.empty[s], 1); mbar_init(&b.full[s], 1); }
#pragma unroll
        for (int i = 0; i < kTcMaxA; ++i) mbar_init(&b.ready[i], kTcSet * CG);
        mbar_init(&b.acc_full, 1);
        mbar_init(&b.acc_empty, kTcEpiWarps * CG);
        b.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 32) {
        __syncwarp();  // the allocation is a warp-wide instruction: re-converge after the single-thread block
        if (CG == 1) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&b.tmem)), "r"(COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&b.tmem)), "r"(COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (CG == 2) cg::this_cluster().sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return b.tmem;
}
__device__ __forceinline__ void tc_fail(int* status, int* failed, int code) { atomicExch(status, code); *reinterpret_cast<volatile int*>(failed) = 1; }

// ---- producer: a step's activations (`rows` rows of shared memory) into a stage ---------------------------------------------
template <int ROWS>
__device__ __forceinline__ void tc_issue(const CUtensorMap* xmap, unsigned stage, unsigned bar, int kt, int tok0) {
    mbar_expect(bar, (unsigned)ROWS * 256u);
    tma_load_2d(stage, xmap, kt * kTcStep, tok0, bar);
    tma_load_2d(stage + ROWS * 128, xmap, kt * kTcStep + 64, tok0, bar);
}
// The same for a pair: both CTAs' copies count on the barrier of the CTA that issues the MMAs (`bar`: a cluster address). The other CTA's
// may get there before the bytes are announced: the phase ends with the announcement at the earliest.
template <int ROWS>
__device__ __forceinline__ void tc_issue_pair(const CUtensorMap* xmap, unsigned stage, unsigned bar, int kt, int tok0) {
    tma_load_2d_pair(stage, xmap, kt * kTcStep, tok0, bar);
    tma_load_2d_pair(stage + ROWS * 128, xmap, kt * kTcStep + 64, tok0, bar);
}
// ---- the eight MMAs of a step; ROWS: activation rows in this CTA's shared memory ----------------------------------------------
template <int CG, int ROWS>
__device__ __forceinline__ void tc_mma_step(unsigned d_tmem, unsigned a_tmem, unsigned stage, bool first) {
    const unsigned lo = umma_desc_lo(stage);
#pragma unroll
    for (int j = 0; j < kTcStep / 16; ++j)   // 16 fp16 = 8 columns of A, 32 bytes along K inside B's 128-byte row
        umma_f16_ta<CG>(d_tmem, a_tmem + 8u * j, lo + (j >> 2) * (ROWS * 8) + 2 * (j & 3), umma_idesc(kTcRows * CG, ROWS * CG), j > 0 ? 1u : first ? 0u : 1u);
}

// ---- dequantising warps: warp w takes row tile 2 (w & 3) + ((w >> 2) & 1) of the eight of the CTA's rows (its lanes of tensor
// memory) in every other step ---------------------------------------------------------------------------------
template <bool F16SB>
__device__ __forceinline__ float tc_scale(unsigned pair) { return F16SB ? __half2float(__ushort_as_half((unsigned short)(pair & 0xFFFFu))) : __uint_as_float(pair << 16); }
template <bool F16SB>
__device__ __forceinline__ float tc_zero(unsigned pair) { return F16SB ? __half2float(__ushort_as_half((unsigned short)(pair >> 16))) : __uint_as_float(pair & 0xFFFF0000u); }
// the scale as an fp16 pair: a bf16 (MLX) scale converts exactly (8 mantissa bits into 11) unless it lies below fp16's normal range,
// where the weights it scales are nil anyway
template <bool F16SB>
__device__ __forceinline__ __half2 tc_scale2(unsigned pair) {
    if (F16SB) { const unsigned v = __byte_perm(pair, 0, 0x1010); return *reinterpret_cast<const __half2*>(&v); }
    return __float2half2_rn(__uint_as_float(pair << 16));
}
// 16 x 64 nibbles -> scale * (q - 8) in fragment order; the low nibble of each byte is row g, the high one row g + 8
__device__ __forceinline__ void tc_unpack(const uint4& wq, __half2 lo, __half2 hi, unsigned (&a)[16]) {
    const unsigned w[4] = {wq.x, wq.y, wq.z, wq.w};
    const unsigned c1032 = 0x64086408u, c16th = 0x2C002C00u, c72 = 0xD480D480u;   // 1024 + 8; 1 / 16; -(64 + 8)
    const __half2 off = *reinterpret_cast<const __half2*>(&c1032), sixteenth = *reinterpret_cast<const __half2*>(&c16th), off16 = *reinterpret_cast<const __half2*>(&c72);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const unsigned v = (r & 1) ? w[j] >> 8 : w[j];
            const unsigned pr = ((r >> 1) ? v & 0x00F000F0u : v & 0x000F000Fu) | 0x64006400u;
            const __half2 m = *reinterpret_cast<const __half2*>(&pr);
            const __half2 h = __hmul2((r >> 1) ? __hfma2(m, sixteenth, off16) : __hsub2(m, off), (r >> 1) ? hi : lo);
            a[4 * j + r] = *reinterpret_cast<const unsigned*>(&h);
        }
}
// The A operand of 64 appended columns, block `blk` of them: c = 64 (zero + 8 scale) of 64 groups as an fp16 pair (hi, lo). Of three
// blocks one after the other the first carries c_hi (against sum_hi), the second c_lo (against sum_hi), the third c_hi (against sum_lo).
// The activation side holds sum / 64 so that neither factor leaves fp16's range.
template <bool F16SB>
__device__ __forceinline__ float tc_const(unsigned pair) { return 64.0f * fmaf(8.0f, tc_scale<F16SB>(pair), tc_zero<F16SB>(pair)); }
template <bool F16SB>
__device__ __forceinline__ void tc_appended(const QGemmTcParams& p, int rt, int blk, unsigned (&a)[16]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int plane = blk % 3, st0 = blk / 3 * 16;   // four groups per 16-byte entry
    if (st0 >= p.kt / 4) {   // (padding to whole steps)
#pragma unroll
        for (int i = 0; i < 16; ++i) a[i] = 0u;
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int st = st0 + 4 * j + t;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (rt < p.row_tiles && st < p.kt / 4) v = __ldg(reinterpret_cast<const uint4*>(p.sb) + ((size_t)rt * (p.kt / 4) + st) * 16 + g + 8 * h);
            const unsigned u[4] = {v.x, v.y, v.z, v.w};
            float c[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float cf = tc_const<F16SB>(u[i]), hi = __half2float(__float2half_rn(cf));
                c[i] = plane == 1 ? cf - hi : hi;
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const __half2 pr = __floats2half2_rn(c[2 * i], c[2 * i + 1]);
                a[4 * j + 2 * h + i] = *reinterpret_cast<const unsigned*>(&pr);
            }
        }
}
// c_hi and c_lo of 64 groups of a row tile at once
template <bool F16SB>
__device__ __forceinline__ void tc_appended_pair(const QGemmTcParams& p, int rt, int block, unsigned (&hi)[16], unsigned (&lo)[16]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int st = block * 16 + 4 * (i >> 1) + t;
        v[i] = st < p.kt / 4 ? __ldg(reinterpret_cast<const uint4*>(p.sb) + ((size_t)rt * (p.kt / 4) + st) * 16 + g + 8 * (i & 1)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const unsigned u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float c0 = tc_const<F16SB>(u[2 * e]), c1 = tc_const<F16SB>(u[2 * e + 1]);
            const __half2 h = __floats2half2_rn(c0, c1);
            const float2 f = __half22float2(h);
            const __half2 l = __floats2half2_rn(c0 - f.x, c1 - f.y);
            hi[2 * i + e] = *reinterpret_cast<const unsigned*>(&h);
            lo[2 * i + e] = *reinterpret_cast<const unsigned*>(&l);
        }
    }
}

// Everything a dequantising warp does: the steps [lo, hi) of tiles `tile`, `tile` + stride, ... below `end`, of all of which it takes
// every other one (counted over the tiles). rt_of(tile): the first row tile of the CTA's rows; w_ring: the CTA's weight rings.
// Returns false when a wait expired. (What bounds a step is this warp's chain of waits, shared-memory reads, unpacking and the store to
// tensor memory, about 1600 clocks with all warps in every step; two sets of warps have twice the time, and the waits and the arrival
// serve two tiles. Weights kept ahead in registers were waited for as if the latest request were needed.)
template <int CG, int SA, int STAGES, bool F16SB, typename RowTile>
__device__ __forceinline__ bool tc_dequant(const QGemmTcParams& p, TcBars<STAGES>& b, unsigned w_ring, unsigned tmem_a, int tile, int stride, int end, int lo, int hi, RowTile rt_of) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, set = warp / kTcSet;
    const int own_rt = 2 * (warp & 3) + ((warp >> 2) & 1);
    const unsigned a_dst = tmem_a + ((unsigned)((warp & 3) * 32 + ((warp >> 2) & 1) * 16) << 16);
    const unsigned full0 = smem_u32(&b.full[0]), empty0 = smem_u32(&b.empty[0]);
    const unsigned ready0 = CG == 1 ? smem_u32(&b.ready[0]) : pair_leader(smem_u32(&b.ready[0]));
    const unsigned ring = w_ring + warp * (kTcAhead * kTcSlotBytes);
    const int real_hi = min(hi, p.real_steps), odd = (hi - lo) & 1;

    // request side: this warp's steps over real weights, in order (rows beyond the last are not stored: what they hold does not matter)
    int f_tile = tile, f_kt = lo + set, f_set = set;
    auto fetch = [&](int slot) {
        while (f_kt >= real_hi && f_tile < end) {   // on to the next tile; with an odd number of steps the sets change places
            f_tile += stride;
            f_set ^= odd;
            f_kt = lo + f_set;
            if (lo >= real_hi) f_tile = end;        // (a CTA whose share of K is appended columns only)
        }
        if (f_tile < end) {
            const int rt = min(rt_of(f_tile) + own_rt, p.row_tiles - 1), kt = 2 * f_kt;
            const unsigned dst = ring + slot * kTcSlotBytes;
            const uint4* w = p.tiles + ((size_t)rt * p.kt + kt) * 32 + lane;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + lane * 16), "l"(w) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 512 + lane * 16), "l"(w + 32) : "memory");
            if (lane < 16) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 1024 + lane * 8), "l"(p.sb + ((size_t)rt * (p.kt / 4) + (kt >> 2)) * 64 + lane * 4 + (kt & 3)) : "memory");
            f_kt += 2;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // this warp's place in the sequence of all steps: `at` is a stage's place, `old` that of the step SA back, a_slot its weight tile
    RingPos<STAGES> at, old;
    at.s = set;
    old.s = (SA & 1) ^ set;                       // the first step of this set that waits is SA + that
    int a_slot = set % SA, fresh = (SA + 1 - set) / 2;   // steps without one SA back
    auto begin = [&]() {   // the MMAs of the step SA back are done (its weight tile may be overwritten)
        if (fresh > 0) { --fresh; return true; }
        const bool ok = mbar_wait_warp(empty0 + 8u * old.s, old.par);
        old.skip2();
        return ok;
    };
    auto finish = [&]() {
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");   // the stores are ordered before the MMAs of the thread that waits
        // the CTA's activations have landed: one warp's arrival covers them for the MMAs (of a pair the MMA warp waits for both CTAs')
        if (CG == 1 && (warp & (kTcSet - 1)) == 0 && !mbar_wait_warp(full0 + 8u * at.s, at.par)) return false;
        __syncwarp();
        if (lane == 0) {
            if (CG == 1) tc_arrive(ready0 + 8u * a_slot);
            else tc_arrive_tmem(ready0 + 8u * a_slot);
        }
        a_slot += 2;
        if (a_slot >= SA) a_slot -= SA;
        at.skip2();
        return true;
    };
    static_assert(SA >= 2 && STAGES >= 2, "steps advance by two");
    // a wait by parity cannot tell a phase from the one two before: when a step is seen to be SA steps behind the MMAs, the copies and
    // MMAs of the step STAGES back (the phase before of its stage's barriers) have to be over
    static_assert(STAGES >= SA, "a stage's phase may not lap a waiting warp");

#pragma unroll
    for (int i = 0; i < kTcAhead - 1; ++i) fetch(i);
    int slot = 0, s_now = set;
    bool ok = true;
    for (; tile < end && ok; tile += stride, s_now ^= odd) {
        int kt = lo + s_now;
        for (; kt < real_hi; kt += 2) {
            fetch(slot == 0 ? kTcAhead - 1 : slot - 1);   // (that slot was read a step ago, by all lanes)
            asm volatile("cp.async.wait_group %0;" ::"n"(kTcAhead - 1) : "memory");
            __syncwarp();
            const unsigned src = ring + slot * kTcSlotBytes;
            if (++slot == kTcAhead) slot = 0;
            uint4 w0, w1;
            uint2 s_lo, s_hi;
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w0.x), "=r"(w0.y), "=r"(w0.z), "=r"(w0.w) : "r"(src + lane * 16));
            asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w1.x), "=r"(w1.y), "=r"(w1.z), "=r"(w1.w) : "r"(src + 512 + lane * 16));
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(s_lo.x), "=r"(s_lo.y) : "r"(src + 1024 + (lane >> 2) * 8));
            asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(s_hi.x), "=r"(s_hi.y) : "r"(src + 1088 + (lane >> 2) * 8));
            unsigned a[16];
            tc_unpack(w0, tc_scale2<F16SB>(s_lo.x), tc_scale2<F16SB>(s_hi.x), a);
            if (!begin()) { ok = false; break; }
            tmem_st_frag(a_dst + (unsigned)a_slot * 64u, a);
            tc_unpack(w1, tc_scale2<F16SB>(s_lo.y), tc_scale2<F16SB>(s_hi.y), a);
            tmem_st_frag(a_dst + (unsigned)a_slot * 64u + 32u, a);
            if (!finish()) { ok = false; break; }
        }
        for (; kt < hi && ok; kt += 2) {
            if (!begin()) { ok = false; break; }
            const int blk = (kt - p.real_steps) * (kTcStep / 64), rt = rt_of(tile) + own_rt;
            if (blk % 3 == 0 && rt < p.row_tiles) {   // hi and lo of the same groups
                unsigned a[16], a_lo[16];
                tc_appended_pair<F16SB>(p, rt, blk / 3, a, a_lo);
                tmem_st_frag(a_dst + (unsigned)a_slot * 64u, a);
                tmem_st_frag(a_dst + (unsigned)a_slot * 64u + 32u, a_lo);
                if (!finish()) ok = false;
                continue;
            }
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                unsigned a[16];
                tc_appended<F16SB>(p, rt, blk + half, a);
                tmem_st_frag(a_dst + (unsigned)a_slot * 64u + half * 32u, a);
            }
            if (!finish()) ok = false;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    return ok;
}

// Where a lane's results go: its weight row of one output, or the row of a gate row and its up row together.
struct TcDst { __nv_bfloat16* y; int stride; bool live; };
__device__ __forceinline__ TcDst tc_dst(const QGemmTcParams& p, int row) {
    if (p.gated) { const int r = (row >> 4) * 8 + (row & 7); return {p.out.y[0] + r, p.out.stride[0], r < p.out.end[0]}; }
    const int q = row < p.out.end[0] ? 0 : row < p.out.end[1] ? 1 : 2;
    return {(q == 0 ? p.out.y[0] : q == 1 ? p.out.y[1] : p.out.y[2]) + (row - (q == 0 ? 0 : q == 1 ? p.out.end[0] : p.out.end[1])),
            q == 0 ? p.out.stride[0] : q == 1 ? p.out.stride[1] : p.out.stride[2], row < p.out.end[2]};
}
// silu(gate) * up
__device__ __forceinline__ float tc_swiglu(float gate, float up) { return 0.25f * gate * four_over(1.0f + expf(-gate)) * up; }
template <bool GELU>
__device__ __forceinline__ void tc_emit_gated(const QGemmTcParams& p, const TcDst& d, const unsigned* v, float fac, int fac0, int token0) {
    // gate rows sit in the lanes of the first eight of 16, up rows in the others: a gate lane finishes even columns, its up lane odd ones.
    // Both are rounded to bf16 first because the reference stores them to bf16 scratch before `swiglu` reads them
    // (Primitives/ElementwiseFragment.swift:49-54).
    const int up_lane = (threadIdx.x >> 3) & 1;
    __nv_bfloat16 res[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const unsigned own = up_lane ? v[2 * i + 1] : v[2 * i], other = __shfl_xor_sync(0xffffffffu, up_lane ? v[2 * i] : v[2 * i + 1], 8);
        const float sc = __shfl_sync(0xffffffffu, fac, fac0 + 2 * i + up_lane);
        const float gate = __bfloat162float(__float2bfloat16_rn(__uint_as_float(up_lane ? other : own) * sc));
        const float up = __bfloat162float(__float2bfloat16_rn(__uint_as_float(up_lane ? own : other) * sc));
        res[i] = __float2bfloat16_rn(GELU ? gated_activation(gate, up, GATED_ACT_GELU_TANH) : tc_swiglu(gate, up));
    }
    if (!d.live) return;
    __nv_bfloat16* y = d.y + (size_t)(token0 + up_lane) * d.stride;
    if (token0 + 16 <= p.m) {
#pragma unroll
        for (int i = 0; i < 8; ++i) y[(size_t)(2 * i) * d.stride] = res[i];
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (token0 + 2 * i + up_lane < p.m) y[(size_t)(2 * i) * d.stride] = res[i];
    }
}
// 16 columns of a warp's 32 rows, tokens token0 on; lane fac0 + i holds the factor of token0 + i. What bounds a tile's end is the chain
// behind its accumulators, which the next tile's MMAs wait for: a load of the factor, a test, an activation and a store for each column
// in turn took as long as 18 steps of 128 columns (gate and up of 16384 x 2048 over 2010 rows: 257 us, 37 per tile). Without a branch
// between the columns and with the factors in registers beforehand they overlap. Prompt of 2011 tokens, 16 layers of width 2048:
// 8298 -> 6335 us; 4096 tokens, 4 layers of width 4096: 10410 -> 9092 us; 14336 x 4096 at 512 rows 64.4 -> 60.6 us.
__device__ __forceinline__ void tc_emit16(const QGemmTcParams& p, const TcDst& d, const unsigned* v, float fac, int fac0, int token0) {
    if (p.gated) {
        if (p.gated_act == GATED_ACT_GELU_TANH) tc_emit_gated<true>(p, d, v, fac, fac0, token0);
        else tc_emit_gated<false>(p, d, v, fac, fac0, token0);
        return;
    }
    __nv_bfloat16 res[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) res[i] = __float2bfloat16_rn(__uint_as_float(v[i]) * __shfl_sync(0xffffffffu, fac, fac0 + i));
    if (!d.live) return;
    __nv_bfloat16* y = d.y + (size_t)token0 * d.stride;
    if (token0 + 16 <= p.m) {
#pragma unroll
        for (int i = 0; i < 16; ++i) y[(size_t)i * d.stride] = res[i];
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (token0 + i < p.m) y[(size_t)i * d.stride] = res[i];
    }
}

// ---- long form: many activation rows. Pairs of CTAs walk tiles of 256 weight rows x 256 activation rows; eight warps of their own
// store a tile's results while the next tile's first stages are fetched and dequantised. ------------------------------------
constexpr int kTcPairRows = 128;   // activation rows in a CTA's shared memory
template <int STAGES, bool F16SB>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__((kTcDeqWarps + 2 + kTcEpiWarps) * 32, 1) qgemm_tc_kernel(const QGemmTcParams p, const __grid_constant__ CUtensorMap xmap) {
    constexpr int SA = 4;
    constexpr unsigned kTmemCols = 512;                      // accumulator 256, four weight tiles
    constexpr unsigned STAGE_BYTES = kTcPairRows * 256;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const unsigned ring = (smem_u32(smem_raw) + 1023u) & ~1023u;   // the swizzle pattern repeats every 1024 bytes
    __shared__ __align__(8) TcBars<STAGES> bars;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = (int)blockIdx.x & 1;
    const int first = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const unsigned tmem_d = tc_setup<STAGES, kTmemCols, 2>(bars);
    pdl_launch_dependents();   // (behind the allocation: a CTA of the next kernel cannot take tensor memory that this one still waits for)
    volatile int* const failed = &bars.failed;

    if (warp == kTcDeqWarps) {
        if (rank == 0) {   // the first CTA issues for both
            const bool el = elect_one();
            RingPos<STAGES> full;
            int a_slot = 0, done = 0;   // done: tiles whose completion has been requested
            unsigned a_par = 0;
            bool ok = true;
            for (int tile = first; tile < p.n_tiles && ok; tile += pairs) {
                // the accumulators of the tile before have been read
                if (done > 0 && !mbar_wait_cluster_warp(&bars.acc_empty, (unsigned)((done - 1) & 1))) { ok = false; break; }
                for (int kt = 0; kt < p.steps; ++kt) {
                    if (!mbar_wait_cluster_warp(&bars.full[full.s], full.par) || !mbar_wait_cluster_warp(&bars.ready[a_slot], a_par)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (el) {
                        tc_mma_step<2, kTcPairRows>(tmem_d, tmem_d + 256u + a_slot * 64u, ring + full.s * STAGE_BYTES, kt == 0);
                        umma_commit_pair(&bars.empty[full.s]);
                    }
                    __syncwarp();
                    if (++a_slot == SA) { a_slot = 0; a_par ^= 1u; }
                    full.next();
                }
                if (ok) { if (el) umma_commit_pair(&bars.acc_full); ++done; }
                __syncwarp();
            }
            if (!ok && el) {   // the MMAs issued so far end before tensor memory is freed
                tc_fail(p.status, &bars.failed, 2);
                umma_commit_pair(&bars.acc_full);
                if (done > 0) mbar_wait(&bars.acc_full, (unsigned)((done - 1) & 1));
                mbar_wait(&bars.acc_full, (unsigned)(done & 1));
            }
        }
        __syncwarp();
    } else if (warp == kTcDeqWarps + 1) {
        if (lane == 0) {
            pdl_wait();                         // the activations come from the kernel just before this one
            RingPos<STAGES> at;
            const unsigned full0 = pair_leader(smem_u32(&bars.full[0]));
            int issued = 0;
            bool ok = true;
            for (int tile = first; tile < p.n_tiles && ok; tile += pairs) {
                const int tok0 = tile % p.tok_tiles * 256 + rank * kTcPairRows;
                for (int kt = 0; kt < p.steps; ++kt) {
                    // the MMAs that read this stage a round ago are done
                    if (*failed || (issued >= STAGES && !mbar_wait(&bars.empty[at.s], at.par ^ 1u))) { ok = false; break; }
                    if (rank == 0) mbar_expect(smem_u32(&bars.full[at.s]), 2u * STAGE_BYTES);
                    tc_issue_pair<kTcPairRows>(&xmap, ring + at.s * STAGE_BYTES, full0 + 8u * at.s, kt, tok0);
                    at.next();
                    ++issued;
                }
            }
            if (!ok) tc_fail(p.status, &bars.failed, 3);
            // every copy of the pair has landed before either CTA leaves: they meet again behind this. Where one of them stopped early the
            // last wait is for a phase that does not end: its limit is the time that the other's copies get.
            if (rank == 0) {
                for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i) mbar_wait(&bars.full[i % STAGES], (unsigned)((i / STAGES) & 1));
                if (!ok) mbar_wait(&bars.full[at.s], at.par);
            }
        }
        __syncwarp();
    } else if (warp < kTcDeqWarps) {
        if (!tc_dequant<2, SA, STAGES, F16SB>(p, bars, ring + STAGES * STAGE_BYTES, tmem_d + 256u, first, pairs, p.n_tiles, 0, p.steps,
                                              [&](int tile) { return tile / p.tok_tiles * 16 + rank * 8; })) tc_fail(p.status, &bars.failed, 1);
        __syncwarp();
    } else {
        // a warp reads the 32 accumulator lanes of its quarter (warp & 3) and half of the columns
        const int half = (warp - kTcDeqWarps - 2) >> 2;
        const unsigned acc_empty = pair_leader(smem_u32(&bars.acc_empty));
        unsigned par = 0;
        pdl_wait();   // (the rows' factors)
        for (int tile = first; tile < p.n_tiles; tile += pairs, par ^= 1u) {
            const int tok0 = tile % p.tok_tiles * 256 + half * 128;
            const TcDst dst = tc_dst(p, tile / p.tok_tiles * 256 + rank * kTcRows + (warp & 3) * 32 + lane);
            float fac = tc_rscale(p, min(tok0 + lane, p.m - 1));   // of 32 tokens, one per lane, requested before they are needed
            if (!mbar_wait_warp(&bars.acc_full, par)) { tc_fail(p.status, &bars.failed, 4); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            float next = 0.f;
#pragma unroll 1
            for (int c = 0; c < 128; c += 16) {
                const int token = tok0 + c;
                unsigned v[16];
                if (!(c & 16)) next = tc_rscale(p, min(token + 32 + lane, p.m - 1));
                if (token < p.m) tmem_ld16(tmem_d + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)(half * 128 + c), v);
                const bool last = c == 112 || token + 16 >= p.m;   // uniform across the warp
                if (last) {   // the accumulators have been read
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) tc_arrive_tmem(acc_empty);
                }
                if (token < p.m) tc_emit16(p, dst, v, fac, c & 16, token);
                if (last) break;
                if (c & 16) fac = next;
            }
        }
        __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cg::this_cluster().sync();   // nobody arrives at a barrier of a CTA that has left, and no MMA reads its tensor memory
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kTmemCols) : "memory");
}

// ---- short form: 65 to 128 activation rows, or few tiles. K is cut over the CTAs of a cluster; each sends its part of a tile's results
// to the CTA that finishes a row, through distributed shared memory (the ring's, which is free by then). 72 registers: what is left of an
// SM's takes the CTAs that turn the next product's rows into fp16 (with 96 of them 2048 x 2048 at 256 rows took 18.3 us, with 72 14.7; 16.6 before
// the end of a tile was worked out for 16 columns at once). ---------------------------------------------------------------------------
template <int BN, int STAGES, bool F16SB>
__global__ void __maxnreg__(72) qgemm_tc_short_kernel(const QGemmTcParams p, const __grid_constant__ CUtensorMap xmap) {
    constexpr unsigned kTmemCols = 512;                      // accumulator, four weight tiles
    constexpr int SA = kTcMaxA;
    static_assert(BN + SA * 64 <= 512, "tensor memory");
    constexpr unsigned STAGE_BYTES = BN * 256;
    static_assert((size_t)STAGES * STAGE_BYTES >= (size_t)BN * kTcRows * 4, "the ring takes what the cluster sends");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* const ring_ptr = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const unsigned ring = smem_u32(ring_ptr);
    __shared__ __align__(8) TcBars<STAGES> bars;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % p.splits, row0 = (int)blockIdx.x / p.splits * kTcRows, tok0 = blockIdx.y * BN;
    const int lo = p.steps * rank / p.splits, hi = p.steps * (rank + 1) / p.splits;
    const unsigned tmem_d = tc_setup<STAGES, kTmemCols, 1>(bars);
    pdl_launch_dependents();   // (behind the allocation: a CTA of the next kernel cannot take tensor memory that this one still waits for)
    volatile int* const failed = &bars.failed;

    if (warp == kTcDeqWarps) {
        const bool el = elect_one();
        RingPos<STAGES> full;
        int a_slot = 0;
        unsigned a_par = 0;
        for (int kt = lo; kt < hi; ++kt) {
            if (!mbar_wait_warp(&bars.ready[a_slot], a_par)) { tc_fail(p.status, &bars.failed, 2); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (el) {
                tc_mma_step<1, BN>(tmem_d, tmem_d + BN + a_slot * 64u, ring + full.s * STAGE_BYTES, kt == lo);
                umma_commit(&bars.empty[full.s]);
            }
            __syncwarp();
            if (++a_slot == SA) { a_slot = 0; a_par ^= 1u; }
            full.next();
        }
        if (el) umma_commit(&bars.acc_full);   // also behind a failure: tensor memory is not freed under MMAs in flight
        __syncwarp();
    } else if (warp == kTcDeqWarps + 1) {
        if (lane == 0) {
            pdl_wait();                         // the activations come from the kernel just before this one
            RingPos<STAGES> at;
            int issued = 0;
            for (int kt = lo; kt < hi; ++kt) {
                if (*failed || (issued >= STAGES && !mbar_wait(&bars.empty[at.s], at.par ^ 1u))) { tc_fail(p.status, &bars.failed, 3); break; }
                tc_issue<BN>(&xmap, ring + at.s * STAGE_BYTES, smem_u32(&bars.full[at.s]), kt, tok0);
                at.next();
                ++issued;
            }
            // every copy has landed before the ring is given to the cluster (also behind a failure)
            for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i) mbar_wait(&bars.full[i % STAGES], (unsigned)((i / STAGES) & 1));
        }
        __syncwarp();
    } else {
        if (!tc_dequant<1, SA, STAGES, F16SB>(p, bars, ring + STAGES * STAGE_BYTES, tmem_d + BN, 0, 1, 1, lo, hi, [&](int) { return row0 / 16; })) tc_fail(p.status, &bars.failed, 1);
        __syncwarp();
    }
    // ---- results: warp w reads the lanes of quarter w & 3 and a quarter of the columns ---------------------------------------
    pdl_wait();   // (the rows' factors)
    const bool done = mbar_wait_warp(&bars.acc_full, 0u);
    if (!done && lane == 0) tc_fail(p.status, &bars.failed, 5);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int r = (warp & 3) * 32 + lane;
    constexpr int CW = 16;                          // columns per read
    const cg::cluster_group cluster = cg::this_cluster();
    const int own = BN / p.splits;                  // columns that a CTA of the cluster finishes: whole reads
    const unsigned lanes = tmem_d + ((unsigned)((warp & 3) * 32) << 16);
    if (p.splits == 1) {
        if (done && warp < kTcDeqWarps) {
            const TcDst dst = tc_dst(p, row0 + r);
#pragma unroll 1
            for (int c0 = (warp >> 2) * CW; c0 < BN; c0 += 4 * CW) {
                if (tok0 + c0 >= p.m) break;
                unsigned v[CW];
                tmem_ld16(lanes + (unsigned)c0, v);
                tc_emit16(p, dst, v, tc_rscale(p, min(tok0 + c0 + (lane & 15), p.m - 1)), 0, tok0 + c0);
            }
        }
    } else {
        cluster.sync();                             // every ring of the cluster is free
        if (done && warp < kTcDeqWarps) {
#pragma unroll 1
            for (int c0 = (warp >> 2) * CW; c0 < BN; c0 += 4 * CW) {
                if (tok0 + c0 >= p.m) break;
                unsigned v[CW];
                tmem_ld16(lanes + (unsigned)c0, v);
                const int owner = c0 / own;
                float* to = reinterpret_cast<float*>(cluster.map_shared_rank(ring_ptr, owner)) + (rank * own + (c0 - owner * own)) * kTcRows + r;
#pragma unroll
                for (int i = 0; i < CW; ++i)
                    if (tok0 + c0 + i < p.m) to[i * kTcRows] = __uint_as_float(v[i]);
            }
        }
        cluster.sync();
        const float* got = reinterpret_cast<const float*>(ring_ptr);
        const int rows = p.gated ? kTcRows / 2 : kTcRows;
        for (int o = threadIdx.x; o < own * rows; o += blockDim.x) {
            const int cl = o / rows, i = o % rows, token = tok0 + rank * own + cl;
            if (token >= p.m) continue;
            const int ra = p.gated ? (i >> 3) * 16 + (i & 7) : i;   // a gate row, its up row eight further on
            const float* src = got + cl * kTcRows + ra;
            float va = 0.f, vb = 0.f;
            for (int z = 0; z < p.splits; ++z) {   // ranges in order
                va += src[z * own * kTcRows];
                if (p.gated) vb += src[z * own * kTcRows + 8];
            }
            const float sc = tc_rscale(p, token);
            if (p.gated) tc_store_gated(p, token, row0 / 2 + i, va * sc, vb * sc);
            else tc_store(p.out, token, row0 + i, va * sc);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kTmemCols) : "memory");
}

// ---- few activation rows (up to 64): persistent CTAs, one on an SM, or clusters of two or four along K ------------------------------
// What bounds it: the dequantising warps (about 330 instructions per 4096 weights; without the subtractions and multiplications a pass of
// eight row tiles would take 0.45 us per step instead of 0.6), before that what surrounds them: in steps of 128 x 128 with a wait, a
// fetch and an arrival for each, appended columns worked out three times, two CTAs on some SMs and one on others, 28672 x 4096 at 41 rows
// took 34 us, 128256 x 4096 139; now 28 and 87. With their rows on the way to fp16, one call after the other: 14336 x 4096 23.9 -> 18.5,
// 4096 x 14336 32 -> 24, 6144 x 4096 21.0 -> 14.7, 2048 x 2048 13.2 -> 9.8. (What the compiler spills lies outside the loop over units: 0.6 % of
// the instructions.) Hence
//   * a unit of work is 16 weight rows x 256 columns, the streaming layout's contiguous 2304 bytes: addresses by addition, one wait, one
//     arrival and one set of scales for 16 words of nibbles per lane. A warp reads a unit into registers and requests the next but one in
//     its place;
//   * row tiles (16 rows) are dealt to the CTAs one by one: passes of eight each over one contiguous window of the matrix, what is left
//     evenly (sl_ctas: as few CTAs as that takes). Row tile j of a pass takes lanes 32 (j & 3) + 16 (j >> 2) of tensor memory, so that four already occupy all four schedulers
//     (a warp reaches the lanes of its quarter only); six warps per quarter, three steps of two row tiles;
//   * two accumulators: four warps of their own store a pass while the next one is multiplied;
//   * the wait for a step's activations is made by a dequantising warp, so that the MMA warp has one wait per step (16 MMAs at 30 clocks,
//     about 200 for a wait). CTAs that start at different places of K, so as not to ask for the same activations at the same time, took
//     longer (12 -> 19 us for 4096 x 4096).
// K over a cluster (few row tiles, long K): one pass, the parts meet in distributed shared memory.
constexpr int kSlCols = 256;                    // columns of K per step
constexpr int kSlWarps = 24;                    // dequantising: six of a quarter, three steps of two row tiles
constexpr int kSlAhead = 2;                     // units of a warp in its ring, behind the one in its registers
constexpr int kSlUnitBytes = 4 * 512 + 256;     // four 16 x 64 tiles and 16 rows' four scale / zero pairs
constexpr int kSlRingBytes = kSlWarps * kSlAhead * kSlUnitBytes;
constexpr int kSlSlots = 3;                     // dequantised 128 x 256 tiles in tensor memory, 128 columns each
constexpr int kSlEpiWarps = 4;
constexpr int kSlThreads = (kSlWarps + 2 + kSlEpiWarps) * 32;

template <int STAGES>
struct SlBars {
    unsigned long long full[STAGES], empty[STAGES];        // activations of a step
    unsigned long long ready[kSlSlots], free[kSlSlots];    // a weight tile is in tensor memory (eight arrivals); its MMAs are done
    unsigned long long acc_full[2], acc_empty[2];
    unsigned tmem;
    int failed;
};
// row tiles of this CTA (group of them along K) in pass `pass`: the first and how many
struct SlPass { int first, count; };
__device__ __forceinline__ SlPass sl_pass(const QGemmTcParams& p, int pass, int cta, int ctas) {
    if (pass < p.whole) return {(pass * ctas + cta) * 8, 8};
    const int lo = (int)((unsigned)(p.left * cta) / (unsigned)ctas);   // (left < 8 ctas)
    return {p.whole * ctas * 8 + lo, (int)((unsigned)(p.left * (cta + 1)) / (unsigned)ctas) - lo};
}

template <int BN, int STAGES, bool F16SB>
__global__ void __launch_bounds__(kSlThreads, 1) qgemm_slab_kernel(const QGemmTcParams p, const __grid_constant__ CUtensorMap xmap) {
    constexpr unsigned kTmemCols = 512;                    // accumulators 2 BN, weight tiles 3 x 128
    static_assert(2 * BN + kSlSlots * 128 <= 512, "tensor memory");
    constexpr unsigned STAGE_BYTES = BN * kSlCols * 2, HALF = BN * 128;   // (boxes of 64 columns)
    static_assert((size_t)STAGES * STAGE_BYTES >= (size_t)BN * kTcRows * 4, "the ring takes what the cluster sends");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* const ring_ptr = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const unsigned ring = smem_u32(ring_ptr);
    __shared__ __align__(8) SlBars<STAGES> bars;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % p.splits, cta = (int)blockIdx.x / p.splits, ctas = (int)gridDim.x / p.splits;
    const int lo = p.steps * rank / p.splits, hi = p.steps * (rank + 1) / p.splits, steps = hi - lo;
    const int passes = p.n_tiles;
    const int real = max(0, min(hi, p.real_steps) - lo);   // steps over weights; those over appended columns, 192 of them each, follow
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&bars.full[s], 1); mbar_init(&bars.empty[s], 1); }
        for (int s = 0; s < kSlSlots; ++s) { mbar_init(&bars.ready[s], 8); mbar_init(&bars.free[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&bars.acc_full[s], 1); mbar_init(&bars.acc_empty[s], kSlEpiWarps); }
        bars.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars.tmem)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_d = bars.tmem, tmem_a = tmem_d + 2 * BN;
    pdl_launch_dependents();   // (behind the allocation: a CTA of the next kernel cannot take tensor memory that this one still waits for)
    volatile int* const failed = &bars.failed;

    if (warp == kSlWarps) {   // ---- MMAs
        const bool el = elect_one();
        RingPos<STAGES> at;
        RingPos<kSlSlots> a;
        bool ok = true;
        for (int pass = 0; pass < passes && ok; ++pass) {
            const int d = pass & 1;
            if (pass >= 2 && !mbar_wait_warp(&bars.acc_empty[d], (unsigned)((pass >> 1) - 1) & 1u)) { ok = false; break; }   // (stored two passes ago)
            for (int k = 0; k < steps; ++k) {
                if (!mbar_wait_warp(&bars.ready[a.s], a.par)) { ok = false; break; }   // (whoever made it ready has waited for the activations)
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (el) {
                    const unsigned b = umma_desc_lo(ring + at.s * STAGE_BYTES);
#pragma unroll
                    for (int j = 0; j < kSlCols / 16; ++j)
                        if (j < 12 || k < real)
                            umma_f16_ta<1>(tmem_d + d * BN, tmem_a + a.s * 128u + 8u * j, b + (j >> 2) * (HALF / 16) + 2 * (j & 3), umma_idesc(kTcRows, BN), j > 0 || k > 0 ? 1u : 0u);
                    umma_commit(&bars.empty[at.s]);
                    umma_commit(&bars.free[a.s]);
                }
                __syncwarp();
                at.next();
                a.next();
            }
            if (ok && el) umma_commit(&bars.acc_full[d]);
            __syncwarp();
        }
        if (!ok) {   // the MMAs issued so far end before tensor memory is freed: an arrival of their own, which nothing else makes
            if (el) { tc_fail(p.status, &bars.failed, 2); umma_commit(&bars.free[a.s]); }
            mbar_wait_warp(&bars.free[a.s], a.par);
        }
        __syncwarp();
    } else if (warp == kSlWarps + 1) {   // ---- activations
        const bool el = elect_one();
        pdl_wait();                         // they come from the kernel just before this one
        RingPos<STAGES> at;
        int issued = 0;
        const int total = passes * steps;
        bool ok = true;
        for (int j = 0; issued < total; ++issued) {
            const bool whole = j < real;
            const int x = whole ? (lo + j) * kSlCols : p.real_steps * kSlCols + (lo + j - p.real_steps) * 192;
            if (issued >= STAGES && !mbar_wait_warp(&bars.empty[at.s], at.par ^ 1u)) { ok = false; break; }
            if (*failed) { ok = false; break; }
            if (el) {
                const unsigned bar = smem_u32(&bars.full[at.s]), stage = ring + at.s * STAGE_BYTES;
                mbar_expect(bar, whole ? STAGE_BYTES : 3 * HALF);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (q < 3 || whole) tma_load_2d(stage + q * HALF, &xmap, x + q * 64, 0, bar);
            }
            __syncwarp();
            at.next();
            if (++j == steps) j = 0;
        }
        if (!ok && el) tc_fail(p.status, &bars.failed, 3);
        // every copy has landed before the ring is given to the cluster, or the CTA leaves
        for (int i = issued > STAGES ? issued - STAGES : 0; i < issued; ++i) mbar_wait_warp(&bars.full[i % STAGES], (unsigned)((i / STAGES) & 1));
        __syncwarp();
    } else if (warp < kSlWarps) {   // ---- dequantising warps: quarter warp & 3 of the lanes, number warp >> 2 of the quarter's six
        const int quarter = warp & 3, number = warp >> 2;
        const int tile_of = number / 3, first = number - 3 * tile_of;
        const unsigned ready0 = smem_u32(&bars.ready[0]), free0 = smem_u32(&bars.free[0]), full0 = smem_u32(&bars.full[0]);
        const unsigned my_ring = ring + STAGES * STAGE_BYTES + warp * (kSlAhead * kSlUnitBytes);
        const int kt4 = p.kt / 4;
        const bool lands = warp == 0 || warp == 4 || warp == 8;   // quarter 0's first tile, present in every pass: waits for the step's activations
        // A warp takes every third step of all passes, and so always the same slot: when it waits for the MMAs of the step three before its
        // own, it has waited for those of the step six before, the slot's phase before, itself. (A wait by parity cannot tell a phase from
        // the one two before.) Where the quarter has one row tile or none, in the last pass, its first three warps make the arrivals of
        // the others.
        // request side: this warp's units over real weights, in order
        int f_pass = 0, f_j = first, f_left = 0;   // f_left: units of the tile still to request
        const uint4* f_w = nullptr;
        const uint4* f_s = nullptr;
        auto f_seek = [&]() {   // on to a pass with a tile and units over real weights
            for (; f_pass < passes; ++f_pass) {
                const SlPass t = sl_pass(p, f_pass, cta, ctas);
                const int at_j = f_j;
                f_j += (steps - f_j + 2) / 3 * 3 - steps;   // its first place in the next pass
                f_left = at_j < real ? (real - at_j + 2) / 3 : 0;
                if (quarter + 4 * tile_of < t.count && f_left > 0) {
                    const size_t at = (size_t)(t.first + quarter + 4 * tile_of) * kt4 + lo + at_j;
                    f_w = p.tiles + at * 128 + lane;
                    f_s = reinterpret_cast<const uint4*>(p.sb) + at * 16 + lane;
                    ++f_pass;
                    return;
                }
            }
            f_left = 0;
        };
        f_seek();
        auto fetch = [&](unsigned dst) {
            if (f_left > 0) {
                asm volatile(
                    "cp.async.cg.shared.global [%0], [%1], 16;\n"
                    "cp.async.cg.shared.global [%0+512], [%1+512], 16;\n"
                    "cp.async.cg.shared.global [%0+1024], [%1+1024], 16;\n"
                    "cp.async.cg.shared.global [%0+1536], [%1+1536], 16;\n" ::"r"(dst), "l"(f_w) : "memory");
                if (lane < 16) asm volatile("cp.async.cg.shared.global [%0+2048], [%1], 16;" ::"r"(dst), "l"(f_s) : "memory");
                f_w += 3 * 128;
                f_s += 3 * 16;
                if (--f_left == 0) f_seek();
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        unsigned src = my_ring;
        fetch(my_ring + lane * 16);
        fetch(my_ring + kSlUnitBytes + lane * 16);
        RingPos<STAGES> stage;
        stage.s = first;
        const unsigned ready_bar = ready0 + 8u * first, free_bar = free0 + 8u * first;
        unsigned free_par = 1u;        // (of the slot's phase before the first one: over from the start)
        int j = first;
        bool ok = true;
        auto begin = [&]() {   // the MMAs that read this slot are done
            const bool done = mbar_wait_warp(free_bar, free_par);
            free_par ^= 1u;
            return done;
        };
        for (int pass = 0; pass < passes && ok; ++pass, j -= steps) {
            const SlPass t = sl_pass(p, pass, cta, ctas);
            const bool there = quarter + 4 * tile_of < t.count, alone = quarter + 4 >= t.count;
            if (alone && tile_of) break;   // (the last pass)
            const unsigned dst = tmem_a + ((unsigned)(quarter * 32 + tile_of * 16) << 16) + first * 128u;
            auto finish = [&]() {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");   // the stores are ordered before the MMAs of the warp that waits
                if (lands && !mbar_wait_warp(full0 + 8u * stage.s, stage.par)) return false;
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(ready_bar), "r"(alone ? 2 : 1) : "memory");
                stage.skip3();
                return true;
            };
            if (!there) {
                for (; j < steps && ok; j += 3) ok = begin() && finish();
                continue;
            }
            for (; j < real && ok; j += 3) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kSlAhead - 1) : "memory");
                __syncwarp();
                uint4 w[4], s_lo, s_hi;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[q].x), "=r"(w[q].y), "=r"(w[q].z), "=r"(w[q].w)   : "r"(src + lane * 16 + q * 512) : "memory");
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s_lo.x), "=r"(s_lo.y), "=r"(s_lo.z), "=r"(s_lo.w)   : "r"(src + 2048 + (lane >> 2) * 16) : "memory");
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s_hi.x), "=r"(s_hi.y), "=r"(s_hi.z), "=r"(s_hi.w)   : "r"(src + 2176 + (lane >> 2) * 16) : "memory");
                __syncwarp();
                fetch(src + lane * 16);   // (read by all lanes)
                src = my_ring + (my_ring + kSlUnitBytes - src);
                if (!begin()) { ok = false; break; }
                const unsigned sl[4] = {s_lo.x, s_lo.y, s_lo.z, s_lo.w}, sh[4] = {s_hi.x, s_hi.y, s_hi.z, s_hi.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    unsigned a[16];
                    tc_unpack(w[q], tc_scale2<F16SB>(sl[q]), tc_scale2<F16SB>(sh[q]), a);
                    tmem_st_frag(dst + 32u * q, a);
                }
                ok = finish();
            }
            for (; j < steps && ok; j += 3) {
                unsigned a[16], a_lo[16];
                tc_appended_pair<F16SB>(p, t.first + quarter + 4 * tile_of, lo + j - p.real_steps, a, a_lo);
                if (!begin()) { ok = false; break; }
                tmem_st_frag(dst, a);
                tmem_st_frag(dst + 32u, a_lo);
                tmem_st_frag(dst + 64u, a);
                ok = finish();
            }
        }
        if (!ok && lane == 0) tc_fail(p.status, &bars.failed, 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
    } else if (p.splits == 1) {   // ---- results of a pass: a warp has its quarter's lanes, two row tiles of 16
        const int quarter = warp & 3;
        pdl_wait();   // (the rows' factors)
        float fac[BN > 32 ? 2 : 1];
#pragma unroll
        for (int i = 0; i < (BN > 32 ? 2 : 1); ++i) fac[i] = tc_rscale(p, min(32 * i + lane, p.m - 1));
        for (int pass = 0; pass < passes; ++pass) {
            const SlPass t = sl_pass(p, pass, cta, ctas);
            const int d = pass & 1, j = quarter + 4 * (lane >> 4);
            TcDst dst = tc_dst(p, (t.first + j) * 16 + (lane & 15));
            dst.live = dst.live && j < t.count;
            if (!mbar_wait_warp(&bars.acc_full[d], (unsigned)(pass >> 1) & 1u)) { if (lane == 0) tc_fail(p.status, &bars.failed, 4); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                if (c0 >= p.m) break;
                unsigned v[16];
                tmem_ld16(tmem_d + ((unsigned)(quarter * 32) << 16) + (unsigned)(d * BN + c0), v);
                tc_emit16(p, dst, v, fac[c0 / 32], c0 & 16, c0);
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) tc_arrive(smem_u32(&bars.acc_empty[d]));
        }
        __syncwarp();
    }
    if (p.splits > 1) {
        // one pass; each CTA of the cluster sends its part of the columns that another one finishes
        pdl_wait();   // (the rows' factors)
        const bool done = mbar_wait_warp(&bars.acc_full[0], 0u);
        if (!done && lane == 0) tc_fail(p.status, &bars.failed, 5);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();                                 // every ring of the cluster is free
        const int own = BN / p.splits;                  // columns that a CTA of the cluster finishes
        const SlPass t = sl_pass(p, 0, cta, ctas);
        if (done && warp < kTcDeqWarps) {
            const int r = (warp & 3) * 32 + lane;
#pragma unroll 1
            for (int c0 = (warp >> 2) * 16; c0 < BN; c0 += 64) {
                if (c0 >= p.m) break;
                unsigned v[16];
                tmem_ld16(tmem_d + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)c0, v);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int c = c0 + i, owner = c / own;
                    if (c < p.m) reinterpret_cast<float*>(cluster.map_shared_rank(ring_ptr, owner))[(rank * own + (c - owner * own)) * kTcRows + r] = __uint_as_float(v[i]);
                }
            }
        }
        cluster.sync();
        const float* got = reinterpret_cast<const float*>(ring_ptr);
        const int rows = p.gated ? kTcRows / 2 : kTcRows;
        for (int o = threadIdx.x; o < own * rows; o += blockDim.x) {
            const int cl = o / rows, i = o % rows, token = rank * own + cl;
            if (token >= p.m) continue;
            // row tile j of the pass and its row; where its lane is (gated: a gate row, its up row eight further on)
            const int j = p.gated ? i >> 3 : i >> 4, in = p.gated ? i & 7 : i & 15, ra = 32 * (j & 3) + 16 * (j >> 2) + in;
            if (j >= t.count) continue;
            const float* src = got + cl * kTcRows + ra;
            float va = 0.f, vb = 0.f;
            for (int z = 0; z < p.splits; ++z) {   // ranges in order
                va += src[z * own * kTcRows];
                if (p.gated) vb += src[z * own * kTcRows + 8];
            }
            const float sc = tc_rscale(p, token);
            if (p.gated) tc_store_gated(p, token, (t.first + j) * 8 + in, va * sc, vb * sc);
            else tc_store(p.out, token, (t.first + j) * 16 + in, va * sc);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_d), "r"(kTmemCols) : "memory");
}

// Activations bf16 -> fp16, one CTA per row: the row's largest magnitude goes to [2^14, 2^15), so that nothing overflows fp16 and
// every element within 2^-28 of the largest converts exactly (bf16 carries 8 significant bits, fp16 11). rscale[row] = the inverse
// factor. Within a group of 64 column 16 t + 4 j + i goes to place 16 j + 4 t + i, the order of the weights' fragments. Behind the k
// values (and zeros up to the weights' padding) the row gets, for every 64 groups, three blocks of 64 columns: sum / 64 of every group of 64 converted values as an fp16
// pair, laid out (hi, hi, lo) to meet the (c_hi, c_lo, c_hi) blocks of the weight side; the rest is zeros.
// CH: eights of a row per thread, held in registers between the two passes (reading 4 bytes per lane twice took 24 us for 2048 x 4096 under
// ncu); 0: a row of more than 16384 values is read twice. Few rows want short chains: two eights and up to 1024 threads; many rows want
// all of them resident at once and no warp without work: four eights. 2010 rows of 2048: 6.4 us under ncu, of 256 threads 9.4.
struct F16Rows { int k, k_pad; __half* xh; int stride; float* rscale; };   // columns, padded; the copy and its pitch
// bf16 magnitudes order like their bit patterns: two 16-bit maxima at a time
__device__ __forceinline__ unsigned f16_top(unsigned mx, const uint4& v) {
    mx = __vmaxu2(mx, v.x & 0x7FFF7FFFu); mx = __vmaxu2(mx, v.y & 0x7FFF7FFFu);
    mx = __vmaxu2(mx, v.z & 0x7FFF7FFFu); return __vmaxu2(mx, v.w & 0x7FFF7FFFu);
}
// the power of two of a row out of its threads' maxima
__device__ __forceinline__ int f16_shift(unsigned mx, unsigned* red) {
    mx = __reduce_max_sync(0xffffffffu, max(mx & 0xFFFFu, mx >> 16));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) mx = max(mx, red[i]);
    const int e = (int)(mx >> 7);                                   // biased exponent of the largest magnitude
    return (e == 0 || e == 255) ? 0 : max(-100, min(100, 141 - e));
}
// eight values, the i-th eight of the row; lanes of eight share a group (k is a multiple of 64)
__device__ __forceinline__ void f16_put(const F16Rows& f, __half* out, int i, const uint4& v, float mul) {
    const unsigned u[4] = {v.x, v.y, v.z, v.w};
    float sum = 0.f;
    unsigned o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(__uint_as_float(u[j] << 16) * mul, __uint_as_float(u[j] & 0xFFFF0000u) * mul);
        o[j] = *reinterpret_cast<const unsigned*>(&h);
        const float2 g = __half22float2(h);
        sum += g.x + g.y;
    }
    // eight columns 8 u .. of a group: t = u / 2, j = 2 (u & 1) and the next one
    __half* dst = out + (i >> 3) * 64 + 32 * (i & 1) + 4 * ((i & 7) >> 1);
    *reinterpret_cast<uint2*>(dst) = make_uint2(o[0], o[1]);
    *reinterpret_cast<uint2*>(dst + 16) = make_uint2(o[2], o[3]);
    const unsigned lane = threadIdx.x & 31, mask = 0xFFu << (lane & 24);
    sum += __shfl_xor_sync(mask, sum, 1);
    sum += __shfl_xor_sync(mask, sum, 2);
    sum += __shfl_xor_sync(mask, sum, 4);
    if ((lane & 7) == 0) {
        const float sc = sum * 0.015625f;
        const __half hi = __float2half_rn(sc), lo = __float2half_rn(sc - __half2float(hi));
        const int group = i >> 3;
        __half* ext = out + f.k_pad + (group >> 6) * 192 + (group & 63);
        ext[0] = hi; ext[64] = hi; ext[128] = lo;
    }
}
// what lies behind the values and behind the last group
__device__ __forceinline__ void f16_pad(const F16Rows& f, __half* out, int row, int sh) {
    for (int i = f.k + threadIdx.x; i < f.k_pad; i += blockDim.x) out[i] = __ushort_as_half(0);
    const int groups = f.k / 64;
    for (int i = threadIdx.x; i < f.stride - f.k_pad; i += blockDim.x)
        if (i / 192 * 64 + (i & 63) >= groups) out[f.k_pad + i] = __ushort_as_half(0);
    if (threadIdx.x == 0) f.rscale[row] = __uint_as_float((unsigned)(127 - sh) << 23);
}

constexpr int f16_max_threads(int ch) { return ch == 4 ? 512 : ch == 2 ? 1024 : 256; }
constexpr int kF16FewRows = 296;   // two per SM
int f16_threads(int k, int ch) { return ch ? (k / 8 + 32 * ch - 1) / (32 * ch) * 32 : 256; }

template <int CH>
__global__ void __launch_bounds__(f16_max_threads(CH)) x_to_f16_kernel(const __nv_bfloat16* x, int x_stride, const F16Rows f) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ unsigned red[32];
    const int row = blockIdx.x, tid = threadIdx.x, n8 = f.k / 8, nt = blockDim.x;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)row * x_stride);
    uint4 held[CH ? CH : 1];
    unsigned mx = 0;
    if (CH) {
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            held[c] = make_uint4(0, 0, 0, 0);
            if (tid + c * nt < n8) held[c] = src[tid + c * nt];
        }
#pragma unroll
        for (int c = 0; c < CH; ++c) mx = f16_top(mx, held[c]);
    } else {
        for (int i = tid; i < n8; i += nt) mx = f16_top(mx, src[i]);
    }
    const int sh = f16_shift(mx, red);
    const float mul = __uint_as_float((unsigned)(127 + sh) << 23);  // 2^sh
    __half* out = f.xh + (size_t)row * f.stride;
    if (CH) {
#pragma unroll
        for (int c = 0; c < CH; ++c)
            if (tid + c * nt < n8) f16_put(f, out, tid + c * nt, held[c], mul);
    } else {
        for (int i = tid; i < n8; i += nt) f16_put(f, out, i, src[i], mul);
    }
    f16_pad(f, out, row, sh);
}

// A norm step (see rmsnorm_kernel) whose result goes to its buffer and, converted, to the product behind it: one pass instead of two
// launches. MODE: 0 copy, 1 residual add and copy, 2 residual add. A row stays in registers, its weights come before the wait for the
// kernel in front; CH as above. 2010 rows of 2048: 9.9 us under ncu; with 256 threads, the row in shared memory and the weights behind the
// first sum 11.3. A decode step of 41 sequences of the 8B transformer is 5 % faster for both, a prompt 1 to 2 %.
template <int MODE, int CH>
__global__ void __launch_bounds__(f16_max_threads(CH)) norm_to_f16_kernel(const __nv_bfloat16* in, int in_stride, __nv_bfloat16* residual, int res_stride,
                                                                          const __nv_bfloat16* weight, float eps, float weight_bias, __nv_bfloat16* y, int y_stride,
                                                                          const F16Rows f) {
    pdl_launch_dependents();
    __shared__ unsigned red[32];
    __shared__ float sums[32];
    const int row = blockIdx.x, tid = threadIdx.x, n8 = f.k / 8, nt = blockDim.x;
    auto pack = [](float a, float b) { const __nv_bfloat162 v = __floats2bfloat162_rn(a, b); return *reinterpret_cast<const unsigned*>(&v); };
    uint4 w[CH], v[CH], r[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        w[c] = make_uint4(0, 0, 0, 0);
        if (tid + c * nt < n8) w[c] = reinterpret_cast<const uint4*>(weight)[tid + c * nt];
    }
    pdl_wait();
    const uint4* in4 = reinterpret_cast<const uint4*>(in + (size_t)row * in_stride);
    uint4* res4 = reinterpret_cast<uint4*>(residual + (size_t)row * res_stride);
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        v[c] = r[c] = make_uint4(0, 0, 0, 0);
        if (tid + c * nt < n8) { v[c] = in4[tid + c * nt]; if (MODE != 0) r[c] = res4[tid + c * nt]; }
    }
    float h[CH][8], ss = 0.f;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const unsigned u[4] = {v[c].x, v[c].y, v[c].z, v[c].w}, q[4] = {r[c].x, r[c].y, r[c].z, r[c].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            h[c][2 * j] = __uint_as_float(u[j] << 16); h[c][2 * j + 1] = __uint_as_float(u[j] & 0xFFFF0000u);
            if (MODE != 0) { h[c][2 * j] += __uint_as_float(q[j] << 16); h[c][2 * j + 1] += __uint_as_float(q[j] & 0xFFFF0000u); }
        }
        if (MODE != 2 && tid + c * nt < n8)
            res4[tid + c * nt] = make_uint4(pack(h[c][0], h[c][1]), pack(h[c][2], h[c][3]), pack(h[c][4], h[c][5]), pack(h[c][6], h[c][7]));
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(h[c][e], h[c][e], ss);
    }
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((tid & 31) == 0) sums[tid >> 5] = ss;
    __syncthreads();
    float total = 0.f;
    for (int i = 0; i < (nt >> 5); ++i) total += sums[i];
    const float rs = rsqrtf(total / (float)f.k + eps);
    unsigned mx = 0;
#pragma unroll
    for (int c = 0; c < CH; ++c) {
        const unsigned u[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
        unsigned o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            o[j] = pack(h[c][2 * j] * rs * (__uint_as_float(u[j] << 16) + weight_bias), h[c][2 * j + 1] * rs * (__uint_as_float(u[j] & 0xFFFF0000u) + weight_bias));
        v[c] = make_uint4(o[0], o[1], o[2], o[3]);
        if (tid + c * nt < n8) {
            reinterpret_cast<uint4*>(y + (size_t)row * y_stride)[tid + c * nt] = v[c];
            mx = f16_top(mx, v[c]);
        }
    }
    const int sh = f16_shift(mx, red);
    const float mul = __uint_as_float((unsigned)(127 + sh) << 23);
    __half* out = f.xh + (size_t)row * f.stride;
#pragma unroll
    for (int c = 0; c < CH; ++c)
        if (tid + c * nt < n8) f16_put(f, out, tid + c * nt, v[c], mul);
    f16_pad(f, out, row, sh);
}

// rows: activation rows in a CTA's shared memory
constexpr size_t tc_smem_bytes(int rows, int stages) { return (size_t)stages * rows * 256 + kTcRingBytes + 1024; }

// fp16 activations X[m][x_stride] as a 2-D tensor (k innermost); box = 64 columns x bn rows, 128-byte swizzle
int make_x_map(const __half* x, int x_stride, int m, int bn, CUtensorMap* map) {
    TensorMapEncodeFn fn = tensor_map_encode_fn();
    if (!fn) { set_error("qgemm (tcgen05): cuTensorMapEncodeTiled is not available"); return SWLM_ERR_CUDA; }
    const cuuint64_t dims[2] = {(cuuint64_t)x_stride, (cuuint64_t)m};
    const cuuint64_t strides[1] = {(cuuint64_t)x_stride * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)bn};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(x), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { set_error("qgemm (tcgen05): cuTensorMapEncodeTiled failed (%d)", (int)r); return SWLM_ERR_CUDA; }
    return SWLM_OK;
}
// stages of the form with 128 activation rows per tile and of the pair's
constexpr int kTcStages128 = 4, kTcStagesPair = 5;
constexpr int kTcSMs = 148;

int ext_blocks(int kt) { return (kt + 63) / 64; }   // blocks of 64 groups
// CTAs (groups of `splits` along K) that share the row tiles. In a single pass as few as keep the largest share: with fewer SMs taken the next
// launch's CTAs start beside them (8192 x 2048 at 41 rows 13.5 us with 148, 10.2 with 128; 4096 x 4096 16.6 and 13.8). Fours: 32 of the 34 to
// 36 clusters that the GPU runs at once.
int sl_ctas(int row_tiles, int splits) {
    const int most = std::min(splits == 4 ? 32 : kTcSMs / splits, row_tiles), share = (row_tiles + most - 1) / most;
    return share <= 8 ? (row_tiles + share - 1) / share : most;
}
// CTAs along K of a product of up to 64 rows: two or four where row tiles are few and K is long. A step of 256 columns takes 0.36 us and 0.05
// for each row tile of the CTA up to four, 0.64 with more; meeting in a cluster 5 to 6. One, two and four, us at 41 rows: 2048 x 8192
// 23.5 / 21.1 / 16.8, 4096 x 14336 36.6 / 29.4 / 24.1, 1000 x 16448 38.6 / 32.5 / 24.4; 4096 x 4096 14.4 / 15.8 / 13.8, 1024 x 4096
// 13.1 / 15.7 / 12.9, 2048 x 2048 9.8 / 13.2 / 11.6.
int sl_splits(int row_tiles, int kt) {
    const int steps = kt / 4 + ext_blocks(kt);
    auto time = [&](int z) {
        const int ctas = sl_ctas(row_tiles, z), whole = row_tiles / (8 * ctas), share = (row_tiles - whole * 8 * ctas + ctas - 1) / ctas;
        const double step = 0.64 * whole + (share > 4 ? 0.64 : share > 0 ? 0.36 + 0.05 * share : 0.0);
        return step * ((steps + z - 1) / z) + (z > 1 ? 6.0 : 0.0);
    };
    int best = 1;
    for (int z = 2; z <= 4; z *= 2)
        if (steps >= z && row_tiles <= 8 * sl_ctas(row_tiles, z) && time(z) < time(best)) best = z;
    return best;
}

constexpr int sl_stages(int bn) { return bn == 32 ? 6 : bn == 48 ? 4 : 3; }
constexpr size_t sl_smem_bytes(int bn) { return (size_t)sl_stages(bn) * bn * kSlCols * 2 + kSlRingBytes + 1024; }
template <typename K>
int tc_init_one(K kernel, size_t smem) {
    SWLM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return SWLM_OK;
}
int tc_launch_short(QGemmTcParams& p, bool f16, const __half* xh, int xh_stride, int splits, cudaStream_t s) {
    constexpr int BN = 128, STAGES = kTcStages128;
    CUtensorMap xmap;
    const int rc = make_x_map(xh, xh_stride, p.m, BN, &xmap);
    if (rc) return rc;
    p.splits = splits;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((p.row_tiles + 7) / 8 * splits), (unsigned)((p.m + BN - 1) / BN));
    cfg.blockDim = dim3((kTcDeqWarps + 2) * 32); cfg.dynamicSmemBytes = tc_smem_bytes(BN, STAGES); cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)splits; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t e = f16 ? cudaLaunchKernelEx(&cfg, qgemm_tc_short_kernel<BN, STAGES, true>, p, xmap)
                              : cudaLaunchKernelEx(&cfg, qgemm_tc_short_kernel<BN, STAGES, false>, p, xmap);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "qgemm_tc short launch");
}
template <int BN>
int sl_launch(QGemmTcParams& p, bool f16, const __half* xh, int xh_stride, int splits, cudaStream_t s) {
    CUtensorMap xmap;
    const int rc = make_x_map(xh, xh_stride, p.m, BN, &xmap);
    if (rc) return rc;
    p.real_steps = p.kt * 64 / kSlCols; p.steps = p.real_steps + ext_blocks(p.kt); p.splits = splits;
    const int ctas = sl_ctas(p.row_tiles, splits);
    p.whole = p.row_tiles / (8 * ctas); p.left = p.row_tiles - p.whole * 8 * ctas;
    p.n_tiles = p.whole + (p.left > 0);
    if (splits > 1 && p.n_tiles > 1) { set_error("qgemm (tcgen05): passes"); return SWLM_ERR_INVALID; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ctas * splits)); cfg.blockDim = dim3(kSlThreads); cfg.dynamicSmemBytes = sl_smem_bytes(BN); cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)splits; attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    const cudaError_t e = f16 ? cudaLaunchKernelEx(&cfg, qgemm_slab_kernel<BN, sl_stages(BN), true>, p, xmap)
                              : cudaLaunchKernelEx(&cfg, qgemm_slab_kernel<BN, sl_stages(BN), false>, p, xmap);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "qgemm_tc slab launch");
}
int tc_launch_long(QGemmTcParams& p, bool f16, const __half* xh, int xh_stride, cudaStream_t s) {
    CUtensorMap xmap;
    const int rc = make_x_map(xh, xh_stride, p.m, kTcPairRows, &xmap);
    if (rc) return rc;
    p.splits = 1;
    p.tok_tiles = (p.m + 255) / 256;
    p.n_tiles = (p.row_tiles + 15) / 16 * p.tok_tiles;
    const dim3 grid((unsigned)(2 * std::min(p.n_tiles, kTcSMs / 2))), block((kTcDeqWarps + 2 + kTcEpiWarps) * 32);
    const size_t smem = tc_smem_bytes(kTcPairRows, kTcStagesPair);
    const cudaError_t e = f16 ? launch_k(qgemm_tc_kernel<kTcStagesPair, true>, grid, block, smem, s, p, xmap)
                              : launch_k(qgemm_tc_kernel<kTcStagesPair, false>, grid, block, smem, s, p, xmap);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "qgemm_tc launch");
}

// appended columns for `kt` groups, in whole steps
int ext_cols(int kt) { return (192 * ext_blocks(kt) + kTcStep - 1) / kTcStep * kTcStep; }
int kt_padded(int k) { return (k / 64 + 3) / 4 * 4; }

// How a product of m rows over `tiles16` row tiles of `kt` groups runs: up to 64 rows the slab form with 32, 48 or 64; with more the form with
// the least time by what was measured over K = 2048 .. 14336, n = 2048 .. 128256 and m = 65 .. 512 (us; graphs of launches, weights from
// memory). A CTA with 128 activation rows takes 0.5 us per step, a pair of the long form 0.87. A launch starts and ends in about 6. Cutting K
// over a cluster costs the exchange: 5 over four CTAs, 9 over two.
struct TcChoice { int bn, splits; };
TcChoice tc_choose(int m, int tiles16, int kt) {
    if (m <= 64) return {m <= 32 ? 32 : m <= 48 ? 48 : 64, sl_splits(tiles16, kt)};
    const int steps = (kt * 64 + ext_cols(kt)) / kTcStep;
    const long long tiles = (long long)((tiles16 + 7) / 8) * ((m + 127) / 128);
    TcChoice best{128, 1};
    double least = 1e30;
    auto offer = [&](double cost, const TcChoice& c) { if (cost < least) { least = cost; best = c; } };
    for (int z = 1; z <= 4 && z <= steps; z *= 2)
        offer((double)((tiles * z + kTcSMs - 1) / kTcSMs) * (0.5 * ((steps + z - 1) / z) + 2) + 4 + (z == 1 ? 0 : z == 4 ? 5 : 9), {128, z});
    if (m > 128) {
        const long long pairs = (long long)((tiles16 + 15) / 16) * ((m + 255) / 256);
        offer((double)((pairs + kTcSMs / 2 - 1) / (kTcSMs / 2)) * (0.87 * steps + 1.5) + 5, {256, 1});
    }
    return best;
}
}  // namespace

template <int BN>
static int sl_init() {
    const int rc = tc_init_one(qgemm_slab_kernel<BN, sl_stages(BN), false>, sl_smem_bytes(BN));
    return rc ? rc : tc_init_one(qgemm_slab_kernel<BN, sl_stages(BN), true>, sl_smem_bytes(BN));
}
int qgemm_tc_init() {
    int rc;
    if ((rc = sl_init<32>()) || (rc = sl_init<48>()) || (rc = sl_init<64>()) ||
        (rc = tc_init_one(qgemm_tc_short_kernel<128, kTcStages128, false>, tc_smem_bytes(128, kTcStages128))) ||
        (rc = tc_init_one(qgemm_tc_short_kernel<128, kTcStages128, true>, tc_smem_bytes(128, kTcStages128))) ||
        (rc = tc_init_one(qgemm_tc_kernel<kTcStagesPair, false>, tc_smem_bytes(kTcPairRows, kTcStagesPair))) ||
        (rc = tc_init_one(qgemm_tc_kernel<kTcStagesPair, true>, tc_smem_bytes(kTcPairRows, kTcStagesPair)))) return rc;
    return SWLM_OK;
}

// [fp16 activations + group sums][one float per row]
static int xh_cols(int k) { return kt_padded(k) * 64 + ext_cols(kt_padded(k)); }
size_t qgemm_tc_scratch_bytes(int m, int k) { return ((size_t)m * xh_cols(k) * 2 + 255) / 256 * 256 + (size_t)m * 4; }

int qgemm_tc_launch_count(bool reuse_x) { return (reuse_x ? 0 : 1) + 1; }

static F16Rows f16_rows(int m, int k, void* scratch) {
    F16Rows f{};
    f.k = k; f.k_pad = kt_padded(k) * 64; f.xh = static_cast<__half*>(scratch); f.stride = xh_cols(k);
    f.rscale = reinterpret_cast<float*>(static_cast<unsigned char*>(scratch) + ((size_t)m * f.stride * 2 + 255) / 256 * 256);
    return f;
}

int launch_norm_to_f16(int mode, int m, int dim, const __nv_bfloat16* in, int in_stride, __nv_bfloat16* residual, int res_stride, const __nv_bfloat16* weight,
                       float eps, float weight_bias, __nv_bfloat16* out, int out_stride, void* scratch, cudaStream_t s) {
    if (dim % 64 || in_stride % 8 || res_stride % 8 || out_stride % 8 || dim > kNormMaxDim) { set_error("rmsnorm: dim=%d", dim); return SWLM_ERR_INVALID; }
    const F16Rows f = f16_rows(m, dim, scratch);
    const int ch = m <= kF16FewRows ? 2 : 4;
    auto go = [&](auto kernel) {
        return launch_k(kernel, dim3((unsigned)m), dim3((unsigned)f16_threads(dim, ch)), 0, s, in, in_stride, residual, res_stride, weight, eps, weight_bias, out, out_stride, f);
    };
    cudaError_t e;
    if (mode == SWLM_STEP_COPY_RMSNORM) e = ch == 2 ? go(norm_to_f16_kernel<0, 2>) : go(norm_to_f16_kernel<0, 4>);
    else if (mode == SWLM_STEP_RESADD_COPY_RMSNORM) e = ch == 2 ? go(norm_to_f16_kernel<1, 2>) : go(norm_to_f16_kernel<1, 4>);
    else e = ch == 2 ? go(norm_to_f16_kernel<2, 2>) : go(norm_to_f16_kernel<2, 4>);
    return e == cudaSuccess ? SWLM_OK : cuda_fail(e, "norm_to_f16 launch");
}

// Y[m][n] = bf16(X[m][k] . W^T). `scratch` (qgemm_tc_scratch_bytes) takes the fp16 copy of the activations; `status` is a device
// word the kernel sets when a bounded wait expires.
int launch_qgemm_tc(const Q4Tiled& w, int m, const __nv_bfloat16* x, int x_stride, const TcSegments& out, int epilogue, int gated_act,
                    void* scratch, int* status, cudaStream_t s, bool reuse_x) {
    const F16Rows f = f16_rows(m, w.k, scratch);
    __half* const xh = f.xh;
    const int xh_stride = f.stride;
    if (w.k % 64 || (x_stride & 7) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(xh) & 15) || !xh) {
        set_error("qgemm (tcgen05): bad shape, alignment or scratch");
        return SWLM_ERR_INVALID;
    }
    QGemmTcParams p{};
    p.tiles = w.tiles; p.sb = reinterpret_cast<const unsigned*>(w.sb); p.row_tiles = w.row_tiles; p.kt = w.kt_pad;
    p.rscale = f.rscale;
    p.m = m; p.status = status;
    p.real_steps = w.kt_pad * 64 / kTcStep; p.steps = xh_stride / kTcStep;
    p.gated = epilogue == QGEMV_EPI_SWIGLU; p.gated_act = gated_act;
    p.out = out;
    if (out.count < 1 || out.count > 3 || (p.gated && (out.count != 1 || !w.interleaved))) { set_error("qgemm (tcgen05): output segments"); return SWLM_ERR_INVALID; }
    for (int q = out.count; q < 3; ++q) p.out.end[q] = p.out.end[out.count - 1];   // never stored to
    // (reuse_x: the scratch still holds the copy of these very rows, made for the product before this one or by their norm)
    if (!reuse_x) {
        const int ch = w.k > 16384 ? 0 : m <= kF16FewRows ? 2 : 4;
        auto go = [&](auto kernel) { return launch_k(kernel, dim3((unsigned)m), dim3((unsigned)f16_threads(w.k, ch)), 0, s, x, x_stride, f); };
        const cudaError_t e = ch == 0 ? go(x_to_f16_kernel<0>) : ch == 2 ? go(x_to_f16_kernel<2>) : go(x_to_f16_kernel<4>);
        if (e != cudaSuccess) return cuda_fail(e, "x_to_f16 launch");
    }
    const TcChoice c = tc_choose(m, w.row_tiles, p.kt);
    switch (c.bn) {
    case 32: return sl_launch<32>(p, w.sb_f16, xh, xh_stride, c.splits, s);
    case 48: return sl_launch<48>(p, w.sb_f16, xh, xh_stride, c.splits, s);
    case 64: return sl_launch<64>(p, w.sb_f16, xh, xh_stride, c.splits, s);
    case 128: return tc_launch_short(p, w.sb_f16, xh, xh_stride, c.splits, s);
    default: return tc_launch_long(p, w.sb_f16, xh, xh_stride, s);
    }
}

}  // namespace swlm

extern "C" int swlm_op_qgemm_form(int m, int n, int k, int gated, int* form) {
    using namespace swlm;
    if (m < kQGemmTcMinRows || n <= 0 || k <= 0 || k % 64 || !form) { set_error("bad argument"); return SWLM_ERR_INVALID; }
    const TcChoice c = tc_choose(m, gated ? (n + 7) / 8 : (n + 15) / 16, kt_padded(k));
    form[0] = c.bn; form[1] = c.splits;
    return SWLM_OK;
}
