// experts_kq.cu - decode-sized grouped experts for the ggml K- and I-quant formats (Q6_K, IQ1_M) read in place: a bandwidth-bound
// weight stream through shared memory with the dot products on the integer tensor cores.
//
// Why integers.  At 1.75 bits a weight (IQ1_M) the stream is so dense that the decode instructions, not HBM, set the pace: a
// warp-per-row fp32 kernel spends ~8 instructions on every weight.  Here a weight costs about two: the codes stay small
// integers, the activations become int8 too, and mma.sync m16n8k32 (u8 x s8 -> s32) does the multiplying.
//   * Activations: a row x becomes two int8 terms under one scale per row, x s ~ q1 + q2 / 254 (|q| <= 127), so the rounding
//     error is ~1e-4 of the row's norm (one int8 term, what Basalt's q8_1 rows carry, would leave ~1e-2).  A pass multiplies 4
//     entries x 2 terms = the 8 columns of the MMA.
//   * IQ1_M (include/basalt/ggml/ggml_common.h:350-362, decode rule src/kernels/cpu/ggml/ggml_quants.c:1266-1314): a weight is
//     d m (g + delta) with g in {-1, 0, 1} from the 2048-point codebook, m = 2 s + 1 (3-bit s per 16 weights), delta = +-1/8
//     per 8 weights, d an fp16 per 256.  With c = g + 1 in {0, 1, 2}:  8 w / d = 8 m c - m (8 -+ 1).  The first term is the
//     MMA operand (one table word per 8 weights gives their c as nibbles; times m they stay below 31); the second is
//     constant over a group of 8, so it multiplies the group's activation SUM: one more k-step per 256 weights whose operands
//     are the 32 group coefficients m (8 -+ 1) <= 135 (u8) and the 32 negated group sums split as 16 hi + lo (s8 each).
//     Everything up to the factor d / 8 is exact integer arithmetic.
//   * Q6_K (ggml_common.h:279-285, ggml_quants.c:1048-1075): a weight is d sc (q - 32), sc an int8 per 16 weights: one
//     m16n8k16 MMA per scale group, its result times sc added up in int32, the 32 taken off by a correction like IQ1_M's.
// Each warp owns 16 weight rows (8 gate rows with their 8 up rows, so SwiGLU stays in the thread; or 16 down rows) and
// streams them through its own cp.async ring in chunks of 512 columns; a block's warps share the pass's activation columns.
// Blocks are persistent; each takes an equal run of the (pass, row block) sequence.
//
// Semantics: Basalt's native_expert_grouped (include/basalt/kernels/iq_kernels.hpp:77-92; its IQ1_M dot src/kernels/cuda/
// iq_kernels.cu:227-257 with the grid table staged in shared memory :1516-1521), minus the single-term q8_1 rounding.
#include <atomic>

#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "formats.cuh"
#include "pdl.cuh"
#include "plan.cuh"

namespace bsx {
namespace {

constexpr int kRowsQ = 16;      // weight rows per warp tile
constexpr int kColsQ = 8;       // MMA n: 4 entries x 2 int8 terms
constexpr int kEntQ = 4;
constexpr float kTerm2 = 1.0f / 254.0f;

enum { QMODE_GU = 0, QMODE_DOWN = 1 };
// Q6_K rows beyond this go to the fp32 kernels: the images hold 15 bits of a row's largest value, not its 24
constexpr int64_t kMaxColsQ6K = 8192;

// What a stage holds of a row: kCB blocks of 256 columns, kRow bytes apart.  IQ1_M: two blocks (112 bytes), copied in 16-byte pieces.  Q6_K:
// one 210-byte block as the 53 words that cover it (every second block starts on 2 bytes, so its copy starts 2 bytes early; none reaches
// past its row), rows 60 words apart, which keeps a quarter-warp's reads in different banks.  One block a stage lets any power-of-two part
// of a row be a warp's own (KS below) and, up to about 5000 columns, two CTAs of eight warps share an SM.
template <int TYPE> struct QT;
template <> struct QT<kTypeIQ1M> {
    static constexpr int kBlock = 56, kPad = 32, kCB = 2, kRow = 112, kCorr = 64;      // kCorr: correction bytes of a column and block
};
template <> struct QT<kTypeQ6K> {
    static constexpr int kBlock = 210, kPad = 16, kCB = 1, kRow = 240, kCorr = 32;
};

__device__ __forceinline__ void cpa16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cpa4(uint32_t dst, const void* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// D (16 x 8, s32) += A (16 x 32, u8, row) x B (32 x 8, s8, col)
__device__ __forceinline__ void mma_u8s8_k32(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D (16 x 8, s32) = A (16 x 16, u8 or s8, row) x B (16 x 8, s8, col)
__device__ __forceinline__ void mma_u8s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};\n"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

// ---------------------------------------------------------------- activation images
// One warp per image row: the row as two int8 terms under one scale, x s ~ q1 + q2 / 254, s = 127 / max|x|; inv[row] = 1 / s.
// Layout: img[row][term][K] int8 in column order.  Q6_K: per 256 columns the 16 negated group-of-16 sums of each term as 16 hi + lo,
// corr[row][term][K / 256][hi 16 bytes | lo 16 bytes].  IQ1_M: per 256 columns the 32 negated group-of-8 sums of each term as
// 16 hi + lo, corr[row][term][K / 256][hi 32 bytes | lo 32 bytes], a group at the byte its coefficient has in the A fragment:
// group 4 u + t (u = 32-column unit, t = group inside it) -> byte 4 t + p (u < 4) or 16 + 4 t + p with p = 0, 2, 1, 3 for
// u % 4 = 0, 1, 2, 3 (the order in which the product kernel can assemble the coefficients cheaply).
// FROM_H = false: rows of x (row i of x when the caller gave the number of x rows, else the row of entry i); true: row e of
// the SwiGLU output.  The last block lists the passes (up to pass_entries consecutive entries of a group).
template <bool FROM_H, int TYPE>
__global__ void __launch_bounds__(256)
kq_image_kernel(ExpertArgs a, int8_t* __restrict__ img, int8_t* __restrict__ corr, float* __restrict__ inv, PassRec* __restrict__ items,
                int* __restrict__ n_items, int pass_entries) {
    pdl_wait();
    pdl_launch_dependents();
    const int ng = min(*a.n_groups, (int) a.cap_groups);
    const int total = min(a.grp_start[ng], (int) a.cap_entries);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == gridDim.x - 1) {
        __shared__ int sh[8];
        __shared__ int s_base;
        if (threadIdx.x == 0) s_base = 0;
        __syncthreads();
        for (int g0 = 0; g0 < ng; g0 += 256) {
            const int g = g0 + threadIdx.x;
            const int s0 = g < ng ? a.grp_start[g] : 0;
            const int cnt = g < ng ? max(0, min(a.grp_start[g + 1], (int) a.cap_entries) - s0) : 0;
            const int np = (cnt + pass_entries - 1) / pass_entries;
            int x = np;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) sh[warp] = x;
            __syncthreads();
            int before = s_base;
            for (int w = 0; w < warp; ++w) before += sh[w];
            for (int p = 0; p < np; ++p) {
                PassRec r;
                r.blob = a.grp_ptr[g];
                r.eb = s0 + p * pass_entries;
                r.ntok = min(pass_entries, cnt - p * pass_entries);
                items[before + x - np + p] = r;
            }
            __syncthreads();
            if (threadIdx.x == 255) s_base = before + x;
            __syncthreads();
        }
        if (threadIdx.x == 0) n_items[0] = s_base;
        return;
    }
    const int i = blockIdx.x * 8 + warp;
    const int n_img = FROM_H ? total : (a.n_x_rows > 0 ? a.n_x_rows : total);
    if (i >= n_img) return;
    const int64_t K = FROM_H ? a.L.n_ff : a.L.n_embd;
    const int64_t row = FROM_H ? (int64_t) i : (a.n_x_rows > 0 ? (int64_t) i : (int64_t) a.ent_tok[i]);
    const void* src = FROM_H ? (const void*) a.h : a.x;
    const int kind = FROM_H ? BSX_X_F32 : a.x_kind;
    const int n_sb = (int) (K >> 4);
    float amax = 0.f;
    for (int sb = lane; sb < n_sb; sb += 32) {
        float v[16];
        load16(src, kind, row, K, sb, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(v[j]));
    }
    amax = warp_max_xor(amax);
    float s = 1.f, iv = 1.f;
    if (amax > 0.f && amax <= 3.0e38f) {
        s = 127.f / amax;
        iv = amax / 127.f;
    }
    if (lane == 0) inv[i] = iv;
    const int nblk = (int) (K >> 8);
    int8_t* q1 = img + (size_t) i * 2 * K;
    int8_t* q2 = q1 + K;
    for (int sb = lane; sb < n_sb; sb += 32) {
        float v[16];
        load16(src, kind, row, K, sb, v);
        uint32_t w1[4], w2[4];
        int sum1[2] = {0, 0}, sum2[2] = {0, 0};
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float xs = v[j] * s;
            int a1 = __float2int_rn(xs);
            a1 = max(-127, min(127, a1));
            int a2 = __float2int_rn((xs - (float) a1) * 254.f);
            a2 = max(-127, min(127, a2));
            if ((j & 3) == 0) { w1[j >> 2] = 0u; w2[j >> 2] = 0u; }
            w1[j >> 2] |= (uint32_t) (a1 & 0xFF) << (8 * (j & 3));
            w2[j >> 2] |= (uint32_t) (a2 & 0xFF) << (8 * (j & 3));
            sum1[j >> 3] += a1;
            sum2[j >> 3] += a2;
        }
        reinterpret_cast<uint4*>(q1)[sb] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        reinterpret_cast<uint4*>(q2)[sb] = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        const int blk = sb >> 4;
        if constexpr (TYPE == kTypeIQ1M) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gi = ((sb & 15) << 1) + h;               // group inside the 256-column block
                const int u = gi >> 2, t = gi & 3;
                const int pos = ((u & 1) << 1) | ((u >> 1) & 1);      // units (0, 1, 2, 3) of a half sit in bytes (0, 2, 1, 3)
                const int slot = (u < 4 ? 0 : 16) + 4 * t + pos;
#pragma unroll
                for (int term = 0; term < 2; ++term) {
                    const int neg = -(term ? sum2[h] : sum1[h]);
                    const int hi = neg >> 4, lo = neg & 15;       // neg = 16 hi + lo, 0 <= lo < 16 (arithmetic shift floors)
                    int8_t* c = corr + (((size_t) i * 2 + term) * nblk + blk) * QT<TYPE>::kCorr;
                    c[slot] = (int8_t) hi;
                    c[32 + slot] = (int8_t) lo;
                }
            }
        } else {
#pragma unroll
            for (int term = 0; term < 2; ++term) {
                const int neg = -(term ? sum2[0] + sum2[1] : sum1[0] + sum1[1]);
                int8_t* c = corr + (((size_t) i * 2 + term) * nblk + blk) * QT<TYPE>::kCorr;
                c[sb & 15] = (int8_t) (neg >> 4);
                c[16 + (sb & 15)] = (int8_t) (neg & 15);
            }
        }
    }
}

// ---------------------------------------------------------------- block decoders
// IQ1_M: one 256-weight block of rows g and g + 8 (raw 56-byte blocks ra, rb in shared memory, 8-byte aligned) against NB times 8
// activation columns; the caller scales: tot[i] += I[i] * d[row] where I is the exact integer
// 8 m c q - coefficient sums described at the top.  bcol: this lane's column, at the block's first byte plus 8 t;
// ccol: the column's 64 correction bytes of this block; bnext / cnext: bytes to the column 8 further; wide: the pass has such columns.
// tab: the lane's copy of the table (NC copies interleaved point by point).
template <int NC, int NB>
__device__ __forceinline__ void iq1m_block(const uint8_t* ra, const uint8_t* rb, const uint2* __restrict__ tab, const uint8_t* bcol,
                                           const uint8_t* ccol, int bnext, int cnext, bool wide, int t, float (&tot)[NB][4]) {
    uint32_t wa[14], wb[14];
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        const uint2 va = reinterpret_cast<const uint2*>(ra)[i], vb = reinterpret_cast<const uint2*>(rb)[i];
        wa[2 * i] = va.x; wa[2 * i + 1] = va.y;
        wb[2 * i] = vb.x; wb[2 * i + 1] = vb.y;
    }
    // words 0-7: qs (unit u = bytes 4u..4u+3), 8-11: qh (unit u = bytes 2u, 2u+1; group t = nibble t), 12-13: four scale words
    int acc[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0;
    const int s4 = 4 * t, s3 = 3 * (t >> 1);
    // a point's index: byte t of the unit's qs word under the three high bits, which byte 0 (even units) or 2 of the masked qh word holds
    const uint32_t sel0 = 0x7740u + (uint32_t) t, sel1 = 0x7760u + (uint32_t) t;
    uint32_t msum[4] = {0u, 0u, 0u, 0u};              // the groups' scales m as bytes, in the correction operand's order (below)
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        uint32_t a[4];
        constexpr int kPos[4] = {0, 2, 1, 3};        // unit u of a half sits in byte kPos[u & 3] of that half's correction word
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t* w = r ? wb : wa;
            const uint32_t hi = (w[8 + (u >> 1)] >> s4) & 0x00070007u;
            const uint2 e = tab[__byte_perm(w[u], hi, (u & 1) ? sel1 : sel0) * NC];
            const uint32_t sw = w[12 + (u >> 2)] >> s3;                                    // the thread's scale field of unit u now sits at a fixed bit
            const int fb = 16 * ((u >> 1) & 1) + 6 * (u & 1);
            const uint32_t m = fb > 0 ? (((sw >> (fb - 1)) & 14u) | 1u) : (((sw << 1) & 14u) | 1u);   // 2 s + 1
            a[r] = e.x * m;
            a[2 + r] = e.y * m;
            msum[(u < 4 ? 0 : 2) + r] += m << (8 * kPos[u & 3]);
        }
        const uint2 b = *reinterpret_cast<const uint2*>(bcol + 32 * u);
        mma_u8s8_k32(acc[0], a[0], a[1], a[2], a[3], b.x, b.y);
        if (NB > 1 && wide) {
#pragma unroll
            for (int n = 1; n < NB; ++n) {
                const uint2 bn = *reinterpret_cast<const uint2*>(bcol + n * bnext + 32 * u);
                mma_u8s8_k32(acc[n], a[0], a[1], a[2], a[3], bn.x, bn.y);
            }
        }
    }
    // the correction operand: byte = m (8 - 8 delta) = 7 m + 2 m [delta = -1/8], four groups at a time.  The delta bits of units
    // (0, 1) are bits 4t+3 and 4t+19 of qh word 0, of units (2, 3) the same bits of qh word 1: shifted and merged they land in bytes
    // 0, 2 and 1, 3 - the order kPos gives the scales.
    uint32_t ca[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t* w = r ? wb : wa;
        const uint32_t dlo = ((w[8] >> (s4 + 3)) & 0x00010001u) | (((w[9] >> (s4 + 3)) & 0x00010001u) << 8);
        const uint32_t dhi = ((w[10] >> (s4 + 3)) & 0x00010001u) | (((w[11] >> (s4 + 3)) & 0x00010001u) << 8);
        ca[r] = 7u * msum[r] + 2u * (msum[r] & (dlo * 0xFFu));
        ca[2 + r] = 7u * msum[2 + r] + 2u * (msum[2 + r] & (dhi * 0xFFu));
    }
    // the fp16 super-scale: the top nibbles of the four scale words
    float d[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t* w = r ? wb : wa;
        const uint32_t bits = ((w[12] >> 12) & 0x000Fu) | ((w[12] >> 24) & 0x00F0u) | ((w[13] >> 4) & 0x0F00u) | ((w[13] >> 16) & 0xF000u);
        d[r] = __half2float(__ushort_as_half((unsigned short) bits));
    }
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        if (n > 0 && !wide) break;
        const uint8_t* cc = ccol + n * cnext;
        int chi[4] = {0, 0, 0, 0}, clo[4] = {0, 0, 0, 0};
        const uint32_t h0 = *reinterpret_cast<const uint32_t*>(cc + 4 * t), h1 = *reinterpret_cast<const uint32_t*>(cc + 16 + 4 * t);
        const uint32_t l0 = *reinterpret_cast<const uint32_t*>(cc + 32 + 4 * t), l1 = *reinterpret_cast<const uint32_t*>(cc + 48 + 4 * t);
        mma_u8s8_k32(chi, ca[0], ca[1], ca[2], ca[3], h0, h1);
        mma_u8s8_k32(clo, ca[0], ca[1], ca[2], ca[3], l0, l1);
#pragma unroll
        for (int i = 0; i < 4; ++i) tot[n][i] = fmaf((float) (8 * acc[n][i] + 16 * chi[i] + clo[i]), d[i >> 1], tot[n][i]);
    }
}

// four bytes of shared memory from an address that is a multiple of four, or two past one (every second 210-byte block)
template <bool ODD>
__device__ __forceinline__ uint32_t ld_word(const uint8_t* p) {
    if (!ODD) return *reinterpret_cast<const uint32_t*>(p);
    return __byte_perm(*reinterpret_cast<const uint32_t*>(p - 2), *reinterpret_cast<const uint32_t*>(p + 2), 0x5432);
}

// Q6_K: one 256-weight block of rows g and g + 8 (raw 210-byte blocks in shared memory) against NB times 8 columns; bcol: this lane's
// column at the block's first byte plus 4 t, ccol: its 32 correction bytes of this block plus 4 t.  All of it up to d is integer: the
// codes go in as they are (0 .. 63), a group's sum times its scale adds up in 32 bits (below 2^29), and the 32 that a code is too
// large by comes off as one MMA pair over the block's 16 scales and the groups' negated activation sums (16 hi + lo).  What bounds the
// kernel is instructions: with signed codes, a scale converted to fp32 for each group and half-words loaded one by one a warp spent
// 794 on a block of 16 rows and the 64-token step of 2048 x 512, 512 experts, took 325 us; now 250.
template <int NB, bool ODD>
__device__ __forceinline__ void q6k_block(const uint8_t* ra, const uint8_t* rb, const uint8_t* bcol, const uint8_t* ccol, int bnext, int cnext, bool wide, int t,
                                          float (&tot)[NB][4]) {
    int sum[NB][4];
#pragma unroll
    for (int n = 0; n < NB; ++n) sum[n][0] = sum[n][1] = sum[n][2] = sum[n][3] = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int lo = 64 * h + 16 * j + 4 * t, hi = 128 + 32 * h + 16 * j + 4 * t;
            const uint32_t qa[2] = {ld_word<ODD>(ra + lo), ld_word<ODD>(ra + lo + 32)}, qah = ld_word<ODD>(ra + hi);
            const uint32_t qb[2] = {ld_word<ODD>(rb + lo), ld_word<ODD>(rb + lo + 32)}, qbh = ld_word<ODD>(rb + hi);
#pragma unroll
            for (int sub = 0; sub < 4; ++sub) {
                const int down = sub >= 2 ? 4 : 0;
                const uint32_t a0 = ((qa[sub & 1] >> down) & 0x0F0F0F0Fu) | ((sub < 2 ? qah << (4 - 2 * sub) : qah >> (2 * sub - 4)) & 0x30303030u);
                const uint32_t a1 = ((qb[sub & 1] >> down) & 0x0F0F0F0Fu) | ((sub < 2 ? qbh << (4 - 2 * sub) : qbh >> (2 * sub - 4)) & 0x30303030u);
                const int is = 8 * h + 2 * sub + j;
                const int sa = (int8_t) ra[192 + is], sb = (int8_t) rb[192 + is];
#pragma unroll
                for (int n = 0; n < NB; ++n) {
                    if (n > 0 && !wide) break;
                    int c[4];
                    mma_u8s8_k16(c, a0, a1, *reinterpret_cast<const uint32_t*>(bcol + n * bnext + 128 * h + 32 * sub + 16 * j));
#pragma unroll
                    for (int i = 0; i < 4; ++i) sum[n][i] += c[i] * (i < 2 ? sa : sb);
                }
            }
        }
    }
    const float da = __half2float(*reinterpret_cast<const __half*>(ra + 208)), db = __half2float(*reinterpret_cast<const __half*>(rb + 208));
    const uint32_t ca = ld_word<ODD>(ra + 192 + 4 * t), cb = ld_word<ODD>(rb + 192 + 4 * t);
#pragma unroll
    for (int n = 0; n < NB; ++n) {
        if (n > 0 && !wide) break;
        int chi[4], clo[4];
        mma_s8_k16(chi, ca, cb, *reinterpret_cast<const uint32_t*>(ccol + n * cnext));
        mma_s8_k16(clo, ca, cb, *reinterpret_cast<const uint32_t*>(ccol + n * cnext + 16));
#pragma unroll
        for (int i = 0; i < 4; ++i) tot[n][i] = fmaf((float) (sum[n][i] + 512 * chi[i] + 32 * clo[i]), i < 2 ? da : db, tot[n][i]);
    }
}

// ---------------------------------------------------------------- the product kernel
// MODE GU: rows = 8 gate rows r0.. with the up rows r0..; columns = the entries' x images; writes h (fp32).
// MODE DOWN: rows = 16 down rows; columns = the entries' h images; writes out rows through ent_dst.
// NB: a pass is up to 4 NB entries, NB column blocks of the MMA over one decoded A fragment; a pass of four or fewer multiplies one block.
// KS > 1: KS neighbouring warps share a row tile, each a part of its columns, and their sums meet in shared memory: a step of the
// block is then W / KS tiles instead of W, so that a small call still divides evenly.
// Work: the row blocks (W / KS tiles) of all passes in one sequence, cut into equal runs, one a block.  A run's part of one pass shares
// its columns and its weight stream, so barriers, activation copies and first loads come once or twice a call.  (Units drawn from a
// counter instead: IQ1_M gate/up of 7168 x 2048 at 64 tokens 765 us, with runs and a look-up index made by one byte permutation 655.)
template <int TYPE, int MODE, int W, int OCC, int KS, int NC, int ST, int NB>
__global__ void __launch_bounds__(W * 32, OCC)
kq_mma_kernel(ExpertArgs a, const int8_t* img, const int8_t* corr, const float* inv, const PassRec* items, const int* n_items, int n_row_blocks) {
    using Q = QT<TYPE>;
    constexpr int kThreads = W * 32, kStages = ST, kEntP = kEntQ * NB, kCols = kColsQ * NB, kTiles = W / KS, CB = Q::kCB;
    constexpr int kChunkBytes = CB * Q::kBlock, kRow = Q::kRow, kStageBytes = kRowsQ * kRow;
    extern __shared__ __align__(128) uint8_t smem[];
    const int64_t K = MODE == QMODE_GU ? a.L.n_embd : a.L.n_ff;
    const int nblk = (int) (K >> 8);
    const int cstride = (int) K + Q::kPad;                                   // bytes between activation columns
    const int xstride = nblk * Q::kCorr + 16;                                // ... and between their correction columns
    uint8_t* xs = smem;                                                        // [kCols][cstride]
    uint8_t* cs = xs + (size_t) kCols * cstride;                               // [kCols][xstride]
    uint2* tab = reinterpret_cast<uint2*>(cs + (size_t) kCols * xstride);      // [2048][NC] (IQ1_M)
    uint8_t* wbase = reinterpret_cast<uint8_t*>(tab) + (TYPE == kTypeIQ1M ? 16384 * NC : 0);
    float2* part = reinterpret_cast<float2*>(wbase + (size_t) W * kStages * kStageBytes);     // [2][tiles][KS - 1][NB][32] (KS > 1)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    uint8_t* wring = wbase + (size_t) warp * kStages * kStageBytes;
    const uint32_t wring_s = (uint32_t) __cvta_generic_to_shared(wring);
    const uint32_t xs_s = (uint32_t) __cvta_generic_to_shared(xs), cs_s = (uint32_t) __cvta_generic_to_shared(cs);
    __shared__ int s_ir[kEntP];

    if (TYPE == kTypeIQ1M) {
        // the codebook as 8 bytes per point, coordinate i's code c = g + 1 in byte i: the two words are the two MMA operand
        // registers of an 8-weight group.  The look-ups are the kernel's scarce resource (16 data-dependent 8-byte reads a lane and
        // block), and what they cost is bank conflicts.  NC copies, interleaved so that a lane's copy (lane % NC) lives in 1 / NC of the
        // banks and only as many lanes compete there: sixteen lanes over sixteen bank pairs collide three deep on average, four
        // over four two deep.  64-token step of the 7168 x 2048 layer: two copies 1602 us, four 1523.
        for (int j = threadIdx.x; j < 2048 * NC; j += kThreads) {
            const int i = j / NC;
            const uint32_t p = a.grid[i];
            uint32_t lo = 0u, hi = 0u;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                lo |= ((p >> (2 * c)) & 3u) << (8 * c);
                hi |= ((p >> (2 * c + 8)) & 3u) << (8 * c);
            }
            tab[j] = make_uint2(lo, hi);
        }
    }
    pdl_wait();
    pdl_launch_dependents();

    const int64_t n_rows = MODE == QMODE_GU ? a.L.n_ff : a.L.n_embd;
    constexpr int kTileRows = MODE == QMODE_GU ? 8 : 16;
    static_assert(W % KS == 0, "");
    constexpr int kStepRows = kTiles * kTileRows;
    const int n_chunks = nblk / CB / KS, chunk0 = (warp % KS) * n_chunks;      // this warp's part of a row
    const size_t row_bytes = MODE == QMODE_GU ? (size_t) a.L.gu_row : (size_t) a.L.d_row;

    const int64_t n_work = (int64_t) n_items[0] * n_row_blocks;
    int work = (int) (n_work * blockIdx.x / gridDim.x);
    const int work_end = (int) (n_work * (blockIdx.x + 1) / gridDim.x);
    PassRec next{0ull, 0, 0};
    if (work < work_end) next = items[work / n_row_blocks];
    while (work < work_end) {
        const PassRec pass = next;
        const int item = work / n_row_blocks, rb = work - item * n_row_blocks;
        const int steps = min(work_end - work, n_row_blocks - rb);
        work += steps;
        if (work < work_end) next = items[item + 1];      // rides under this pass
        const int64_t r0 = (int64_t) rb * kStepRows + warp / KS * kTileRows;
        int live_tiles = 0;
        if (r0 < n_rows) live_tiles = (int) min((int64_t) steps, (n_rows - r0 + kStepRows - 1) / kStepRows);
        const int n_units = live_tiles * n_chunks;
        const uint8_t* blob = reinterpret_cast<const uint8_t*>(pass.blob);
        const int eb = pass.eb, ntok = pass.ntok;
        const int ncol = 2 * ntok;
        const bool wide = NB > 1 && ntok > kEntQ;
        __syncthreads();   // the previous pass is done with xs, cs and s_ir
        if (threadIdx.x < ntok) s_ir[threadIdx.x] = (MODE == QMODE_GU && a.n_x_rows > 0) ? a.ent_tok[eb + threadIdx.x] : eb + (int) threadIdx.x;
        __syncthreads();
        // the pass's activation columns (and their correction bytes): column c = 2 entry + term.  Columns beyond ncol keep
        // whatever they held: an MMA column depends on its own B column only, and those results are never stored.
        {
            const int per_col = (int) (K >> 4);
            for (int i = threadIdx.x; i < ncol * per_col; i += kThreads) {
                const int c = i / per_col, q = i - c * per_col;
                cpa16(xs_s + (uint32_t) (c * cstride + q * 16), img + ((size_t) s_ir[c >> 1] * 2 + (c & 1)) * K + (size_t) q * 16);
            }
            const int per_cc = nblk * (QT<TYPE>::kCorr / 16);
            for (int i = threadIdx.x; i < ncol * per_cc; i += kThreads) {
                const int c = i / per_cc, q = i - c * per_cc;
                cpa16(cs_s + (uint32_t) (c * xstride + q * 16), corr + ((size_t) s_ir[c >> 1] * 2 + (c & 1)) * nblk * QT<TYPE>::kCorr + (size_t) q * 16);
            }
            cpa_commit();
        }
        // the weight stream: (tile, chunk) stages of this warp's 16 rows; rows 0-7 `pitch` apart, row 8 `half` past row 0
        const uint8_t* row0 = MODE == QMODE_GU ? blob + (size_t) r0 * a.L.gu_row : blob + a.L.down_off + (size_t) r0 * a.L.d_row;
        const size_t pitch0 = row_bytes, pitch1 = MODE == QMODE_GU ? (size_t) a.L.up_row : row_bytes;
        const size_t half = MODE == QMODE_GU ? (size_t) a.L.up_off + (size_t) r0 * (a.L.up_row - a.L.gu_row) : 8 * row_bytes;
        const size_t tile_bytes = (size_t) kStepRows * row_bytes;
        int iss_unit = 0, iss_chunk = 0;
        size_t iss_tile = 0;
        auto issue = [&]() {
            if (iss_unit < n_units) {
                const uint32_t dst = wring_s + (uint32_t) (iss_unit % kStages) * kStageBytes;
                if constexpr (TYPE == kTypeIQ1M) {
                    const uint8_t* src = row0 + iss_tile + (size_t) (chunk0 + iss_chunk) * kChunkBytes;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {                    // 7 pieces a row, 112 in all
                        const int p = lane + 32 * j, row = p / 7, off = (p - row * 7) * 16;
                        if (p < 112) cpa16(dst + (uint32_t) (row * kRow + off), src + (row < 8 ? row * pitch0 : half + (row - 8) * pitch1) + off);
                    }
                } else {
                    const uint8_t* src = row0 + iss_tile + (size_t) (chunk0 + iss_chunk) * kChunkBytes - 2 * ((chunk0 + iss_chunk) & 1) + 4 * lane;
                    auto row_at = [&](int row) { return src + (row < 8 ? row * pitch0 : half + (row - 8) * pitch1); };
#pragma unroll
                    for (int row = 0; row < kRowsQ; ++row) {
                        const uint8_t* r = row_at(row);
                        const uint32_t d = dst + (uint32_t) (row * kRow + 4 * lane);
                        cpa4(d, r);
                        if (lane < 53 - 32) cpa4(d + 128, r + 128);
                    }
                }
                ++iss_unit;
                if (++iss_chunk == n_chunks) {
                    iss_chunk = 0;
                    iss_tile += tile_bytes;
                }
            }
            cpa_commit();
        };
#pragma unroll
        for (int c = 0; c < kStages - 1; ++c) issue();
        cpa_wait<kStages - 1>();   // the activation group (the oldest) has landed
        __syncthreads();

        // epilogue constants of this thread's entries (columns 2 t, 2 t + 1 of each column block)
        float f[NB];
        int64_t orow[NB];
#pragma unroll
        for (int n = 0; n < NB; ++n) {
            const int j = kEntQ * n + t;
            f[n] = 0.f;
            orow[n] = 0;
            if (j < ntok) {
                f[n] = inv[s_ir[j]] * (TYPE == kTypeIQ1M ? 0.125f : 1.f);
                orow[n] = MODE == QMODE_GU ? (int64_t) (eb + j) * a.L.n_ff : (int64_t) a.ent_dst[eb + j] * a.L.n_embd;
            }
        }
        float tot[NB][4];
#pragma unroll
        for (int n = 0; n < NB; ++n) tot[n][0] = tot[n][1] = tot[n][2] = tot[n][3] = 0.f;
        const uint8_t* bcol = xs + (size_t) g * cstride + (TYPE == kTypeIQ1M ? 8 * t : 4 * t);
        const uint8_t* ccol = cs + (size_t) g * xstride + (TYPE == kTypeIQ1M ? 0 : 4 * t);
        int tile = 0, chunk = 0;
        for (int unit = 0; unit < n_units; ++unit) {
            issue();
            cpa_wait<kStages - 1>();
            __syncwarp();
            const uint8_t* st = wring + (size_t) (unit % kStages) * kStageBytes;
#pragma unroll
            for (int b = 0; b < CB; ++b) {
                const int blk = (chunk0 + chunk) * CB + b;
                const int at = TYPE == kTypeIQ1M ? b * Q::kBlock : 2 * (blk & 1);
                const uint8_t* ra = st + g * kRow + at;
                const uint8_t* rbp = st + (g + 8) * kRow + at;
                const uint8_t *bc = bcol + 256 * blk, *cc = ccol + QT<TYPE>::kCorr * blk;
                if constexpr (TYPE == kTypeIQ1M) iq1m_block<NC, NB>(ra, rbp, tab + (lane & (NC - 1)), bc, cc, kColsQ * cstride, kColsQ * xstride, wide, t, tot);
                else if (blk & 1) q6k_block<NB, true>(ra, rbp, bc, cc, kColsQ * cstride, kColsQ * xstride, wide, t, tot);
                else q6k_block<NB, false>(ra, rbp, bc, cc, kColsQ * cstride, kColsQ * xstride, wide, t, tot);
            }
            __syncwarp();   // every lane is done with this stage before a later issue overwrites it
            if (++chunk != n_chunks) continue;
            const int64_t rt = r0 + (int64_t) tile * kStepRows;
            chunk = 0;
            float2 v[NB];
#pragma unroll
            for (int n = 0; n < NB; ++n) {
                v[n] = make_float2(tot[n][0] + tot[n][1] * kTerm2, tot[n][2] + tot[n][3] * kTerm2);
                tot[n][0] = tot[n][1] = tot[n][2] = tot[n][3] = 0.f;
            }
            if constexpr (KS > 1) {
                // the tile's other warps hand their sums to its first; two buffers, so one barrier of the tile's warps is enough: a
                // buffer is written again only after the barrier of the tile in between, which its reader has passed
                float2* buf = part + ((size_t) (tile & 1) * kTiles + warp / KS) * (KS - 1) * NB * 32 + lane;
                if (warp % KS != 0)
#pragma unroll
                    for (int n = 0; n < NB; ++n) buf[((warp % KS - 1) * NB + n) * 32] = v[n];
                asm volatile("bar.sync %0, %1;\n" ::"r"(1 + warp / KS), "n"(KS * 32) : "memory");
                if (warp % KS == 0)
#pragma unroll
                    for (int n = 0; n < NB; ++n)
#pragma unroll
                        for (int k = 0; k < KS - 1; ++k) {
                            const float2 o = buf[(k * NB + n) * 32];
                            v[n].x += o.x;
                            v[n].y += o.y;
                        }
            }
            ++tile;
            if (KS == 1 || warp % KS == 0) {
#pragma unroll
                for (int n = 0; n < NB; ++n) {
                    if (kEntQ * n + t < ntok) {
                        if (MODE == QMODE_GU) {
                            a.h[orow[n] + rt + g] = swiglu(v[n].x * f[n], v[n].y * f[n], a.L);
                        } else {
                            store_out(a.out, a.out_kind, orow[n] + rt + g, v[n].x * f[n]);
                            store_out(a.out, a.out_kind, orow[n] + rt + g + 8, v[n].y * f[n]);
                        }
                    }
                }
            }
        }
        cpa_wait<0>();
    }
}

size_t al256q(size_t v) { return (v + 255) & ~(size_t) 255; }

// shared memory that a block may ask for, alone on its SM or one of two (227 and 113 KB less the static words)
constexpr size_t kSmemOne = 232448 - 256, kSmemTwo = 115712 - 256;

template <int TYPE>
size_t kq_smem(int64_t K, int W, int KS, int NC, int ST, int NB) {
    using Q = QT<TYPE>;
    return (size_t) kColsQ * NB * (K + Q::kPad) + (size_t) kColsQ * NB * ((K >> 8) * QT<TYPE>::kCorr + 16) + (TYPE == kTypeIQ1M ? (size_t) 16384 * NC : 0) +
           (size_t) W * ST * kRowsQ * Q::kRow + (size_t) W / KS * (KS - 1) * NB * 512 + 128;
}

template <int TYPE, int MODE, int W, int OCC, int KS, int NC, int ST, int NB>
int32_t kq_launch_as(const ExpertArgs& a, const int8_t* img, const int8_t* corr, const float* inv, const PassRec* items, const int* n_items, cudaStream_t st) {
    const size_t smem = kq_smem<TYPE>(MODE == QMODE_GU ? a.L.n_embd : a.L.n_ff, W, KS, NC, ST, NB);
    static std::atomic<bool> configured[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(kq_mma_kernel<TYPE, MODE, W, OCC, KS, NC, ST, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int) (OCC == 2 ? kSmemTwo : kSmemOne));
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    const int64_t rows = MODE == QMODE_GU ? a.L.n_ff : a.L.n_embd, step_rows = (MODE == QMODE_GU ? 8 : 16) * W / KS;
    launch_k(kq_mma_kernel<TYPE, MODE, W, OCC, KS, NC, ST, NB>, dim3((unsigned) (OCC * sm_count())), dim3(W * 32), smem, st, a, img, corr, inv, items, n_items,
             (int) ((rows + step_rows - 1) / step_rows));
    return launch_status();
}

// The shape of a product's launch: OCC blocks an SM, KS warps to a row tile, NB column blocks (4 NB entries) a pass.  Q6_K: two blocks of
// eight warps where shared memory holds two (K up to about 5000), which hide each other's first loads (2048 x 512, 512 experts, 64 tokens:
// one block of 16 warps 365 us, two of eight 312); wider rows one block of 16 warps (7168 x 2048: 2178 us, of eight 2668).  Two column
// blocks where they fit, for a pass of four or fewer entries multiplies one; four, or two and twelve warps, only where the groups are deep
// (a shared expert of 64 tokens, 7168 x 2048: gate/up 113 us with one, 76 with two).
struct KqShape { int OCC, KS, NB; };

// cap_groups and cap_entries bound the passes on the host.
template <int TYPE>
KqShape kq_shape(const ExpertArgs& a, bool gu) {
    const int64_t K = gu ? a.L.n_embd : a.L.n_ff, rows = gu ? a.L.n_ff : a.L.n_embd;
    const bool deep = a.cap_entries >= 8 * a.cap_groups;
    KqShape s{1, 1, 1};
    int W = 16, most = 2;
    if (TYPE == kTypeIQ1M) {
        if (kq_smem<TYPE>(K, 16, 2, 4, 3, 2) <= kSmemOne) s.NB = 2;
    } else {
        W = 8;
        if (deep && kq_smem<TYPE>(K, 8, 2, 1, 2, 4) <= kSmemTwo) { s.OCC = 2; s.NB = 4; }
        else if (kq_smem<TYPE>(K, 8, 8, 1, 2, 2) <= kSmemTwo) { s.OCC = 2; s.NB = 2; most = 8; }
        else if (!deep && kq_smem<TYPE>(K, 8, 4, 1, 2, 1) <= kSmemTwo) { s.OCC = 2; most = 4; }
        else {
            s.NB = deep && kq_smem<TYPE>(K, 12, 4, 1, 2, 2) <= kSmemOne ? 2 : 1;
            W = s.NB == 2 ? 12 : 16;
            most = 4;
        }
    }
    // Columns are split where whole rows would leave a block fewer than four steps, until it has eight: the last, partial one then weighs
    // little.  Where there are more steps the split costs more than it evens out (16 tokens of 2048 x 512: with 64 experts, 2.2 steps, 77 us
    // split in four and 84 in two; with 512, 4.9 steps, 150 us split in two and 137 whole).
    const int64_t chunks = K / (TYPE == kTypeIQ1M ? 512 : 256), step_rows = (gu ? 8 : 16) * W;
    const int64_t steps = (a.cap_groups + a.cap_entries / (kEntQ * s.NB)) * ((rows + step_rows - 1) / step_rows);
    const int64_t blocks = (int64_t) s.OCC * sm_count();
    if (steps < 4 * blocks)
        while (s.KS < most && chunks % (2 * s.KS) == 0 && steps * s.KS < 8 * blocks) s.KS *= 2;
    return s;
}

template <int TYPE, int MODE>
int32_t kq_launch(const KqShape& s, const ExpertArgs& a, const int8_t* img, const int8_t* corr, const float* inv, const PassRec* items, const int* n_items, cudaStream_t st) {
    const int64_t K = MODE == QMODE_GU ? a.L.n_embd : a.L.n_ff;
#define KQ_AS(W, OCC, KS, NC, ST, NB) return kq_launch_as<TYPE, MODE, W, OCC, KS, NC, ST, NB>(a, img, corr, inv, items, n_items, st)
    if constexpr (TYPE == kTypeQ6K) {
        if (s.OCC == 2 && s.NB == 4) {
            if (s.KS == 2) KQ_AS(8, 2, 2, 1, 2, 4);
            KQ_AS(8, 2, 1, 1, 2, 4);
        }
        if (s.OCC == 2 && s.NB == 2) {
            if (s.KS == 8) KQ_AS(8, 2, 8, 1, 2, 2);
            if (s.KS == 4) KQ_AS(8, 2, 4, 1, 2, 2);
            if (s.KS == 2) KQ_AS(8, 2, 2, 1, 2, 2);
            KQ_AS(8, 2, 1, 1, 2, 2);
        }
        if (s.OCC == 2) {
            if (s.KS == 4) KQ_AS(8, 2, 4, 1, 2, 1);
            if (s.KS == 2) KQ_AS(8, 2, 2, 1, 2, 1);
            KQ_AS(8, 2, 1, 1, 2, 1);
        }
        if (s.NB == 2) {
            if (s.KS == 4) KQ_AS(12, 1, 4, 1, 2, 2);
            if (s.KS == 2) KQ_AS(12, 1, 2, 1, 2, 2);
            KQ_AS(12, 1, 1, 1, 2, 2);
        }
        if (s.KS == 4) KQ_AS(16, 1, 4, 1, 2, 1);
        if (s.KS == 2) KQ_AS(16, 1, 2, 1, 2, 1);
        KQ_AS(16, 1, 1, 1, 2, 1);
    } else {
        if (s.NB == 2) {
            if (s.KS == 2) KQ_AS(16, 1, 2, 4, 3, 2);
            KQ_AS(16, 1, 1, 4, 3, 2);
        }
        // four copies of the codebook where they fit beside the columns and the stages (K up to 7680), else two
        if (kq_smem<TYPE>(K, 16, 2, 4, 3, 1) <= kSmemOne) {
            if (s.KS == 2) KQ_AS(16, 1, 2, 4, 3, 1);
            KQ_AS(16, 1, 1, 4, 3, 1);
        }
        KQ_AS(16, 1, 1, 2, 3, 1);
    }
#undef KQ_AS
}

bool kq_type(int t) { return t == kTypeIQ1M || t == kTypeQ6K; }

// the layout's K dimension works for the stream: whole 512-column chunks, 16-byte aligned rows where the copies are 16 bytes
bool kq_dim_ok(int type, int64_t K, int64_t rows) {
    if (K % 512 || rows % 8) return false;
    const int64_t rb = K / 256 * (type == kTypeIQ1M ? 56 : 210);
    return rb % (type == kTypeIQ1M ? 16 : 4) == 0;
}

}  // namespace

// scratch beyond the SwiGLU buffer: x images, h images (2 int8 terms each), their correction bytes, inverse scales, pass list
size_t experts_kq_scratch_bytes(int64_t cap, int64_t H, int64_t I) {
    return al256q((size_t) cap * 2 * H) + al256q((size_t) cap * 2 * I) + al256q((size_t) cap * 2 * (H / 256) * 64) + al256q((size_t) cap * 2 * (I / 256 + 1) * 64) +
           2 * al256q((size_t) cap * 4) + al256q((size_t) (cap + 1) * 16 + 16);
}

int32_t experts_grouped_kq(const ExpertArgs& a, cudaStream_t st) {
    const bsx_expert_layout& L = a.L;
    if (!kq_type(L.gu_type) || L.up_type != L.gu_type || !kq_type(L.d_type)) return BSX_E_TYPE;
    if (!kq_dim_ok(L.gu_type, L.n_embd, L.n_ff) || !kq_dim_ok(L.d_type, L.n_ff, L.n_embd) || L.n_embd % 16) return BSX_E_TYPE;
    if (L.gu_type == kTypeIQ1M ? kq_smem<kTypeIQ1M>(L.n_embd, 16, 1, 2, 3, 1) > kSmemOne : L.n_embd > kMaxColsQ6K) return BSX_E_TYPE;
    if (L.d_type == kTypeIQ1M ? kq_smem<kTypeIQ1M>(L.n_ff, 16, 1, 2, 3, 1) > kSmemOne : L.n_ff > kMaxColsQ6K) return BSX_E_TYPE;
    const int64_t cap = a.cap_entries, H = L.n_embd, I = L.n_ff;
    uint8_t* p = reinterpret_cast<uint8_t*>(a.h) + al256q((size_t) cap * I * 4);
    int8_t* ximg = reinterpret_cast<int8_t*>(p);
    p += al256q((size_t) cap * 2 * H);
    int8_t* himg = reinterpret_cast<int8_t*>(p);
    p += al256q((size_t) cap * 2 * I);
    int8_t* xcorr = reinterpret_cast<int8_t*>(p);
    p += al256q((size_t) cap * 2 * (H / 256) * 64);
    int8_t* hcorr = reinterpret_cast<int8_t*>(p);
    p += al256q((size_t) cap * 2 * (I / 256 + 1) * 64);
    float* xinv = reinterpret_cast<float*>(p);
    p += al256q((size_t) cap * 4);
    float* hinv = reinterpret_cast<float*>(p);
    p += al256q((size_t) cap * 4);
    int* n_items = reinterpret_cast<int*>(p);
    PassRec* items = reinterpret_cast<PassRec*>(n_items + 4);
    const int phase = experts_phase(a.L);
    const int64_t x_rows = a.n_x_rows > 0 ? a.n_x_rows : cap;
    const unsigned nbx = (unsigned) ((x_rows + 7) / 8 + 1), nbh = (unsigned) ((cap + 7) / 8 + 1);
    int32_t rc = BSX_OK;
    const KqShape gu = L.gu_type == kTypeIQ1M ? kq_shape<kTypeIQ1M>(a, true) : kq_shape<kTypeQ6K>(a, true);
    const KqShape dn = L.d_type == kTypeIQ1M ? kq_shape<kTypeIQ1M>(a, false) : kq_shape<kTypeQ6K>(a, false);
    if (phase != 2) {
        if (L.gu_type == kTypeIQ1M) {
            launch_k(kq_image_kernel<false, kTypeIQ1M>, dim3(nbx), dim3(256), 0, st, a, ximg, xcorr, xinv, items, n_items, kEntQ * gu.NB);
            rc = kq_launch<kTypeIQ1M, QMODE_GU>(gu, a, ximg, xcorr, xinv, items, n_items, st);
        } else {
            launch_k(kq_image_kernel<false, kTypeQ6K>, dim3(nbx), dim3(256), 0, st, a, ximg, xcorr, xinv, items, n_items, kEntQ * gu.NB);
            rc = kq_launch<kTypeQ6K, QMODE_GU>(gu, a, ximg, xcorr, xinv, items, n_items, st);
        }
    }
    if (rc != BSX_OK || phase == 1) return rc;
    if (L.d_type == kTypeIQ1M) {
        rc = launch_spread<kq_image_kernel<true, kTypeIQ1M>>(nbh, st, a, himg, hcorr, hinv, items, n_items, kEntQ * dn.NB);
        if (rc != BSX_OK) return rc;
        return kq_launch<kTypeIQ1M, QMODE_DOWN>(dn, a, himg, hcorr, hinv, items, n_items, st);
    }
    rc = launch_spread<kq_image_kernel<true, kTypeQ6K>>(nbh, st, a, himg, hcorr, hinv, items, n_items, kEntQ * dn.NB);
    if (rc != BSX_OK) return rc;
    return kq_launch<kTypeQ6K, QMODE_DOWN>(dn, a, himg, hcorr, hinv, items, n_items, st);
}

}  // namespace bsx
